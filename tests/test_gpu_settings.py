"""Settings that change after a step has been captured: the next advance runs
with the new setting, alone or in an ensemble."""
import math

import numpy as np
import pytest

from chapsim import gpu
from chapsim.mesh import channel_setup
from chapsim.fields import initial_field

pytestmark = pytest.mark.gpu


def _channel(shape, seed, precision="fp64"):
    s = channel_setup(*shape, 2 * math.pi, math.pi, 2.0, 2800.0)
    Q, PR = initial_field(s, seed, 0.1)
    c = gpu.ChannelTG(s, precision=precision)
    c.upload(Q, PR)
    c.set_dt(2e-3)
    c.SOLVERRK3_MOM_tg(0)
    return c


# 64 | 256: another right-hand side beside the same y-solve table (64^3 starts with 64 | 256 | 4); 0: the hybrid
# y-solve, whose choice frees the table of the scan solve that the context starts with; 1 and 16: another table
@pytest.mark.parametrize("force", [64 | 256, 0, 1, 16])
def test_ensemble_follows_its_members_settings(force):
    shapes = [(64, 64, 64), (32, 64, 96)]
    solo = [_channel(sh, 61 + k) for k, sh in enumerate(shapes)]
    grp = [_channel(sh, 61 + k) for k, sh in enumerate(shapes)]
    e = gpu.Ensemble(grp)
    e.advance(2, 2e-3, 1e-6, 0.5)
    for c in solo:
        c.advance(2, 2e-3, 1e-6, 0.5)
    for c in (solo[0], grp[0]):
        assert c.autotune(force=force)[0] == force
    e.advance(3, 2e-3, 1e-6, 0.5)
    for c in solo:
        c.advance(3, 2e-3, 1e-6, 0.5)
    for a, b in zip(solo, grp):
        for x, y in zip(a.download(want_h0=True), b.download(want_h0=True)):
            assert np.array_equal(x, y)
    e.close()
    for c in solo + grp:
        c.close()
