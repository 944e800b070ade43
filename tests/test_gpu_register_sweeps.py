"""The FP64 z and y sweeps in registers, at every line length and both tile
widths, against the oracle's sequential line solves.

REN = 2 makes the implicit operators stiff (|a| = F / dz^2 from 1 to 190 at
these grids, where the recurrences' ratio rho approaches 1 and carries travel
across every segment); the velocities after the projection and one step stay
within 1e-11 of the oracle, the bound of the step tests: the operators'
condition number 1 + 4|a| < 800 times 2^-53 is 1e-13 per sweep.
"""
import math

import numpy as np
import pytest

from oracle import Oracle
from chapsim import gpu
from chapsim.mesh import channel_setup
from chapsim.fields import initial_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 32, 32), (32, 64, 96), (64, 96, 64), (32, 128, 128), (96, 192, 192),
                                   (32, 256, 256), (64, 384, 384)])
def test_stiff_sweeps_match_oracle(shape):
    L, M, N = shape
    HX, HZ, REN, DT = 2 * math.pi, math.pi, 2.0, 0.05
    s = channel_setup(L, M, N, HX, HZ, 2.0, REN)
    Q, PR = initial_field(s, 41, 0.1)
    o = Oracle(L, M, N, HX, HZ, 2.0, REN, DT0=DT, DTMIN=1e-6, CFLGV=0.5, threads=8)
    o.set_fields(Q, PR)
    o.set_dt(DT)
    o.substep(0)
    assert o.run_steps(1)[0] == 0
    Qo = o.get_fields()[0]
    o.close()
    for force in (0, 256):
        c = gpu.ChannelTG(s)
        assert c.autotune(force=force)[0] == force
        c.upload(Q, PR)
        c.set_dt(DT)
        c.SOLVERRK3_MOM_tg(0)
        c.advance(1, DT, 1e-6, 0.5)
        Qg = c.download()[0]
        c.close()
        for i in range(3):
            e = float(np.abs(Qg[i] - Qo[i]).max() / np.abs(Qo[i]).max())
            assert e <= 1e-11, (force, i, e)
