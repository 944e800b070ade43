"""Settings that change after a step has been captured: the next advance runs
with the new setting, alone or in an ensemble."""
import math

import numpy as np
import pytest

from chapsim import gpu, thermo
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


def test_ensemble_error_is_not_carried_into_the_next_call():
    """Two of three members report a NaN; with good fields in all of them the ensemble advances as new members do."""
    shapes = [(32, 32, 32), (64, 32, 32), (32, 64, 32)]
    out = []
    for bad in (False, True):
        grp = [_channel(sh, 91 + k) for k, sh in enumerate(shapes)]
        e = gpu.Ensemble(grp)
        if bad:
            good = [c.download() for c in grp]
            for c, (Q, PR) in zip(grp[::2], good[::2]):
                Qn = Q.copy()
                Qn[0, 3, 5, 7] = float("nan")
                c.upload(Qn, PR)
            with pytest.raises(gpu.ChapsimError) as err:
                e.advance(1, 2e-3, 1e-6, 0.5)
            assert err.value.code == -2
            for c, (Q, PR) in zip(grp, good):
                c.upload(Q, PR)
                c.set_dt(2e-3)
        else:
            for c in grp:  # as the others, through the host
                c.upload(*c.download())
        e.advance(2, 2e-3, 1e-6, 0.5)
        out.append([x for c in grp for x in c.download()])
        e.close()
        for c in grp:
            c.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)


def _heated(seed=63):
    L = M = N = 32
    s = channel_setup(L, M, N, 2 * math.pi, math.pi, 2.0, 2800.0)
    Q, PR = initial_field(s, seed, 0.1)
    rows, T0 = thermo.synthetic_table()
    tab = thermo.SplineTable.from_rows(rows, T0)
    c = gpu.ChannelIO(s, ivisscheme=gpu.VIS_IMPLICIT)
    ones = np.ones(c.field_shape())
    c.upload_io(Q, PR, ones, ones, ones)
    DH = np.zeros(c.field_shape())
    DH[:, 1:M + 1] = 1e-3 * np.random.default_rng(seed).uniform(-1.0, 1.0, (N, M, L))
    c.thermal_init(tab, DH, 0.5, 0.5, 1.0 / 2800.0 / (tab.ref["M0"] * tab.ref["CP0"] / tab.ref["K0"]))
    c.set_dt(1e-3)
    return c, tab


@pytest.mark.parametrize("what", ["table", "mlp"])
def test_new_property_source_reaches_the_captured_step(what):
    """A second property table, or a model of another range, after the first captured step.  The second context is told
    a setting that it already has besides, which asks for a new capture by itself."""
    out = []
    for again in (False, True):
        c, tab = _heated()
        lo, hi = float(tab.lists["DH"][0]), float(tab.lists["DH"][-1])
        if what == "mlp":
            c.mlp_init(lo + 0.02 * (hi - lo), hi - 0.02 * (hi - lo), seed=5)
            c.thermal_use_mlp(True)
        c.advance(1, 1e-3, 1e-6, 0.5)
        if what == "table":
            c.prop_table_init(tab, fix_swap=True)
        else:
            c.mlp_init(lo + 0.2 * (hi - lo), hi - 0.2 * (hi - lo), seed=5)
        if again:
            c.set_buoyancy(0, 0.0)
        c.advance(2, 1e-3, 1e-6, 0.5)
        out.append(list(c.download_io()) + list(c.download_thermal().values()))
        c.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
