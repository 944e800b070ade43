"""What a context says about the step it runs: the kernels per step, and the kernel variants."""
import math

import numpy as np
import pytest

from chapsim import gpu, thermo
from chapsim.mesh import channel_setup, xinout_setup
from chapsim.fields import initial_field, xinout_fields_from_tg

pytestmark = pytest.mark.gpu

HX, HZ, REN, DT = 2 * math.pi, math.pi, 2800.0, 1e-3


def _tg(L, M, N, precision="fp64", force=None):
    s = channel_setup(L, M, N, HX, HZ, 2.0, REN)
    c = gpu.ChannelTG(s, precision=precision)
    if force is not None:
        c.autotune(force=force)
    c.upload(*initial_field(s, 71, 0.1))
    c.set_dt(DT)
    return c


def _thermal(c, M):
    rows, T0 = thermo.synthetic_table()
    tab = thermo.SplineTable.from_rows(rows, T0)
    DH = np.zeros(c.field_shape())
    DH[:, 1:M + 1] = 1e-3
    c.thermal_init(tab, DH, 0.5, 0.5, 1.0 / REN / (tab.ref["M0"] * tab.ref["CP0"] / tab.ref["K0"]))


def _io(L, M, N, precision="fp64", ivisscheme=gpu.VIS_EXPLICIT, thermal=False, force=None):
    s = channel_setup(L, M, N, HX, HZ, 2.0, REN)
    c = gpu.ChannelIO(s, ivisscheme=ivisscheme, precision=precision)
    if force is not None:
        c.autotune(force=force)
    Q, PR = initial_field(s, 73, 0.1)
    ones = np.ones(c.field_shape())
    c.upload_io(Q, PR, ones, ones, ones)
    c.set_dt(DT)
    if thermal:
        _thermal(c, M)
    return c


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_kernels_per_step(precision):
    ctxs = [_tg(64, 32, 64, precision, force) for force in (None, 0, 2, 4, 6, 8, 64)]
    ctxs += [_io(32, 32, 32, precision, iv, th) for iv in (gpu.VIS_EXPLICIT, gpu.VIS_IMPLICIT) for th in (False, True)]
    for c in ctxs:
        before = c.launch_count()
        c.advance(3, DT, 1e-6, 0.5)
        assert c.launch_count() - before == 3 * c.kernels_per_step()
        c.close()


@pytest.mark.parametrize("thermal", [False, True])
def test_kernels_per_step_xinout(thermal):
    LT, L, M, N = 32, 64, 32, 32
    tg = _tg(LT, M, N)
    io = gpu.ChannelXinout(xinout_setup(L, M, N, 2 * HX, HZ, 2.0, REN), tg=tg)
    G, P = xinout_fields_from_tg(tg.download()[0], L)
    ones = np.ones(io.field_shape())
    io.upload_io(G, P, ones, ones, ones)
    io.set_dt(DT)
    if thermal:
        _thermal(io, M)
        io.thermal_inlet([1.0, 0.0, 1.0, 1.0, 1.0, 1.0, 0.0])
    before = io.launch_count()
    io.advance(2, DT, 1e-6, 0.5)
    assert io.launch_count() - before == 2 * io.kernels_per_step()
    io.close()
    tg.close()


@pytest.mark.parametrize("kind,shape,precision", [
    ("tg", (32, 32, 32), "fp64"), ("tg", (64, 32, 32), "fp64"), ("tg", (128, 32, 64), "fp64"), ("tg", (192, 32, 32), "fp64"),
    ("tg", (64, 32, 32), "mixed"), ("io", (64, 32, 32), "fp64"), ("io", (32, 32, 192), "fp64"), ("io", (64, 32, 32), "mixed")])
def test_starting_choice_is_what_runs(kind, shape, precision):
    """Forcing the choice that a new context names changes no bit of its fields."""
    make = _tg if kind == "tg" else _io
    a = make(*shape, precision=precision)
    b = make(*shape, precision=precision, force=a.choice)
    assert b.choice == a.choice
    for c in (a, b):
        c.advance(3, DT, 1e-6, 0.5)
    get = (lambda c: c.download()) if kind == "tg" else (lambda c: c.download_io())
    for x, y in zip(get(a), get(b)):
        assert np.array_equal(x, y)
    a.close()
    b.close()


@pytest.mark.parametrize("shape", [(32, 32, 32), (32, 32, 384)])
def test_main_domain_keeps_a_forced_choice(shape):
    """The bits of the periodic channel's kernels stay clear in a main-domain context."""
    c = _io(*shape)
    assert c.choice & ~(1 | 16 | 32 | 64) == 0
    for force in (0, 1, 16, 64):
        assert c.autotune(force=force)[0] == force
    c.close()
