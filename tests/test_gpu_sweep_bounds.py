"""Bounds of the line solves that the other tests leave wide or to one variant.

* The untuned FP64 step at REN = 2 (stiff sweeps, every default variant: fused, bulk-staged and wide right-hand sides,
  the register y-solve), velocities and pressure against the oracle.  Velocities 1e-11 as in the forced variants' test.
  Pressure: a sweep's 1e-13 of |u| < 2 reaches DPH through div / (alpha dt) and the inverse Laplacian as
  1e-13 |u| / (alpha dt k), alpha dt >= 6.7e-3 and k >= 1, 3e-11 of |PR| about 1, over two substeps; 1e-10.
* The Poisson entry of a mixed-precision context solves an FP64 spectrum: the scan y-solve at every line length
  within 1e-12 of the oracle, as the FP64 contexts' solves.
* The mixed-precision step with the scan y-solve (its FP32 spectrum) against the warp solve at every line length: each
  solves in FP64 and rounds once, so five steps differ by a few FP32 roundings; 1e-5 as for the sequential solve.
"""
import math

import numpy as np
import pytest

from oracle import Oracle
from chapsim import gpu
from chapsim.mesh import channel_setup
from chapsim.fields import initial_field

pytestmark = pytest.mark.gpu

LENGTHS = [(64, 32, 32), (32, 64, 96), (384, 96, 64), (96, 128, 384), (128, 192, 128), (256, 256, 192), (192, 384, 256)]


def _rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("shape", [(32, 32, 32), (64, 96, 64), (128, 64, 192), (96, 192, 256), (192, 128, 96),
                                   (256, 64, 384), (384, 256, 64), (32, 384, 128)])
def test_stiff_default_step_matches_oracle(shape):
    L, M, N = shape
    HX, HZ, REN, DT = 2 * math.pi, math.pi, 2.0, 0.05
    s = channel_setup(L, M, N, HX, HZ, 2.0, REN)
    Q, PR = initial_field(s, 83, 0.1)
    o = Oracle(L, M, N, HX, HZ, 2.0, REN, DT0=DT, DTMIN=1e-6, CFLGV=0.5, threads=8)
    o.set_fields(Q, PR)
    o.set_dt(DT)
    o.substep(0)
    assert o.run_steps(1)[0] == 0
    Qo, Po = o.get_fields()[:2]
    o.close()
    c = gpu.ChannelTG(s)
    c.upload(Q, PR)
    c.set_dt(DT)
    c.SOLVERRK3_MOM_tg(0)
    c.advance(1, DT, 1e-6, 0.5)
    Qg, Pg = c.download()
    c.close()
    for i in range(3):
        assert _rel(Qg[i], Qo[i]) <= 1e-11
    assert _rel(Pg[:, 1:M + 1], Po[:, 1:M + 1]) <= 1e-10


@pytest.mark.parametrize("shape", LENGTHS)
def test_mixed_context_poisson_solve_matches_oracle(shape):
    L, M, N = shape
    s = channel_setup(L, M, N, 2 * math.pi, math.pi, 2.0, 2800.0)
    o = Oracle(L, M, N, 2 * math.pi, math.pi, 2.0, 2800.0, threads=8)
    rhs = np.random.default_rng(89).standard_normal((N, M, L))
    full = np.zeros((N, M + 2, L))
    full[:, 1:M + 1, :] = rhs
    ref = o.poisson(full)
    o.close()
    c = gpu.ChannelTG(s, precision="mixed")
    assert c.autotune(force=64)[0] == 64
    got = c.FFT99_POIS3D_periodicxz(rhs)
    c.close()
    assert _rel(got[:, 1:M + 1], ref[:, 1:M + 1]) <= 1e-12


@pytest.mark.parametrize("shape", LENGTHS)
def test_mixed_step_scan_matches_warp_solve(shape):
    L, M, N = shape
    s = channel_setup(L, M, N, 2 * math.pi, math.pi, 2.0, 2800.0)
    Q, PR = initial_field(s, 97, 0.1)
    out = []
    for force in (0, 64):
        c = gpu.ChannelTG(s, precision="mixed")
        assert c.autotune(force=force)[0] == force
        c.upload(Q, PR)
        c.set_dt(2e-3)
        c.SOLVERRK3_MOM_tg(0)
        c.advance(5, 2e-3, 1e-6, 0.5)
        out.append(c.download())
        c.close()
    for i in range(3):
        assert _rel(out[1][0][i], out[0][0][i]) <= 1e-5
