"""The line solves in registers at every line length, against the oracle's
sequential ones: the FP64 z and y sweeps of the periodic channel (both tile
widths), the Crank-Nicolson sweeps of the main domain, the FP64 Poisson
y-solve with the register transforms, and the scan y-solve of mixed-precision
contexts; and the energy equation's tiles.

REN = 2 makes the implicit operators stiff (|a| = F / dz^2 from 1 to 190 at
these grids, where the recurrences' ratio rho approaches 1 and carries travel
across every segment); the velocities after the projection and one step stay
within 1e-11 of the oracle, the bound of the step tests: the operators'
condition number 1 + 4|a| < 800 times 2^-53 is 1e-13 per sweep.
"""
import math

import numpy as np
import pytest

import oracle as orc
from oracle import Oracle
from chapsim import gpu, thermo
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


@pytest.mark.parametrize("shape", [(32, 384, 64), (64, 32, 32), (96, 64, 96), (128, 96, 384), (192, 128, 128),
                                   (256, 192, 192), (384, 256, 256)])
def test_stiff_main_domain_sweeps_match_oracle(shape):
    """Non-uniform density and viscosity (each row has its own coefficients), two steps at REN = 2."""
    L, M, N = shape
    HX, HZ, REN, DT = 2 * math.pi, math.pi, 2.0, 5e-3
    s = channel_setup(L, M, N, HX, HZ, 2.0, REN)
    G, PR = initial_field(s, 43, 0.1)
    k, j, i = np.meshgrid(np.arange(N), np.arange(M + 2), np.arange(L), indexing="ij")
    rho = 1.0 + 0.05 * np.sin(2 * np.pi * i / L) * np.cos(2 * np.pi * k / N) + 0.02 * np.cos(np.pi * j / (M + 2))
    mu0 = 1.0 + 0.1 * np.cos(2 * np.pi * i / L + 0.3) * np.sin(np.pi * j / (M + 2))
    mu = mu0 * (1.0 + 0.03 * np.sin(2 * np.pi * k / N + 0.7))
    o = Oracle(L, M, N, HX, HZ, 2.0, REN, DT0=DT, DTMIN=1e-6, CFLGV=1e9, threads=8)
    o.io_set_fields(G, PR, rho, mu0, mu)
    o.io_set_vis_scheme(1)
    o.set_dt(DT)
    assert o.io_run_steps(2)[0] == 0
    Go = o.io_get_fields()[0]
    o.close()
    c = gpu.ChannelIO(s, ivisscheme=gpu.VIS_IMPLICIT)
    c.upload_io(G, PR, rho, mu0, mu)
    c.set_dt(DT)
    c.advance(2, DT, 1e-6, 1e9)
    Gg = c.download_io()[0]
    c.close()
    for q in range(3):
        e = float(np.abs(Gg[q] - Go[q]).max() / np.abs(Go[q]).max())
        assert e <= 1e-11, (q, e)


@pytest.mark.parametrize("shape", [(64, 32, 32), (32, 64, 96), (384, 96, 64), (96, 128, 384), (128, 192, 128),
                                   (256, 256, 192), (192, 384, 256)])
def test_poisson_solve_matches_oracle(shape):
    """The default FP64 solve (inverse x and both z transforms on registers, the y-solve by affine maps in
    registers) at every line length, 1e-12 of the oracle as for the other y-solves."""
    L, M, N = shape
    s = channel_setup(L, M, N, 2 * math.pi, math.pi, 2.0, 2800.0)
    o = Oracle(L, M, N, 2 * math.pi, math.pi, 2.0, 2800.0, threads=8)
    rhs = np.random.default_rng(19).standard_normal((N, M, L))
    full = np.zeros((N, M + 2, L))
    full[:, 1:M + 1, :] = rhs
    ref = o.poisson(full)
    o.close()
    c = gpu.ChannelTG(s)
    got = c.FFT99_POIS3D_periodicxz(rhs)
    c.close()
    assert float(np.abs(got[:, 1:M + 1] - ref[:, 1:M + 1]).max() / np.abs(ref[:, 1:M + 1]).max()) <= 1e-12


@pytest.mark.parametrize("shape", [(64, 32, 32), (32, 64, 96), (384, 96, 64), (96, 128, 384), (128, 192, 128),
                                   (256, 256, 192), (192, 384, 256)])
def test_mixed_scan_matches_warp_solve(shape):
    """The scan y-solve of a mixed-precision context against its warp solve at every line length, the FP64
    spectrum of the Poisson entry included; held to the bound that an FP32 spectrum would meet, one ulp a
    mode and log2(L N) 2^-24 < 1.1e-6 of the inverse transforms' rounding (2e-6)."""
    L, M, N = shape
    s = channel_setup(L, M, N, 2 * math.pi, math.pi, 2.0, 2800.0)
    rhs = np.random.default_rng(23).standard_normal((N, M, L))
    p = []
    for force in (0, 64):
        c = gpu.ChannelTG(s, precision="mixed")
        assert c.autotune(force=force)[0] == force
        p.append(c.FFT99_POIS3D_periodicxz(rhs)[:, 1:M + 1])
        c.close()
    assert float(np.abs(p[1] - p[0]).max() / np.abs(p[0]).max()) <= 2e-6


@pytest.mark.parametrize("shape", [(32, 32, 32), (96, 64, 192), (128, 32, 384), (256, 96, 64), (384, 192, 32)])
def test_energy_tiles_match_oracle(shape):
    """Two heated steps over grids whose z chunks are short, long or uneven, constant flux at both walls; 1e-10 as
    in the thermal step tests (which hold the isothermal walls)."""
    L, M, N = shape
    HX, HZ, REN = 2 * math.pi, math.pi, 2800.0
    s = channel_setup(L, M, N, HX, HZ, 2.0, REN)
    Q, PR = initial_field(s, 47, 0.1)
    rows, T0 = thermo.synthetic_table()
    tab = thermo.SplineTable.from_rows(rows, T0)
    cthecd = 1.0 / REN / (tab.ref["M0"] * tab.ref["CP0"] / tab.ref["K0"])
    DH = np.zeros((N, M + 2, L))
    DH[:, 1:M + 1, :] = 1e-3 * np.random.default_rng(29).uniform(-1.0, 1.0, (N, M, L))
    ones = np.ones((N, M + 2, L))
    o = Oracle(L, M, N, HX, HZ, 2.0, REN, DT0=1e-3, DTMIN=1e-6, CFLGV=0.5, threads=8)
    o.io_set_fields(Q, PR, ones, ones, ones)
    ot = orc.PropTable(tab.lists)
    o.thermal_enable(ot, DH, 0.5, 0.5, cthecd)
    o.set_dt(1e-3)
    assert o.io_run_steps(2)[0] == 0
    to = o.thermal_get()
    o.close()
    c = gpu.ChannelIO(s)
    c.upload_io(Q, PR, ones, ones, ones)
    c.thermal_init(tab, DH, 0.5, 0.5, cthecd)
    c.set_dt(1e-3)
    c.advance(2, 1e-3, 1e-6, 0.5)
    tg = c.download_thermal()
    c.close()
    for q in ("DH", "H", "T", "D", "M", "K", "CP"):
        assert float(np.abs(tg[q] - to[q]).max() / np.abs(to[q]).max()) <= 1e-10, q
