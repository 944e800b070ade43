"""PRCALC_tg: PR + DPH - alpha dt nu / 2 RHSLLPHI, with RHSLLPHI the divergence that the Poisson solve was given.

The FP64 update takes the discrete Laplacian of DPH for it, which holds for the reference's Poisson operator only: the
caller's wavenumbers AK1 and AK3 need not be the second difference's, nor the rows AMPH, ACPH, APPH conservative with
Neumann walls.  With the exact second derivative's wavenumbers, and with an upper wall row of a fixed pressure, the FP64
context is held to the mixed-precision one (which keeps RHSLLPHI) at REN = 2, where the term is of DPH's own size.  Bound:
the FP32 velocities' rounding, 2^-24, enters RHSLLPHI times alpha dt nu / 2 as 2^-24 |u| nu 3 / dx < 1e-6 and DPH by less,
relative to |PR| about 0.1 to 1; 1e-4.
"""
import math

import numpy as np
import pytest

from chapsim import gpu
from chapsim.mesh import channel_setup
from chapsim.fields import initial_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,force", [((64, 64, 64), None), ((64, 32, 96), 64 | 8), ((256, 32, 256), 64 | 8),
                                         ((384, 32, 32), 0)])
@pytest.mark.parametrize("operator", ["wavenumbers", "wall row"])
def test_pressure_update_with_other_operators(shape, force, operator):
    L, M, N = shape
    HX, HZ = 2 * math.pi, math.pi
    s = channel_setup(L, M, N, HX, HZ, 2.0, 2.0)
    if operator == "wavenumbers":
        kx = np.minimum(np.arange(L), L - np.arange(L)) * 2 * math.pi / HX
        kz = np.minimum(np.arange(N), N - np.arange(N)) * 2 * math.pi / HZ
        s.AK1, s.AK3 = kx * kx, kz * kz
    else:
        s.ACPH[M] -= 2.0 * s.AMPH[M]
    Q, PR = initial_field(s, 53, 0.1)
    got = []
    for precision in ("fp64", "mixed"):
        c = gpu.ChannelTG(s, precision=precision)
        if force is not None:
            assert c.autotune(force=force)[0] == force
        c.upload(Q, PR)
        c.set_dt(0.05)
        c.SOLVERRK3_MOM_tg(0)
        got.append(c.download()[1][:, 1:M + 1])
        c.close()
    assert float(np.abs(got[0] - got[1]).max() / np.abs(got[1]).max()) <= 1e-4
