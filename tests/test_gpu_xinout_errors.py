"""The coupled step when the periodic domain reports a non-finite field: both domains are idle when the call returns,
and neither carries the error into the next one."""
import math

import numpy as np
import pytest
import torch

from chapsim import gpu
from chapsim.mesh import channel_setup, xinout_setup
from chapsim.fields import initial_field, xinout_fields_from_tg

pytestmark = pytest.mark.gpu

LT, L, M, N = 32, 256, 128, 128


def _start(tg, io, Q, PR):
    tg.upload(Q, PR)
    tg.set_dt(1e-3)
    G, P = xinout_fields_from_tg(Q, L)
    ones = np.ones(io.field_shape())
    io.upload_io(G, P, ones, ones, ones)
    io.set_dt(1e-3)


def test_tg_error_leaves_both_domains_idle_and_clean():
    HZ, REN, DX = math.pi, 2800.0, 2 * math.pi / 64
    st, sx = channel_setup(LT, M, N, LT * DX, HZ, 2.0, REN), xinout_setup(L, M, N, L * DX, HZ, 2.0, REN)
    Q, PR = initial_field(st, 67, 0.1)
    out = []
    for bad in (False, True):
        tg = gpu.ChannelTG(st)
        io = gpu.ChannelXinout(sx, tg=tg)
        if bad:
            _start(tg, io, Q, PR)
            Qn = Q.copy()
            Qn[0, 3, 5, 7] = float("nan")
            tg.upload(Qn, PR)
            with pytest.raises(gpu.ChapsimError) as e:
                io.advance(1, 1e-3, 1e-6, 0.5)
            assert torch.cuda.ExternalStream(io.stream_handle()).query()
            assert e.value.code == -2 and "TG domain" in str(e.value)
        _start(tg, io, Q, PR)
        io.advance(2, 1e-3, 1e-6, 0.5)
        out.append(io.download_io() + tg.download())
        io.close()
        tg.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
