"""A context on a device with room for its fields but not for the pivots of the scan y-solve."""
import math

import numpy as np
import pytest
import torch

from chapsim import gpu
from chapsim.mesh import channel_setup
from chapsim.fields import initial_field

pytestmark = pytest.mark.gpu


def test_context_without_room_for_the_pivots():
    L, M, N = 384, 128, 384
    s = channel_setup(L, M, N, 2 * math.pi, math.pi, 2.0, 2800.0)
    pivots = (L // 2 + 1) * M * N * 8
    Q, PR = initial_field(s, 79, 0.1)
    out = []
    filler = None
    for full in (False, True):
        if full:
            torch.cuda.empty_cache()
            free = torch.cuda.mem_get_info()[0]
            filler = torch.empty(free - need + pivots // 2, dtype=torch.uint8, device="cuda")
        before = torch.cuda.mem_get_info()[0]
        c = gpu.ChannelTG(s)
        need = before - torch.cuda.mem_get_info()[0]
        assert bool(c.choice & 64) != full
        filler = None
        torch.cuda.empty_cache()
        if not full:
            c.autotune(force=c.choice & ~64)  # the hybrid here too
        c.upload(Q, PR)
        c.set_dt(1e-3)
        c.advance(2, 1e-3, 1e-6, 0.5)
        out.append(c.download())
        c.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
