"""Caller buffers on the GPU (V_on_device = 1): the same values as through host memory, whichever way
the call writes them."""
from __future__ import annotations

import ctypes as C
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import cases  # noqa: E402
import cudaem_b200 as cb  # noqa: E402

pytestmark = pytest.mark.gpu


def fptr(address):
    return C.cast(C.c_void_p(address), C.POINTER(C.c_float))


@pytest.mark.parametrize("offset", [0, 4, 12, 2])
def test_projected_potential(ctx, offset):
    """Any byte offset: the kernel stores into aligned memory itself, the rest goes through a copy."""
    p, at = cases.hrtem_small(n=128)
    want = ctx.projected_potential(p, at, conf=1)
    guard = 64
    raw = torch.full((want.nbytes + 2 * guard,), 0xA5, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ns = C.c_int()
    cp, ca = p.c(), at.c()
    ctx.check(cb.lib().ms_projected_potential(ctx.handle, C.byref(cp), C.byref(ca), 1,
                                              fptr(raw.data_ptr() + guard + offset), want.size, 1, C.byref(ns)))
    host = raw.cpu().numpy()
    lo, hi = guard + offset, guard + offset + want.nbytes
    assert ns.value == want.shape[0]
    assert np.array_equal(host[lo:hi].view(np.float32).reshape(want.shape), want)
    assert (host[:lo] == 0xA5).all() and (host[hi:] == 0xA5).all()
