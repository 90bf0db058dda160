"""Sizes that a call chooses by the free device memory: the same on every call, although the buffers of the
call before it stay; and memory that only makes a call faster gives way to a call that needs it.  The
device is filled up to a few hundred megabytes for this; a call's launch count shows how it was split."""
from __future__ import annotations

import contextlib
import ctypes as C
import os
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import cases  # noqa: E402
import cudaem_b200 as cb  # noqa: E402
from cudaem_b200 import _abi as abi  # noqa: E402

pytestmark = pytest.mark.gpu
MB = 1 << 20


@contextlib.contextmanager
def only_free(nbytes):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    ballast = torch.empty(torch.cuda.mem_get_info()[0] - int(nbytes), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del ballast
        torch.cuda.empty_cache()


def fptr(t):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_float))


def probes(p, n):
    return np.ascontiguousarray(p.lx / 2 + np.random.default_rng(3).uniform(-1.5, 1.5, (n, 2)))


def forward(ctx, p, V, xy):
    I = np.empty((len(xy), p.n_det), np.float32)
    cp = p.c()
    ctx.check(cb.lib().ms_stem_forward_potential(ctx.handle, C.byref(cp), fptr(V), V.shape[0], 1, 0.5,
                                                 xy.ctypes.data_as(C.POINTER(C.c_double)), len(xy),
                                                 I.ctypes.data_as(C.POINTER(C.c_float))))
    return I, ctx.last_launch_count


def phases(p, S):
    g = torch.Generator(device="cuda").manual_seed(5)
    return torch.rand((S, p.ny, p.nx), generator=g, device="cuda") * 0.02


@pytest.fixture
def fixed():
    """A context on one tile shape (no tuner launches in the counts)."""
    with cb.Context(0) as c:
        c.set_tile_shape(0)
        yield c


def test_forward_keeps_its_route_and_yields_its_store(fixed):
    p, _ = cases.stem_small(n=128)
    p.set_detectors([(0.0, 0.012)])
    free, N = 600 * MB, 128 * 128
    S = int(0.225 * free) // (8 * N)   # its transmission: above a fifth of the free memory, below a quarter
    V = phases(p, S)
    xy = probes(p, 4)
    p2, _ = cases.stem_small(n=512)
    p2.set_detectors([(0.0, 0.012)])
    big = np.zeros((int(0.88 * free) // (4 * 512 * 512), 512, 512), np.float32)
    few = fixed.stem_forward_potential(p2, big[:3], 0.5, xy[:1])
    forward(fixed, p, V[:2], xy)       # the grid's tables, whose launches would count in the first call
    with only_free(free):
        calls = [forward(fixed, p, V, xy) for _ in range(3)]
        assert calls[0][1] == calls[1][1] == calls[2][1]
        assert np.array_equal(calls[0][0], calls[1][0]) and np.array_equal(calls[0][0], calls[2][0])
        # one probe on host slices that need nearly all of the memory: the store gives way
        vacuum = fixed.stem_forward_potential(p2, big, 0.5, xy[:1])
    assert np.allclose(vacuum, few, rtol=1e-3)   # empty slices keep the band-limited probe


def test_forward_without_room_for_its_store(fixed):
    """Above a quarter of the free memory, or when the allocation fails, t is formed probe by probe: the same
    values."""
    p, _ = cases.stem_small(n=128)
    p.probe_batch = 2
    free = 300 * MB
    V = phases(p, int(0.4 * free) // (8 * 128 * 128))
    xy = probes(p, 4)
    forward(fixed, p, V[:2], xy[:3])
    with only_free(free):
        tight, n_tight = forward(fixed, p, V, xy)
    few = V[:40]
    fixed.set_fault_injection(abi.MS_INJECT_ALLOC_FAIL)
    failed, n_failed = forward(fixed, p, few, xy)
    fixed.set_fault_injection(abi.MS_INJECT_NONE)
    with_store, n_store = forward(fixed, p, few, xy)
    assert np.array_equal(failed, with_store) and n_failed == n_store - 1
    roomy, n_roomy = forward(fixed, p, V, xy)
    assert np.array_equal(tight, roomy) and n_tight == n_roomy - 1


def gradient(ctx, p, V, xy, n):
    target = np.zeros((len(xy), p.n_det), np.float32)
    gV = torch.empty_like(V)
    loss, g10, g30 = C.c_double(), C.c_double(), C.c_double()
    cp = p.c()
    ctx.check(cb.lib().ms_stem_backward(
        ctx.handle, C.byref(cp), fptr(V), n, 1, 0.5, xy.ctypes.data_as(C.POINTER(C.c_double)), len(xy),
        target.ctypes.data_as(C.POINTER(C.c_float)), C.byref(loss), fptr(gV), C.byref(g10), C.byref(g30)))
    return loss.value, gV[:n].cpu().numpy(), ctx.last_launch_count


def test_gradient_after_one_of_another_checkpoint_interval(fixed):
    """Checkpoints of every slice leave one buffer large that another interval hardly uses: what it holds is
    not room for the other buffers."""
    p, _ = cases.stem_small(n=256)
    p.set_detectors([(0.0, 0.012)])
    V, xy = phases(p, 64), probes(p, 24)
    gradient(fixed, p, V, xy, 9)
    out = []
    with only_free(600 * MB):
        for k in (1, 32, 1, 8):
            p.ckpt_interval = k
            out.append(gradient(fixed, p, V, xy, 64))
    assert all(abs(o[0] - out[0][0]) <= 1e-12 * out[0][0] and np.array_equal(o[1], out[0][1]) for o in out)


def test_backward_keeps_its_batch(fixed):
    p, _ = cases.stem_small(n=256)
    p.set_detectors([(0.0, 0.012)])
    p.ckpt_interval = 8
    V, xy = phases(p, 64), probes(p, 24)

    def call(n):
        return gradient(fixed, p, V, xy, n)

    call(9)
    with only_free(400 * MB):   # room for about 18 of the 24 probes
        first, second, third = call(64), call(64), call(64)
    assert first[2] == second[2] == third[2]
    assert first[0] == second[0] == third[0]
    assert np.array_equal(first[1], second[1]) and np.array_equal(first[1], third[1])


def test_thickness_keeps_its_groups(fixed):
    p, at = cases.thickness_small(n=512, nconf=6)
    at2 = cases.hrtem_small(n=512, cells=(4, 4, 12), nconf=6)[1]
    sim = cb.ThicknessSimulator(ctx=fixed)
    sim.run(p, at)
    N = 512 * 512
    est = (at2.z.max() - at2.z.min() + 12 * at2.sigma.max()) / p.dz + 3
    with only_free(4.5 * est * N * 8 / 0.6):   # four of the six configurations at a time
        runs = []
        for _ in range(3):
            frames = sim.run(p, at2).thickness_frames.copy()
            runs.append((frames, fixed.last_launch_count))
    assert runs[0][1] == runs[1][1] == runs[2][1]
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][0], runs[2][0])
