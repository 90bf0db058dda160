"""Forward and gradient calls on caller potentials replay their batches from graphs: one for the full
batches and one for the last, whatever the number of batches, the lens, the potential, the probes and the
targets, with the values of direct launches bit for bit, from host and from device memory."""
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
from conftest import rel_l2  # noqa: E402
from oracle import oracle as orc  # noqa: E402

pytestmark = pytest.mark.gpu


def problem(seed, n=128, S=5, n_probe=23, batch=5):
    p, _ = cases.stem_small(n=n)
    p.set_detectors([(0.0, 0.012), (0.025, 0.06)])
    p.cond_lens.c10, p.cond_lens.c30 = -30.0 - seed, 2.0e4 + 100.0 * seed
    p.ckpt_interval, p.probe_batch = 2, batch
    rng = np.random.default_rng(seed)
    V = cases.random_phase_slices(p, S, seed=seed, amp=0.4)
    xy = np.ascontiguousarray(p.lx / 2 + rng.uniform(-1.5, 1.5, (n_probe, 2)))
    return p, V, xy


def device_calls(ctx, p, V, xy, T):
    """Forward and gradient with the slices and the gradient in device memory."""
    dV = torch.from_numpy(V).cuda()
    gV = torch.full_like(dV, float("nan"))
    I = np.empty((len(xy), p.n_det), np.float32)
    loss, g10, g30 = C.c_double(), C.c_double(), C.c_double()
    cp, L = p.c(), cb.lib()

    def f(t):
        return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_float))
    xyp = xy.ctypes.data_as(C.POINTER(C.c_double))
    torch.cuda.synchronize()
    ctx.check(L.ms_stem_forward_potential(ctx.handle, C.byref(cp), f(dV), V.shape[0], 1, 0.5, xyp, len(xy),
                                          I.ctypes.data_as(C.POINTER(C.c_float))))
    ctx.check(L.ms_stem_backward(ctx.handle, C.byref(cp), f(dV), V.shape[0], 1, 0.5, xyp, len(xy),
                                 T.ctypes.data_as(C.POINTER(C.c_float)), C.byref(loss), f(gV), C.byref(g10),
                                 C.byref(g30)))
    return I, (loss.value, gV.cpu().numpy(), g10.value, g30.value)


def same(a, b):
    return a[0] == b[0] and np.array_equal(a[1], b[1]) and a[2] == b[2] and a[3] == b[3]


def test_two_graphs_serve_every_batch_and_call():
    counts = []
    with cb.Context(0) as ctx:
        for seed in (1, 2, 3):
            p, V, xy = problem(seed)
            T = np.zeros((len(xy), p.n_det), np.float32)
            ctx.stem_forward_potential(p, V, 0.5, xy)
            counts.append(ctx.last_graph_captures)
            ctx.stem_backward(p, V, 0.5, xy, T)
            counts.append(ctx.last_graph_captures)
    assert counts == [2, 2, 0, 0, 0, 0]


@pytest.mark.parametrize("n,n_probe,batch", [(128, 23, 5), (256, 4, 0), (128, 8, 4)])
def test_replays_follow_their_inputs(n, n_probe, batch):
    with cb.Context(0) as ctx, cb.Context(0) as direct:
        direct.set_graphs(False)
        for seed in (1, 2, 1):
            p, V, xy = problem(seed, n=n, n_probe=n_probe, batch=batch)
            I = ctx.stem_forward_potential(p, V, 0.5, xy)
            T = (I * (1 + 0.05 * np.random.default_rng(seed).standard_normal(I.shape))).astype(np.float32)
            g = ctx.stem_backward(p, V, 0.5, xy, T)
            assert np.array_equal(I, direct.stem_forward_potential(p, V, 0.5, xy))
            assert same(g, direct.stem_backward(p, V, 0.5, xy, T))
            Id, gd = device_calls(ctx, p, V, xy, T)
            assert np.array_equal(I, Id) and same(g, gd)
            assert rel_l2(I, orc.stem_forward_potential(p, V, 0.5, xy)) < 1e-5
            ref = orc.stem_backward(p, V, 0.5, xy, T)
            assert rel_l2(g[1], ref[1]) < 1e-4 and abs(g[2] - ref[2]) < 1e-4 * abs(ref[2])


def test_more_kinds_of_call_than_graphs_are_kept():
    """Ten grids' graphs in turn, twice: the oldest make room, and the values stay."""
    with cb.Context(0) as ctx:
        sizes = [(128, 128 << k) for k in range(5)] + [(256, 128 << k) for k in range(5)]
        first = []
        for rep in range(2):
            for i, (nx, ny) in enumerate(sizes):
                p, V, xy = problem(i, n=nx, S=2, n_probe=4, batch=4)
                p.ny = ny
                V = cases.random_phase_slices(p, 2, seed=i, amp=0.4)
                I = ctx.stem_forward_potential(p, V, 0.5, xy)
                assert ctx.last_graph_captures == 1
                if rep == 0:
                    first.append(I)
                else:
                    assert np.array_equal(I, first[i])
        ctx.stem_forward_potential(p, V, 0.5, xy)
        assert ctx.last_graph_captures == 0


def test_thickness_series_graph_serves_every_probe():
    p, at = cases.thickness_small(n=128, nconf=2)
    p.iw_type = cb._abi.MS_IW_CONVERGENT
    p.cond_lens.outer_aper_ang = 0.02
    p.iw_x = p.iw_y = p.lx / 2
    with cb.Context(0) as ctx:
        sim = cb.ThicknessSimulator(ctx=ctx)
        for i, c10 in enumerate((-20.0, -60.0)):
            p.cond_lens.c10 = c10
            out = sim.run(p, at).thickness_frames
            assert ctx.last_graph_captures == (1 if i == 0 else 0)
            assert rel_l2(out, orc.simulate_thickness(p, at)) < 1e-5
