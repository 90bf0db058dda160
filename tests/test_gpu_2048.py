"""The slice steps of 2048 points (64-thread teams) on each axis and both, on both slice stores,
with waves of different slice counts, against the FP64 oracle; and in an uneven batch.  The
tolerance is the parity tests' 1e-5: the transforms' error per slice is that of the other lengths
(2e-7 on a random wave)."""
from __future__ import annotations

import numpy as np
import pytest

import cudaem_b200 as cb
from cudaem_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, float) - b) / np.linalg.norm(b)


def problem(nx, ny, nconf, cells_z=2):
    p, at = wl.cbed_si(cells=(max(2, nx // 128), max(2, ny // 128), cells_z), n=nx, nconf=nconf)
    p.ny = ny
    return p, at


@pytest.mark.parametrize("store", [True, False])
@pytest.mark.parametrize("nx,ny,nconf", [(2048, 128, 3), (128, 2048, 2), (2048, 512, 1), (2048, 2048, 1)])
def test_axes(nx, ny, nconf, store):
    p, at = problem(nx, ny, nconf)
    with cb.Context() as ctx:
        ctx.set_transmission_store(store)
        out = cb.MulSimulator(ctx=ctx).executionCBED(p, at)
    assert rel(out.image_intensity, orc.simulate_cbed(p, at)) < 1e-5


def test_uneven_batch(ctx):
    jobs = [problem(2048, 2048, 1, 1), problem(256, 256, 2, 3), problem(2048, 2048, 2, 3)]
    outs, _ = cb.MulSimulator(ctx=ctx).executionMany(jobs)
    for (p, at), o in zip(jobs, outs):
        assert rel(o.image_intensity, orc.simulate_cbed(p, at)) < 1e-5


@pytest.mark.parametrize("nx,ny,n_probe", [(2048, 128, 4), (128, 2048, 4), (2048, 2048, 1), (128, 128, 5)])
def test_gradient_sees_the_forward_call_s_intensities(ctx, nx, ny, n_probe):
    """At its own forward intensities the loss is what rounding the targets to float leaves, at every length
    and on both slice stores (fewer than four probes read sigma V): at most half a unit in the last place
    per intensity.  Gradients as far from the oracle's as at the other lengths (1e-4)."""
    p, _ = wl.stem_sto(cells=(3, 3, 2), n=nx, nconf=1, scan=(1, 1), step=0.4, batch=0)
    p.ny = ny
    p.set_detectors([(0.0, 0.012), (0.025, 0.06)])
    p.ckpt_interval = 2
    rng = np.random.default_rng(nx + n_probe)
    V = rng.uniform(0, 0.4, (5, ny, nx)).astype(np.float32)
    xy = p.lx / 2 + rng.uniform(-1.0, 1.0, (n_probe, 2))
    I = ctx.stem_forward_potential(p, V, 0.5, xy)
    loss = ctx.stem_backward(p, V, 0.5, xy, I)[0]
    assert loss <= np.sum((I.astype(float) * 2.0 ** -24) ** 2) * 1.0001
    if nx * ny < 2048 * 2048:
        T = (I * (1 + 0.05 * rng.standard_normal(I.shape))).astype(np.float32)
        _, gV, g10, _ = ctx.stem_backward(p, V, 0.5, xy, T)
        _, gVo, g10o, _ = orc.stem_backward(p, V, 0.5, xy, T)
        assert rel(gV, gVo) < 1e-4 and abs(g10 - g10o) < 1e-4 * abs(g10o)
