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
