"""The short slice steps of small batches (128, 256 and 512 points) against the FP64 oracle: each length
as rows and as columns, both slice stores, batches at and beyond the size where the longer forms take
over, waves of different slice counts, and the filtered column step of the thickness series.  The
tolerance is the parity tests' 1e-5: both twiddles are carried as hi + lo, so a slice's error is that
of the other forms (2e-7 on a random wave)."""
from __future__ import annotations

import numpy as np
import pytest

import cudaem_b200 as cb
from cudaem_b200 import _abi as abi
from cudaem_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, float) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("convergent", [False, True])
@pytest.mark.parametrize("store", [True, False])
@pytest.mark.parametrize("nx,ny,nconf", [(128, 128, 1), (128, 128, 9), (256, 128, 2), (128, 256, 5), (256, 256, 3),
                                         (512, 128, 2), (128, 512, 1), (512, 512, 1), (512, 512, 3), (512, 1024, 1)])
def test_images(nx, ny, nconf, store, convergent):
    p, at = wl.hrtem_sto(cells=(max(2, nx // 64), max(2, ny // 64), 3), n=nx, nconf=nconf)
    p.ny = ny
    if convergent:
        p.iw_type = abi.MS_IW_CONVERGENT
        p.cond_lens.outer_aper_ang = 0.02
        p.iw_x, p.iw_y = p.lx / 2, p.ly / 2
    with cb.Context() as ctx:
        ctx.set_transmission_store(store)
        out = cb.MulSimulator(ctx=ctx).executionTEM(p, at)
    assert rel(out.image_intensity, orc.simulate_tem(p, at)) < 1e-5


@pytest.mark.parametrize("nx,ny", [(128, 128), (256, 128), (128, 512)])
def test_filtered_steps(ctx, nx, ny):
    p, at = wl.hrtem_sto(cells=(3, 3, 4), n=nx, nconf=2)
    p.ny = ny
    p.set_detectors([(0.004, 0.020)])
    out = cb.ThicknessSimulator(ctx=ctx).run(p, at)
    assert rel(out.thickness_frames, orc.simulate_thickness(p, at)) < 1e-5
