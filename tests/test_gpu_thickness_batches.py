"""Thickness series whose filtered spectra span several chunks and configurations, on wide and
narrow tiles, against the FP64 oracle: 512 x 256, six configurations, 45 slices (42 slices of
spectra fit the store, so the second chunk holds a remainder).  The tolerance is the parity tests'
1e-5: the images go through the same FP32 transforms as before."""
from __future__ import annotations

import numpy as np
import pytest

import cudaem_b200 as cb
from cudaem_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    p, at = wl.hrtem_sto(cells=(6, 3, 22), n=512, nconf=6)
    p.ny = 256
    p.set_detectors([(0.0, 0.020), (0.004, 0.030)])
    p.thick_det = 1
    return p, at, orc.simulate_thickness(p, at)


@pytest.mark.parametrize("shape", [0, 3, -1])
def test_chunked_series(case, shape):
    p, at, ref = case
    with cb.Context() as ctx:
        ctx.set_tile_shape(shape)
        out = cb.ThicknessSimulator(ctx=ctx).run(p, at).thickness_frames
    assert out.shape == ref.shape and out.shape[0] > 42
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) < 1e-5
