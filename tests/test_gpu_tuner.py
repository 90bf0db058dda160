"""The autotuners run the steps of the call they tune: on its slice store, its L2 mode and its kernel
forms, and only where the choice is used."""
from __future__ import annotations

import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import cases  # noqa: E402
import cudaem_b200 as cb  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(128, 128), (256, 128), (2048, 128)])
def test_probe_batch_tuned_on_the_sigma_v_store(nx, ny):
    """An 8 x 8 scan has two candidate batches, so the tuner runs; on the sigma V store it must read that
    store (a wave has none of its own).  Both stores give the same values bit for bit."""
    p, at = cases.stem_small(n=nx, cells=(max(2, nx // 64), max(2, ny // 64), 2), scan=(8, 8), nconf=1, batch=0)
    p.ny = ny
    out = []
    for store in (True, False):
        with cb.Context(0) as ctx:
            ctx.set_transmission_store(store)
            out.append(cb.MulSimulator(ctx=ctx).executionSTEM(p, at).stem_intensity)
            assert ctx.last_probe_batch in (32, 64)
    assert np.array_equal(out[0], out[1])
