"""The autotuners run the steps of the call they tune: on its slice store, its L2 mode and its kernel
forms, and only where the choice is used."""
from __future__ import annotations

import json
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


def entries(ctx_calls, tmp_path):
    path = str(tmp_path / "tune.json")
    with cb.Context(0) as ctx:
        ctx.set_tune_cache(path)
        ctx_calls(ctx)
    with open(path) as f:
        return json.load(f)


def test_choices_are_kept_per_slice_store(tmp_path):
    """Steps on a sigma V store are other kernels than those on a transmission store: a choice timed on
    one does not stand for the other."""
    p, at = cases.stem_small(n=128, scan=(8, 8), nconf=1, batch=0)

    def calls(ctx):
        sim = cb.MulSimulator(ctx=ctx)
        for store in (True, False):
            ctx.set_transmission_store(store)
            sim.executionSTEM(p, at)

    keys = entries(calls, tmp_path)
    for kind in ("tile|", "batch|"):
        mine = [k for k in keys if k.startswith(kind)]
        assert len(mine) == 2 and sum(k.endswith(",v") for k in mine) == 1


def test_nothing_is_timed_where_the_steps_have_no_tiles(tmp_path):
    """2048 x 2048 simulations run one row and one column kernel: no entry, and the wide shape reported."""
    p, at = cases.cbed_small(n=2048, cells=(3, 3, 1), nconf=1)
    q, at_q = cases.cbed_small(n=256, cells=(3, 3, 1), nconf=1)
    last = []

    def calls(ctx):
        sim = cb.MulSimulator(ctx=ctx)
        for prob in ((p, at), (q, at_q)):
            sim.executionCBED(*prob)
            last.append(ctx.last_tile_shape)

    keys = entries(calls, tmp_path)
    assert [k.split("|")[-1] for k in keys if k.startswith("tile|")] == ["256,256,1"]
    assert last[0] == 0
