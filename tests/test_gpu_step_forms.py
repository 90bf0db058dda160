"""The forms of the slice steps that a call reaches only by its size, its tile shape or its launch mode:
each gives the bits of the others.  (Tile shapes and slice stores of simulations at sizes without tiles
compare a kernel with itself, so the sizes here are those that have them.)"""
from __future__ import annotations

import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import cases  # noqa: E402
import cudaem_b200 as cb  # noqa: E402
from cudaem_b200 import _abi as abi  # noqa: E402
from conftest import rel_l2  # noqa: E402
from oracle import oracle as orc  # noqa: E402

pytestmark = pytest.mark.gpu

WIDE, NARROW_ROWS, NARROW_COLS, NARROW, WARP_COLS = 0, 1, 2, 3, 4


@pytest.mark.parametrize("nx,ny,n_probe", [(128, 128, 2), (128, 128, 5), (256, 512, 3), (512, 256, 4), (1024, 1024, 1),
                                           (1024, 1024, 4), (2048, 128, 4), (128, 2048, 2), (2048, 2048, 4)])
def test_gradient_on_every_tile_shape(nx, ny, n_probe):
    """Forward, transmitted-wave, adjoint and conjugate steps on both slice stores (fewer than four probes:
    sigma V)."""
    p, _ = cases.stem_small(n=nx)
    p.ny = ny
    p.ckpt_interval = 2
    V = cases.random_phase_slices(p, 5, seed=nx + ny, amp=0.4)
    rng = np.random.default_rng(n_probe)
    xy = p.lx / 2 + rng.uniform(-1.5, 1.5, (n_probe, 2))
    ref = None
    shapes = [WIDE, NARROW_ROWS, NARROW_COLS, NARROW]
    if ny == 1024:
        shapes += [WARP_COLS, WARP_COLS | NARROW_ROWS]
    with cb.Context(0) as ctx:
        for shape in shapes:
            ctx.set_tile_shape(shape)
            I = ctx.stem_forward_potential(p, V, 0.5, xy)
            if ref is None:
                T = (I * (1 + 0.05 * rng.standard_normal(I.shape))).astype(np.float32)
            g = ctx.stem_backward(p, V, 0.5, xy, T)
            if ref is None:
                ref = I, g
                if nx * ny <= 512 * 256:
                    o = orc.stem_backward(p, V, 0.5, xy, T)
                    assert rel_l2(g[1], o[1]) < 1e-4
            assert np.array_equal(I, ref[0])
            assert g[0] == ref[1][0] and np.array_equal(g[1], ref[1][1]) and g[2:] == ref[1][2:]


@pytest.mark.parametrize("nx,ny,nconf", [(512, 512, 3), (256, 1024, 3), (1024, 512, 1)])
def test_hrtem_batches_with_tiles(nx, ny, nconf):
    """HRTEM beyond the short steps: every tile shape, both slice stores."""
    p, at = cases.hrtem_small(n=nx, nconf=nconf)
    p.ny = ny
    out = []
    with cb.Context(0) as ctx:
        sim = cb.MulSimulator(ctx=ctx)
        for store in (True, False):
            ctx.set_transmission_store(store)
            for shape in (WIDE, NARROW_ROWS, NARROW_COLS, NARROW):
                ctx.set_tile_shape(shape)
                out.append(sim.executionTEM(p, at).image_intensity)
    assert all(np.array_equal(o, out[0]) for o in out)
    assert rel_l2(out[0], orc.simulate_tem(p, at)) < 1e-5


@pytest.mark.parametrize("kind,nx,ny,nconf", [("tem", 128, 128, 2), ("tem", 512, 512, 1), ("ed", 256, 128, 3),
                                              ("cbed", 128, 128, 2), ("cbed", 256, 512, 1), ("stem", 128, 128, 1),
                                              ("stem", 2048, 128, 1), ("thickness", 256, 256, 2),
                                              ("thickness", 128, 512, 1)])
def test_chained_steps_equal_plain_ones(kind, nx, ny, nconf):
    """Steps that start before the one ahead has ended, against one launch after another (per-launch timing
    launches them so)."""
    if kind == "stem":
        p, at = cases.stem_small(n=nx, scan=(3, 1), nconf=nconf)
    elif kind == "cbed":
        p, at = cases.cbed_small(n=nx, nconf=nconf)
    elif kind == "thickness":
        p, at = cases.thickness_small(n=nx, nconf=nconf)
    else:
        p, at = cases.hrtem_small(n=nx, nconf=nconf)
        if kind == "ed":
            p.simulation_type = abi.MS_SIM_ED
    p.ny = ny
    out = []
    with cb.Context(0) as ctx:
        ctx.set_tile_shape(WIDE)
        sim = cb.ThicknessSimulator(ctx=ctx)
        run = {"stem": lambda: sim.executionSTEM(p, at).stem_intensity,
               "cbed": lambda: sim.executionCBED(p, at).image_intensity,
               "thickness": lambda: sim.run(p, at).thickness_frames}.get(
                   kind, lambda: sim.executionTEM(p, at).image_intensity)
        for profiling in (False, True, False):
            ctx.set_profiling(profiling)
            out.append(run().copy())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


def test_specimens_about_the_size_of_the_pinned_memory(ctx):
    """Atoms go through pinned memory where they fit beside the call's other copies and straight from the
    caller's arrays where not: atoms far outside the box change nothing but that."""
    p, at = cases.hrtem_small(n=128)
    sim = cb.MulSimulator(ctx=ctx)
    want = sim.executionTEM(p, at).image_intensity
    row = (2 << 20) // 24   # atoms whose six values fill the pinned memory
    for total in [*range(row - 600, row + 20, 20), 2 * row]:
        pad = total - len(at.x)
        far = cb.Atoms(Z=np.concatenate([at.Z, np.full(pad, at.Z[0])]),
                       x=np.concatenate([at.x, np.full(pad, -1.0e3, np.float32)]),
                       y=np.concatenate([at.y, np.full(pad, -1.0e3, np.float32)]),
                       z=np.concatenate([at.z, np.full(pad, at.z.mean(), np.float32)]),
                       sigma=np.concatenate([at.sigma, np.zeros(pad, np.float32)]),
                       occ=np.concatenate([at.occ, np.ones(pad, np.float32)]))
        assert np.array_equal(sim.executionTEM(p, far).image_intensity, want)
