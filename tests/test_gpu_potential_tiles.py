"""Projected potentials of specimens whose tiles hold few, many and very many candidate atoms (one
warp of candidates, several warps, several rounds of the block's list), on square and rectangular
grids, with and without periodic images, against the FP64 oracle.  The tolerance is the potential
tests' 2e-6: sums of FP32 splines, each good to a few 1e-7."""
from __future__ import annotations

import numpy as np
import pytest

import cudaem_b200 as cb
from cudaem_b200 import _abi as abi
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wrap", [0, 1])
@pytest.mark.parametrize("n_atoms,nx,ny,lx,ly", [(3, 128, 128, 11.0, 11.0), (90, 256, 128, 23.0, 13.0),
                                                  (900, 128, 256, 12.5, 20.0), (6000, 128, 128, 15.0, 14.0)])
def test_candidate_counts(ctx, n_atoms, nx, ny, lx, ly, wrap):
    rng = np.random.default_rng(n_atoms)
    # half a pixel off the grid and beyond the box's edges by up to a cut-off
    x = (np.floor(rng.uniform(-2.0, lx + 2.0, n_atoms) / (lx / nx)) + 0.5) * (lx / nx)
    y = (np.floor(rng.uniform(-2.0, ly + 2.0, n_atoms) / (ly / ny)) + 0.5) * (ly / ny)
    if wrap:
        x, y = x % lx, y % ly
    at = cb.Atoms(rng.choice([6, 22, 79], n_atoms), x, y, rng.uniform(0.0, 3.0, n_atoms),
                  np.zeros(n_atoms), rng.uniform(0.3, 1.0, n_atoms))
    p = cb.MultisliceParams(simulation_type=abi.MS_SIM_CBED, nx=nx, ny=ny, lx=lx, ly=ly, dz=1.6, E0=200.0, pot_wrap=wrap)
    V = ctx.projected_potential(p, at)
    ref = orc.potential(p, at)
    ref = np.asarray(ref[0] if isinstance(ref, tuple) else ref)
    assert V.shape == ref.shape
    assert np.linalg.norm(V - ref) / np.linalg.norm(ref) < 2e-6
