"""Density pass over blocks of cells: block sizes, blocks that are split or not
staged because they are too dense, and particles without a position."""
import numpy as np
import pytest

import wcsph
from parity import dam_break_scene, run_one_step
from test_gpu_parity import check_step

pytestmark = pytest.mark.gpu


# one row more or less than a unit's warps hold, and one scene per block size
# (2x2x2 cells below 2^18 particles, 4x4x2 below 2^19, 4x4x4 from there on)
@pytest.mark.parametrize("dims", [(4, 4, 4), (9, 11, 5), (64, 64, 65), (81, 81, 81)])
def test_block_sizes(dims):
    n = int(np.prod(dims))
    p, bx, pos, bpos = dam_break_scene(dims=dims, r=0.01 if n < 100000 else 0.003, jitter_frac=0.3,
                                       walls=n < 100000)
    vel = wcsph.make_velocities(n, 0.2, seed=4)
    check_step(p, bx, pos, vel, bpos, 1e-3, nbr_cap=n * 128)


# particles per cell: 20 and 32 split the units, at 120 not even one cell's 27
# neighbour cells fit (rows are then summed from global memory)
@pytest.mark.parametrize("per_cell,side", [(20, 6), (32, 4), (120, 3)])
def test_dense_blocks(per_cell, side):
    rng = np.random.default_rng(per_cell)
    n = per_cell * side ** 3
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = (0.33 + rng.random((n, 3)) * (0.04 * side)).astype(np.float32)
    p = wcsph.default_params(particle_radius=0.01, max_time_step=1e-3, cfl_factor=0.0)
    check_step(p, wcsph.box((0, 0, 0), (1, 1, 1)), pos, np.zeros_like(pos), None, 1e-3)


def test_particle_without_position_is_nobodys_neighbour():
    # a NaN position lies in cell (0, 0, 0) and within h of nothing: the other
    # particles' densities are those of the scene without it, bit for bit
    p, bx, pos, _ = dam_break_scene(dims=(7, 6, 5), walls=False)
    bad = np.concatenate([pos, np.full((1, 4), np.nan, np.float32)])
    a = run_one_step(p, bx, pos, np.zeros_like(pos), None, 1e-3)
    b = run_one_step(p, bx, bad, np.zeros_like(bad), None, 1e-3)
    n = len(pos)
    da, db = np.empty(n, np.float32), np.empty(n + 1, np.float32)
    da[a["permutation"]] = a["density"]
    db[b["permutation"]] = b["density"]
    assert np.array_equal(da, db[:n])
    counts = np.empty(n + 1, np.uint32)
    counts[b["permutation"]] = b["neighbors"][0]
    assert counts[n] == 0
