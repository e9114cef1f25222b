"""Density units of 4x4x2 and 4x4x4 cells that hold more candidates than their
buffer: split once, several times, down to single cells (a batch's smaller
buffers: test_gpu_list_spills)."""
import numpy as np
import pytest

import wcsph
from test_gpu_parity import check_step

pytestmark = pytest.mark.gpu


# the units' 144 and 216 cells against 2048 and 2560 candidates: 20 particles a
# cell (split once), 45 in a part of the fluid (to 2x1x1 cells), 100 in one corner
# (single cells that do not fit either), beside rest density
@pytest.mark.parametrize("n,side", [(270000, 25), (530000, 31)])
def test_large_units_are_split(n, side):
    r, h = 0.004, 0.016
    rng = np.random.default_rng(side)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = (0.2 + rng.random((n, 3)) * (h * side)).astype(np.float32)
    at = 0
    for cells, per_cell in ((6, 25), (3, 90)):   # on top of the 17 a cell
        k = cells ** 3 * per_cell
        pos[at:at + k, :3] = (0.2 + h * 8 * (at > 0) + rng.random((k, 3)) * (h * cells)).astype(np.float32)
        at += k
    p = wcsph.default_params(particle_radius=r, max_time_step=1e-4, cfl_factor=0.0)
    check_step(p, wcsph.box((0, 0, 0), (2, 2, 2)), pos, np.zeros_like(pos), None, 1e-4, nbr_cap=n * 128)
