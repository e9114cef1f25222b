"""The one-launch cluster sort: permutations of given keys and of scenes at the
edges of its block counts, items per thread and digit passes."""
import numpy as np
import pytest

import wcsph
from test_zz_no_alloc import _device_sort

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# one, two and sixteen blocks; one to four items a thread, full and one over
@pytest.mark.parametrize("n", [1, 31, 1024, 1025, 2049, 16384, 16385, 32769, 49153, 65536])
# no differing bit; one partial digit; three digits; low and high bits only; all 64
@pytest.mark.parametrize("mask", [0x0, 0x3F, 0xFFFFFF, 0x7F00000000000F01, 0xFFFFFFFFFFFFFFFF])
def test_keys(n, mask):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 64, n, dtype=np.uint64) & np.uint64(mask) | np.uint64(0x10) & ~np.uint64(mask)
    perm = _device_sort(torch, keys, calls=1)[0]
    assert np.array_equal(perm, np.argsort(keys, kind="stable").astype(np.uint32))


# eight items a thread and the first size past the cluster's; around the origin
# (a sign bit per axis), at positive coordinates only, and far out (64-bit keys)
@pytest.mark.parametrize("n", [65537, 98305, 131072, 131073])
@pytest.mark.parametrize("where", [0.0, 1.0, 100.0])
def test_scene_permutation(n, where):
    rng = np.random.default_rng(n)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = (where + rng.random((n, 3)) - 0.5).astype(np.float32)
    p = wcsph.default_params(particle_radius=0.004, max_time_step=1e-4, cfl_factor=0.0)
    side = abs(where) + 1.0
    sim = wcsph.CUDASPHSimulator(p, pos, wcsph.box((-side,) * 3, (side,) * 3))
    sim.update(1e-4)
    keys = sim.field("morton_keys")
    cell = np.floor(pos[:, :3] / np.float32(np.float32(2) * (np.float32(2) * np.float32(p.particle_radius))))
    u = (cell.astype(np.int64) + (1 << 20)).astype(np.uint64)
    want = np.zeros(n, np.uint64)
    for b in range(21):
        for d in range(3):
            want |= ((u[:, d] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + d)
    assert np.array_equal(keys, want)
    assert np.array_equal(sim.field("permutation"), np.argsort(keys, kind="stable").astype(np.uint32))
    sim.close()
