"""The large scenes' sort (the onesweep passes) at sizes that the cluster sort takes
otherwise: the path of devices on which the cluster does not fit."""
import numpy as np
import pytest

import wcsph
from test_zz_no_alloc import _device_sort

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# one key, one tile less one, full and one over, several, the most; no deciding
# bit, one digit, three, all
@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 13824, 65536])
@pytest.mark.parametrize("mask", [0x0, 0x3F, 0xFFFFFF, 0xFFFFFFFFFFFFFFFF])
def test_static_sort_on_the_scratch(n, mask):
    keys = np.random.default_rng(n).integers(0, 1 << 64, n, dtype=np.uint64) & np.uint64(mask)
    want = np.argsort(keys, kind="stable").astype(np.uint32)
    with wcsph.large_sort():
        for got in _device_sort(torch, keys):   # two calls in a row share the scratch
            assert np.array_equal(got, want)
    with wcsph.stall_sort():                    # a call that fails leaves the scratch to be cleared
        stalled = _device_sort(torch, keys, calls=1)[0]
    assert n <= 2048 or (stalled == np.uint32(wcsph.STATIC_SORT_FAILED)).all() or not mask
    with wcsph.large_sort():
        assert np.array_equal(_device_sort(torch, keys, calls=1)[0], want)


def test_static_sort_on_the_scratch_allocates_no_device_memory():
    n = wcsph.STATIC_SORT_MAX_KEYS
    d_keys = torch.from_numpy(np.random.default_rng(8).integers(0, 1 << 62, n, dtype=np.int64)).cuda()
    d_perm = torch.empty(n, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    with wcsph.large_sort():
        wcsph.sort_keys_static(d_keys.data_ptr(), n, d_perm.data_ptr(), stream)
        torch.cuda.synchronize()
        free_before, _ = torch.cuda.mem_get_info()
        for _ in range(8):
            wcsph.sort_keys_static(d_keys.data_ptr(), n, d_perm.data_ptr(), stream)
        torch.cuda.synchronize()
        free_after, _ = torch.cuda.mem_get_info()
    assert free_after == free_before


# near the origin the sort's keys are 32-bit words, far out 64-bit ones
@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 13824, 131072])
@pytest.mark.parametrize("where", [0.0, 100.0])
def test_step_matches_the_cluster_sort(n, where):
    rng = np.random.default_rng(n)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = (where + rng.random((n, 3)) - 0.5).astype(np.float32)
    p = wcsph.default_params(particle_radius=0.004, max_time_step=1e-4, cfl_factor=0.0, table_size_mult=4)
    side = abs(where) + 1.0

    def run():
        with wcsph.CUDASPHSimulator(p, pos, wcsph.box((-side,) * 3, (side,) * 3)) as sim:
            sim.step_n(3, 1e-4)
            return [sim.field(k) for k in ("morton_keys", "permutation", "density", "position", "velocity")]

    want = run()
    with wcsph.large_sort():
        got = run()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_staged_batch_matches_the_cluster_sort():
    pres = [wcsph.preset_ensemble(3, k) for k in range(3)]
    specs = [wcsph.BatchSceneSpec(fluid_pos=q.pos, fluid_vel=q.vel, box=q.box, gravity=tuple(q.params.gravity),
                                  viscosity=q.params.viscosity, boundary_pos=q.bpos) for q in pres]

    def run():
        b = wcsph.BatchSimulator(pres[0].params, specs)
        b.set_persistent(False)
        b.step_n(3, 1e-3)
        out = [a for k in range(len(pres)) for a in b.get_state(k)]
        b.close()
        return out

    want = run()
    with wcsph.large_sort():
        got = run()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_launches_per_step_are_those_of_the_path():
    pos = np.ones((3000, 4), np.float32)
    pos[:, :3] = np.random.default_rng(0).random((3000, 3))
    p = wcsph.default_params(particle_radius=0.02, max_time_step=1e-4, cfl_factor=0.0)
    for hook, want in ((None, 5), (wcsph.large_sort, 15)):
        with wcsph.CUDASPHSimulator(p, pos, wcsph.box((0, 0, 0), (1, 1, 1))) as sim:
            if hook:
                with hook():
                    sim.update(1e-4)
            else:
                sim.update(1e-4)
            sim.synchronize()
            assert sim.launches_per_step() == want
