"""Density units that hold a few particles each: a scattered fluid and spray
around a bulk (their rows are summed without staging where there are many), and
the same bits in a batch, whose kernels draw that line elsewhere."""
import numpy as np
import pytest

import wcsph
from test_gpu_parity import check_step

pytestmark = pytest.mark.gpu


def params(r, **kw):
    kw = dict(particle_radius=r, stiffness=1000.0 * (4 * r) ** 6, viscosity=0.01, max_time_step=1e-3,
              cfl_factor=0.0, table_size_mult=16) | kw
    return wcsph.default_params(**kw)


def scattered(n, extent, seed=0):
    rng = np.random.default_rng(seed)
    pos = np.ones((n, 4), np.float32)
    pos[:, :3] = rng.random((n, 3)) * np.asarray(extent)
    return pos


def block(dims, r, at):
    g = np.stack(np.meshgrid(*[np.arange(d) for d in dims], indexing="ij"), -1).reshape(-1, 3)
    pos = np.ones((len(g), 4), np.float32)
    pos[:, :3] = np.asarray(at) + 2 * r * g
    return pos


# units of 2x2x2, 4x4x2 and 4x4x4 cells; a particle or a few of them in a unit,
# alone, around a bulk, beside walls
@pytest.mark.parametrize("n,extent", [(30000, (4, 4, 4)), (30000, (1, 0.6, 0.6)), (270000, (2, 2, 2)),
                                      (530000, (3, 3, 3))])
@pytest.mark.parametrize("bulk,walls", [(None, False), ((24, 24, 24), False), ((24, 24, 24), True)])
def test_scattered_fluid(n, extent, bulk, walls):
    if walls and extent[0] != 1:
        pytest.skip("walls of the small box only")
    r = 0.004
    pos = scattered(n, extent)
    if bulk:
        pos = np.concatenate([pos, block(bulk, r, (0.3, 0.2, 0.2))])
    bpos = wcsph.sample_box_walls((0, 0, 0), extent, 2 * r) if walls else None
    vel = wcsph.make_velocities(len(pos), 0.2, seed=1)
    check_step(params(r), wcsph.box((0, 0, 0), extent), pos, vel, bpos, 1e-3, nbr_cap=len(pos) * 64)


@pytest.mark.parametrize("persistent", [True, False])
def test_scattered_batch_matches_single_scenes(persistent):
    r = 0.01
    p = params(r)
    bx = wcsph.box((0, 0, 0), (2.5, 2.5, 2.5))
    scenes = [np.concatenate([scattered(12000, (2.4, 2.4, 2.4), seed=k), block((9, 8, 7), r, (0.5, 0.5, 0.5))])
              for k in range(3)]
    b = wcsph.BatchSimulator(p, [wcsph.BatchSceneSpec(fluid_pos=x, box=bx) for x in scenes])
    b.set_persistent(persistent)
    b.step_n(3, 1e-3)
    for k, x in enumerate(scenes):
        with wcsph.CUDASPHSimulator(p, x, bx) as sim:
            sim.step_n(3, 1e-3)
            want = sim.get_state()
        got = b.get_state(k)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    b.close()


def test_scattered_fluid_is_not_slow():
    """Unit by unit a scattered fluid took 14 times the step of a block with the
    same number of particles; by rows it takes about the same."""
    r = 0.01

    def step_ms(pos):
        lo, hi = pos[:, :3].min(0) - 1, pos[:, :3].max(0) + 1
        with wcsph.CUDASPHSimulator(params(r, max_time_step=1e-6, min_time_step=1e-7), pos, wcsph.box(lo, hi)) as sim:
            sim.time_steps(3, 1e-6)
            return min(sim.time_steps(5, 1e-6) for _ in range(5))

    assert step_ms(scattered(400000, (20, 20, 20))) < 4 * step_ms(block((80, 80, 63), r, (0, 0, 0)))
