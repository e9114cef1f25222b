"""Rows whose neighbours do not fit their list: alone, all of them, several of a
cell together, shared between warps; the same sums whoever takes them."""
import numpy as np
import pytest

import wcsph
from parity import dam_break_scene
from test_gpu_parity import check_step

pytestmark = pytest.mark.gpu


# one warp's rows shared by four, and not (2^14 particles); one and three
# neighbours at a time (2^17); a few rows without a list, most, all
@pytest.mark.parametrize("dims", [(9, 11, 5), (25, 26, 25), (26, 26, 25), (50, 52, 50), (51, 52, 50)])
@pytest.mark.parametrize("width", [8, 24, 32])
def test_spilled_rows(dims, width):
    n = int(np.prod(dims))
    p, bx, pos, bpos = dam_break_scene(dims=dims, r=0.01 if n < 20000 else 0.004, jitter_frac=0.3, walls=n < 20000)
    vel = wcsph.make_velocities(n, 0.2, seed=4)
    check_step(p, bx, pos, vel, bpos, 1e-3, nbr_cap=n * 64, config={"neighbour_list_width": width})


def test_spilled_rows_with_two_cells_a_radius():
    # cell size h / 2: 125 cells, four a lane
    p, bx, pos, bpos = dam_break_scene(dims=(12, 11, 10), jitter_frac=0.3, cell_size_mult=0.5, table_size_mult=8)
    vel = wcsph.make_velocities(len(pos), 0.2, seed=4)
    check_step(p, bx, pos, vel, bpos, 1e-3, config={"neighbour_list_width": 16})


def test_spilled_rows_same_bits_in_a_batch():
    # denser than 64 neighbours; below 2^14 particles alone, above in the batch
    pres = [wcsph.preset_ensemble(3, k) for k in range(4)]
    p = pres[0].params
    for q in pres:
        q.pos[:, :3] *= np.float32(0.72)
    specs = [wcsph.BatchSceneSpec(fluid_pos=q.pos, fluid_vel=q.vel, box=q.box, gravity=tuple(q.params.gravity),
                                  viscosity=q.params.viscosity, boundary_pos=q.bpos) for q in pres]
    states = []
    for persistent in (True, False):
        b = wcsph.BatchSimulator(p, specs)
        b.set_persistent(persistent)
        b.step_n(2, 1e-5)
        states.append([b.get_state(k) for k in range(len(pres))])
        b.close()
    for k, q in enumerate(pres):
        sim = wcsph.CUDASPHSimulator(q.params, q.pos, q.box, fluid_vel=q.vel, boundary_pos=q.bpos)
        sim.step_n(2, 1e-5)
        want = sim.get_state()
        sim.close()
        for s in states:
            assert np.array_equal(s[k][0], want[0]) and np.array_equal(s[k][1], want[1])


def test_spilled_rows_of_a_small_scene_are_not_slow(tmp_path):
    """One warp took 32 rows without a usable list one after the other: 4 times
    the step of a scene whose lists hold (2 k particles); shared, 1.7 times."""
    p, bx, pos, bpos = dam_break_scene(dims=(16, 16, 8), max_time_step=1e-6, min_time_step=1e-7)
    pos[:, :3] *= np.float32(0.92)

    def step_ms(width):
        cfg = tmp_path / f"{width}.json"
        cfg.write_text('[{"Name": "neighbour_list_width", "Value": %d, "ValueType": "UnsignedInt"}]' % width)
        with wcsph.CUDASPHSimulator(p, pos, bx) as sim:
            sim.set_tuning(wcsph.SEARCH_MCMC, 0.0, cfg)
            sim.time_steps(3, 1e-6)
            return min(sim.time_steps(10, 1e-6) for _ in range(5))

    assert step_ms(16) < 3 * step_ms(64)
