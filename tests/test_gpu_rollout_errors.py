"""Error paths of the differentiable rollout: a step whose sort fails, and a
forward pass that fails before it has run. Nothing here faults or hangs."""
import numpy as np
import pytest

import wcsph
from test_gpu_adjoint import rollout_scene

pytestmark = pytest.mark.gpu


def rollout(sim, target, steps=6, every=3):
    loss = sim.rollout_forward(steps, 1e-3, every, target)
    return loss, sim.rollout_backward()[0]


# the failed steps run in the context's buffers, in their own sets, or both; on
# a context that has no rollout's workspaces yet, and on one that has
@pytest.mark.parametrize("every", [1, 3, 6])
@pytest.mark.parametrize("used", [False, True])
def test_sort_timeout_in_a_rollout(every, used):
    p, bx, pos, walls, target = rollout_scene(dims=(16, 16, 24))   # 6,144 particles: 3 sort tiles
    with wcsph.CUDASPHSimulator(p, pos, bx, boundary_pos=walls) as sim:
        want = rollout(sim, target)
    with wcsph.CUDASPHSimulator(p, pos, bx, boundary_pos=walls) as sim:
        if used:
            rollout(sim, target, 2, every)
            sim.set_state(pos)
        with wcsph.stall_sort():
            with pytest.raises(wcsph.WcsphError) as e:
                sim.rollout_forward(6, 1e-3, every, target)
        assert e.value.status == wcsph.ERR_DEVICE_TIMEOUT
        with pytest.raises(wcsph.WcsphError) as e:
            sim.rollout_backward()
        assert e.value.status == wcsph.ERR_STATE
        x, v = sim.get_state()
        assert np.array_equal(x, pos) and not v.any()   # the failed steps left the state as it was
        got = rollout(sim, target)                      # and the context works on
    assert got[0] == want[0] and np.array_equal(got[1], want[1])


# the second forward fails before it has run (its checkpoints would take 8 TB:
# the allocation is refused at once); the rollout before it is no longer there
def test_forward_out_of_memory_leaves_no_rollout_behind():
    p, bx, pos, walls, target = rollout_scene(dims=(8, 8, 8))
    with wcsph.CUDASPHSimulator(p, pos, bx, boundary_pos=walls) as sim:
        want = rollout(sim, target)
        sim.set_state(pos)
        with pytest.raises(wcsph.WcsphError) as e:
            sim.rollout_forward(1 << 30, 1e-3, 1, target)
        assert e.value.status == wcsph.ERR_OUT_OF_MEMORY
        with pytest.raises(wcsph.WcsphError) as e:
            sim.rollout_backward()
        assert e.value.status == wcsph.ERR_STATE
        x, v = sim.get_state()
        assert np.array_equal(x, pos) and not v.any()
        got = rollout(sim, target)
    assert got[0] == want[0] and np.array_equal(got[1], want[1])


def other_parameters(sim, p, bx):
    q = wcsph.Params.from_buffer_copy(p)
    q.cell_size_mult, q.table_size_mult = 0.5, 8    # another sort order, another table
    q.viscosity *= 3
    q.rest_density *= 1.1                           # other boundary masses
    sim.set_params(q)


def other_box(sim, p, bx):
    sim.set_box(wcsph.box((0, 0, 0), (0.25, 0.2, 0.15), wcsph.rotation_z(0.2)))


# what is set between forward and backward changes neither the gradients nor,
# afterwards, what was set: the next step is that of a context that had no backward
@pytest.mark.parametrize("every", [2, 5])
@pytest.mark.parametrize("between", [other_parameters, other_box, lambda sim, p, bx: sim.update(1e-3)])
def test_backward_is_the_forwards(every, between):
    p, bx, pos, walls, target = rollout_scene(dims=(10, 9, 8))

    def run(change, backward):
        with wcsph.CUDASPHSimulator(p, pos, bx, boundary_pos=walls) as sim:
            sim.rollout_forward(5, 1e-3, every, target)
            if change:
                between(sim, p, bx)
            grads = sim.rollout_backward() if backward else None
            if change and backward:   # from the rollout's end, under what was set
                sim.rollout_forward(2, 1e-3, 1, target)
            return grads, sim.get_state()

    def forward_again():
        with wcsph.CUDASPHSimulator(p, pos, bx, boundary_pos=walls) as sim:
            sim.rollout_forward(5, 1e-3, every, target)
            x, v = sim.get_state()
            between(sim, p, bx)
            sim.set_state(x, v)
            sim.rollout_forward(2, 1e-3, 1, target)
            return sim.get_state()

    (gv0, gnu0, gk0), _ = run(False, True)
    (gv, gnu, gk), after = run(True, True)
    assert np.array_equal(gv, gv0)
    # the two scalars are double sums in arrival order, rounded to float
    assert abs(gnu - gnu0) <= 2e-7 * abs(gnu0) and abs(gk - gk0) <= 2e-7 * abs(gk0)
    want = forward_again()
    assert np.array_equal(after[0], want[0]) and np.array_equal(after[1], want[1])
