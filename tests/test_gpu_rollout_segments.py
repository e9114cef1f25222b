"""Rollout gradients do not depend on where the segments end, on which steps
the forward left for the backward, or on a backward that re-runs them all."""
import numpy as np
import pytest

import wcsph
from parity import dam_break_scene

pytestmark = pytest.mark.gpu


def gradients(every, steps=7, between=None, twice=False):
    p, bx, pos, bpos = dam_break_scene(dims=(10, 9, 8), surface_tension=0.0)
    vel = wcsph.make_velocities(len(pos), 0.3, seed=2)
    target = pos + np.float32(0.05)
    sim = wcsph.CUDASPHSimulator(p, pos, bx, fluid_vel=vel, boundary_pos=bpos)
    loss = sim.rollout_forward(steps, 1e-3, every, target)
    fields = sim.field("density"), sim.field("permutation")
    if between:
        between(sim, p, bx)
    g = sim.rollout_backward()
    if twice:
        g = sim.rollout_backward()
    sim.close()
    return (loss, *g), fields


# one segment, segments with a whole and a partial last one, one longer than the rollout
@pytest.mark.parametrize("every", [1, 3, 6, 7, 20])
@pytest.mark.parametrize("between,twice", [(None, False), (None, True),
                                           (lambda sim, p, bx: sim.set_box(bx), False),
                                           (lambda sim, p, bx: sim.set_params(p), False)])
def test_segments(every, between, twice):
    (loss0, gv0, gnu0, gk0), fields0 = gradients(4)
    (loss, gv, gnu, gk), fields = gradients(every, between=between, twice=twice)
    assert loss == loss0
    assert np.array_equal(gv, gv0)
    # the two scalars are double sums in arrival order, rounded to float
    assert abs(gnu - gnu0) <= 2e-7 * abs(gnu0) and abs(gk - gk0) <= 2e-7 * abs(gk0)
    assert all(np.array_equal(a, b) for a, b in zip(fields, fields0))   # the last step's
