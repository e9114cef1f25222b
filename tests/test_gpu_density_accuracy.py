"""Accuracy of the density sums against 64 bits.

Radius 1/64 makes h, its reciprocal and the particle mass exact, so what is left
are the roundings of the sums: three of the result (the sum's value, W(0) + sum,
times the mass), each uniform within 2^-24 of it, 2^-24 / sqrt(3) RMS, together
2^-24; and the pairs' own (q within 2 ulp), averaged over some 57 neighbours to
0.3 of that. The bound is 1.3 * 2^-24; a plain chain of 57 additions comes to
1.9 * 2^-24 (emulated in numpy, as is 0.83 * 2^-24 for sums that carry their error).
"""
import numpy as np
import pytest

import wcsph

pytestmark = pytest.mark.gpu


def test_density_rms_error():
    r, side = 1.0 / 64, 16
    rng = np.random.default_rng(0)
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = np.ones((len(g), 4), np.float32)
    pos[:, :3] = g * (1.6 * r) + 2 * r + rng.uniform(-0.35 * r, 0.35 * r, g.shape)
    p = wcsph.default_params(particle_radius=r, max_time_step=1e-4, cfl_factor=0.0)
    with wcsph.CUDASPHSimulator(p, pos, wcsph.box((0, 0, 0), (1, 1, 1))) as sim:
        sim.update(1e-4)
        rho = np.empty(len(pos))
        rho[sim.field("permutation")] = sim.field("density")
    x = pos[:, :3].astype(np.float64)
    h = 4 * r
    q = np.sqrt(((x[:, None] - x[None]) ** 2).sum(-1)) / h
    w = np.where(q <= 0.5, 6 * q ** 3 - 6 * q ** 2 + 1, np.where(q <= 1, 2 * (1 - q) ** 3, 0))   # the row's own pair: W(0)
    want = 1000.0 * (2 * r) ** 3 * 0.8 * 8 / (np.pi * h ** 3) * w.sum(1)
    err = (rho - want) / want
    # about its mean: the spline's factor is rounded once for all rows
    assert abs(err.mean()) < 4 * 2.0 ** -24
    assert err.std() < 1.3 * 2.0 ** -24, f"{err.std() * 2 ** 24:.2f} * 2^-24"
