"""The autotuner's space: every configuration is a launch of its own, and the walk
over it moves."""
import json

import pytest

import wcsph
from parity import dam_break_scene

pytestmark = pytest.mark.gpu

DENSITY = ("compute_rho_p_block", "mask_words", "particles_per_warp")


def searched(searcher, updates, tmp_path):
    p, bx, pos, _ = dam_break_scene(dims=(6, 6, 6), walls=False)
    with wcsph.CUDASPHSimulator(p, pos, bx) as sim:
        sim.set_tuning(searcher, 1.0)
        for _ in range(updates):
            sim.update(1e-5)
        sim.save_tuning_results(tmp_path / "r.json")
    results = json.loads((tmp_path / "r.json").read_text())["Results"]
    return [{e["Name"]: e["Value"] for e in r["Configuration"]} for r in results]


def test_full_search_times_each_launch_once(tmp_path):
    # force and surface blocks (9) by cell sizes 1, 1.5 and 2 with 6 table sizes each;
    # two cells a radius (h / 2, tables from 8) with 45 density configurations
    configs = searched(wcsph.SEARCH_FULL, 3200, tmp_path)
    one = [c for c in configs if c["CELL_SIZE_MULT"] >= 0.99]
    assert len({tuple(c[k] for k in DENSITY) for c in one}) == 1
    two = {tuple(sorted(c.items())) for c in configs if c["CELL_SIZE_MULT"] < 0.6}
    assert len({tuple(sorted(c.items())) for c in one}) == 9 * 3 * 6
    assert len(two) == 9 * 45 * 3
    first = {tuple(sorted(c.items())) for c in configs[:9 * 3 * 6]}
    assert len(first) == 9 * 3 * 6   # nothing twice before all


def test_walk_proposes_other_configurations(tmp_path):
    configs = searched(wcsph.SEARCH_MCMC, 60, tmp_path)
    assert len({tuple(sorted(c.items())) for c in configs}) >= 15
