"""Small grids in large batches on a B200: a Newton run of few systems goes to one launch that holds a system a block, a run
of many small systems to the level launches over all of them. The two sides of the rule by their launch counts, and the
systems of a large run against the same systems in small ones: statuses, iterations and violations identical, voltages within
the parity bar of 1e-8 pu and 1e-8 rad of each other."""
import numpy as np
import pytest

from gridsim_b200 import _abi, synthetic
from gridsim_b200.engine import ContingencyAnalysis, PowerFlowOptions, SparseNewtonRaphsonPowerFlow

pytestmark = pytest.mark.gpu

LINE = {"fp64": 4000, "mixed": 6000}  # the most systems of these grids in one launch


@pytest.mark.parametrize("n_bus,precision", [(6, "fp64"), (30, "fp64"), (30, "mixed"), (60, "fp64")])
def test_large_batches_of_small_systems_go_level_by_level(n_bus, precision):
    m = synthetic.make_grid(n_bus, n_bus + n_bus // 3 + 1, max(1, n_bus // 8), seed=3)
    pairs = m.in_service_branches()
    pairs = np.array([(i, j) for i in pairs for j in pairs if i < j], np.int32)
    sets = np.resize(pairs, (8001, 2))  # repeated where the grid has fewer
    opt = PowerFlowOptions(precision=precision, max_iterations=20, warm_start_from_base=True)
    solver = SparseNewtonRaphsonPowerFlow(precision)
    large = ContingencyAnalysis.screen_sets_raw(m, sets, solver, opt, keep_states=True)
    small = ContingencyAnalysis.screen_sets_raw(m, sets[:1001], solver, opt, keep_states=True)
    solved = int((large["status"] != _abi.PF_UNSOLVABLE_PART).sum())  # sets without a solution by topology are not run
    assert small["kernel_launches"] < 20 and (large["kernel_launches"] > 20) == (solved > LINE[precision])
    k = 1001
    for key in ("status", "iterations", "islanded"):
        assert (large[key][:k] == small[key]).all(), key
    assert (large["viol_ptr"][:k + 1] == small["viol_ptr"]).all()
    v = small["viol_ptr"][-1]
    assert (large["viol_kind"][:v] == small["viol_kind"]).all() and (large["viol_element"][:v] == small["viol_element"]).all()
    ok = small["status"] == 0
    assert ok.any()
    assert np.abs(large["vm"][:k] - small["vm"])[ok].max() <= 1e-8
    assert np.radians(np.abs(large["va_deg"][:k] - small["va_deg"])[ok]).max() <= 1e-8
    again = ContingencyAnalysis.screen_sets_raw(m, sets[-300:], solver, opt, keep_states=True)
    assert (large["status"][-300:] == again["status"]).all()


def test_larger_systems_stay_in_one_launch():
    m = synthetic.make_grid(160, 214, 20, seed=3)
    scale = np.random.default_rng(1).uniform(0.97, 1.03, size=(8001, 1)) * np.ones((1, m.n_bus))
    opt = PowerFlowOptions(max_iterations=20)
    solver = SparseNewtonRaphsonPowerFlow("fp64")
    large = solver.solve_batch(m, load_scale=scale, options=opt, keep_states=True)
    part = solver.solve_batch(m, load_scale=scale[:40], options=opt, keep_states=True)
    assert (large["status"][:40] == part["status"]).all() and (large["iterations"][:40] == part["iterations"]).all()
    assert np.abs(large["vm"][:40] - part["vm"]).max() <= 1e-12  # the same kernel
