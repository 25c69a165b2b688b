"""The classification's chunks of 256 items (branches, then buses) on a B200: grids whose item count lies one short of, at
and one past a chunk's edge, systems one short of, at and past a group of 32, limits tight enough that most items violate.
Violations (order, kind, element) equal the oracle's; values within 1e-6 of them (states agree within 1e-8 pu, and a
loading or voltage is at most 1e2 times as sensitive)."""
import numpy as np
import pytest

import oracle
from gridsim_b200 import synthetic
from gridsim_b200.engine import ContingencyAnalysis, PowerFlowOptions, SparseNewtonRaphsonPowerFlow

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("items", [255, 256, 257, 513])
@pytest.mark.parametrize("count", [31, 32, 33])
def test_violations_match_the_oracle(items, count):
    n_bus = 2 * items // 5
    m = synthetic.make_grid(n_bus, items - n_bus, max(1, n_bus // 8), seed=4)
    assert m.n_bus + len(m.br_from) == items
    m.rate_a = np.asarray(m.rate_a) * 0.05
    idx = m.in_service_branches()[:count]
    opt = PowerFlowOptions(max_iterations=20, warm_start_from_base=True)
    ref = oracle.screen(m, idx, opt.to_c())
    got = ContingencyAnalysis.screen_raw(m, idx, SparseNewtonRaphsonPowerFlow("fp64"), opt)
    assert (got["status"] == ref["status"]).all()
    total = int(ref["viol_ptr"][-1])
    assert total > count
    assert (got["viol_ptr"] == ref["viol_ptr"]).all()
    for key in ("viol_kind", "viol_element"):
        assert (np.asarray(got[key])[:total] == np.asarray(ref[key])[:total]).all()
    for key in ("viol_value", "max_loading_pct", "min_vm", "max_vm"):
        a, b = np.asarray(got[key]), np.asarray(ref[key])
        k = total if key == "viol_value" else count
        assert np.abs(a[:k] - b[:k]).max() <= 1e-6 * max(1.0, np.abs(b[:k]).max())
