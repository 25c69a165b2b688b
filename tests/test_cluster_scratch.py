"""The memory of the cluster solves' exchange is allocated with a call's workspace on a B200, not between two Newton steps
(where an allocation makes a first call wait, milliseconds at times): a call that stops before its first step leaves nothing
for the next one to allocate."""
import numpy as np
import pytest
import torch

from gridsim_b200 import synthetic
from gridsim_b200.engine import PowerFlowOptions, SparseNewtonRaphsonPowerFlow

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_bus,count", [(1000, 288), (2000, 256)])  # two and four blocks; more systems than one wave
def test_no_step_allocates(n_bus, count):
    m = synthetic.make_grid(n_bus, n_bus + n_bus // 3 + 1, n_bus // 8, seed=5)
    solver = SparseNewtonRaphsonPowerFlow("fp64")
    none = np.full(count, -1, np.int32)
    scale = np.full((count, n_bus), 1.02)
    r = solver.solve_batch(m, load_scale=scale, outage=none, options=PowerFlowOptions(max_iterations=0))
    assert (r["iterations"] == 0).all() and (r["status"] != 0).all()
    before = torch.cuda.mem_get_info()[0]
    r = solver.solve_batch(m, load_scale=scale, outage=none, options=PowerFlowOptions(max_iterations=20))
    assert (r["status"] == 0).all()
    assert torch.cuda.mem_get_info()[0] == before
