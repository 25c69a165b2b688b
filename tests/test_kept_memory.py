"""Device arrays that a call leaves allocated for the next one are bounded on a B200: those of a sparse pattern and the
staging of a batch's load scales are given back past 1 GiB each. Measured as the device memory missing after a call; the
workspaces that stay grow with the number of systems."""
import numpy as np
import pytest
import torch

from gridsim_b200 import synthetic
from gridsim_b200.engine import CudaContext, CudaSparseLinearSolver, PowerFlowOptions, SparseNewtonRaphsonPowerFlow

pytestmark = pytest.mark.gpu

GIB = float(1 << 30)


def _free():
    return float(torch.cuda.mem_get_info()[0])


def test_a_patterns_arrays_past_the_bound_are_given_back():
    n = 2000
    solver = CudaSparseLinearSolver(CudaContext(0))  # a context of its own: no pattern kept from before

    def taken(order, count):
        """Device memory missing after `count` systems on a path graph through the unknowns in `order`."""
        nxt = np.full((2, n), -1)
        nxt[0, order[:-1]], nxt[1, order[1:]] = order[1:], order[:-1]
        rows = [np.sort([c for c in (i, nxt[0, i], nxt[1, i]) if c >= 0]) for i in range(n)]
        ip = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
        ci = np.concatenate(rows).astype(np.int32)
        v = np.where(ci == np.repeat(np.arange(n), np.diff(ip)), 4.0, -1.0)
        b = np.ones(n)
        before = _free()
        x = solver.solve_batch([(ip, ci, v)] * count, [b] * count)
        r = 4.0 * x[-1]
        r[order[1:]] -= x[-1][order[:-1]]
        r[order[:-1]] -= x[-1][order[1:]]
        assert np.abs(r - b).max() < 1e-12
        return before - _free()

    few = taken(np.arange(n), 16000)  # values of 0.72 GiB
    values = 8.0 * (3 * n - 2) * 24000
    assert values > 1.05 * GIB
    many = taken(np.random.default_rng(1).permutation(n), 24000)
    assert many < 1.5 * few - 0.8 * values  # all kept: 1.5 few
    solver.ctx.close()


def test_a_batchs_staging_past_the_bound_is_given_back():
    n, count = 200, 800_000
    m = synthetic.make_grid(n, 267, 25, seed=3)
    solver = SparseNewtonRaphsonPowerFlow("fp64")
    opt = PowerFlowOptions(max_iterations=20)
    solver.solve_batch(m, outage=np.full(count, -1, np.int32), options=opt)
    before = _free()
    scale = np.ones((count, n))
    r = solver.solve_batch(m, load_scale=scale, options=opt)
    assert (r["status"] == 0).all()
    assert scale.nbytes > 1.1 * GIB
    # the scales of every system stay with the workspace, their staging does not
    assert before - _free() < 1.5 * scale.nbytes
