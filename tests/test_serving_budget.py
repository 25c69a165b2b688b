"""The request loop's device-memory budget on a B200: grids solved in shared memory hold their slots in FP64, but a mixed
loop's budget is booked in its own precision first. Eight mixed grids in a budget that their FP32 slots just fill are all
registered, stay on the walk over L2, and answer as the oracle; in a wide budget the same grids move to FP64 slots when the
loop starts."""
import numpy as np
import pytest
import torch

import oracle
from gridsim_b200 import _abi, synthetic
from gridsim_b200.engine import EngineError, PowerFlowOptions
from gridsim_b200.serving import LoadFlowServer, drain

pytestmark = pytest.mark.gpu

GRIDS = 8


def _opts():
    return PowerFlowOptions(precision="mixed", max_iterations=20, warm_start_from_base=True)


def _server(budget):
    free, _ = torch.cuda.mem_get_info()
    return LoadFlowServer(_opts(), slots_per_grid=128, hbm_fraction=budget / free)


@pytest.mark.parametrize("n_bus", [300, 1000])  # a block's program, a cluster's
def test_grids_that_fit_in_fp32_are_accepted(n_bus):
    m = synthetic.make_grid(n_bus, n_bus + n_bus // 3 + 1, n_bus // 8, seed=3)
    # the booking of 32 FP32 slots: the smallest budget that takes the grid, within 20 % (128 FP64 slots take far more)
    one, budget = None, 2e5
    while one is None:
        srv = _server(budget)
        try:
            srv.add_grid(m)
            one = srv.stats()["slot_bytes"]
        except EngineError:
            budget *= 1.2
        finally:
            srv.close()
    assert 0.8 * budget < one <= budget
    idx = np.nonzero(~synthetic.bridges(m) & (m.br_in_service != 0))[0][:20].astype(np.int32)
    ref = oracle.screen(m, idx, PowerFlowOptions(max_iterations=20, warm_start_from_base=True).to_c(), keep_states=True)
    vm, va = np.asarray(ref["vm"]).reshape(len(idx), -1), np.asarray(ref["va_deg"]).reshape(len(idx), -1)
    for budget, wide in ((GRIDS * one * 1.01, False), (GRIDS * one * 100, True)):
        srv = _server(budget)
        try:
            for _ in range(GRIDS):
                srv.add_grid(m)
            assert srv.stats()["slot_bytes"] == pytest.approx(GRIDS * one)
            srv.start()
            assert (srv.stats()["slot_bytes"] > 1.2 * GRIDS * one) == wide
            reqs = [(k % GRIDS, int(idx[k // GRIDS]), 1) for k in range(GRIDS * len(idx))]
            tickets = srv.submit(reqs)
            got = {r.ticket: r for r in drain(srv, len(reqs))}
        finally:
            srv.close()
        for k, t in enumerate(tickets):
            r, j = got[int(t)], k // GRIDS
            assert r.status == ref["status"][j]
            if r.status == _abi.PF_CONVERGED:
                assert np.abs(r.vm - vm[j]).max() <= 1e-8
                assert np.radians(np.abs(r.va_deg - va[j])).max() <= 1e-8
