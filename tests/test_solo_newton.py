"""Newton runs held in one block's shared memory (k_solo) on a B200, through the C ABI: the smallest grid, one of odd
size, the largest that fit and the first that does not, plain and under StudyOptions (Q-limit passes in the kernel),
against the oracle on the same inputs: statuses, iterations and violations identical, converged voltages within the
parity bar of 1e-8 pu and 1e-8 rad."""
import numpy as np
import pytest

import oracle
from gridsim_b200 import _abi, synthetic
from gridsim_b200.engine import ContingencyAnalysis, PowerFlowOptions, SparseNewtonRaphsonPowerFlow, study_options
from gridsim_b200.serving import LoadFlowServer, drain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("study", [False, True])
@pytest.mark.parametrize("n_bus", [6, 31, 120, 640, 1000])
def test_screens_match_the_oracle(n_bus, study):
    m = synthetic.make_grid(n_bus, n_bus + n_bus // 3 + 1, max(1, n_bus // 8), seed=3)
    idx = m.in_service_branches()[:33]
    opt = study_options("fp64") if study else PowerFlowOptions(max_iterations=20, warm_start_from_base=True)
    if study:  # limits that bind on some units, so that passes switch buses
        m.qmin, m.qmax = m.qmin * 0.1, m.qmax * 0.1
    ref = oracle.screen(m, idx, opt.to_c(), keep_states=True)
    got = ContingencyAnalysis.screen_raw(m, idx, SparseNewtonRaphsonPowerFlow("fp64"), opt, keep_states=True)
    assert (got["status"] == ref["status"]).all()
    # where both singular-step fallbacks fail the reference stops at step 0, the engine at its cap: steps of the others
    conv = ref["status"] == _abi.PF_CONVERGED
    assert (got["iterations"][conv] == ref["iterations"][conv]).all()
    assert (got["viol_ptr"] == ref["viol_ptr"]).all()
    ok = np.nonzero((ref["status"] == _abi.PF_CONVERGED) & ~synthetic.bridges(m)[idx])[0]
    assert len(ok)
    vm, va = np.asarray(ref["vm"]).reshape(len(idx), -1), np.asarray(ref["va_deg"]).reshape(len(idx), -1)
    assert np.abs(got["vm"][ok] - vm[ok]).max() <= 1e-8
    assert np.radians(np.abs(got["va_deg"][ok] - va[ok])).max() <= 1e-8


@pytest.mark.parametrize("count", [1, 37, 400])
def test_batches_of_more_systems_than_blocks(count):
    m = synthetic.make_grid(57, 80, 7, seed=9)
    scale = np.random.default_rng(1).uniform(0.95, 1.05, size=(count, m.n_bus))
    opt = PowerFlowOptions(max_iterations=20)
    got = SparseNewtonRaphsonPowerFlow("fp64").solve_batch(m, load_scale=scale, options=opt, keep_states=True)
    for k in {0, count // 2, count - 1}:
        one = m.copy()
        one.pd, one.qd = m.pd * scale[k], m.qd * scale[k]
        ref = oracle.solve(one, opt.to_c())
        assert got["status"][k] == ref["status"] and got["iterations"][k] == ref["iterations"]
        assert np.abs(got["vm"][k] - ref["vm"]).max() <= 1e-8


# the few last systems of a batch on clusters of two, four, eight and sixteen blocks: a single solve (one system), and a
# batch of more systems than clusters are resident at once
@pytest.mark.parametrize("n_bus,count", [(1000, 1), (1000, 90), (2000, 1), (2000, 45), (4000, 1), (4000, 21), (10000, 3)])
def test_cluster_solves_match_the_oracle(n_bus, count):
    m = synthetic.make_grid(n_bus, n_bus + n_bus // 3 + 1, n_bus // 8, seed=5)
    scale = np.random.default_rng(2).uniform(0.97, 1.03, size=(count, m.n_bus))
    opt = PowerFlowOptions(max_iterations=20)
    got = SparseNewtonRaphsonPowerFlow("fp64").solve_batch(m, load_scale=scale, options=opt, keep_states=True)
    for k in {0, count // 2, count - 1}:
        one = m.copy()
        one.pd, one.qd = m.pd * scale[k], m.qd * scale[k]
        ref = oracle.solve(one, opt.to_c())
        assert got["status"][k] == ref["status"] and got["iterations"][k] == ref["iterations"]
        assert np.abs(got["vm"][k] - ref["vm"]).max() <= 1e-8
        assert np.radians(np.abs(got["va_deg"][k] - ref["va_deg"])).max() <= 1e-8


# the request loop's steps: a block's program (k_solo_step) at its smallest, an odd size and near its largest, a cluster's of
# two and four blocks, and the first size whose lanes stay on the walk (eight blocks and 128 slots)
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n_bus", [6, 31, 640, 1000, 2000, 4000])
def test_request_steps_match_the_oracle(n_bus, precision):
    m = synthetic.make_grid(n_bus, n_bus + n_bus // 3 + 1, max(1, n_bus // 8), seed=3)
    ok = np.nonzero(~synthetic.bridges(m) & (m.br_in_service != 0))[0][:40]
    opt = PowerFlowOptions(precision=precision, max_iterations=20, warm_start_from_base=True)
    ref = oracle.screen(m, ok, PowerFlowOptions(max_iterations=20, warm_start_from_base=True).to_c(), keep_states=True)
    srv = LoadFlowServer(opt, slots_per_grid=128)
    srv.add_grid(m)
    srv.start()
    try:
        tickets = srv.submit([(0, int(k), 1) for k in ok])
        got = {r.ticket: r for r in drain(srv, len(ok))}
    finally:
        srv.close()
    vm, va = np.asarray(ref["vm"]).reshape(len(ok), -1), np.asarray(ref["va_deg"]).reshape(len(ok), -1)
    for k, t in enumerate(tickets):
        r = got[int(t)]
        assert r.status == ref["status"][k]
        if ref["status"][k] == _abi.PF_CONVERGED:
            assert r.iterations == ref["iterations"][k]
            assert np.abs(r.vm - vm[k]).max() <= 1e-8
            assert np.radians(np.abs(r.va_deg - va[k])).max() <= 1e-8
