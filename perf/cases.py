"""The work users have this engine do, as measurable cases through its public entry points.

Grids come from ``gridsim_b200.synthetic`` (the construction of the benchmark configurations); a case fixes the grid's
topology (bus count and grid seed) and the call, and the seed of :func:`prepare` makes the call's inputs: the operating
point's loads (a lognormal factor per bus around the stored ones), the load scalings of a batch, the outages screened,
the values of a sparse matrix. States that do not converge have no result (the engine reports their status), so a
pass returns their status and leaves their last iterate out; a solve's closing mismatch is rounding noise below the
tolerance and is left out likewise.
"""
import functools
import math
from dataclasses import replace

import numpy as np
import torch

from gridsim_b200 import synthetic
from gridsim_b200.engine import (ContingencyAnalysis, CudaSparseLinearSolver, PowerFlowOptions,
                                 SparseNewtonRaphsonPowerFlow, UnevenBatch, study_options)
from gridsim_b200.serving import LoadFlowServer, drain

LOAD_SIGMA = 0.05  # lognormal factor per bus on the stored loads
VIOLATION_ROWS = 96  # rows of a study's violation table per outage: about twice what these screens report


def listed():
    return [
        # an operator's single load flow of a small network (a substation area, a teaching case): pure latency
        {"name": "solve_120_fp64", "kind": "solve", "n_bus": 120, "precision": "fp64"},
        # the same call on a regional grid, and on a national one in mixed precision
        {"name": "solve_2000_fp64", "kind": "solve", "n_bus": 2000, "precision": "fp64"},
        {"name": "solve_10000_mixed", "kind": "solve", "n_bus": 10000, "precision": "mixed"},
        # Monte Carlo load scalings of one grid with every state read back (planning studies, training data)
        {"name": "batch_300_fp64", "kind": "batch", "n_bus": 300, "precision": "fp64", "count": 200},
        {"name": "batch_2750_mixed", "kind": "batch", "n_bus": 2750, "precision": "mixed", "count": 777},
        # the N-1 screen of the 2,000-bus grid, every branch that does not split it
        {"name": "screen_2000_fp64", "kind": "screen", "n_bus": 2000, "precision": "fp64", "count": 2500},
        # the N-1 screens of the 10,000-bus grid: the benchmark's, and the plain double-precision one
        {"name": "screen_10000_mixed", "kind": "screen", "n_bus": 10000, "precision": "mixed", "count": 5000},
        {"name": "screen_10000_fp64", "kind": "screen", "n_bus": 10000, "precision": "fp64", "count": 5000},
        # a contingency study under the reference's StudyOptions (Q limits enforced, DC-angle retry)
        {"name": "study_300_fp64", "kind": "study", "n_bus": 300, "precision": "fp64", "count": 400},
        # load flows of grids of uneven size in one launch
        {"name": "uneven_mixed", "kind": "uneven", "n_bus": 4000, "precision": "mixed", "grids": 8, "count": 24},
        # the batched sparse linear seam: one pattern, many matrices
        {"name": "sparse_1500", "kind": "sparse", "n_bus": 1500, "precision": "fp64", "count": 48},
        # the request loop: a burst of single-outage requests on four resident grids
        {"name": "serve_burst", "kind": "serve", "n_bus": 2000, "precision": "mixed", "grids": 4, "count": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "batch", "batch", "screen", "screen", "screen", "study", "uneven", "sparse"])
    precision = rng.choice(["fp64", "mixed"])
    grid = rng.randrange(1, 1000)
    if kind == "solve":
        return {"kind": kind, "n_bus": _log_int(rng, 100, 10000), "precision": precision, "grid": grid}
    if kind == "batch":
        n = _log_int(rng, 100, 4000)
        return {"kind": kind, "n_bus": n, "precision": precision, "grid": grid,
                "count": _log_int(rng, 2, min(3000, 4_000_000 // n))}
    if kind == "screen":
        n = _log_int(rng, 200, 10000)
        return {"kind": kind, "n_bus": n, "precision": precision, "grid": grid, "count": _log_int(rng, 10, 5000)}
    if kind == "study":
        return {"kind": kind, "n_bus": _log_int(rng, 100, 1000), "precision": precision, "grid": grid,
                "count": _log_int(rng, 20, 400)}
    if kind == "uneven":
        return {"kind": kind, "n_bus": _log_int(rng, 500, 4000), "precision": precision, "grid": grid,
                "grids": rng.randint(3, 8), "count": _log_int(rng, 1, 24)}
    return {"kind": kind, "n_bus": _log_int(rng, 50, 2000), "precision": "fp64", "grid": grid,
            "count": _log_int(rng, 1, 64)}


# ---- inputs ---------------------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _grid(n_bus, grid):
    """The network a user's program has loaded: 1.35 branches and 0.12 PV buses per bus, as the benchmark grids."""
    known = {120: (180, 20), 2000: (2800, 250), 10000: (13500, 1200)}
    branches, pv = known.get(n_bus, (int(round(1.37 * n_bus)), max(1, int(round(0.12 * n_bus)))))
    return synthetic.make_grid(n_bus, branches, pv, grid)


def _sizes(case):
    """Bus counts of an uneven population, spaced evenly over their logarithm up to the case's n_bus."""
    k = case["grids"]
    lo = min(100, case["n_bus"])
    return [int(round(lo * (case["n_bus"] / lo) ** (j / (k - 1)))) for j in range(k)]


def _rng(seed, salt):
    return np.random.Generator(np.random.PCG64([int(seed), salt]))


def _operating_point(n_bus, grid, rng):
    m = _grid(n_bus, grid).copy()
    f = np.exp(LOAD_SIGMA * rng.standard_normal(m.n_bus))
    m.pd = m.pd * f
    m.qd = m.qd * f
    m.vmin, m.vmax = np.full(m.n_bus, 0.90), np.full(m.n_bus, 1.10)  # a post-contingency (emergency) band
    return m


def _options(case):
    p = case["precision"]
    if case["kind"] == "study":
        return replace(study_options(p), per_bus_voltage_limits=True)
    warm = case["kind"] in ("screen", "serve")
    return PowerFlowOptions(precision=p, max_iterations=20, warm_start_from_base=warm, per_bus_voltage_limits=warm)


def _scalings(rng, count, n):
    """Load multipliers of one grid's cases: a global factor and a lognormal one per bus."""
    return rng.uniform(0.97, 1.03, size=(count, 1)) * np.exp(LOAD_SIGMA * rng.standard_normal((count, n)))


def _outages(m, count, rng):
    cand = np.nonzero((~synthetic.bridges(m)) & (m.br_in_service != 0))[0].astype(np.int32)
    return np.sort(rng.choice(cand, size=min(count, cand.shape[0]), replace=False)).astype(np.int32)


@functools.lru_cache(maxsize=None)
def _pattern(n_bus, grid):
    """CSR pattern of a grid's bus admittance matrix."""
    m = synthetic.make_grid(n_bus, int(round(1.37 * n_bus)), max(1, n_bus // 8), grid, operating_point=False)
    i = np.concatenate([m.br_from, m.br_to, np.arange(n_bus)]).astype(np.int64)
    j = np.concatenate([m.br_to, m.br_from, np.arange(n_bus)]).astype(np.int64)
    key = np.unique(i * n_bus + j)
    rows, cols = key // n_bus, (key % n_bus).astype(np.int32)
    indptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n_bus))]).astype(np.int32)
    return indptr, cols, rows


def _sparse_inputs(case, seed):
    n = case["n_bus"]
    indptr, cols, rows = _pattern(n, case.get("grid", 0))
    rng = _rng(seed, 5)
    matrices, rhs = [], []
    for _ in range(case["count"]):
        v = -rng.uniform(0.2, 2.0, size=cols.shape[0])  # unsymmetric off-diagonals, a loaded diagonal
        v[rows == cols] = 0.0
        s = np.zeros(n)
        np.add.at(s, rows, -v)
        v[rows == cols] = s * rng.uniform(1.01, 1.3, size=n) + 0.1
        matrices.append((indptr, cols, v))
        rhs.append(rng.standard_normal(n))
    return matrices, rhs


class _Server:
    """A request loop with its grids resident, stopped when the program drops it."""

    def __init__(self, models, options):
        self.server = LoadFlowServer(options)
        for m in models:
            self.server.add_grid(m)
        self.server.start()

    def __del__(self):
        self.server.close()


def prepare(case, seed):
    kind, grid = case["kind"], case.get("grid", 0)
    opt = _options(case)
    st = {"case": case, "options": opt}
    if kind == "sparse":
        st["matrices"], st["rhs"] = _sparse_inputs(case, seed)
        st["solver"] = CudaSparseLinearSolver()
        return st
    if kind in ("uneven", "serve"):
        rng = _rng(seed, 3)
        models = [_operating_point(n, grid + k, rng) for k, n in enumerate(_sizes(case))]
        if kind == "uneven":
            st["batch"] = UnevenBatch(models)
            st["counts"] = [case["count"]] * len(models)
            st["scale"] = [_scalings(rng, case["count"], m.n_bus) for m in models]
        else:
            st["server"] = _Server(models, opt)
            st["models"] = models
            lists = [_outages(m, 64, rng) for m in models]
            st["requests"] = [(k, int(lists[k][rng.integers(len(lists[k]))]), 1)
                              for k in (q % len(models) for q in range(case["count"]))]
        return st
    rng = _rng(seed, 1)
    m = _operating_point(case["n_bus"], grid, rng)
    st["model"] = m
    st["solver"] = SparseNewtonRaphsonPowerFlow(case["precision"])
    st["solver"].grid_for(m, opt)
    if kind == "batch":
        st["scale"] = _scalings(rng, case["count"], m.n_bus)
    elif kind in ("screen", "study"):
        st["outages"] = _outages(m, case["count"], rng)
    return st


# ---- one pass -------------------------------------------------------------------------------------------------------

def run(state):
    kind = state["case"]["kind"]
    opt = state["options"]
    if kind == "solve":
        r = state["solver"].solve(state["model"], opt)
        return {"status": r.status, "iterations": r.iterations, "vm": r.vm, "va_deg": r.va_deg, "p": r.p_inj_mw,
                "q": r.q_inj_mvar, "loading": r.loading_percent, "sf": r.sf_mva, "st": r.st_mva}
    if kind == "batch":
        r = state["solver"].solve_batch(state["model"], load_scale=state["scale"], options=opt, keep_states=True)
        ok = r["status"] == 0
        return {"status": r["status"], "iterations": r["iterations"], "vm": _kept(r["vm"], ok),
                "va_deg": _kept(r["va_deg"], ok)}
    if kind in ("screen", "study"):
        r = ContingencyAnalysis.screen_raw(state["model"], state["outages"], state["solver"], opt)
        out = {k: r[k] for k in ("status", "iterations", "min_vm", "max_vm", "max_loading_pct", "viol_ptr", "islanded")}
        rows = VIOLATION_ROWS * len(state["outages"])
        return out | {k: _table(r[k], rows) for k in ("viol_kind", "viol_element", "viol_value")}
    if kind == "uneven":
        r = state["batch"].solve(state["counts"], load_scale=state["scale"], options=opt, keep_states=True)
        ok = [s == 0 for s in r["status"]]
        return {"status": np.concatenate(r["status"]), "iterations": np.concatenate(r["iterations"]),
                "vm": [_kept(v, o) for v, o in zip(r["vm"], ok)], "va_deg": [_kept(v, o) for v, o in zip(r["va_deg"], ok)]}
    if kind == "sparse":
        return np.concatenate(state["solver"].solve_batch(state["matrices"], state["rhs"]))
    server, reqs = state["server"].server, state["requests"]
    tickets = server.submit(reqs)
    got = {r.ticket: r for r in drain(server, len(reqs))}
    rs = [got[int(t)] for t in tickets]
    return {"status": np.array([r.status for r in rs]), "iterations": np.array([r.iterations for r in rs]),
            "vm": np.concatenate([r.vm if r.converged else np.zeros_like(r.vm) for r in rs]),
            "va_deg": np.concatenate([r.va_deg if r.converged else np.zeros_like(r.vm) for r in rs])}


def _table(v, rows):
    """A screen's violation list in a table of a fixed number of rows (the report a study keeps), zeros after its end."""
    out = np.zeros(rows, v.dtype)
    out[:min(rows, v.shape[0])] = v[:rows]
    return out


def _kept(states, converged):
    """States of the cases that converged; a case that did not has none."""
    return states if converged.all() else np.where(converged[:, None], states, 0.0)


# ---- the least a pass has to move and compute ------------------------------------------------------------------------

def work(case):
    n, kind = case["n_bus"], case["kind"]
    if kind == "sparse":
        nnz = 3.74 * n
        return {"bytes": case["count"] * (8 * nnz + 16 * n) + 4 * nnz,
                "flops": case["count"] * (2 * 3.0 * n * math.log2(n) + 4 * 3 * n)}
    sizes = _sizes(case) if kind in ("uneven", "serve") else [n]
    per = 1 if kind == "solve" else case["count"]
    if kind == "serve":
        per = case["count"] / len(sizes)
    elif kind in ("screen", "study"):
        per = min(per, int(1.1 * n))
    steps = {"solve": 3, "batch": 3, "uneven": 3, "screen": 2.4, "serve": 2.4, "study": 4}[kind]
    bytes_, flops = 0.0, 0.0
    for m in sizes:
        grid = 3.74 * m * 20 + 1.37 * m * 80 + 100 * m  # Y, branches, buses
        states = 16 * m if kind not in ("screen", "study") else 64  # a state, or a row of results, per system
        scale = 8 * m if kind in ("batch", "uneven") else 4
        bytes_ += grid + per * (states + scale)
        # a step: 12 n log2 n multiply-adds of the factorisation, two sweeps over the factors, mismatch and Jacobian
        flops += per * steps * (2 * 12 * m * math.log2(m) + 4 * 26 * m + 3.74 * m * 60)
    return {"bytes": bytes_, "flops": flops}


# ---- 64-bit values ---------------------------------------------------------------------------------------------------

def _ybus(m):
    n = m.n_bus
    y = np.zeros((n, n), complex)
    on = m.br_in_service != 0
    f, t = m.br_from[on], m.br_to[on]
    ys = 1.0 / (m.r[on] + 1j * m.x[on])
    bc = 0.5j * m.b[on]
    a = m.tap[on] * np.exp(1j * np.deg2rad(m.shift_deg[on]))
    np.add.at(y, (f, f), (ys + bc) / np.abs(a) ** 2)
    np.add.at(y, (t, t), ys + bc)
    np.add.at(y, (f, t), -ys / np.conj(a))
    np.add.at(y, (t, f), -ys / a)
    y[np.arange(n), np.arange(n)] += (m.gs + 1j * m.bs) / m.base_mva
    return y, (f, t, ys, bc, a)


def _root(m, y, scale):
    """The load flow's solution for one row of load multipliers, by a dense Newton iteration to rounding level."""
    pv, pq, ref = (np.nonzero(m.bus_type == k)[0] for k in (2, 1, 3))
    ang = np.sort(np.concatenate([pv, pq]))
    vm = m.vm.astype(float).copy()
    held = np.concatenate([pv, ref])
    set_point = dict(zip(m.gen_bus.tolist(), m.vg.tolist()))
    for i in held:
        vm[i] = set_point.get(int(i), vm[i])
    v = vm * np.exp(1j * np.deg2rad(m.va_deg))
    s = -(m.pd + 1j * m.qd) * scale / m.base_mva
    np.add.at(s, m.gen_bus, (m.pg + 1j * m.qg) / m.base_mva)
    yt = torch.from_numpy(y)
    for _ in range(12):
        i = (yt @ torch.from_numpy(v)).numpy()
        mis = v * np.conj(i) - s
        fvec = np.concatenate([mis[ang].real, mis[pq].imag])
        if not np.isfinite(fvec).all():
            return None
        if np.abs(fvec).max() < 1e-12:
            return v
        u = v / np.abs(v)
        dvm = v[:, None] * np.conj(y * u[None, :])
        dvm[np.arange(v.size), np.arange(v.size)] += np.conj(i) * u
        dva = -1j * v[:, None] * np.conj(y * v[None, :])
        dva[np.arange(v.size), np.arange(v.size)] += 1j * v * np.conj(i)
        top = np.concatenate([dva[np.ix_(ang, ang)].real, dvm[np.ix_(ang, pq)].real], 1)
        low = np.concatenate([dva[np.ix_(pq, ang)].imag, dvm[np.ix_(pq, pq)].imag], 1)
        j = torch.from_numpy(np.concatenate([top, low], 0))
        dx = torch.linalg.solve(j, torch.from_numpy(-fvec)).numpy()
        va, vmag = np.angle(v), np.abs(v)
        va[ang] += dx[:ang.size]
        vmag[pq] += dx[ang.size:]
        v = vmag * np.exp(1j * va)
    return v if np.abs(fvec).max() < 1e-9 else None


def exact(case, seed):
    """Values in 64 bits by dense algebra: states of single solves and small batches, sparse solutions. Screens, whole
    populations and the largest grids would take minutes."""
    kind, n = case["kind"], case["n_bus"]
    if kind == "sparse":
        if case["count"] * (n / 1500.0) ** 3 > 64:
            return None
        out = []
        for (indptr, cols, v), b in zip(*_sparse_inputs(case, seed)):
            a = torch.zeros((n, n), dtype=torch.float64)
            rows = np.repeat(np.arange(n), np.diff(indptr))
            a[torch.from_numpy(rows), torch.from_numpy(cols.astype(np.int64))] = torch.from_numpy(v)
            out.append(torch.linalg.solve(a, torch.from_numpy(b)).numpy())
        return np.concatenate(out)
    if kind not in ("solve", "batch") or n > 2500:
        return None
    if kind == "batch" and case["count"] * (n / 300.0) ** 3 > 200:
        return None
    rng = _rng(seed, 1)
    m = _operating_point(n, case.get("grid", 0), rng)
    y, (f, t, ys, bc, a) = _ybus(m)
    if kind == "batch":
        scale = _scalings(rng, case["count"], n)
        vs = [_root(m, y, sc) for sc in scale]
        if any(v is None for v in vs):
            return None
        va = np.stack([np.degrees(np.angle(v)) for v in vs])
        return {"status": None, "iterations": None, "vm": np.stack([np.abs(v) for v in vs]), "va_deg": va}
    v = _root(m, y, 1.0)
    if v is None:
        return None
    s = v * np.conj(y @ v) * m.base_mva
    sf = v[f] * np.conj((ys + bc) / np.abs(a) ** 2 * v[f] - ys / np.conj(a) * v[t]) * m.base_mva
    st = v[t] * np.conj(-ys / a * v[f] + (ys + bc) * v[t]) * m.base_mva
    rate = m.rate_a
    loading = np.where(rate > 0, 100.0 * np.maximum(np.abs(sf), np.abs(st)) / np.where(rate > 0, rate, 1.0), 0.0)
    return {"status": None, "iterations": None, "vm": np.abs(v), "va_deg": np.degrees(np.angle(v)), "p": s.real,
            "q": s.imag, "loading": loading, "sf": sf, "st": st}
