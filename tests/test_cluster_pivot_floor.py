"""The pivot floor of the cluster's program (k_shared) above its cut: a pivot collapses when it falls below 1e-12 of the
matrix's own diagonal (at least 1), whatever other blocks' sums were added to that diagonal first. A grid is built so that
one pivot of a higher tier, whose diagonal of about 1e4 per unit is cancelled by a subtree of another block, comes out just
below its floor or just above it: a branch of 1e-4 per unit reactance to a bus of that subtree, and a shunt that moves the
pivot by twice its susceptance. Which pivot that is, and its value, come from the analysis and an elimination in extended
precision on the host.

Rounding: a pivot of 3e-9 (below the floor of 1e-8) or 3e-8 (above) against errors of about 16 roundings of values of 1e4,
2e-11. With the floor taken from what is left of the diagonal (below 500, so 5e-10) the first would pass unseen."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gridsim_b200 import synthetic
from gridsim_b200.engine import ContingencyAnalysis, CudaContext, PowerFlowOptions, SparseNewtonRaphsonPowerFlow

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gridsim_b200", "csrc")

HARNESS = r'''
#include <cmath>
#include <vector>
#include "gs_host.h"
using namespace gs;

// Per pivot step: its bus and kind (0 P, 1 Q), block and tier in the cluster's program, the matrix's diagonal at the start
// state, what other blocks' sums leave of it, the pivot, its parent. Returns the number of steps, or below 0: no program,
// or a diagonal that the program does not keep for its pivot's floor.
extern "C" int pivots(const gs_grid_desc* d, int* bus, int* kind, int* block, int* tier, double* diag, double* left, double* pivot,
                      int* parent) {
    HostGrid h;
    Symbolic s;
    if (!CopyGrid(d, h).empty() || !Analyze(h, s, false).empty()) return -1;
    const SharedProgram P = BuildShared(s);
    if (!P.on) return -2;
    std::vector<long double> a(s.nnzLU, 0.0L), inv(s.m);
    for (int i = 0; i < s.n; i++) {
        if (s.busP[i] >= 0) { bus[s.busP[i]] = i; kind[s.busP[i]] = 0; }
        if (s.busQ[i] >= 0) { bus[s.busQ[i]] = i; kind[s.busQ[i]] = 1; }
        long double pi = 0, qi = 0, G0 = 0, B0 = 0;
        const long double v = s.vm0[i];
        int own = -1;
        auto put = [&](int p, long double H, long double N, long double M, long double L) {
            const long double x[4] = {H, N, M, L};
            for (int k = 0; k < 4; k++) if (s.ySlot[4 * p + k] >= 0) a[s.ySlot[4 * p + k]] = x[k];
        };
        for (int p = s.yRowPtr[i]; p < s.yRowPtr[i + 1]; p++) {
            const int j = s.yCol[p];
            const long double G = s.yG[p], B = s.yB[p], u = s.vm0[j], t = (long double)s.va0[i] - s.va0[j];
            const long double c = G * std::cos(t) + B * std::sin(t), q = G * std::sin(t) - B * std::cos(t);
            pi += u * c;
            qi += u * q;
            if (j == i) { own = p; G0 = G; B0 = B; continue; }
            put(p, v * u * q, v * c, -v * u * c, v * q);
        }
        if (own >= 0) put(own, -v * qi - B0 * v * v, pi + G0 * v, v * pi - G0 * v * v, qi - B0 * v);
    }
    for (int q = 0; q < P.ctas; q++) {
        const SharedBlock& b = P.blocks[q];
        if ((int)b.diagAt.size() != b.nDinv - 1) return -3;
        std::vector<int> at(b.nVal, -1);  // the node of a right-hand side's place
        for (size_t k = 0; k < b.yNode.size(); k++) {
            block[b.yNode[k]] = q;
            tier[b.yNode[k]] = 0;
            at[b.yAt[k]] = b.yNode[k];
            if (b.from[b.diagAt[k]] != (int)s.luBase[b.yNode[k]]) return -3;
        }
        for (size_t t = 1; t < b.tier.size(); t++)
            for (int y : b.tier[t].ownAt) tier[at[y]] = (int)t;
        // a pivot's sum starts from the diagonal kept for it
        const int32_t* c = b.chunks.data();
        for (size_t n = b.chunks.size() / kSoloWords; n-- > 0; c += kSoloWords)
            for (int lane = 0; lane < 32; lane++) {
                auto w = [&](int r) { return c[(r * 32 + lane) * 4 + 3]; };
                if ((w(2) & kSoloExport) || (w(2) & 15) != kSoloDiag) continue;
                if (w(0) / 8 != b.diagAt[w(1) / 8 - b.nVal] || w(1) != w(3)) return -3;
            }
    }
    std::vector<int> nodeOf(s.nnzLU);
    for (int k = 0; k < s.m; k++)
        for (int64_t x = s.luBase[k]; x <= s.luBase[k] + 2 * s.luCnt[k]; x++) nodeOf[x] = k;
    std::vector<std::vector<int>> ents(s.m);
    for (size_t e = 0; e < s.entSlot.size(); e++) if (s.entKind[e] != kFwd) ents[s.entNode[e]].push_back((int)e);
    for (int k = 0; k < s.m; k++) {
        parent[k] = s.parent[k];
        for (int e : ents[k]) {
            long double v = a[s.entSlot[e]], l = v;
            for (int64_t x = s.entPairPtr[e]; x < s.entPairPtr[e + 1]; x++) {
                const int j = nodeOf[s.pairs[2 * x]];
                const long double p = a[s.pairs[2 * x]] * a[s.pairs[2 * x + 1]] * inv[j];
                v -= p;
                if (block[j] != block[k]) l -= p;
            }
            if (s.entKind[e] == kDiag) { diag[k] = (double)a[s.entSlot[e]]; left[k] = (double)l; pivot[k] = (double)v; inv[k] = 1.0L / v; }
            else a[s.entSlot[e]] = v;
        }
    }
    return s.m;
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("floor")
    src, so = d / "floor.cpp", d / "floor.so"
    src.write_text(HARNESS)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-pthread", "-I", CSRC, "-o", str(so), str(src)]
                          + [os.path.join(CSRC, f) for f in ("gs_symbolic.cpp", "gs_solo.cpp", "gs_host.cpp",
                                                             "gs_topology.cpp", "gs_dc.cpp")])
    return ctypes.CDLL(str(so))


def _pivots(lib, m):
    k = 2 * m.n_bus
    i = {f: np.zeros(k, np.int32) for f in ("bus", "kind", "block", "tier", "parent")}
    v = {f: np.zeros(k) for f in ("diag", "left", "pivot")}
    d = m.desc()
    arg = [x.ctypes.data_as(ctypes.c_void_p) for x in (i["bus"], i["kind"], i["block"], i["tier"], v["diag"], v["left"],
                                                       v["pivot"], i["parent"])]
    rc = lib.pivots(ctypes.byref(d), *arg)
    assert rc > 0, rc
    return {f: x[:rc] for f, x in {**i, **v}.items()}


def _crafted(lib, n_bus, target):
    """The grid, its step with the pivot, the outages that leave that pivot alone (both ends' steps outside its subtree)."""
    base = synthetic.make_grid(n_bus, n_bus + n_bus // 3 + 1, n_bus // 8, seed=5)
    p = _pivots(lib, base)
    step = np.full((base.n_bus, 2), -1)
    step[p["bus"], p["kind"]] = np.arange(len(p["bus"]))
    for k in np.nonzero((p["tier"] > 0) & (p["kind"] == 1))[0]:
        a = p["bus"][k]
        for e in np.nonzero(((base.br_from == a) | (base.br_to == a)) & (base.br_in_service != 0))[0]:
            b = base.br_to[e] if base.br_from[e] == a else base.br_from[e]
            ps, qs = step[b]
            if base.bus_type[b] != 1 or max(ps, qs) > k or (p["block"][[ps, qs]] == p["block"][k]).any():
                continue
            m = base.copy()
            m.r[e], m.x[e], m.b[e], m.tap[e], m.shift_deg[e] = 0.0, 1e-4, 0.0, 0.0, 0.0
            m.vm[b], m.va_deg[b] = m.vm[a], m.va_deg[a]
            for _ in range(3):
                got = _pivots(lib, m)
                m.bs[a] += (got["pivot"][k] - target) / (2.0 * m.vm[a]) * m.base_mva
            got = _pivots(lib, m)
            if not (abs(got["diag"][k]) > 5e3 and abs(got["left"][k]) < 500 and abs(got["pivot"][k] - target) < 1e-11):
                continue
            below = np.zeros(len(got["bus"]), bool)
            below[k] = True
            for j in range(k - 1, -1, -1):
                below[j] = got["parent"][j] >= 0 and below[got["parent"][j]]
            touched = np.zeros(m.n_bus, bool)
            touched[got["bus"][below]] = True
            free = ~touched[m.br_from] & ~touched[m.br_to] & ~synthetic.bridges(m) & (m.br_in_service != 0)
            out = np.nonzero(free)[0][:8].astype(np.int32)
            others = np.delete(np.abs(got["pivot"]) / np.maximum(1.0, np.abs(got["diag"])), k).min()
            if len(out) == 8 and others > 1e-6:
                return m, out
    raise AssertionError("no step fits")


@pytest.mark.parametrize("n_bus", [1000, 2000, 4000])
def test_the_program_keeps_the_diagonals(lib, n_bus):
    p = _pivots(lib, synthetic.make_grid(n_bus, n_bus + n_bus // 3 + 1, n_bus // 8, seed=5, operating_point=False))
    assert (p["tier"] > 0).any() and (p["left"] != p["diag"]).any()


@pytest.mark.gpu
@pytest.mark.parametrize("target,collapses", [(3e-9, True), (3e-8, False)])
@pytest.mark.parametrize("n_bus", [1000, 2000])
def test_collapsed_pivots_above_the_cut_are_found(lib, monkeypatch, n_bus, target, collapses):
    m, out = _crafted(lib, n_bus, target)
    opt = PowerFlowOptions(max_iterations=20)  # every outage starts at the case's state
    here = ContingencyAnalysis.screen_raw(m, out, SparseNewtonRaphsonPowerFlow("fp64"), opt)
    monkeypatch.setenv("GS_NO_CLUSTER_TAIL", "1")  # a context without clusters: the walks over L2
    ctx = CudaContext(0)
    monkeypatch.delenv("GS_NO_CLUSTER_TAIL")
    try:
        solver = SparseNewtonRaphsonPowerFlow("fp64", ctx)
        walk = ContingencyAnalysis.screen_raw(m, out, solver, opt)
        solver._grid.close()
    finally:
        ctx.close()
    for r in (here, walk):
        assert r["n_partial_pivot"] + r["n_singular_pivot"] == (len(out) if collapses else 0)
    if collapses:  # both solve again with row partial pivoting, from the same start
        assert (here["status"] == walk["status"]).all() and (here["iterations"] == walk["iterations"]).all()
