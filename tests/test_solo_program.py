"""The shared-memory program of one system's linear solve (gs::SoloProgram), run on the CPU from its bundles the way the
kernel runs it: between two barriers every bundle reads only the values from before the first of them (so a dependency
within a level changes the result), lanes of a bundle summed in groups. A random diagonally dominant matrix on the
matrix's own cells must be solved to rounding level, with no value or reciprocal pivot written twice in a factorisation
and every warp arriving at every barrier."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gridsim_b200 import synthetic
from conftest import golden_model

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gridsim_b200", "csrc")

HARNESS = r'''
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>
#include "gs_host.h"

using gs::SoloProgram;
using gs::SharedProgram;
using gs::Symbolic;

struct Out { double resid; int32_t on, warps, levels, rewrites, badBarriers, badIndex, wideLanes, bundles; };

// One stream set (first table `first`) over `val` (nVal values; zero and scratch indices) and `dinv`, level by level.
void Walk(const int32_t* chunks, const int32_t* first, int nVal, int zero, std::vector<double>& val, std::vector<double>& dinv,
          std::vector<int>& wrote, std::vector<int>& wroteD, bool& back, std::vector<double>* ext, std::vector<int>* extN, Out* o) {
    const int W = gs::kSoloWarps;
    std::vector<int> left(W), wait(W);
    std::vector<const int32_t*> at(W);                 // each warp's next chunk
    for (int w = 0; w < W; w++) {
        at[w] = chunks + (size_t)first[3 * w] * gs::kSoloWords;
        left[w] = first[3 * w + 1];
        wait[w] = first[3 * w + 2];
        o->bundles += left[w];
    }
    for (bool live = true; live;) {
        live = false;
        const std::vector<double> v0 = val, d0 = dinv;  // the values before this level
        int arrived = 0, ended = 0;
        for (int w = 0; w < W; w++) {
            if (wait[w] > 0) { wait[w]--; arrived++; continue; }
            if (left[w] == 0) { ended++; continue; }
            std::vector<double> acc(32, 0.0);
            for (;;) {
                if (left[w] == 0) { o->badBarriers++; break; }
                const int32_t* r = at[w];
                auto word = [&](int lane, int q, int i) { return r[(q * 32 + lane) * 4 + i]; };
                const int meta = word(0, 2, 3), G = 1 << ((meta >> 4) & 15), barriers = meta >> 12;
                const bool last = meta & gs::kSoloLast;
                if (G > 1) o->wideLanes++;
                for (int lane = 0; lane < 32; lane++) {
                    if ((word(lane, 2, 3) & ~15) != (meta & ~15)) o->badIndex++;  // the chunk's head is one for all lanes
                    for (int k = 0; k < gs::kSoloRounds; k++) {
                        const int a_ = word(lane, k, 0) / 8, c_ = word(lane, k, 1) / 8, j_ = word(lane, k, 2) / 8 - nVal;
                        if (a_ < 0 || a_ >= nVal || c_ < 0 || c_ >= nVal || j_ < 0 || j_ >= (int)dinv.size()) { o->badIndex++; continue; }
                        acc[lane] += a_ == zero ? 0.0 : v0[a_] * v0[c_] * d0[j_];
                    }
                }
                for (int lane = 0; lane < 32 && last; lane++) {
                    if (meta & gs::kSoloExport) {
                        const int to = word(lane, 1, 3);
                        if ((to >= 0) != ((word(lane, 2, 3) & 15) == gs::kSoloEntry)) o->badIndex++;
                        if (to < 0) continue;
                        double sum = 0.0;
                        for (int j = 0; j < G; j++) sum += acc[lane + j];
                        (*ext)[to] = -sum;
                        (*extN)[to]++;
                        continue;
                    }
                    const int from = word(lane, 0, 3) / 8, to = word(lane, 1, 3) / 8, kind = word(lane, 2, 3) & 15;
                    if (kind == gs::kSoloNone) { if (to != zero + 1) o->badIndex++; continue; }
                    if (lane % G) { o->badIndex++; continue; }
                    double sum = 0.0;
                    for (int j = 0; j < G; j++) sum += acc[lane + j];
                    double v = v0[from] - sum;
                    if (kind == gs::kSoloDiag) {
                        if (!(meta & gs::kSoloHasDiag)) o->badIndex++;
                        dinv[to - nVal] = 1.0 / v;
                        wroteD[to - nVal]++;
                        continue;
                    }
                    if ((kind == gs::kSoloBack) != ((meta & gs::kSoloIsBack) != 0)) o->badIndex++;
                    if (kind == gs::kSoloBack) {
                        if (!back) { back = true; std::fill(wrote.begin(), wrote.end(), 0); }
                        v *= d0[word(lane, 3, 3) / 8 - nVal];
                    }
                    if (to != from) o->badIndex++;
                    val[to] = v;
                    wrote[to]++;
                }
                if (last) std::fill(acc.begin(), acc.end(), 0.0);
                at[w] += gs::kSoloWords;
                left[w]--;
                if (barriers > 0) {
                    if (!last) o->badBarriers++;
                    wait[w] = barriers - 1;
                    arrived++;
                    break;
                }
            }
        }
        for (int x : wrote) o->rewrites += x > 1;
        for (int x : wroteD) o->rewrites += x > 1;
        if (arrived) { live = true; if (arrived != W || ended) o->badBarriers++; }
    }
}

int Run(const Symbolic& s, unsigned long long seed, Out* o) {
    const SoloProgram P = gs::BuildSolo(s);
    std::memset(o, 0, sizeof *o);
    o->on = P.on; o->warps = gs::kSoloWarps; o->levels = P.levels; 
    if (!P.on) return 0;
    std::mt19937_64 rng(seed);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    std::vector<double> val(P.nVal, 0.0), dinv(P.m + 1, std::nan("")), rowAbs(s.m, 0.0), b(s.m);
    for (int l = 0; l < s.m; l++)
        for (int p = s.aColPtr[l]; p < s.aColPtr[l + 1]; p++) {
            if (s.aRow[p] == l) continue;
            val[s.aSlot[p]] = U(rng);
            rowAbs[s.aRow[p]] += std::fabs(val[s.aSlot[p]]);
        }
    for (int l = 0; l < s.m; l++) val[s.luBase[l]] = (rowAbs[l] + 1.0) * (U(rng) < 0 ? -1.0 : 1.0);
    for (int k = 0; k < s.m; k++) val[P.yBase + k] = b[k] = U(rng);
    dinv[P.one] = 1.0;
    const std::vector<double> a = val;
    std::vector<int> wrote(P.nVal, 0), wroteD(P.m + 1, 0);
    bool back = false;
    Walk(P.chunks.data(), P.first.data(), P.nVal, P.zero, val, dinv, wrote, wroteD, back, nullptr, nullptr, o);
    double num = 0, den = 0;
    std::vector<double> r(b);
    for (int l = 0; l < s.m; l++)
        for (int p = s.aColPtr[l]; p < s.aColPtr[l + 1]; p++) r[s.aRow[p]] -= a[s.aSlot[p]] * val[P.yBase + l];
    for (int i = 0; i < s.m; i++) { num = std::fmax(num, std::isnan(r[i]) ? 1e300 : std::fabs(r[i])); den = std::fmax(den, std::fabs(b[i])); }
    o->resid = num / den;
    return 0;
}

// A cluster's program: its blocks' tiers, exports and upper solutions through arrays poisoned before each solve.
int RunShared(const Symbolic& s, unsigned long long seed, int reverse, Out* o) {
    const SharedProgram P = gs::BuildShared(s);
    std::memset(o, 0, sizeof *o);
    o->on = P.on; o->warps = P.ctas; o->levels = P.tiers;
    if (!P.on) return 0;
    if (P.smem > gs::kSoloSmemMax) return -5;
    std::mt19937_64 rng(seed);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    std::vector<double> lu(s.nnzLU, std::nan("")), rowAbs(s.m, 0.0), y(s.m);
    for (int l = 0; l < s.m; l++)
        for (int p = s.aColPtr[l]; p < s.aColPtr[l + 1]; p++) {
            if (s.aRow[p] == l) continue;
            lu[s.aSlot[p]] = U(rng);
            rowAbs[s.aRow[p]] += std::fabs(lu[s.aSlot[p]]);
        }
    for (int l = 0; l < s.m; l++) lu[s.luBase[l]] = (rowAbs[l] + 1.0) * (U(rng) < 0 ? -1.0 : 1.0);
    for (auto& v : y) v = U(rng);
    const std::vector<double> b = y;
    const int C = P.ctas;
    std::vector<std::vector<double>> val(C), dinv(C);
    std::vector<std::vector<int>> wrote(C), wroteD(C);
    std::vector<double> ext(P.nExport, std::nan("")), up(P.nUpper, std::nan(""));
    std::vector<int> extN(P.nExport, 0);
    std::vector<char> back(C, 0);
    for (int q = 0; q < C; q++) {
        const gs::SharedBlock& B = P.blocks[q];
        val[q].assign(B.nVal, 0.0);
        dinv[q].assign(B.nDinv, std::nan(""));
        dinv[q].back() = 1.0;
        wrote[q].assign(B.nVal, 0);
        wroteD[q].assign(B.nDinv, 0);
        for (size_t k = 0; k < B.from.size(); k++) if (B.from[k] >= 0) val[q][k] = lu[B.from[k]];
        for (size_t k = 0; k < B.yAt.size(); k++) val[q][B.yAt[k]] = y[B.yNode[k]];
        if (gs::SoloSmem(B.nVal, B.nDinv - 1) > P.smem) return -6;
    }
    auto walk = [&](int q, const std::vector<int32_t>& first) {
        bool bk = back[q];
        Walk(P.blocks[q].chunks.data(), first.data(), P.blocks[q].nVal, P.blocks[q].nVal - 2, val[q], dinv[q], wrote[q], wroteD[q], bk,
             &ext, &extN, o);
        back[q] = bk;
    };
    auto each = [&](auto&& f) { for (int k = 0; k < C; k++) f(reverse ? C - 1 - k : k); };
    for (int t = 0; t < P.tiers; t++)
        each([&](int q) {
            const gs::SharedTier& R = P.blocks[q].tier[t];
            for (size_t k = 0; k < R.importAt.size(); k++)
                for (int p = R.importPtr[k]; p < R.importPtr[k + 1]; p++) val[q][R.importAt[k]] += ext[R.importIdx[p]];
            walk(q, R.down);
        });
    for (int t = P.tiers - 1; t >= 0; t--) {
        each([&](int q) {
            const gs::SharedTier& R = P.blocks[q].tier[t];
            if (t == P.tiers - 1 && !R.ghostAt.empty()) o->badIndex++;
            for (size_t k = 0; k < R.ghostAt.size(); k++) val[q][R.ghostAt[k]] = up[R.ghostUp[k]];
            walk(q, R.up);
        });
        for (int q = 0; q < C; q++) {
            const gs::SharedTier& R = P.blocks[q].tier[t];
            for (size_t k = 0; k < R.ownAt.size(); k++) up[R.ownUp[k]] = val[q][R.ownAt[k]];
        }
    }
    for (int v : extN) o->rewrites += v != 1;
    std::vector<int> seen(s.m, 0);
    for (int q = 0; q < C; q++)
        for (size_t k = 0; k < P.blocks[q].yAt.size(); k++) { y[P.blocks[q].yNode[k]] = val[q][P.blocks[q].yAt[k]]; seen[P.blocks[q].yNode[k]]++; }
    for (int v : seen) o->badIndex += v != 1;
    double num = 0, den = 0;
    std::vector<double> r(b);
    for (int l = 0; l < s.m; l++)
        for (int p = s.aColPtr[l]; p < s.aColPtr[l + 1]; p++) r[s.aRow[p]] -= lu[s.aSlot[p]] * y[l];
    for (int i = 0; i < s.m; i++) { num = std::fmax(num, std::isnan(r[i]) ? 1e300 : std::fabs(r[i])); den = std::fmax(den, std::fabs(b[i])); }
    o->resid = num / den;
    return 0;
}

extern "C" int shared_grid(const gs_grid_desc* d, int qlim, unsigned long long seed, int reverse, Out* o) {
    gs::HostGrid g;
    if (!gs::CopyGrid(d, g).empty()) return -1;
    Symbolic s;
    if (!gs::Analyze(g, s, qlim != 0).empty()) return -2;
    return RunShared(s, seed, reverse, o);
}
extern "C" int solo_grid(const gs_grid_desc* d, int qlim, unsigned long long seed, Out* o) {
    gs::HostGrid g;
    if (!gs::CopyGrid(d, g).empty()) return -1;
    Symbolic s;
    if (!gs::Analyze(g, s, qlim != 0).empty()) return -2;
    return Run(s, seed, o);
}
extern "C" int solo_matrix(int n, const int* rp, const int* ci, unsigned long long seed, Out* o) {
    Symbolic s;
    std::vector<int> aSlot;
    if (!gs::AnalyzeMatrix(n, rp, ci, s, aSlot).empty()) return -2;
    return Run(s, seed, o);
}
'''


class Out(ctypes.Structure):
    _fields_ = [("resid", ctypes.c_double)] + [(k, ctypes.c_int32) for k in (
        "on", "warps", "levels", "rewrites", "badBarriers", "badIndex", "wideLanes", "bundles")]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("solo")
    src, so = d / "solo.cpp", d / "solo.so"
    src.write_text(HARNESS)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)]
                          + [os.path.join(CSRC, f) for f in ("gs_symbolic.cpp", "gs_solo.cpp", "gs_host.cpp",
                                                             "gs_topology.cpp", "gs_dc.cpp")])
    return ctypes.CDLL(str(so))


def check(o):
    assert o.on == 1
    assert o.rewrites == 0 and o.badBarriers == 0 and o.badIndex == 0
    # diagonally dominant, growth below 2: rounding of about n eps of the largest entries
    assert o.resid < 1e-12, o.resid


# up to the largest grid whose factors fit a block's shared memory (about 750 buses)
@pytest.mark.parametrize("qlim", [0, 1])
@pytest.mark.parametrize("size", [(6, 7, 1), (30, 45, 5), (120, 180, 20), (300, 411, 36), (700, 959, 84)],
                         ids=lambda s: str(s[0]))
def test_grid_programs(lib, size, qlim):
    m = synthetic.make_grid(*size, seed=1, operating_point=False)
    d = m.desc()
    o = Out()
    assert lib.solo_grid(ctypes.byref(d), qlim, ctypes.c_ulonglong(7), ctypes.byref(o)) == 0
    check(o)


@pytest.mark.parametrize("case", ["case9", "case14", "case24_ieee_rts", "case57", "case118", "case300"])
def test_golden_cases(lib, case):
    m, _ = golden_model(case)
    d = m.desc()
    o = Out()
    assert lib.solo_grid(ctypes.byref(d), 0, ctypes.c_ulonglong(3), ctypes.byref(o)) == 0
    check(o)


def _band(n, k):
    rows = [[j for j in range(max(0, i - k), min(n, i + k + 1))] for i in range(n)]
    rp = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
    return rp, np.concatenate([np.array(r, np.int32) for r in rows])


# one value, single-lane sums only, sums longer than a round of every group width
@pytest.mark.parametrize("n,k", [(1, 0), (2, 1), (9, 2), (40, 39), (140, 139), (1500, 3)])
def test_matrix_programs(lib, n, k):
    rp, ci = _band(n, k)
    o = Out()
    assert lib.solo_matrix(n, rp.ctypes.data_as(ctypes.c_void_p), ci.ctypes.data_as(ctypes.c_void_p),
                           ctypes.c_ulonglong(5), ctypes.byref(o)) == 0
    check(o)
    assert n < 40 or k < 39 or o.wideLanes > 0


# clusters of two, four, eight and sixteen blocks, with two and three tiers
@pytest.mark.parametrize("qlim", [0, 1])
@pytest.mark.parametrize("size", [(120, 180, 20), (1000, 1370, 120), (2000, 2800, 250), (4000, 5480, 480), (10000, 13500, 1200)],
                         ids=lambda s: str(s[0]))
def test_cluster_programs(lib, size, qlim):
    m = synthetic.make_grid(*size, seed=1, operating_point=False)
    d = m.desc()
    for reverse in (0, 1):
        o = Out()
        assert lib.shared_grid(ctypes.byref(d), qlim, ctypes.c_ulonglong(7), reverse, ctypes.byref(o)) == 0
        if size[0] == 10000 and qlim and not o.on:
            continue  # every bus's P and Q rows: past a cluster
        check(o)
        assert o.warps == {120: 2, 1000: 2, 2000: 4, 4000: 8, 10000: 16}[size[0]]


def test_a_system_too_large_for_a_block_has_none(lib):
    m = synthetic.make_grid(2000, 2800, 250, seed=1, operating_point=False)
    d = m.desc()
    o = Out()
    assert lib.solo_grid(ctypes.byref(d), 0, ctypes.c_ulonglong(7), ctypes.byref(o)) == 0
    assert o.on == 0
