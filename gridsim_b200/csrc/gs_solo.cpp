// gs_solo.cpp — the program of one system's linear solve held in a block's shared memory (SoloProgram, gs_internal.h):
// the entries of every elimination level cut into warp-sized bundles and dealt to the warps.
#include <algorithm>

#include "gs_internal.h"

namespace gs {
namespace {

struct Task {
    int out, kind, node;
    std::vector<SoloPair> pairs;
};

// Cycles of a bundle, for the choice of a level's split: a fixed part, one per chunk, one per halving of the group's sum.
constexpr int kBundleCycles = 90, kChunkCycles = 55, kSumCycles = 40;

int Lanes(int pairs, int chunks) {  // the lanes whose share of `pairs` takes at most `chunks` chunks
    int g = 1;
    while (g < 32 && (pairs + g - 1) / g > chunks * kSoloRounds) g *= 2;
    return g;
}

// A warp's chunks so far, and the levels it waits out before the first.
struct Stream {
    std::vector<int32_t> chunks;
    int before = 0;
    bool worked = false;  // in the level before
    void barrier() {
        if (chunks.empty()) { before++; return; }
        int32_t* c = chunks.data() + chunks.size() - kSoloWords;
        for (int lane = 0; lane < 32; lane++) c[(2 * 32 + lane) * 4 + 3] += 1 << 12;
    }
};

// A level's tasks (all independent) into bundles, dealt to the warps, a barrier after each warp's last one.
void AddLevel(const SoloProgram& P, std::vector<Stream>& warps, const std::vector<Task>& tasks) {
    const int W = (int)warps.size();
    int best = 1;
    int64_t bestCost = INT64_MAX;
    for (int r : {1, 2, 3, 4, 6, 8, 12, 16}) {
        int64_t lanes = 0, most = 0, sums = 0;
        for (const Task& t : tasks) {
            const int g = Lanes((int)t.pairs.size(), r);
            lanes += g;
            most = std::max<int64_t>(most, ((int)t.pairs.size() + g * kSoloRounds - 1) / (g * kSoloRounds));
            int h = 0;
            for (int x = g; x > 1; x /= 2) h++;
            sums = std::max<int64_t>(sums, h);
        }
        const int64_t perWarp = ((lanes + 31) / 32 + W - 1) / W;
        const int64_t c = perWarp * (kBundleCycles + std::max<int64_t>(1, most) * kChunkCycles) + sums * kSumCycles;
        if (c < bestCost) { bestCost = c; best = r; }
    }
    struct Bundle { int lg, chunks; std::vector<int> t; };
    std::vector<Bundle> bundles;
    std::vector<std::vector<int>> byG(6);
    for (size_t q = 0; q < tasks.size(); q++) {
        const int g = Lanes((int)tasks[q].pairs.size(), best);
        int e = 0;
        while ((1 << e) < g) e++;
        byG[e].push_back((int)q);
    }
    for (int e = 5; e >= 0; e--) {
        std::vector<int>& v = byG[e];
        std::stable_sort(v.begin(), v.end(), [&](int a, int b) { return tasks[a].pairs.size() > tasks[b].pairs.size(); });
        const int per = 32 >> e, share = kSoloRounds << e;
        for (size_t q = 0; q < v.size(); q += per) {
            Bundle b;
            b.lg = e;
            b.t.assign(v.begin() + q, v.begin() + std::min(v.size(), q + per));
            b.chunks = std::max(1, ((int)tasks[b.t[0]].pairs.size() + share - 1) / share);
            bundles.push_back(std::move(b));
        }
    }
    std::stable_sort(bundles.begin(), bundles.end(), [](const Bundle& a, const Bundle& b) { return a.chunks > b.chunks; });
    // a warp that worked in the level before is the last to be given work: another one has its next chunk at hand already
    std::vector<int64_t> load(W, 0);
    for (int w = 0; w < W; w++) load[w] = warps[w].worked ? kBundleCycles : 0;
    for (Stream& s : warps) s.worked = false;
    for (const Bundle& b : bundles) {
        const int w = (int)(std::min_element(load.begin(), load.end()) - load.begin());
        load[w] += kBundleCycles + b.chunks * kChunkCycles;
        warps[w].worked = true;
        int32_t head = b.lg << 4;
        for (int q : b.t) head |= tasks[q].kind == kSoloDiag ? kSoloHasDiag : tasks[q].kind == kSoloBack ? kSoloIsBack : 0;
        std::vector<int32_t>& out = warps[w].chunks;
        for (int k = 0; k < b.chunks; k++)
            for (int r = 0; r < kSoloRounds; r++)
                for (int lane = 0; lane < 32; lane++) {
                    const int q = lane >> b.lg, j = lane & ((1 << b.lg) - 1);
                    const Task* t = q < (int)b.t.size() ? &tasks[b.t[q]] : nullptr;
                    const size_t at = (size_t)j + ((size_t)(k * kSoloRounds + r) << b.lg);
                    const SoloPair p = t && at < t->pairs.size() ? t->pairs[at] : SoloPair{P.zero, P.zero, P.one};
                    const int pivot = 8 * (P.nVal + (t ? t->node : P.one));
                    const int extra[4] = {8 * (t ? t->out : P.zero),
                                          !t || j > 0 ? 8 * (P.zero + 1) : t->kind == kSoloDiag ? pivot : 8 * t->out,
                                          (t && j == 0 ? t->kind : kSoloNone) | head | (k + 1 == b.chunks ? kSoloLast : 0), pivot};
                    out.insert(out.end(), {8 * p.a, 8 * p.c, 8 * (P.nVal + p.j), extra[r]});
                }
    }
    for (Stream& s : warps) s.barrier();
}

}  // namespace

SoloProgram BuildSolo(const Symbolic& s) {
    SoloProgram P;
    const int64_t values = s.nnzLU + s.m + 2;
    if (s.m <= 0 || values > 65535 || SoloSmem(values, s.m) > kSoloSmemMax) return P;
    P.m = s.m;
    P.nVal = (int)values;
    P.yBase = (int)s.nnzLU;
    P.zero = (int)s.nnzLU + s.m;
    P.one = s.m;
    std::vector<int> nodeOf(s.nnzLU);  // the node whose row and column a slot is in
    for (int k = 0; k < s.m; k++)
        for (int64_t x = s.luBase[k]; x <= s.luBase[k] + 2 * s.luCnt[k]; x++) nodeOf[x] = k;
    std::vector<std::vector<int>> byLevel(s.nLevels);
    for (size_t e = 0; e < s.entSlot.size(); e++) byLevel[s.level[s.entNode[e]]].push_back((int)e);
    std::vector<Stream> warps(kSoloWarps);
    std::vector<Task> tasks;
    for (int l = 0; l < s.nLevels; l++) {
        tasks.clear();
        for (int e : byLevel[l]) {
            const bool fwd = s.entKind[e] == kFwd;
            Task t;
            t.node = s.entNode[e];
            t.out = fwd ? P.yBase + s.entSlot[e] : s.entSlot[e];
            t.kind = s.entKind[e] == kDiag ? kSoloDiag : kSoloEntry;
            for (int64_t q = s.entPairPtr[e]; q < s.entPairPtr[e + 1]; q++) {
                const int a = s.pairs[2 * q], c = s.pairs[2 * q + 1];
                t.pairs.push_back({a, fwd ? P.yBase + c : c, nodeOf[a]});
            }
            if (t.kind == kSoloEntry && t.pairs.empty()) continue;  // it keeps its matrix value
            tasks.push_back(std::move(t));
        }
        AddLevel(P, warps, tasks);
    }
    for (int l = s.nLevels - 1; l >= 0; l--) {
        tasks.clear();
        for (int q = s.levelNodePtr[l]; q < s.levelNodePtr[l + 1]; q++) {
            const int k = s.levelNodes[q];
            Task t;
            t.node = k;
            t.out = P.yBase + k;
            t.kind = kSoloBack;
            for (int j = 0; j < s.luCnt[k]; j++)
                t.pairs.push_back({(int)s.luBase[k] + 1 + j, P.yBase + s.pRows[s.pRowPtr[k] + j], P.one});
            tasks.push_back(std::move(t));
        }
        AddLevel(P, warps, tasks);
    }
    P.levels = s.nLevels;
    for (const Stream& st : warps) {
        P.first.push_back((int)(P.chunks.size() / kSoloWords));
        P.first.push_back((int)(st.chunks.size() / kSoloWords));
        P.first.push_back(st.before);
        P.chunks.insert(P.chunks.end(), st.chunks.begin(), st.chunks.end());
    }
    P.on = true;
    return P;
}

}  // namespace gs
