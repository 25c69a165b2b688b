// gs_solo.cpp — the program of one system's linear solve held in a block's shared memory (SoloProgram, gs_internal.h):
// the entries of every elimination level cut into warp-sized bundles and dealt to the warps.
#include <algorithm>
#include <atomic>
#include <future>
#include <thread>

#include "gs_internal.h"

namespace gs {
namespace {

struct Task {
    int out, kind, node, level;
    int p0, p1;  // its pairs in the task list's
    int size() const { return p1 - p0; }
};
struct TaskList {
    std::vector<Task> tasks;
    std::vector<SoloPair> pairs;
    void begin(int out, int kind, int node, int level) {
        tasks.push_back({out, kind, node, level, (int)pairs.size(), (int)pairs.size()});
    }
    void pair(int a, int c, int j) {
        pairs.push_back({a, c, j});
        tasks.back().p1++;
    }
    void drop() { tasks.pop_back(); }  // a task without pairs
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
// zero: the zero's value index (the scratch value follows it); pivots: the reciprocal pivots' index, one: a one among them.
struct Place { int zero, pivots, one; };
void AddLevel(const Place& P, std::vector<Stream>& warps, const SoloPair* pairs, const Task* tasks, int nTasks,
              bool isExport = false) {
    const int W = (int)warps.size();
    int longest = 0;
    std::vector<int> count;  // tasks by number of pairs
    for (int q = 0; q < nTasks; q++) {
        longest = std::max(longest, tasks[q].size());
        if ((int)count.size() <= tasks[q].size()) count.resize(tasks[q].size() + 1, 0);
        count[tasks[q].size()]++;
    }
    int best = 1;
    int64_t bestCost = INT64_MAX;
    for (int r : {1, 2, 3, 4, 6, 8, 12, 16}) {
        int64_t lanes = 0;
        for (int n = 0; n <= longest; n++) lanes += (int64_t)count[n] * Lanes(n, r);
        const int g = Lanes(longest, r);
        int h = 0;
        for (int x = g; x > 1; x /= 2) h++;
        const int64_t most = std::max(1, (longest + g * kSoloRounds - 1) / (g * kSoloRounds));
        const int64_t perWarp = ((lanes + 31) / 32 + W - 1) / W;
        const int64_t c = perWarp * (kBundleCycles + most * kChunkCycles) + h * kSumCycles;
        if (c < bestCost) { bestCost = c; best = r; }
        if (r * kSoloRounds >= longest) break;
    }
    // longest first, the lanes of a sum with it: every power of two a class of its own
    std::vector<int> order(nTasks);
    for (int q = 0; q < nTasks; q++) order[q] = q;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return tasks[a].size() > tasks[b].size(); });
    struct Bundle { int lg, chunks, t0, t1; };
    std::vector<Bundle> bundles;
    for (int q = 0; q < nTasks;) {
        const int g = Lanes(tasks[order[q]].size(), best);
        int e = 0;
        while ((1 << e) < g) e++;
        int end = q + 1;
        while (end < nTasks && end - q < (32 >> e) && Lanes(tasks[order[end]].size(), best) == g) end++;
        const int share = kSoloRounds << e;
        bundles.push_back({e, std::max(1, (tasks[order[q]].size() + share - 1) / share), q, end});
        q = end;
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
        int32_t head = (b.lg << 4) | (isExport ? kSoloExport : 0);
        for (int q = b.t0; q < b.t1; q++)
            head |= tasks[order[q]].kind == kSoloDiag ? kSoloHasDiag : tasks[order[q]].kind == kSoloBack ? kSoloIsBack : 0;
        std::vector<int32_t>& out = warps[w].chunks;
        size_t at = out.size();
        out.resize(at + (size_t)b.chunks * kSoloWords);
        const int none = isExport ? -1 : 8 * (P.zero + 1);  // where a lane without a result stores
        for (int k = 0; k < b.chunks; k++)
            for (int r = 0; r < kSoloRounds; r++)
                for (int lane = 0; lane < 32; lane++, at += 4) {
                    const int q = b.t0 + (lane >> b.lg), j = lane & ((1 << b.lg) - 1);
                    const Task* t = q < b.t1 ? &tasks[order[q]] : nullptr;
                    const int x = t ? t->p0 + j + ((k * kSoloRounds + r) << b.lg) : 0;
                    const SoloPair p = t && x < t->p1 ? pairs[x] : SoloPair{P.zero, P.zero, P.one};
                    const int pivot = 8 * (P.pivots + (t ? t->node : P.one));
                    int extra;
                    if (r == 0) extra = 8 * (t && !isExport ? t->out : P.zero);  // an export starts from the zero
                    else if (r == 1) extra = !t || j > 0 ? none : t->kind == kSoloDiag ? pivot : isExport ? t->out : 8 * t->out;
                    else if (r == 2) extra = (t && j == 0 ? t->kind : kSoloNone) | head | (k + 1 == b.chunks ? kSoloLast : 0);
                    else extra = pivot;
                    int32_t* o = out.data() + at;
                    o[0] = 8 * p.a;
                    o[1] = 8 * p.c;
                    o[2] = 8 * (P.pivots + p.j);
                    o[3] = extra;
                }
    }
    for (Stream& s : warps) s.barrier();
}

// The levels of a task list, ascending by level number.
void AddLevels(const Place& P, std::vector<Stream>& warps, TaskList& L) {
    std::stable_sort(L.tasks.begin(), L.tasks.end(), [](const Task& a, const Task& b) { return a.level < b.level; });
    for (size_t q = 0; q < L.tasks.size();) {
        size_t e = q + 1;
        while (e < L.tasks.size() && L.tasks[e].level == L.tasks[q].level) e++;
        AddLevel(P, warps, L.pairs.data(), L.tasks.data() + q, (int)(e - q));
        q = e;
    }
}

void Emit(const std::vector<Stream>& warps, std::vector<int32_t>& chunks, std::vector<int32_t>& first) {
    for (const Stream& st : warps) {
        first.push_back((int)(chunks.size() / kSoloWords));
        first.push_back((int)(st.chunks.size() / kSoloWords));
        first.push_back(st.before);
        chunks.insert(chunks.end(), st.chunks.begin(), st.chunks.end());
    }
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
    const Place at{P.zero, P.nVal, P.one};
    std::vector<Stream> warps(kSoloWarps);
    TaskList L;
    for (size_t e = 0; e < s.entSlot.size(); e++) {
        const bool fwd = s.entKind[e] == kFwd;
        const int k = s.entNode[e], kind = s.entKind[e] == kDiag ? kSoloDiag : kSoloEntry;
        if (kind == kSoloEntry && s.entPairPtr[e] == s.entPairPtr[e + 1]) continue;  // it keeps its matrix value
        L.begin(fwd ? P.yBase + s.entSlot[e] : s.entSlot[e], kind, k, s.level[k]);
        for (int64_t q = s.entPairPtr[e]; q < s.entPairPtr[e + 1]; q++) {
            const int a = s.pairs[2 * q], c = s.pairs[2 * q + 1];
            L.pair(a, fwd ? P.yBase + c : c, nodeOf[a]);
        }
    }
    for (int k = 0; k < s.m; k++) {  // the backward levels after the others, from the top down
        L.begin(P.yBase + k, kSoloBack, k, 2 * s.nLevels - s.level[k]);
        for (int j = 0; j < s.luCnt[k]; j++) L.pair((int)s.luBase[k] + 1 + j, P.yBase + s.pRows[s.pRowPtr[k] + j], P.one);
    }
    AddLevels(at, warps, L);
    P.levels = s.nLevels;
    Emit(warps, P.chunks, P.first);
    P.on = true;
    return P;
}

// ---- a cluster's program -----------------------------------------------------------------------------------------------

namespace {

// part: a subtree is dealt out whole once it is at most 1 / part of a block's even share of the work
bool BuildSharedOn(const Symbolic& s, int C, double part, SharedProgram& P) {
    const int m = s.m;
    // values a block can hold, some kept for the zero, the scratch and the solution entries it reads of higher tiers
    const int cap = (int)((kSoloSmemMax - SoloSmem(0, 0)) / 8) - 1024;
    std::vector<int64_t> size(m), weight(m, 0), subSize(m, 0), subWeight(m, 0);
    for (int k = 0; k < m; k++) size[k] = 2 * s.luCnt[k] + 3;
    for (size_t e = 0; e < s.entSlot.size(); e++) weight[s.entNode[e]] += s.entPairPtr[e + 1] - s.entPairPtr[e] + 4;
    std::vector<std::vector<int>> kids(m);
    std::vector<int> heap;
    int64_t total = 0, all = 0;
    for (int k = 0; k < m; k++) {
        subSize[k] += size[k];
        subWeight[k] += weight[k];
        total += weight[k];
        all += size[k];
        if (s.parent[k] >= 0) {
            kids[s.parent[k]].push_back(k);
            subSize[s.parent[k]] += subSize[k];
            subWeight[s.parent[k]] += subWeight[k];
        } else {
            heap.push_back(k);
        }
    }
    if (all > (int64_t)C * cap) return false;
    // the tiers above 0: the heaviest subtrees' roots, until the rest can be dealt out evenly; the first of them, as many
    // as block 0 holds, are the last tier
    std::vector<char> tier(m, 0);
    int64_t topSize = 0;
    bool full = false;
    auto lighter = [&](int a, int b) { return subWeight[a] != subWeight[b] ? subWeight[a] < subWeight[b] : a < b; };
    std::make_heap(heap.begin(), heap.end(), lighter);
    while (!heap.empty()) {
        const int k = heap.front();
        if (part * C * (double)subWeight[k] <= (double)total && 1.5 * part * (double)subSize[k] <= (double)cap) break;
        std::pop_heap(heap.begin(), heap.end(), lighter);
        heap.pop_back();
        full = full || topSize + size[k] > cap - 256;
        const bool last = !full && (s.parent[k] < 0 || tier[s.parent[k]] == 2);
        tier[k] = last ? 2 : 1;
        if (last) topSize += size[k];
        for (int c : kids[k]) { heap.push_back(c); std::push_heap(heap.begin(), heap.end(), lighter); }
    }
    // what is dealt out: tier 0 subtrees, and the middle tier's pieces (connected parts below the last tier)
    struct Item { int root, t; int64_t size, weight; };
    std::vector<Item> items;
    for (int r : heap) items.push_back({r, 0, subSize[r], subWeight[r]});
    std::vector<int> piece(m, -1), itemCta;
    bool middle = false;
    for (int k = m - 1; k >= 0; k--) {  // parents have higher steps
        if (tier[k] != 1) continue;
        middle = true;
        if (s.parent[k] < 0 || tier[s.parent[k]] != 1) { piece[k] = (int)items.size(); items.push_back({k, 1, 0, 0}); }
        else piece[k] = piece[s.parent[k]];
        items[piece[k]].size += size[k];
        items[piece[k]].weight += weight[k];
    }
    std::vector<int> order(items.size());
    for (size_t q = 0; q < order.size(); q++) order[q] = (int)q;
    std::sort(order.begin(), order.end(), [&](int a, int b) {
        return items[a].size != items[b].size ? items[a].size > items[b].size : items[a].root < items[b].root;
    });
    std::vector<int64_t> load(2 * C, 0), used(C, 0);  // work per block and tier
    used[0] = topSize;
    itemCta.assign(items.size(), -1);
    std::vector<int> rootCta(m, -1), cta(m, -1);
    for (int q : order) {
        const Item& it = items[q];
        int best = -1;
        for (int x = 0; x < C; x++)
            if (used[x] + it.size <= cap && (best < 0 || load[it.t * C + x] < load[it.t * C + best])) best = x;
        if (best < 0) return false;
        load[it.t * C + best] += it.weight;
        used[best] += it.size;
        itemCta[q] = best;
        if (it.t == 0) rootCta[it.root] = best;
    }
    for (int k = m - 1; k >= 0; k--)
        cta[k] = tier[k] == 2 ? 0 : tier[k] == 1 ? itemCta[piece[k]] : rootCta[k] >= 0 ? rootCta[k] : cta[s.parent[k]];
    const int T = middle ? 3 : 2;
    if (!middle)
        for (int k = 0; k < m; k++) if (tier[k] == 2) tier[k] = 1;
    P.ctas = C;
    P.tiers = T;
    P.blocks.assign(C, SharedBlock());
    // ---- values of each block ----
    std::vector<int> luAt(s.nnzLU, -1), yAt(m, -1), dAt(m, -1), upIdx(m, -1), nodeOf(s.nnzLU);
    std::vector<char> hasA(s.nnzLU, 0);
    for (size_t e = 0; e < s.entSlot.size(); e++)
        if (s.entKind[e] != kFwd && s.entHasA[e]) hasA[s.entSlot[e]] = 1;
    for (int k = 0; k < m; k++) {
        SharedBlock& b = P.blocks[cta[k]];
        for (int64_t x = s.luBase[k]; x <= s.luBase[k] + 2 * s.luCnt[k]; x++) {
            nodeOf[x] = k;
            luAt[x] = (int)b.from.size();
            b.from.push_back(hasA[x] ? (int32_t)x : -1);
        }
        dAt[k] = b.nDinv++;
        b.diagAt.push_back(luAt[s.luBase[k]]);
        if (tier[k] > 0) upIdx[k] = P.nUpper++;
    }
    for (SharedBlock& b : P.blocks) { b.nVal = (int)b.from.size(); b.tier.resize(T); }
    for (int k = 0; k < m; k++) {
        SharedBlock& b = P.blocks[cta[k]];
        yAt[k] = b.nVal++;
        b.yNode.push_back(k);
        b.yAt.push_back(yAt[k]);
        if (tier[k] > 0) { b.tier[tier[k]].ownUp.push_back(upIdx[k]); b.tier[tier[k]].ownAt.push_back(yAt[k]); }
    }
    // solution entries of other blocks' higher tiers that a block's rows read, each copied before the highest tier of its
    // readers here (their own tier is above it in any case)
    std::vector<std::vector<int>> ghost(C, std::vector<int>(P.nUpper, -1));
    for (int t = T - 1; t >= 0; t--)
        for (int k = 0; k < m; k++) {
            if (tier[k] != t) continue;
            SharedBlock& b = P.blocks[cta[k]];
            for (int j = 0; j < s.luCnt[k]; j++) {
                const int r = s.pRows[s.pRowPtr[k] + j];
                if (cta[r] == cta[k] || ghost[cta[k]][upIdx[r]] >= 0) continue;
                ghost[cta[k]][upIdx[r]] = b.nVal;
                b.tier[t].ghostUp.push_back(upIdx[r]);
                b.tier[t].ghostAt.push_back(b.nVal++);
            }
        }
    std::vector<Place> place;
    for (SharedBlock& b : P.blocks) {
        b.nVal += 2;
        b.nDinv += 1;
        place.push_back({b.nVal - 2, b.nVal, b.nDinv - 1});
        P.smem = std::max(P.smem, SoloSmem(b.nVal, b.nDinv - 1));
    }
    if (P.smem > kSoloSmemMax) return false;
    // ---- sums towards entries of higher tiers in other blocks ----
    std::vector<TaskList> exports((size_t)C * T);
    {
        std::vector<std::vector<std::pair<int, SoloPair>>> of((size_t)C * T);  // scratch: pairs by block and tier of their node
        struct Import { int block, tier, at, e; };
        std::vector<int> touched;
        for (size_t e = 0; e < s.entSlot.size(); e++) {
            const int k = s.entNode[e];
            if (tier[k] == 0) continue;
            const bool fwd = s.entKind[e] == kFwd;
            touched.clear();
            for (int64_t x = s.entPairPtr[e]; x < s.entPairPtr[e + 1]; x++) {
                const int a = s.pairs[2 * x], c = s.pairs[2 * x + 1], j = nodeOf[a];
                if (cta[j] == cta[k]) continue;
                const int b = cta[j] * T + tier[j];
                if (of[b].empty()) touched.push_back(b);
                of[b].push_back({0, {luAt[a], fwd ? yAt[c] : luAt[c], dAt[j]}});
            }
            if (touched.empty()) continue;
            SharedTier& t = P.blocks[cta[k]].tier[tier[k]];
            if (t.importPtr.empty()) t.importPtr.push_back(0);
            t.importAt.push_back(fwd ? yAt[s.entSlot[e]] : luAt[s.entSlot[e]]);
            std::sort(touched.begin(), touched.end());
            for (int b : touched) {
                exports[b].begin(P.nExport, kSoloEntry, place[b / T].one, 0);
                for (auto& p : of[b]) exports[b].pair(p.second.a, p.second.c, p.second.j);
                of[b].clear();
                t.importIdx.push_back(P.nExport++);
            }
            t.importPtr.push_back((int)t.importIdx.size());
        }
    }
    // ---- streams: every block by itself ----
    std::vector<std::vector<int>> nodesOf(C);
    std::vector<int> firstEnt(m, -1);
    for (size_t e = s.entSlot.size(); e-- > 0;) firstEnt[s.entNode[e]] = (int)e;
    for (int k = 0; k < m; k++) nodesOf[cta[k]].push_back(k);
    auto build = [&](int q) {
        SharedBlock& B = P.blocks[q];
        std::vector<TaskList> down(T), up(T);
        for (int k : nodesOf[q]) {
            TaskList& D = down[tier[k]];
            for (int e = firstEnt[k]; e < (int)s.entSlot.size() && s.entNode[e] == k; e++) {
                const bool fwd = s.entKind[e] == kFwd;
                const int kind = s.entKind[e] == kDiag ? kSoloDiag : kSoloEntry;
                D.begin(fwd ? yAt[s.entSlot[e]] : luAt[s.entSlot[e]], kind, dAt[k], s.level[k]);
                for (int64_t x = s.entPairPtr[e]; x < s.entPairPtr[e + 1]; x++) {
                    const int a = s.pairs[2 * x], c = s.pairs[2 * x + 1], j = nodeOf[a];
                    if (cta[j] == q) D.pair(luAt[a], fwd ? yAt[c] : luAt[c], dAt[j]);
                }
                if (kind == kSoloEntry && D.tasks.back().size() == 0) D.drop();  // it keeps its matrix value and imports
            }
            TaskList& U = up[tier[k]];
            U.begin(yAt[k], kSoloBack, dAt[k], -s.level[k]);
            for (int j = 0; j < s.luCnt[k]; j++) {
                const int r = s.pRows[s.pRowPtr[k] + j];
                U.pair(luAt[s.luBase[k] + 1 + j], cta[r] == q ? yAt[r] : ghost[q][upIdx[r]], place[q].one);
            }
        }
        for (int t = 0; t < T; t++) {
            std::vector<Stream> d(kSoloWarps), u(kSoloWarps);
            AddLevels(place[q], d, down[t]);
            const TaskList& X = exports[(size_t)q * T + t];
            if (!X.tasks.empty()) AddLevel(place[q], d, X.pairs.data(), X.tasks.data(), (int)X.tasks.size(), true);
            Emit(d, B.chunks, B.tier[t].down);
            AddLevels(place[q], u, up[t]);
            Emit(u, B.chunks, B.tier[t].up);
        }
    };
    std::atomic<int> next{0};
    auto work = [&]() { for (int q; (q = next++) < C;) build(q); };
    std::vector<std::future<void>> threads;
    for (int w = 1; w < std::min(C, std::max(1, (int)std::thread::hardware_concurrency())); w++)
        threads.push_back(std::async(std::launch::async | std::launch::deferred, work));  // deferred: no thread to be had
    work();
    for (auto& t : threads) t.get();
    P.on = true;
    return true;
}

}  // namespace

SharedProgram BuildShared(const Symbolic& s) {
    for (int C : {2, 4, 8, 16})
        for (double part : {2.0, 1.5, 1.0}) {
            SharedProgram P;
            if (s.m > 0 && BuildSharedOn(s, C, part, P)) return P;
        }
    return SharedProgram();
}

}  // namespace gs
