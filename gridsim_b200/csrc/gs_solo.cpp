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
    std::vector<int> order;  // the levels' tasks as they are dealt, level after level
    void begin(int out, int kind, int node, int level) {
        tasks.push_back({out, kind, node, level, (int)pairs.size(), (int)pairs.size()});
    }
    void pair(int a, int c, int j) { pairs.push_back({a, c, j}); }
    void end() { tasks.back().p1 = (int)pairs.size(); }
    void drop() { tasks.pop_back(); }  // a task without pairs
};

// Cycles of a bundle, for the choice of a level's split: a fixed part, one per chunk, one per halving of the group's sum.
constexpr int kBundleCycles = 90, kChunkCycles = 55, kSumCycles = 40;

int Lanes(int pairs, int chunks) {  // the lanes whose share of `pairs` takes at most `chunks` chunks
    int g = 1;
    while (g < 32 && (pairs + g - 1) / g > chunks * kSoloRounds) g *= 2;
    return g;
}

// The sums order[t0 .. t1) of a list, 2^lg lanes each, as consecutive chunks of one warp; the barriers after them.
struct Bundle {
    const TaskList* list;
    int t0, t1, lg, chunks, head, bars;
};
// A warp's bundles so far, and the levels it waits out before the first.
struct Stream {
    std::vector<Bundle> bundles;
    int before = 0, chunks = 0;
    bool worked = false;  // in the level before
    void barrier() {
        if (bundles.empty()) before++;
        else bundles.back().bars++;
    }
};

// Where a program's values are. zero: the zero's value index (the scratch value follows it); pivots: the reciprocal pivots'
// index, one: a one among them.
struct Place { int zero, pivots, one; };

// The tasks of one level (all independent; `order`'s from q0 on) into bundles, dealt to the warps, a barrier after each
// warp's last one.
void AddLevel(std::vector<Stream>& warps, TaskList& L, int q0, bool isExport = false) {
    const int W = (int)warps.size(), q1 = (int)L.order.size();
    int* order = L.order.data();
    // longest first
    thread_local std::vector<int> count, start, sizes, sorted;
    int longest = 0;
    for (int q = q0; q < q1; q++) longest = std::max(longest, L.tasks[order[q]].size());
    count.assign(longest + 1, 0);
    for (int q = q0; q < q1; q++) count[L.tasks[order[q]].size()]++;
    start.resize(longest + 1);
    sizes.clear();
    for (int n = longest, at = 0; n >= 0; at += count[n--]) {
        start[n] = at;
        if (count[n]) sizes.push_back(n);
    }
    sorted.resize(q1 - q0);
    for (int q = q0; q < q1; q++) sorted[start[L.tasks[order[q]].size()]++] = order[q];
    std::copy(sorted.begin(), sorted.end(), order + q0);
    int best = 1;
    int64_t bestCost = INT64_MAX;
    for (int r : {1, 2, 3, 4, 6, 8, 12, 16}) {
        int64_t lanes = 0;
        for (int n : sizes) lanes += (int64_t)count[n] * Lanes(n, r);
        const int g = Lanes(longest, r);
        int h = 0;
        for (int x = g; x > 1; x /= 2) h++;
        const int64_t most = std::max(1, (longest + g * kSoloRounds - 1) / (g * kSoloRounds));
        const int64_t perWarp = ((lanes + 31) / 32 + W - 1) / W;
        const int64_t c = perWarp * (kBundleCycles + most * kChunkCycles) + h * kSumCycles;
        if (c < bestCost) { bestCost = c; best = r; }
        if (r * kSoloRounds >= longest) break;
    }
    // the lanes of a sum with its length: every power of two a class of its own
    thread_local std::vector<Bundle> bundles;
    bundles.clear();
    for (int q = q0; q < q1;) {
        const int longestHere = L.tasks[order[q]].size(), g = Lanes(longestHere, best);
        int e = 0;
        while ((1 << e) < g) e++;
        int end = q + 1;
        while (end < q1 && end - q < (32 >> e) && Lanes(L.tasks[order[end]].size(), best) == g) end++;
        const int share = kSoloRounds << e;
        int head = (e << 4) | (isExport ? kSoloExport : 0);
        for (int t = q; t < end; t++) {
            const int kind = L.tasks[order[t]].kind;
            head |= kind == kSoloDiag ? kSoloHasDiag : kind == kSoloBack ? kSoloIsBack : 0;
        }
        bundles.push_back({&L, q, end, e, std::max(1, (longestHere + share - 1) / share), head, 0});
        q = end;
    }
    std::stable_sort(bundles.begin(), bundles.end(), [](const Bundle& a, const Bundle& b) { return a.chunks > b.chunks; });
    // a warp that worked in the level before is the last to be given work: another one has its next chunk at hand already
    int64_t load[kSoloWarps];
    for (int w = 0; w < W; w++) load[w] = warps[w].worked ? kBundleCycles : 0;
    for (Stream& s : warps) s.worked = false;
    for (const Bundle& b : bundles) {
        const int w = (int)(std::min_element(load, load + W) - load);
        load[w] += kBundleCycles + b.chunks * kChunkCycles;
        warps[w].worked = true;
        warps[w].bundles.push_back(b);
        warps[w].chunks += b.chunks;
    }
    for (Stream& s : warps) s.barrier();
}

// A bundle's chunks as the kernel reads them.
int32_t* Write(const Place& P, const Bundle& b, int32_t* out) {
    const bool isExport = (b.head & kSoloExport) != 0;
    const int zero = 8 * P.zero, one = 8 * (P.pivots + P.one), g = 1 << b.lg;
    const int none = isExport ? -1 : 8 * (P.zero + 1);  // where a lane without a result stores
    for (int lane = 0; lane < 32; lane++) {
        const int q = b.t0 + (lane >> b.lg), j = lane & (g - 1);
        const Task* t = q < b.t1 ? &b.list->tasks[b.list->order[q]] : nullptr;
        const int pivot = t ? 8 * (P.pivots + t->node) : one;
        const int from = t && !isExport ? 8 * t->out : zero;  // an export starts from the zero
        const int to = !t || j > 0 ? none : t->kind == kSoloDiag ? pivot : isExport ? t->out : 8 * t->out;
        const int head = (t && j == 0 ? t->kind : kSoloNone) | b.head;
        const SoloPair *p = t ? b.list->pairs.data() + t->p0 + j : nullptr, *end = t ? b.list->pairs.data() + t->p1 : nullptr;
        int left = t ? (int)(end - p + g - 1) / g : 0;  // this lane's pairs
        int32_t* o = out + 4 * lane;
        for (int k = 0; k < b.chunks; k++) {
            const int32_t extra[4] = {from, to, k + 1 == b.chunks ? head | kSoloLast | b.bars << 12 : head, pivot};
            for (int r = 0; r < kSoloRounds; r++, o += 4 * 32) {
                if (left-- > 0) {
                    o[0] = 8 * p->a;
                    o[1] = 8 * p->c;
                    o[2] = 8 * (P.pivots + p->j);
                    p += g;
                } else {
                    o[0] = o[1] = zero;
                    o[2] = one;
                }
                o[3] = extra[r];
            }
        }
    }
    return out + (size_t)b.chunks * kSoloWords;
}
static_assert(kSoloRounds == 4, "a round carries one of the four further words");

// The levels of a task list, ascending by level number.
void AddLevels(std::vector<Stream>& warps, TaskList& L) {
    const int n = (int)L.tasks.size();
    if (n == 0) return;
    int lo = L.tasks[0].level, hi = lo;
    for (const Task& t : L.tasks) { lo = std::min(lo, t.level); hi = std::max(hi, t.level); }
    std::vector<int> ptr(hi - lo + 2, 0), byLevel(n);
    for (const Task& t : L.tasks) ptr[t.level - lo + 1]++;
    for (int l = 0; l <= hi - lo; l++) ptr[l + 1] += ptr[l];
    std::vector<int> at(ptr.begin(), ptr.end() - 1);
    for (int q = 0; q < n; q++) byLevel[at[L.tasks[q].level - lo]++] = q;
    L.order.reserve(n);
    for (int l = 0; l <= hi - lo; l++) {
        if (ptr[l] == ptr[l + 1]) continue;
        L.order.insert(L.order.end(), byLevel.begin() + ptr[l], byLevel.begin() + ptr[l + 1]);
        AddLevel(warps, L, ptr[l]);
    }
}

size_t Words(const std::vector<Stream>& warps) {
    size_t n = 0;
    for (const Stream& s : warps) n += (size_t)s.chunks * kSoloWords;
    return n;
}

// The warps' streams behind what `chunks` holds (which has room for them).
void Emit(const Place& P, const std::vector<Stream>& warps, std::vector<int32_t>& chunks, std::vector<int32_t>& first) {
    size_t at = chunks.size();
    chunks.resize(at + Words(warps));
    for (const Stream& st : warps) {
        first.push_back((int)(at / kSoloWords));
        first.push_back(st.chunks);
        first.push_back(st.before);
        int32_t* out = chunks.data() + at;
        for (const Bundle& b : st.bundles) out = Write(P, b, out);
        at += (size_t)st.chunks * kSoloWords;
    }
}

}  // namespace

SoloProgram BuildSolo(const Symbolic& s) {
    SoloProgram P;
    const int64_t values = s.nnzLU + s.m + 2;
    if (s.m <= 0 || SoloSmem(values, s.m) > kSoloSmemMax) return P;
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
    L.tasks.reserve(s.entSlot.size() + s.m);
    L.pairs.reserve(s.pairs.size() / 2 + s.nnzLU / 2);
    for (size_t e = 0; e < s.entSlot.size(); e++) {
        const bool fwd = s.entKind[e] == kFwd;
        const int k = s.entNode[e], kind = s.entKind[e] == kDiag ? kSoloDiag : kSoloEntry;
        if (kind == kSoloEntry && s.entPairPtr[e] == s.entPairPtr[e + 1]) continue;  // it keeps its matrix value
        L.begin(fwd ? P.yBase + s.entSlot[e] : s.entSlot[e], kind, k, s.level[k]);
        for (int64_t q = s.entPairPtr[e]; q < s.entPairPtr[e + 1]; q++) {
            const int a = s.pairs[2 * q], c = s.pairs[2 * q + 1];
            L.pair(a, fwd ? P.yBase + c : c, nodeOf[a]);
        }
        L.end();
    }
    for (int k = 0; k < s.m; k++) {  // the backward levels after the others, from the top down
        L.begin(P.yBase + k, kSoloBack, k, 2 * s.nLevels - s.level[k]);
        for (int j = 0; j < s.luCnt[k]; j++) L.pair((int)s.luBase[k] + 1 + j, P.yBase + s.pRows[s.pRowPtr[k] + j], P.one);
        L.end();
    }
    AddLevels(warps, L);
    P.levels = s.nLevels;
    Emit(at, warps, P.chunks, P.first);
    P.on = true;
    return P;
}

// ---- a cluster's program -----------------------------------------------------------------------------------------------

namespace {

// What the cut is chosen by, per node and per subtree: values held and work.
struct Tree {
    std::vector<int64_t> size, weight, subSize, subWeight;
    std::vector<std::vector<int>> kids;
    std::vector<int> roots;
    int64_t total = 0;  // work
};

// part: a subtree is dealt out whole once it is at most 1 / part of a block's even share of the work
bool BuildSharedOn(const Symbolic& s, const Tree& tree, int C, int cap, double part, SharedProgram& P) {
    const int m = s.m;
    const std::vector<int64_t>&size = tree.size, &weight = tree.weight, &subSize = tree.subSize, &subWeight = tree.subWeight;
    const std::vector<std::vector<int>>& kids = tree.kids;
    const int64_t total = tree.total;
    std::vector<int> heap = tree.roots;
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
        std::vector<std::vector<SoloPair>> of((size_t)C * T);  // scratch: pairs by block and tier of their node
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
                of[b].push_back({luAt[a], fwd ? yAt[c] : luAt[c], dAt[j]});
            }
            if (touched.empty()) continue;
            SharedTier& t = P.blocks[cta[k]].tier[tier[k]];
            if (t.importPtr.empty()) t.importPtr.push_back(0);
            t.importAt.push_back(fwd ? yAt[s.entSlot[e]] : luAt[s.entSlot[e]]);
            std::sort(touched.begin(), touched.end());
            for (int b : touched) {
                exports[b].begin(P.nExport, kSoloEntry, place[b / T].one, 0);
                for (const SoloPair& p : of[b]) exports[b].pair(p.a, p.c, p.j);
                exports[b].end();
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
                D.end();
                if (kind == kSoloEntry && D.tasks.back().size() == 0) D.drop();  // it keeps its matrix value and imports
            }
            TaskList& U = up[tier[k]];
            U.begin(yAt[k], kSoloBack, dAt[k], -s.level[k]);
            for (int j = 0; j < s.luCnt[k]; j++) {
                const int r = s.pRows[s.pRowPtr[k] + j];
                U.pair(luAt[s.luBase[k] + 1 + j], cta[r] == q ? yAt[r] : ghost[q][upIdx[r]], place[q].one);
            }
            U.end();
        }
        std::vector<std::vector<Stream>> d(T, std::vector<Stream>(kSoloWarps)), u(d);
        size_t words = 0;
        for (int t = 0; t < T; t++) {
            AddLevels(d[t], down[t]);
            TaskList& X = exports[(size_t)q * T + t];
            X.order.resize(X.tasks.size());
            for (size_t x = 0; x < X.order.size(); x++) X.order[x] = (int)x;
            if (!X.tasks.empty()) AddLevel(d[t], X, 0, true);
            AddLevels(u[t], up[t]);
            words += Words(d[t]) + Words(u[t]);
        }
        B.chunks.reserve(words);
        for (int t = 0; t < T; t++) {
            Emit(place[q], d[t], B.chunks, B.tier[t].down);
            Emit(place[q], u[t], B.chunks, B.tier[t].up);
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
    // values a block can hold, some kept for the zero, the scratch and the solution entries it reads of higher tiers
    const int cap = (int)((kSoloSmemMax - SoloSmem(0, 0)) / 8) - 1024;
    const int m = s.m;
    const int64_t all = s.nnzLU + 2 * (int64_t)m;
    if (m <= 0 || all > 16 * (int64_t)cap) return SharedProgram();
    Tree t;
    t.size.resize(m);
    t.weight.assign(m, 0);
    t.kids.resize(m);
    for (int k = 0; k < m; k++) t.size[k] = 2 * s.luCnt[k] + 3;
    for (size_t e = 0; e < s.entSlot.size(); e++) t.weight[s.entNode[e]] += s.entPairPtr[e + 1] - s.entPairPtr[e] + 4;
    t.subSize = t.size;
    t.subWeight = t.weight;
    for (int k = 0; k < m; k++) {  // parents have higher steps
        t.total += t.weight[k];
        if (s.parent[k] < 0) { t.roots.push_back(k); continue; }
        t.kids[s.parent[k]].push_back(k);
        t.subSize[s.parent[k]] += t.subSize[k];
        t.subWeight[s.parent[k]] += t.subWeight[k];
    }
    for (int C : {2, 4, 8, 16})
        for (double part : {2.0, 1.5, 1.0}) {
            SharedProgram P;
            if (all <= (int64_t)C * cap && BuildSharedOn(s, t, C, cap, part, P)) return P;
        }
    return SharedProgram();
}

}  // namespace gs
