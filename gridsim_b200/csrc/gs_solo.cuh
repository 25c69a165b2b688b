// gs_solo.cuh — whole Newton runs of systems whose factors fit one block's shared memory (SoloProgram), sm_100a.
//
// The batched step costs a small system a chain of launches, a host round trip an iteration, and two barriers (of a
// cluster, over L2) per elimination level. Here a block takes a system and runs its Newton iterations to the end:
// mismatch and Jacobian straight into shared memory, the status test (the Q-limit passes too), the linear solve from
// the program's bundles, the damped update. A level of the solve costs one block barrier, one round of shared-memory
// operand loads, a short sum and a store; the index data of the next bundle (from L2) is loaded while this one is summed.
// Bound by that chain: a run of a 120-bus grid, 3 steps of 44 levels down and up and 4 mismatch evaluations, takes 78 us, so at
// most 0.3 us a level.
#pragma once

namespace gs {

__device__ __forceinline__ double blockMaxD(double v, double* red) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    double r = red[0];
    for (int k = 1; k < nw; k++) r = fmax(r, red[k]);
    return r;
}

__device__ __forceinline__ int blockOrI(int v, int* red) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, off);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    int r = 0;
    for (int k = 0; k < nw; k++) r |= red[k];
    return r;
}

// SoloProgram on the device.
struct DevSolo {
    int on, m, nVal, yBase, one;
    const int4* chunks;
    const int* first;
};

__device__ __forceinline__ void cpAsync16(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpAsyncWait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

extern __shared__ __align__(16) unsigned char soloSmem[];

// This warp's stream of a program (first: its first table). Chunks come
// through the warp's ring in shared memory three ahead (each lane copies and reads its own words, so the copies need no
// barrier and no register waits for L2) and into registers before the barrier that ends the level before. After a
// barrier every operand of a chunk is loaded at once: a level costs the barrier, one shared-memory latency, the products,
// the halvings of the sum, and on the factorisation's levels the reciprocal. A pivot's floor is relative to the matrix's
// diagonal: the value the sum starts from, or (Imported: that value may hold other blocks' sums too) what is in the
// reciprocal pivot's place before it.
template <bool Imported>
__device__ __forceinline__ void soloRun(const int4* chunks, const int* first, int ringOff, int* collapsed, double* exports) {
    constexpr int Q = kSoloRounds, kBytes = kSoloWords * 4;
    constexpr unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int4* src = chunks + (size_t)__ldg(first + 3 * w) * (kSoloWords / 4) + lane;
    const int n = __ldg(first + 3 * w + 1);
    const int before = __ldg(first + 3 * w + 2);
    // operands straight from the shared array by byte offset: one instruction each
    const int mine = ringOff + w * kSoloSlots * kBytes + lane * 16;
    auto value = [&](int off) { return *reinterpret_cast<const double*>(soloSmem + off); };
    const int4* end = src + (size_t)n * (kSoloWords / 4);
    auto copy = [&](int slot) {
        if (src < end) {
#pragma unroll
            for (int q = 0; q < Q; q++) cpAsync16(soloSmem + mine + slot * kBytes + q * 512, src + q * 32);
            src += kSoloWords / 4;
        }
        cpAsyncCommit();
    };
    int4 c[Q];
    int head;  // of the chunk in c, without the lane's kind: the same in every lane
    auto load = [&](int slot) {
#pragma unroll
        for (int q = 0; q < Q; q++) c[q] = *reinterpret_cast<const int4*>(soloSmem + mine + slot * kBytes + q * 512);
        head = (int)__reduce_or_sync(full, (unsigned)c[2].w & ~15u);
    };
    copy(0);
    copy(1);
    copy(2);
    cpAsyncWait<2>();
    if (n > 0) load(0);
    auto barrier = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kSoloWarps) : "memory"); };  // the program's warps
    for (int q = before; q > 0; q--) barrier();
    double acc0 = 0.0, acc1 = 0.0;
    auto step = [&](int slot) {  // the chunk in registers came from `slot`
        double l[kSoloRounds], u[kSoloRounds], d[kSoloRounds];
#pragma unroll
        for (int k = 0; k < kSoloRounds; k++) {
            l[k] = value(c[k].x);
            u[k] = value(c[k].y);
            d[k] = value(c[k].z);
        }
        const double base = value(c[0].w), dn = value(c[3].w);
        const int target = c[1].w, h = head;
        const bool diag = (c[2].w & 15) == kSoloDiag;
        const double mag = fabs(Imported ? dn : base), fl = diag ? pivotFloor<double>() * (mag > 1.0 ? mag : 1.0) : 0.0;
        acc0 += l[0] * (u[0] * d[0]);
        acc1 += l[1] * (u[1] * d[1]);
        acc0 += l[2] * (u[2] * d[2]);
        acc1 += l[3] * (u[3] * d[3]);
        if (h & kSoloLast) {
            double acc = acc0 + acc1;
            acc0 = acc1 = 0.0;
            for (int o = (1 << ((h >> 4) & 15)) >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(full, acc, o);
            double v = base - acc;
            if (h & kSoloHasDiag) {
                double pv = diag ? v : 1.0;
                if (!(fabs(pv) > fl)) { *collapsed = 1; pv = (pv < 0.0) ? -fl : fl; }
                v = diag ? 1.0 / pv : v;
            }
            if (h & kSoloIsBack) v *= dn;
            if (h & kSoloExport) {  // base is the zero: the sum itself, negated
                if (target >= 0) exports[target] = v;
            } else {
                *reinterpret_cast<double*>(soloSmem + target) = v;
            }
        }
        int bars = h >> 12;
        if (bars > 0) barrier();
        copy(slot);        // the chunk three on
        cpAsyncWait<2>();  // the next one is in the ring
        load(slot == 2 ? 0 : slot + 1);
        for (; bars > 1; bars--) barrier();
    };
    for (int i = 0; i < n; i += 3) {
        step(0);
        if (i + 1 >= n) break;
        step(1);
        if (i + 2 >= n) break;
        step(2);
    }
    cpAsyncWait<0>();
}

// Newton runs of the active systems of batch b (started by k_init), a block at a time each; next: the next system to
// take, maxSteps: the most steps any of them took.
// kSoloThreads: the program's warps and as many more for the work around it (mismatch, update).
constexpr int kSoloThreads = 384;
__global__ void __launch_bounds__(kSoloThreads, 2) k_solo(DevGrid g, DevSolo P, DevBatch b, int* next, double tol, double divLimit,
                                              int maxIter, int maxLoop, int* maxSteps) {
    __shared__ int sItem, sGo, sCollapsed, sCount[2];
    __shared__ double redD[32];
    __shared__ int redI[32];
    double* val = reinterpret_cast<double*>(soloSmem);
    double* dinv = val + P.nVal;
    const int ring = (P.nVal + P.m + 2) / 2 * 16;
    const int tid = threadIdx.x, bd = blockDim.x, n = g.n;
    DevBatch o = b;  // this system's Jacobian and right-hand side are in shared memory
    o.lu = val;
    o.y = val + P.yBase;
    o.z = nullptr;
    o.rhs64 = nullptr;
    o.refine = nullptr;
    o.activeCount = sCount;
    for (;;) {
        __syncthreads();
        if (tid == 0) sItem = atomicAdd(next, 1);
        __syncthreads();
        const int s = sItem;
        if (s >= b.count) return;
        if (!b.active[s]) continue;
        for (int iter = 0; iter <= maxLoop; iter++) {
            for (int q = tid; q < P.nVal; q += bd) val[q] = 0.0;
            if (tid == 0) { dinv[P.one] = 1.0; sCollapsed = 0; }
            __syncthreads();
            double mx = 0.0;
            int bad = 0;
            for (int q = tid; q < 2 * n; q += bd) busMismatchJac<double, 2, true>(g, o, q >> 1, s, mx, bad);
            mx = blockMaxD(mx, redD);
            bad = blockOrI(bad, redI);
            if (tid == 0) {
                b.maxMis[s] = (unsigned long long)__double_as_longlong(mx);
                if (bad) b.flags[s] |= (bad & 1 ? kFlagNonFinite : 0) | (bad & 2 ? kFlagJacBad : 0);
                if (g.qlim) statusQStep(o, s, tol, divLimit, maxIter);
                else statusStep(o, s, iter, tol, divLimit, maxIter);
                sGo = b.active[s] ? (g.qlim && (b.qState[s] & kQPending) ? 2 : 1) : 0;
            }
            __syncthreads();
            if (sGo == 2) {  // a converged pass: the Q limits decide whether another follows
                for (int i = tid; i < n; i += bd) qApplyBus(g, b, i, s);
                __syncthreads();
                for (int i = tid; i < n; i += bd) qRevertBus(g, b, i, s);
                __syncthreads();
                if (tid == 0) {
                    qFinishStep(o, s, g.qlimMaxPasses);
                    sGo = b.active[s] ? 2 : 0;
                }
                __syncthreads();
            }
            if (sGo == 0) break;
            if (sGo == 2) continue;  // the next pass starts from this state, no step taken
            if (tid < 32 * kSoloWarps) soloRun<false>(P.chunks, P.first, ring, &sCollapsed, nullptr);
            __syncthreads();
            const double* x = val + P.yBase;
            double dx = 0.0;
            int badStep = 0;
            for (int k = tid; k < P.m; k += bd) {
                const double v = x[k];
                badStep |= isfinite(v) ? 0 : 1;
                dx = fmax(dx, fabs(v));
            }
            dx = blockMaxD(dx, redD);
            badStep = blockOrI(badStep, redI);
            if (tid == 0) {
                const int fl = (sCollapsed ? kFlagPivotPerturbed : 0) | (badStep ? kFlagStepBad : 0);
                if (fl) b.flags[s] |= fl;
            }
            if (!badStep) {
                const double damp = dx > kMaxUndampedStep ? kMaxUndampedStep / dx : 1.0;
                const size_t B = (size_t)b.B;
                for (int i = tid; i < n; i += bd) {
                    const int kp = g.busP[i], kq = g.busQ[i];
                    if (kp >= 0) b.va[i * B + s] += damp * x[kp];
                    if (kq >= 0) {
                        double v = b.vm[i * B + s] + damp * x[kq];
                        if (v < kVmFloorPu) v = kVmFloorPu;
                        b.vm[i * B + s] = v;
                    }
                }
                if (tid == 0) {
                    b.iters[s] += 1;
                    if (b.passIter) b.passIter[s] += 1;
                }
            }
            __syncthreads();
        }
        if (tid == 0) atomicMax(maxSteps, b.iters[s]);
    }
}

// The linear solves of the listed systems of batch b (FP64, batch-interleaved), a block each: the Jacobian's values in lu
// (read only), the right-hand side in y, which becomes the solution. Steps of the request loop, whose systems join and
// leave between steps: the block's memory is refilled for each.
__global__ void __launch_bounds__(kSoloThreads, 2) k_solo_step(DevGrid g, DevSolo P, DevBatch b, const int* list) {
    __shared__ int sCollapsed;
    double* val = reinterpret_cast<double*>(soloSmem);
    const int tid = threadIdx.x, s = list[blockIdx.x];
    const size_t B = (size_t)b.B;
    const double* lu = (const double*)b.lu + s;
    double* y = (double*)b.y + s;
    for (int q = tid; q < P.nVal; q += kSoloThreads) val[q] = 0.0;
    if (tid == 0) { val[P.nVal + P.one] = 1.0; sCollapsed = 0; }
    __syncthreads();
    for (int p = tid; p < 4 * g.yRowPtr[g.n]; p += kSoloThreads) {
        const int at = g.ySlot[p];
        if (at >= 0) val[at] = lu[at * B];
    }
    for (int k = tid; k < P.m; k += kSoloThreads) val[P.yBase + k] = y[k * B];
    __syncthreads();
    if (tid < 32 * kSoloWarps) soloRun<false>(P.chunks, P.first, (P.nVal + P.m + 2) / 2 * 16, &sCollapsed, nullptr);
    __syncthreads();
    for (int k = tid; k < P.m; k += kSoloThreads) y[k * B] = val[P.yBase + k];
    if (tid == 0 && sCollapsed) atomicOr(&b.flags[s], kFlagPivotPerturbed);
}

// One linear system a block: vals / rhs a system a row, its entries' slots, the pivot positions of the right-hand side's
// rows and of the unknowns; x a system a row.
__global__ void __launch_bounds__(kSoloThreads, 2) k_solo_linear(DevSolo P, int nnz, int n, const int* __restrict__ aSlot,
                                                                 const int* __restrict__ pinv, const int* __restrict__ xinv,
                                                                 const double* __restrict__ vals, const double* __restrict__ rhs,
                                                                 double* __restrict__ x, int* flags) {
    __shared__ int sCollapsed;
    double* val = reinterpret_cast<double*>(soloSmem);
    const int tid = threadIdx.x;
    const size_t s = blockIdx.x;
    for (int q = tid; q < P.nVal; q += kSoloThreads) val[q] = 0.0;
    if (tid == 0) { val[P.nVal + P.one] = 1.0; sCollapsed = 0; }
    __syncthreads();
    for (int q = tid; q < nnz; q += kSoloThreads) val[aSlot[q]] = vals[s * nnz + q];
    for (int i = tid; i < n; i += kSoloThreads) val[P.yBase + pinv[i]] = rhs[s * n + i];
    __syncthreads();
    if (tid < 32 * kSoloWarps) soloRun<false>(P.chunks, P.first, (P.nVal + P.m + 2) / 2 * 16, &sCollapsed, nullptr);
    __syncthreads();
    for (int i = tid; i < n; i += kSoloThreads) x[s * n + i] = val[P.yBase + xinv[i]];
    if (tid == 0) flags[s] = sCollapsed ? kFlagPivotPerturbed : 0;
}

}  // namespace gs
