// gs_shared.cuh — the linear solve of a few systems whose factors fit the shared memory of a cluster (SharedProgram),
// sm_100a: one cluster a system, every block's part of the tree walked with block barriers only, the cluster meeting
// between tiers only: twice with two tiers, four times with three.
//
// The walk over L2 (gs_cluster.cuh) meets at a cluster barrier twice per elimination level and loads every operand from
// L2. Here the operands are in the block's own shared memory; what crosses blocks is the sums of the subtrees towards the
// entries of higher tiers, once, and the higher tiers' solution entries, once, both through L2.
#pragma once

namespace gs {

// A block's program on the device; lists as offsets into DevShared::ints.
struct DevSharedTier {
    int down, up;                           // first tables
    int nImport, importAt, importPtr, importIdx;
    int nGhost, ghostUp, ghostAt;
    int nOwn, ownUp, ownAt;
};
struct DevSharedBlock {
    int nVal, nDinv, nLu, nY;
    int from, yNode, yAt, diagAt;
    size_t chunks;                          // the block's first chunk
    DevSharedTier tier[3];
};
struct DevShared {
    int on, ctas, tiers, nUpper, nExport;
    size_t smem;
    const DevSharedBlock* blocks;
    const int* ints;
    const int4* chunks;
};

// The linear solves of the listed systems of batch b (FP64, batch-interleaved), a cluster each: matrix values in lu, the
// right-hand side in y, which becomes the solution. scratch: per cluster the exports, then the upper nodes' solution.
__global__ void __launch_bounds__(kSoloThreads, 1) k_shared(DevGrid g, DevShared P, DevBatch b, const int* list, double* scratch) {
    __shared__ int sCollapsed;
    const int tid = threadIdx.x, q = clusterRank(), sys = blockIdx.x / P.ctas, s = list[sys];
    const DevSharedBlock& B = P.blocks[q];
    const int* ints = P.ints;
    double* val = reinterpret_cast<double*>(soloSmem);
    const int nVal = B.nVal, ring = (nVal + B.nDinv + 1) / 2 * 16;
    double* ext = scratch + (size_t)sys * (P.nExport + P.nUpper);
    double* up = ext + P.nExport;
    const size_t S = (size_t)b.B;
    const double* lu = (const double*)b.lu + s;
    double* y = (double*)b.y + s;
    for (int k = tid; k < B.nLu; k += kSoloThreads) {
        const int from = __ldg(ints + B.from + k);
        val[k] = from >= 0 ? lu[from * S] : 0.0;
    }
    for (int k = B.nLu + tid; k < nVal; k += kSoloThreads) val[k] = 0.0;
    if (tid == 0) { val[nVal + B.nDinv - 1] = 1.0; sCollapsed = 0; }
    __syncthreads();
    for (int k = tid; k < B.nY; k += kSoloThreads) {  // a node's right-hand side, and its diagonal for the pivot's floor
        const int at = __ldg(ints + B.yAt + k), diag = __ldg(ints + B.diagAt + k);
        val[at] = y[__ldg(ints + B.yNode + k) * S];
        val[nVal + k] = val[diag];
    }
    __syncthreads();
    const int4* chunks = P.chunks + B.chunks * (kSoloWords / 4);
    auto meet = [&]() {
        __syncthreads();
        clusterArrive();
        clusterWait();
    };
    for (int t = 0; t < P.tiers; t++) {
        const DevSharedTier& R = B.tier[t];
        if (t > 0) {
            meet();
            for (int k = tid; k < R.nImport; k += kSoloThreads) {
                const int p0 = __ldg(ints + R.importPtr + k), p1 = __ldg(ints + R.importPtr + k + 1);
                double sum = 0.0;  // in the order of the blocks: the same every time
                for (int p = p0; p < p1; p++) sum += __ldcg(ext + __ldg(ints + R.importIdx + p));
                val[__ldg(ints + R.importAt + k)] += sum;
            }
            __syncthreads();
        }
        if (tid < 32 * kSoloWarps) soloRun<true>(chunks, ints + R.down, ring, &sCollapsed, ext);
    }
    for (int t = P.tiers - 1; t >= 0; t--) {
        const DevSharedTier& R = B.tier[t];
        if (t < P.tiers - 1) {
            meet();
            for (int k = tid; k < R.nGhost; k += kSoloThreads)
                val[__ldg(ints + R.ghostAt + k)] = __ldcg(up + __ldg(ints + R.ghostUp + k));
        }
        __syncthreads();
        if (tid < 32 * kSoloWarps) soloRun<true>(chunks, ints + R.up, ring, &sCollapsed, ext);
        __syncthreads();
        for (int k = tid; k < R.nOwn; k += kSoloThreads) up[__ldg(ints + R.ownUp + k)] = val[__ldg(ints + R.ownAt + k)];
    }
    for (int k = tid; k < B.nY; k += kSoloThreads) y[__ldg(ints + B.yNode + k) * S] = val[__ldg(ints + B.yAt + k)];
    if (tid == 0 && sCollapsed) atomicOr(&b.flags[s], kFlagPivotPerturbed);
}

}  // namespace gs
