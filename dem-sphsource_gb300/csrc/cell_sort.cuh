// The sort by cell inside one launch: the scan of the cell counts
// and the phases of the solids' sort, separated by barriers over its blocks (grid.cu's
// sorts, and the contact pairs' rebuild in dem.cu).
#pragma once
#include "kernels.cuh"

namespace demsph {

// Final slot of the element at sorted position p: its cell start plus the
// number of elements of the same cell with a smaller original index.
__device__ __forceinline__ int stableRank(int p, const int* __restrict__ sorted, const int* __restrict__ key,
                                          const int* __restrict__ cellStart, const int* __restrict__ ident, int& e)
{
    e = sorted[p];
    const int k = key[e];
    const int s = cellStart[k], t = cellStart[k + 1];
    const int me = ident ? ident[e] : e;
    int rank = 0;
    for (int q = s; q < t; ++q) {
        const int o = sorted[q];
        rank += (ident ? ident[o] : o) < me;
    }
    return s + rank;
}

// ---- the barrier between two phases ----
// Large scenes sort in a cooperative launch over the GPU (GridWait).  Such a
// launch starts only when the kernel before it has drained, which costs a step
// that does not sort a microsecond more than an ordinary step launch; small
// scenes sort in ONE thread-block cluster (ClusterWait), such a launch, whose
// barrier is the hardware's.
constexpr int SORT_THREADS = 256;
struct GridWait {
    static constexpr int THREADS = SORT_THREADS;
    unsigned *bar, gen;
    int* status;
    __device__ __forceinline__ explicit GridWait(const DeviceState& d)
        : bar(d.gridBar), gen(((volatile unsigned*)d.gridBar)[1]), status(d.status)
    {
    }
    __device__ __forceinline__ bool operator()() { return gridBarrier(bar, gen, status); }
};
constexpr int SORT_CLUSTER = 8;  // blocks
struct ClusterWait {
    static constexpr int THREADS = 1024;
    __device__ __forceinline__ explicit ClusterWait(const DeviceState&) {}
    __device__ __forceinline__ bool operator()()
    {
        __threadfence();
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        return true;
    }
};

// Whether the solids are sorted in one cluster: one thread a solid, and two
// tiles of cells per block.  Steps with the cluster and with the cooperative
// launch: 17.0 and 18.3 us with 500 grains, 26.8 and 28.4 with 8k (112 and 134
// where every step sorts), 31.6 and 29.7 with 16k (177 and 145).
inline bool sortInCluster(const DeviceState& d)
{
    return d.ns <= SORT_CLUSTER * ClusterWait::THREADS && d.grid.num <= 1 << 18;
}

// Exclusive scan of counts[0..num) into starts[0..num] by all blocks: tile
// sums, a barrier, then each tile scanned from the sum of the tiles before it,
// and a closing barrier.  False when a barrier gave up (the caller returns).
template <class Wait>
__device__ __forceinline__ bool cooperativeScan(const int* __restrict__ counts, int* __restrict__ starts, int num, int* tileSum,
                                Wait& wait)
{
    constexpr int SORT_TILE = Wait::THREADS * 16;
    const int tiles = (num + SORT_TILE - 1) / SORT_TILE;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int first = t * SORT_TILE + threadIdx.x * 16;
        int sum = 0;
        for (int k = 0; k < 16; ++k)
            if (first + k < num) sum += counts[first + k];
        int total;
        blockScan<Wait::THREADS>(sum, total);
        if (threadIdx.x == 0) tileSum[t] = total;
    }
    if (!wait()) return false;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        int before = 0;
        for (int q = threadIdx.x; q < t; q += blockDim.x) before += tileSum[q];
        int offset;
        blockScan<Wait::THREADS>(before, offset);
        const int first = t * SORT_TILE + threadIdx.x * 16;
        int v[16];
        int sum = 0;
        for (int k = 0; k < 16; ++k) {
            v[k] = first + k < num ? counts[first + k] : 0;
            sum += v[k];
        }
        int total;
        int run = offset + blockScan<Wait::THREADS>(sum, total);
        for (int k = 0; k < 16; ++k) {
            if (first + k < num) starts[first + k] = run;
            run += v[k];
        }
        if (t == tiles - 1 && threadIdx.x == 0) starts[num] = offset + total;
    }
    return wait();
}

// The solids' sort by cell from the keys of the last integration: the slots in
// the cells, the scan of the counts into the cell starts, the scatter and the
// stable rank, as phases of one launch.  False when a barrier gave up.
template <class Wait>
__device__ __forceinline__ bool solidSortPhases(const DeviceState& d, Wait& wait)
{
    const int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.ns; i += stride)
        d.sslotInCell[i] = atomicAdd(&d.scellCount[d.skey[i]], 1);
    if (!wait()) return false;
    if (!cooperativeScan(d.scellCount, d.scellStart, d.grid.num, d.scanWork, wait)) return false;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.ns; i += stride)
        d.ssortTmp[d.scellStart[d.skey[i]] + d.sslotInCell[i]] = i;
    if (!wait()) return false;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < d.ns; p += stride) {
        int e;
        const int q = stableRank(p, d.ssortTmp, d.skey, d.scellStart, nullptr, e);
        d.ssorted[q] = e;
        d.scellCount[d.skey[e]] = 0;  // the counts are consumed: clear them for the next sort
    }
    return true;
}

}  // namespace demsph
