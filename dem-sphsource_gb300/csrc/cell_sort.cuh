// The sort by cell inside one cooperative launch: the scan of the cell counts
// and the phases of the solids' sort, separated by grid barriers (grid.cu's
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

constexpr int SORT_THREADS = 256;
constexpr int SORT_TILE = SORT_THREADS * 16;

// Exclusive scan of counts[0..num) into starts[0..num] by all blocks of a
// cooperative launch: tile sums, a grid barrier, then each tile scanned from
// the sum of the tiles before it, and a closing barrier.  False when a
// barrier gave up (the caller returns).
__device__ __forceinline__ bool cooperativeScan(const int* __restrict__ counts, int* __restrict__ starts, int num, int* tileSum,
                                unsigned* bar, unsigned& gen, int* status)
{
    const int tiles = (num + SORT_TILE - 1) / SORT_TILE;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int first = t * SORT_TILE + threadIdx.x * 16;
        int sum = 0;
        for (int k = 0; k < 16; ++k)
            if (first + k < num) sum += counts[first + k];
        int total;
        blockScan<SORT_THREADS>(sum, total);
        if (threadIdx.x == 0) tileSum[t] = total;
    }
    if (!gridBarrier(bar, gen, status)) return false;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        int before = 0;
        for (int q = threadIdx.x; q < t; q += blockDim.x) before += tileSum[q];
        int offset;
        blockScan<SORT_THREADS>(before, offset);
        const int first = t * SORT_TILE + threadIdx.x * 16;
        int v[16];
        int sum = 0;
        for (int k = 0; k < 16; ++k) {
            v[k] = first + k < num ? counts[first + k] : 0;
            sum += v[k];
        }
        int total;
        int run = offset + blockScan<SORT_THREADS>(sum, total);
        for (int k = 0; k < 16; ++k) {
            if (first + k < num) starts[first + k] = run;
            run += v[k];
        }
        if (t == tiles - 1 && threadIdx.x == 0) starts[num] = offset + total;
    }
    return gridBarrier(bar, gen, status);
}

// The solids' sort by cell from the keys of the last integration: the slots in
// the cells, the scan of the counts into the cell starts, the scatter and the
// stable rank, as phases of a cooperative launch.  False when a barrier gave up.
__device__ __forceinline__ bool solidSortPhases(const DeviceState& d, unsigned& gen)
{
    const int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.ns; i += stride)
        d.sslotInCell[i] = atomicAdd(&d.scellCount[d.skey[i]], 1);
    if (!gridBarrier(d.gridBar, gen, d.status)) return false;
    if (!cooperativeScan(d.scellCount, d.scellStart, d.grid.num, d.scanWork, d.gridBar, gen, d.status)) return false;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.ns; i += stride)
        d.ssortTmp[d.scellStart[d.skey[i]] + d.sslotInCell[i]] = i;
    if (!gridBarrier(d.gridBar, gen, d.status)) return false;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < d.ns; p += stride) {
        int e;
        const int q = stableRank(p, d.ssortTmp, d.skey, d.scellStart, nullptr, e);
        d.ssorted[q] = e;
        d.scellCount[d.skey[e]] = 0;  // the counts are consumed: clear them for the next sort
    }
    return true;
}

}  // namespace demsph
