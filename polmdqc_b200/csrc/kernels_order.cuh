// kernels_order.cuh -- cell order of the sites by counting.
#pragma once
#include "kernels_setup.cuh"

namespace amg {

// Cell order by counting, where cells are many and small: a site counts itself
// in its cell (`slot`: how many were there before), a scan over the cells
// gives each its run, the sites go to their slots in any order and a warp per
// cell puts its ids in ascending order, so the result is that of a stable
// sort of the cell indices.  Four short kernels, each a few dependent memory
// trips (the radix sort's eight and the clearing took 40 us at 12,288 sites,
// these 12).  count[] is zero between uses.
__global__ void k_cell_count(int n, const double* __restrict__ xyz, CellGrid cg, Box bx, unsigned* __restrict__ keys,
                             int* __restrict__ slot, int* __restrict__ count) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned k = cell_of(cg, bx, xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]);
    keys[i] = k;
    slot[i] = atomicAdd(count + k, 1);
}

// one block: start and end of every cell's run
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) k_cell_scan(int ncell, const int* __restrict__ count,
                                                            int* __restrict__ start, int* __restrict__ end) {
    __shared__ int part[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int carry = 0;
    for (int c0 = 0; c0 < ncell; c0 += kScanThreads) {
        const int c = c0 + threadIdx.x, v = c < ncell ? count[c] : 0;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) part[w] = incl;
        __syncthreads();
        int before = 0, total = 0;  // of the warps below, of all
        for (int q = 0; q < 32; q++) {
            const int p = part[q];
            before += q < w ? p : 0;
            total += p;
        }
        if (c < ncell) {
            start[c] = carry + before + incl - v;
            end[c] = carry + before + incl;
        }
        carry += total;
        __syncthreads();
    }
}

__global__ void k_cell_scatter(int n, const unsigned* __restrict__ keys, const int* __restrict__ slot,
                               const int* __restrict__ start, int* __restrict__ ids) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ids[start[keys[i]] + slot[i]] = i;
}

// The m ids at `a`, all different, in ascending order by one warp, in O(m log^2 m):
// runs of 32 by counting, then each pass merges pairs of runs, every id finding
// its place by its own place in its run and a bisection of the other run.  `b`:
// scratch of the same size.  Returns the one of the two that holds the result.
__device__ __forceinline__ int* warp_merge_sort(int* a, int* b, int m) {
    const int lane = threadIdx.x & 31;
    for (int e0 = 0; e0 < m; e0 += 32) {
        const int len = min(32, m - e0), v = lane < len ? a[e0 + lane] : 0x7fffffff;
        int r = 0;
        for (int q = 0; q < len; q++) r += __shfl_sync(0xffffffffu, v, q) < v;
        if (lane < len) b[e0 + r] = v;
    }
    __syncwarp();
    int *src = b, *dst = a;
    for (int w = 32; w < m; w *= 2) {
        for (int e = lane; e < m; e += 32) {
            const int v = src[e], pair = e / (2 * w) * (2 * w), mid = min(pair + w, m);
            const bool left = e < mid;
            int lo = left ? mid : pair, hi = left ? min(pair + 2 * w, m) : mid;
            const int other = lo;
            while (lo < hi) {  // first id of the other run above v
                const int h = (lo + hi) / 2;
                if (src[h] < v) lo = h + 1;
                else hi = h;
            }
            dst[pair + (left ? e - pair : e - mid) + (lo - other)] = v;
        }
        __syncwarp();
        int* t = src;
        src = dst;
        dst = t;
    }
    return src;
}

// a warp per cell: the cell's ids in ascending order, and what k_cell_bounds
// writes of each site; clears the cell's count.  Up to kRankCell ids by
// counting the smaller ones, m^2 / 32 steps of a lane (a cell of an ordinary
// liquid has ~40 ids at a 7 A cutoff, ~100 at 9 A); a crowded cell, as a droplet
// in a large box or a long cutoff has, by merging (a droplet of 6,303 sites at a
// 22 A cutoff, 1,460 of them in one cell: 6.93 -> 6.56 ms per evaluation; 212 in a
// cell: 563 -> 560 us).  sids is scratch here until it is written.
constexpr int kRankCell = 128;
__global__ void k_cell_order(int ncell, int* ids, const double* __restrict__ xyz, const int* __restrict__ start,
                             const int* __restrict__ end, int* __restrict__ count, unsigned* __restrict__ skeys,
                             int* sids, double4* __restrict__ spos, int* __restrict__ rank,
                             const double* __restrict__ pdamp, const double* __restrict__ thole,
                             double2* __restrict__ sdt) {
    const int cell = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (cell >= ncell) return;
    const int s = start[cell], m = end[cell] - s;
    if (lane == 0) count[cell] = 0;
    const int* sorted = m > kRankCell ? warp_merge_sort(ids + s, sids + s, m) : nullptr;
    for (int e = lane; e < m; e += 32) {
        int a, p = s;
        if (sorted) {
            a = sorted[e];
            p += e;
        } else {
            a = ids[s + e];
            for (int q = 0; q < m; q++) p += ids[s + q] < a;
        }
        skeys[p] = (unsigned)cell;
        sids[p] = a;
        spos[p] = make_double4(xyz[3 * a], xyz[3 * a + 1], xyz[3 * a + 2], 0.0);
        rank[a] = p;
        if (sdt) sdt[p] = make_double2(pdamp[a], thole[a]);
    }
}

}  // namespace amg
