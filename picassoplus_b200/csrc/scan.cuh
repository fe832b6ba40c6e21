// Exclusive prefix sums of int32 arrays in two launches: tile totals, then one pass in which every block adds up the
// totals in front of its tile for itself (a few thousand values out of the L2) and does whatever it needs the prefixes
// for.  No serial kernel over the totals and no pass that only adds offsets: as three dependent launches those were most
// of the time of a scan that fits the chip.
#pragma once
#include "common.cuh"

namespace pb {
namespace scan {

constexpr int THREADS = 256, ITEMS = 8, TILE = THREADS * ITEMS;
static inline int tiles(int64_t n) { return (int)ceil_div(n > 0 ? n : 1, TILE); }

// sum over the block, in every thread; sh: 8 ints of shared memory, reusable after the call
__device__ __forceinline__ int block_sum(int v, int* sh) {
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    int s = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) s += sh[w];
    __syncthreads();
    return s;
}

// sum of the values of the threads in front of this one
__device__ __forceinline__ int block_exclusive(int v, int* sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) sh[warp] = inc;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += sh[w];
    __syncthreads();
    return before + inc - v;
}

__device__ __forceinline__ int tiles_before(const int32_t* __restrict__ tile_sum, int tile, int* sh) {
    int v = 0;
    for (int i = threadIdx.x; i < tile; i += THREADS) v += tile_sum[i];
    return block_sum(v, sh);
}

// the thread's ITEMS consecutive values (0 past the end)
__device__ __forceinline__ void load_items(const int32_t* __restrict__ in, int64_t n, int64_t base, int (&v)[ITEMS]) {
    if (base + ITEMS <= n && (reinterpret_cast<uintptr_t>(in) & 15) == 0) {
        const int4 a = *reinterpret_cast<const int4*>(in + base), b = *reinterpret_cast<const int4*>(in + base + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) v[j] = base + j < n ? in[base + j] : 0;
    }
}

static __global__ void __launch_bounds__(THREADS)
tile_totals_kernel(const int32_t* __restrict__ in, int64_t n, int32_t* __restrict__ tile_sum) {
    __shared__ int sh[THREADS / 32];
    int v[ITEMS], s = 0;
    load_items(in, n, (int64_t)blockIdx.x * TILE + (int64_t)threadIdx.x * ITEMS, v);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) s += v[j];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = s;
}

// rowptr[0..n] = exclusive prefix of cnt[0..n); cursor (may be cnt itself) = a copy of rowptr[0..n), counts (may be NULL) =
// a copy of cnt
static __global__ void __launch_bounds__(THREADS)
row_starts_kernel(const int32_t* cnt, int64_t n, const int32_t* __restrict__ tile_sum, int32_t* __restrict__ rowptr, int32_t* cursor,
                  int32_t* __restrict__ counts) {
    __shared__ int sh[THREADS / 32];
    const int before = tiles_before(tile_sum, blockIdx.x, sh);
    const int64_t base = (int64_t)blockIdx.x * TILE + (int64_t)threadIdx.x * ITEMS;
    int v[ITEMS], s = 0;
    load_items(cnt, n, base, v);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) s += v[j];
    int run = before + block_exclusive(s, sh);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        if (base + j < n) {
            rowptr[base + j] = run;
            cursor[base + j] = run;
            if (counts) counts[base + j] = v[j];
        }
        run += v[j];
        if (base + j + 1 == n) rowptr[n] = run;
    }
}

}  // namespace scan
}  // namespace pb
