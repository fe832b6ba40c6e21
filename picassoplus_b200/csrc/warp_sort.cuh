// Radix sort of a list in global memory by one warp: the way out for the few long lists of a kernel that gives a thread to a list
// (members of a large cluster), where anything quadratic takes seconds for lists of 10^4.
#pragma once
#include <stdint.h>

namespace pb {

constexpr int WARP_SORT_BINS = 256;

// Sorts a[0..n) ascending by its low `bits` bits (stable); b: n more words; hist: WARP_SORT_BINS words of shared memory of this
// warp.  Returns where the result lies, a or b.  Called by a whole warp; a is complete before (a __syncwarp), the result after.
__device__ __forceinline__ uint32_t* warp_sort(uint32_t* a, uint32_t* b, int n, int bits, int32_t* hist) {
    const int lane = threadIdx.x & 31;
    for (int shift = 0; shift < bits; shift += 8) {
        for (int i = lane; i < WARP_SORT_BINS; i += 32) hist[i] = 0;
        __syncwarp();
        for (int i = lane; i < n; i += 32) atomicAdd(&hist[(a[i] >> shift) & 255u], 1);
        __syncwarp();
        int c[WARP_SORT_BINS / 32], s = 0;
#pragma unroll
        for (int j = 0; j < WARP_SORT_BINS / 32; ++j) { c[j] = hist[lane * (WARP_SORT_BINS / 32) + j]; s += c[j]; }
        int inc = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += t; }
        int run = inc - s;
#pragma unroll
        for (int j = 0; j < WARP_SORT_BINS / 32; ++j) { hist[lane * (WARP_SORT_BINS / 32) + j] = run; run += c[j]; }
        __syncwarp();
        for (int i0 = 0; i0 < n; i0 += 32) {
            const bool on = i0 + lane < n;
            const uint32_t x = on ? a[i0 + lane] : 0u;
            const int d = (int)((x >> shift) & 255u);
            const unsigned same = __match_any_sync(0xffffffffu, on ? d : -1);
            if (on) b[hist[d] + __popc(same & ((1u << lane) - 1u))] = x;
            __syncwarp();
            if (on && lane == 31 - __clz(same)) hist[d] += __popc(same);
            __syncwarp();
        }
        uint32_t* t = a; a = b; b = t;
    }
    return a;
}

}  // namespace pb
