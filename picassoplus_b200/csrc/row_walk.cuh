// Walk of a team of TL threads over rows of a CSR (vertices v, v + stride, ...): bounds are asked for two rows ahead, the
// first entries one row ahead, so that a row costs the latency of what its entries point to and not three of them in turn.
#pragma once
#include "common.cuh"

namespace pb {

template <int TL, int B>                 // B: entries handed out together
struct RowWalk {
    static constexpr int EPT = (B + TL - 1) / TL;            // of the first B entries, per thread
    const int32_t *rowptr, *entries;
    int64_t v, stride, n;
    int beg, end, beg1, end1;
    int mine[EPT];
    unsigned mask;
    int lane;

    __device__ __forceinline__ RowWalk(const int32_t* rowptr_, const int32_t* entries_, int64_t first, int64_t stride_, int64_t n_)
        : rowptr(rowptr_), entries(entries_), v(first), stride(stride_), n(n_) {
        lane = threadIdx.x % TL;
        mask = TL == 32 ? 0xffffffffu : (((1u << (TL % 32)) - 1u) << ((threadIdx.x & 31) / TL * TL));
        bounds(v, beg, end);
        bounds(v + stride, beg1, end1);
        first_entries(beg, end);
    }
    __device__ __forceinline__ void bounds(int64_t at, int& b, int& e) const {
        b = at < n ? __ldg(rowptr + at) : 0;
        e = at < n ? __ldg(rowptr + at + 1) : 0;
    }
    __device__ __forceinline__ void first_entries(int b, int e) {
#pragma unroll
        for (int i = 0; i < EPT; ++i) {
            const int at = b + lane + i * TL;
            mine[i] = (TL <= B || lane < B) && at < e ? __ldg(entries + at) : -1;
        }
    }
    // f(ent) for every batch of the row in turn; missing entries are -1.  The next row's first entries and the bounds of the one
    // behind it are asked for once this row's first batch is known.
    template <typename F>
    __device__ __forceinline__ void rows(F&& f) {
        int ent[B];
#pragma unroll
        for (int u = 0; u < B; ++u) ent[u] = __shfl_sync(mask, mine[u / TL % EPT], u % TL, TL);
        first_entries(beg1, end1);
        const int b = beg, e = end;
        beg = beg1; end = end1;
        bounds(v + 2 * stride, beg1, end1);
        f(ent);
        for (int base = b + B; base < e; base += B) {
#pragma unroll
            for (int u = 0; u < B; ++u) ent[u] = base + u < e ? __ldg(entries + base + u) : -1;
            f(ent);
        }
    }
    __device__ __forceinline__ void step() { v += stride; }
};

}  // namespace pb
