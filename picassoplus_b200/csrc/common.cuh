// Shared plumbing of libpicasso_b200: status codes, per-thread error text, the launch
// wrapper (launch counter + optional CUDA-event bracketing) and small device helpers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include "../../include/picasso_b200.h"

namespace pb {

void set_error(const char* fmt, ...);
int  cuda_fail(cudaError_t e, const char* what);

// Brackets one kernel launch: counts it and, when timing is enabled, records a CUDA event
// on the launch stream before and after it.
struct LaunchScope {
    const char* name;
    cudaStream_t stream;
    void* slot;
    LaunchScope(const char* name, cudaStream_t s);
    ~LaunchScope();
};

int sm_count();           // SMs of the current device (cached per device)

#define PB_REQUIRE(cond, code, ...)                      \
    do { if (!(cond)) { pb::set_error(__VA_ARGS__); return (code); } } while (0)

// launch + error check; `name` is the label the timing table reports
#define PB_LAUNCH(name, kern, grid, block, smem, stream, ...)                              \
    do {                                                                                   \
        { pb::LaunchScope _scope(name, stream);                                            \
          kern<<<(grid), (block), (smem), (stream)>>>(__VA_ARGS__); }                      \
        cudaError_t _e = cudaGetLastError();                                               \
        if (_e != cudaSuccess) return pb::cuda_fail(_e, name);                             \
    } while (0)

#define PB_CUDA(call)                                                                      \
    do { cudaError_t _e = (call); if (_e != cudaSuccess) return pb::cuda_fail(_e, #call); } while (0)

static inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
// n as the bound of 32-bit indices: (uint32_t)index < index_range(n) also refuses negative ones
static inline uint32_t index_range(int64_t n) { return n < (1LL << 31) ? (uint32_t)n : 1u << 31; }
static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
static inline int pow2_ceil(int x) { int p = 1; while (p < x) p <<= 1; return p; }

// ---- vector helpers -------------------------------------------------------------------
__device__ __forceinline__ float4 ldg4(const float4* p) { return __ldg(p); }
__device__ __forceinline__ void fma4(float4& acc, const float4& a, const float4& b) {
    acc.x = fmaf(a.x, b.x, acc.x); acc.y = fmaf(a.y, b.y, acc.y);
    acc.z = fmaf(a.z, b.z, acc.z); acc.w = fmaf(a.w, b.w, acc.w);
}
__device__ __forceinline__ void fma4s(float4& acc, float s, const float4& b) {
    acc.x = fmaf(s, b.x, acc.x); acc.y = fmaf(s, b.y, acc.y);
    acc.z = fmaf(s, b.z, acc.z); acc.w = fmaf(s, b.w, acc.w);
}
__device__ __forceinline__ float4 mul4(const float4& a, const float4& b) {
    return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w);
}
__device__ __forceinline__ float4 scale4(const float4& a, float s) {
    return make_float4(a.x * s, a.y * s, a.z * s, a.w * s);
}
__device__ __forceinline__ void add4(float4& acc, const float4& a) {
    acc.x += a.x; acc.y += a.y; acc.z += a.z; acc.w += a.w;
}
__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }

// ---- packed pairs: two fp32 operations in one instruction, each rounded as its own ------
__device__ __forceinline__ uint64_t pair2(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 unpair2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void add2(uint64_t& acc, uint64_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(a)); }
struct F4x2 { uint64_t a, b; };          // a float4 as two pairs
__device__ __forceinline__ F4x2 ldg4x2(const float4* p) {
    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(p));
    return F4x2{v.x, v.y};
}
__device__ __forceinline__ F4x2 pair4(const float4& v) { return F4x2{pair2(v.x, v.y), pair2(v.z, v.w)}; }
__device__ __forceinline__ float4 unpair4(const F4x2& v) {
    const float2 a = unpair2(v.a), b = unpair2(v.b);
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void add2(F4x2& acc, const F4x2& v) { add2(acc.a, v.a); add2(acc.b, v.b); }
__device__ __forceinline__ void add2_if(bool on, F4x2& acc, const F4x2& v) {
    asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %4, 0;\n\t@p add.rn.f32x2 %0, %0, %2;\n\t@p add.rn.f32x2 %1, %1, %3;\n\t}"
        : "+l"(acc.a), "+l"(acc.b) : "l"(v.a), "l"(v.b), "r"((int)on));
}
__device__ __forceinline__ void fma2(F4x2& acc, const F4x2& x, const F4x2& y) { fma2(acc.a, x.a, y.a); fma2(acc.b, x.b, y.b); }

// The vectorised kernels give each item (a face or a vertex) to a team of TL threads
// (TL a power of two <= 32); a thread owns one float4 channel group of the item, and
// gridDim.y walks channel chunks of 32 groups (128 channels).
struct TeamGeom {
    int TL;            // threads per item
    int chunks;        // gridDim.y
    int teams;         // items per block (blockDim 256)
};
static inline TeamGeom team_geom(int CV) {
    TeamGeom g;
    g.TL = pow2_ceil(CV < 32 ? CV : 32);
    g.chunks = (int)ceil_div(CV, 32);
    g.teams = 256 / g.TL;
    return g;
}
static inline int persistent_blocks(int64_t items, int per_block, int blocks_per_sm) {
    int64_t need = ceil_div(items, per_block);
    int64_t cap = (int64_t)sm_count() * blocks_per_sm;
    if (need < 1) need = 1;
    return (int)(need < cap ? need : cap);
}

#define PB_DISPATCH_TL(TLv, ...)                                   \
    switch (TLv) {                                                 \
        case 1:  { constexpr int TL = 1;  __VA_ARGS__; } break;    \
        case 2:  { constexpr int TL = 2;  __VA_ARGS__; } break;    \
        case 4:  { constexpr int TL = 4;  __VA_ARGS__; } break;    \
        case 8:  { constexpr int TL = 8;  __VA_ARGS__; } break;    \
        case 16: { constexpr int TL = 16; __VA_ARGS__; } break;    \
        default: { constexpr int TL = 32; __VA_ARGS__; } break;    \
    }

// out[i] = sum_b partial[b*n + i], b ascending: the fixed-order second stage of every
// filter-gradient reduction.  From `sliced_from` partials on 32 slices of them are summed side by side and then in order; one chain of
// additions costs some 40 ns per partial.  FEW_PARTIALS is for the callers whose grids end below the default: 222 partials of
// facet2vertex's 25 x 128 values 13.3 -> 20.6 us with the chain (8 570 faces), 199 of 16 x 32 11.9 -> 14.6.
constexpr int FEW_PARTIALS = 64;
int reduce_partials(const float* partial, int nparts, int64_t n, float* out, cudaStream_t stream, int sliced_from = 256);

}  // namespace pb
