// vertex2facet: forward (pure gather) and backward (vertex-centred pull over the CSR that
// yields the input gradient and the filter gradient in one pass, no float atomics).
#include "common.cuh"
#include "row_walk.cuh"

#include <mutex>

namespace pb {

// Rows in flight and blocks per SM of the backward kernel: six rows, three sums, filter and filter gradient fill the 85 registers of
// three blocks; most vertices have six faces (batch of 32 height fields, 128 channels: 2.49 ms; eight rows 3.02, four rows and four
// blocks 3.19).
constexpr int V2F_BWD_BATCH = 6, V2F_BWD_BLOCKS = 3;

// ------------------------------------------------------------------- forward, vectorised
// r == 1, C % 4 == 0.  A team of TL threads owns two faces behind one another at a time; a thread owns one float4 of
// channels.  HBM traffic per face: 12 B of indices, 16*CV B written; the three vertex rows are gathers that mostly hit L2
// (every vertex row is shared by ~6 faces; two faces in a row mostly share an edge).  What bounds it is the latency of index
// and row loads: the next pair's indices are asked for before this pair's six rows are used (one face at a time, eight blocks
// per SM: 172 us for 1.76 M faces of 64 channels, now 122, copy floor 110; 7.4 M faces of 128 channels 1.51 ms, now 1.05).
// A corner outside the vertices is not read and contributes nothing: forward passes run on indices that nothing has checked yet.
template <int TL>
__global__ void __launch_bounds__(256, 4)
v2f_fwd_vec_kernel(int64_t Nf, uint32_t Nv, int CV, const int32_t* __restrict__ face, const float4* __restrict__ in,
                   const float4* __restrict__ filt, float4* __restrict__ out) {
    const int lane = threadIdx.x % TL;
    const int team = threadIdx.x / TL;
    const int cg = blockIdx.y * 32 + lane;
    if (cg >= CV) return;
    const float4 f0 = filt[cg], f1 = filt[CV + cg], f2 = filt[2 * CV + cg];
    const int teams = blockDim.x / TL;
    const int64_t step = 2 * (int64_t)gridDim.x * teams;
    int64_t f = 2 * ((int64_t)blockIdx.x * teams + team);
    int n[6];
    auto indices = [&](int64_t at) {                           // past the end: vertex 0, read and not used
#pragma unroll
        for (int j = 0; j < 6; ++j) n[j] = 3 * at + j < 3 * Nf ? __ldg(face + 3 * at + j) : 0;
    };
    if (f < Nf) indices(f);
    for (; f < Nf; f += step) {
        bool all = true;                                       // the team's faces: uniform among its threads
#pragma unroll
        for (int j = 0; j < 6; ++j) all = all && (uint32_t)n[j] < Nv;
        if (!all) {                                            // not for an odd last face: 0.6 us at the end of every such call
#pragma unroll 1
            for (int64_t g = f; g < Nf && g < f + 2; ++g) {
                float4 o = zero4();
#pragma unroll 1
                for (int k = 0; k < 3; ++k) {
                    const int v = __ldg(face + 3 * g + k);
                    if ((uint32_t)v < Nv) fma4(o, ldg4(filt + (int64_t)k * CV + cg), ldg4(in + (int64_t)v * CV + cg));
                }
                __stcs(out + g * CV + cg, o);
            }
            indices(f + step);
            continue;
        }
        float4 x[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) x[j] = ldg4(in + (int64_t)n[j] * CV + cg);
        indices(f + step);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            float4 o = zero4();
            fma4(o, f0, x[3 * u]);      // same k-ascending fused-multiply-add chain as the reference
            fma4(o, f1, x[3 * u + 1]);
            fma4(o, f2, x[3 * u + 2]);
            if (f + u < Nf) __stcs(out + (f + u) * CV + cg, o);
        }
    }
}

// ---------------------------------------------------------------------- forward, generic
__global__ void v2f_fwd_generic_kernel(int64_t Nf, uint32_t Nv, int C, int r, const int32_t* __restrict__ face,
                                       const float* __restrict__ in, const float* __restrict__ filt,
                                       float* __restrict__ out) {
    const int Cr = C * r;
    int64_t total = Nf * Cr;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t f = i / Cr;
        int co = (int)(i - f * Cr);
        int c = co / r;
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int v = face[3 * f + k];
            if ((uint32_t)v < Nv) acc = fmaf(__ldg(filt + k * Cr + co), __ldg(in + (int64_t)v * C + c), acc);
        }
        out[i] = acc;
    }
}

// ------------------------------------------------------------------ backward, vectorised
__device__ __forceinline__ bool finite4(const float4& a) { return isfinite(a.x) && isfinite(a.y) && isfinite(a.z) && isfinite(a.w); }
__device__ __forceinline__ void take_where_infinite(float4& a, const float4& b) {
    if (!isfinite(a.x)) a.x = b.x;
    if (!isfinite(a.y)) a.y = b.y;
    if (!isfinite(a.z)) a.z = b.z;
    if (!isfinite(a.w)) a.w = b.w;
}

// A team owns one vertex v: it walks the CSR row of v in ascending (face, corner) order and sums the gradOutput rows of its
// corners by the corner's number k in the face, s[k] = sum over (f, k) of gradOutput[f]; then
//     gradInput[v]   = sum_k s[k] * filter[k]        (fixed order -> deterministic)
//     gradFilter[k] += s[k] * input[v]               (per-thread registers)
// The per-thread filter-gradient partials are summed over the teams of the block in team
// order and written to partial[blockIdx.x][3][C]; a second kernel adds the blocks in order.
// What bounds it: instructions per corner and the threefold row gather from L2.  Sums by corner number cost a corner two packed
// additions; multiplying every row by its filter row and by input[v] cost it twelve instructions, and bounds, entries and rows
// one behind another three latencies per vertex: 980 000 vertices, 64 channels 341 us (now 248, copy floor 146); 4.15 M
// vertices, 128 channels 3.13 ms (2.49, floor 1.24).
template <int TL>
__global__ void __launch_bounds__(256, V2F_BWD_BLOCKS)
v2f_bwd_vec_kernel(int64_t Nv, int CV, const int32_t* __restrict__ rowptr, const int32_t* __restrict__ entries,
                   const float4* __restrict__ gout, const float4* __restrict__ in, const float4* __restrict__ filt,
                   float4* __restrict__ gin, float4* __restrict__ partial) {
    __shared__ float4 red[3][256];
    const int lane = threadIdx.x % TL;
    const int team = threadIdx.x / TL;
    const int teams = blockDim.x / TL;
    constexpr int B = V2F_BWD_BATCH;
    const int cg = blockIdx.y * 32 + lane;
    const bool active = cg < CV;
    F4x2 gf0{0, 0}, gf1{0, 0}, gf2{0, 0}, f0{0, 0}, f1{0, 0}, f2{0, 0};
    if (active) { f0 = pair4(filt[cg]); f1 = pair4(filt[CV + cg]); f2 = pair4(filt[2 * CV + cg]); }
    RowWalk<TL, B> walk(rowptr, entries, (int64_t)blockIdx.x * teams + team, (int64_t)gridDim.x * teams, Nv);
    for (; walk.v < Nv; walk.step()) {
        const F4x2 x = active ? ldg4x2(in + walk.v * CV + cg) : F4x2{0, 0};
        F4x2 s0{0, 0}, s1{0, 0}, s2{0, 0};
        walk.rows([&](const int (&ent)[B]) {
            F4x2 g[B];
#pragma unroll
            for (int u = 0; u < B; ++u) g[u] = active && ent[u] >= 0 ? ldg4x2(gout + (int64_t)(ent[u] >> 2) * CV + cg) : F4x2{0, 0};
#pragma unroll
            for (int u = 0; u < B; ++u) {              // a missing entry (-1) is no corner 0, 1, 2
                const int k = ent[u] & 3;
                add2_if(k == 0, s0, g[u]);
                add2_if(k == 1, s1, g[u]);
                add2_if(k == 2, s2, g[u]);
            }
        });
        F4x2 acc{0, 0};
        fma2(acc, s0, f0); fma2(acc, s1, f1); fma2(acc, s2, f2);
        fma2(gf0, s0, x); fma2(gf1, s1, x); fma2(gf2, s2, x);
        if (active) gin[walk.v * CV + cg] = unpair4(acc);
    }
    float4 r0 = unpair4(gf0), r1 = unpair4(gf1), r2 = unpair4(gf2);
    // The loop above also multiplies the empty sums of corner numbers that a vertex does not have, which is right for finite factors.
    // With an infinite filter value, or where a sum came out infinite, a thread does its channels again, corner by corner.  (Keeping
    // note in the loop of the corner numbers that occur cost every call 15 %: 245 -> 286 us, 2.14 -> 2.48 ms.)
    const float4 w0 = unpair4(f0), w1 = unpair4(f1), w2 = unpair4(f2);
    const bool filters = finite4(w0) && finite4(w1) && finite4(w2), sums = finite4(r0) && finite4(r1) && finite4(r2);
    if (active && !(filters && sums)) {
        float4 q0 = zero4(), q1 = zero4(), q2 = zero4();
#pragma unroll 1
        for (int64_t v = (int64_t)blockIdx.x * teams + team; v < Nv; v += (int64_t)gridDim.x * teams) {
            const int end = __ldg(rowptr + v + 1);
            float4 acc = zero4();
#pragma unroll 1
            for (int e = __ldg(rowptr + v); e < end; ++e) {
                const int ent = __ldg(entries + e), k = ent & 3;
                const float4 g = ldg4(gout + (int64_t)(ent >> 2) * CV + cg);
                fma4(acc, g, k == 0 ? w0 : k == 1 ? w1 : w2);
                const float4 t = mul4(g, ldg4(in + v * CV + cg));
                if (k == 0) add4(q0, t); else if (k == 1) add4(q1, t); else add4(q2, t);
            }
            if (!filters) gin[v * CV + cg] = acc;
        }
        take_where_infinite(r0, q0); take_where_infinite(r1, q1); take_where_infinite(r2, q2);
    }
    red[0][threadIdx.x] = r0; red[1][threadIdx.x] = r1; red[2][threadIdx.x] = r2;
    __syncthreads();
    if (team == 0 && active) {
        float4 s0 = zero4(), s1 = zero4(), s2 = zero4();
        for (int t = 0; t < teams; ++t) {
            add4(s0, red[0][t * TL + lane]); add4(s1, red[1][t * TL + lane]); add4(s2, red[2][t * TL + lane]);
        }
        float4* p = partial + (int64_t)blockIdx.x * 3 * CV;
        p[cg] = s0; p[CV + cg] = s1; p[2 * CV + cg] = s2;
    }
}

// --------------------------------------------------------------------- backward, generic
__global__ void v2f_bwd_input_generic_kernel(int64_t Nv, int C, int r, const int32_t* __restrict__ rowptr,
                                             const int32_t* __restrict__ entries, const float* __restrict__ gout,
                                             const float* __restrict__ filt, float* __restrict__ gin) {
    const int Cr = C * r;
    int64_t total = Nv * C;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t v = i / C;
        int c = (int)(i - v * C);
        int beg = rowptr[v], end = rowptr[v + 1];
        float acc = 0.f;
        for (int e = beg; e < end; ++e) {
            int ent = entries[e];
            int k = ent & 3;
            const float* g = gout + (int64_t)(ent >> 2) * Cr + c * r;
            const float* w = filt + k * Cr + c * r;
            for (int m = 0; m < r; ++m) acc = fmaf(__ldg(g + m), __ldg(w + m), acc);
        }
        gin[i] = acc;
    }
}

// thread = output channel co, block row = a contiguous chunk of faces walked in order
__global__ void v2f_bwd_filter_generic_kernel(int64_t Nf, uint32_t Nv, int C, int r, int64_t faces_per_chunk,
                                              const int32_t* __restrict__ face, const float* __restrict__ in,
                                              const float* __restrict__ gout, float* __restrict__ partial) {
    const int Cr = C * r;
    int co = blockIdx.y * blockDim.x + threadIdx.x;
    if (co >= Cr) return;
    int c = co / r;
    int64_t f0 = (int64_t)blockIdx.x * faces_per_chunk;
    int64_t f1 = f0 + faces_per_chunk < Nf ? f0 + faces_per_chunk : Nf;
    float a0 = 0.f, a1 = 0.f, a2 = 0.f;
    for (int64_t f = f0; f < f1; ++f) {
        float g = __ldg(gout + f * Cr + co);
        const int v0 = face[3 * f], v1 = face[3 * f + 1], v2 = face[3 * f + 2];
        if ((uint32_t)v0 < Nv) a0 = fmaf(g, __ldg(in + (int64_t)v0 * C + c), a0);
        if ((uint32_t)v1 < Nv) a1 = fmaf(g, __ldg(in + (int64_t)v1 * C + c), a1);
        if ((uint32_t)v2 < Nv) a2 = fmaf(g, __ldg(in + (int64_t)v2 * C + c), a2);
    }
    float* p = partial + (int64_t)blockIdx.x * 3 * Cr;
    p[co] = a0; p[Cr + co] = a1; p[2 * Cr + co] = a2;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
static bool vec_ok(int C, int r) { return r == 1 && C % 4 == 0; }

struct V2FBwdPlan { bool vec; int grid_x; int64_t faces_per_chunk; };
static V2FBwdPlan v2f_bwd_plan(int64_t Nf, int64_t Nv, int C, int r) {
    V2FBwdPlan p;
    p.vec = vec_ok(C, r);
    if (p.vec) {
        TeamGeom g = team_geom(C / 4);
        p.grid_x = persistent_blocks(Nv, g.teams, 8);
        p.faces_per_chunk = 0;
    } else {
        int64_t chunks = ceil_div(Nf, 64);
        int64_t cap = (int64_t)sm_count() * 8;
        if (chunks > cap) chunks = cap;
        if (chunks < 1) chunks = 1;
        p.faces_per_chunk = ceil_div(Nf > 0 ? Nf : 1, chunks);
        p.grid_x = (int)ceil_div(Nf > 0 ? Nf : 1, p.faces_per_chunk);
    }
    return p;
}

}  // namespace pb

using namespace pb;

extern "C" {

int pb200_vertex2facet_forward(int64_t Nf, int64_t Nv, int C, int r, const float* input, const float* filter,
                               const int32_t* face, float* output, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(Nf >= 0 && Nv >= 0 && C > 0 && r > 0, PB200_EINVAL, "vertex2facet_forward: bad sizes");
    if (Nf == 0) return PB200_OK;
    PB_REQUIRE(input && filter && face && output, PB200_EINVAL, "vertex2facet_forward: null pointer");
    const uint32_t vertices = index_range(Nv);
    if (vec_ok(C, r) && aligned16(input) && aligned16(filter) && aligned16(output)) {
        int CV = C / 4;
        TeamGeom g = team_geom(CV);
        dim3 grid(persistent_blocks(ceil_div(Nf, 2), g.teams, 4), g.chunks);
        PB_DISPATCH_TL(g.TL, PB_LAUNCH("v2f_fwd", v2f_fwd_vec_kernel<TL>, grid, 256, 0, stream, Nf, vertices, CV,
                                       face, (const float4*)input, (const float4*)filter, (float4*)output));
    } else {
        int grid = persistent_blocks(Nf * C * r, 256, 16);
        PB_LAUNCH("v2f_fwd_generic", v2f_fwd_generic_kernel, grid, 256, 0, stream, Nf, vertices, C, r, face, input, filter, output);
    }
    return PB200_OK;
}

size_t pb200_vertex2facet_backward_workspace_bytes(int64_t Nf, int64_t Nv, int C, int r) {
    if (Nf < 0 || Nv < 0 || C <= 0 || r <= 0) return 0;
    V2FBwdPlan p = v2f_bwd_plan(Nf, Nv, C, r);
    return align_up(sizeof(float) * (size_t)p.grid_x * 3 * C * r, 256);
}

int pb200_vertex2facet_backward(int64_t Nf, int64_t Nv, int C, int r, const float* gradOutput, const float* input,
                                const float* filter, const int32_t* face, const int32_t* rowptr,
                                const int32_t* entries, float* gradInput, float* gradFilter, void* workspace,
                                size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(Nf >= 0 && Nv >= 0 && C > 0 && r > 0, PB200_EINVAL, "vertex2facet_backward: bad sizes");
    PB_REQUIRE(gradFilter && (Nv == 0 || (gradInput && rowptr && input)), PB200_EINVAL,
               "vertex2facet_backward: null pointer");
    const int Cr = C * r;
    if (Nf == 0 || Nv == 0) {
        PB_CUDA(cudaMemsetAsync(gradFilter, 0, sizeof(float) * 3 * Cr, stream));
        if (Nv > 0) PB_CUDA(cudaMemsetAsync(gradInput, 0, sizeof(float) * Nv * C, stream));
        return PB200_OK;
    }
    PB_REQUIRE(gradOutput && filter && face && entries, PB200_EINVAL, "vertex2facet_backward: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_vertex2facet_backward_workspace_bytes(Nf, Nv, C, r),
               PB200_EWORKSPACE, "vertex2facet_backward: workspace too small");
    V2FBwdPlan p = v2f_bwd_plan(Nf, Nv, C, r);
    float* partial = (float*)workspace;
    bool vec = p.vec && aligned16(gradOutput) && aligned16(input) && aligned16(filter) && aligned16(gradInput);
    if (vec) {
        int CV = C / 4;
        TeamGeom g = team_geom(CV);
        int gx = V2F_BWD_BLOCKS * sm_count() / g.chunks;       // the blocks that run side by side
        if (gx < 1) gx = 1;
        if (gx > p.grid_x) gx = p.grid_x;
        dim3 grid(gx, g.chunks);
        PB_DISPATCH_TL(g.TL, PB_LAUNCH("v2f_bwd", v2f_bwd_vec_kernel<TL>, grid, 256, 0, stream, Nv, CV, rowptr,
                                       entries, (const float4*)gradOutput, (const float4*)input,
                                       (const float4*)filter, (float4*)gradInput, (float4*)partial));
        return reduce_partials(partial, gx, 3 * Cr, gradFilter, stream, FEW_PARTIALS);
    }
    // generic path (any C, r): plan for the non-vector layout even if only alignment failed
    V2FBwdPlan q = p;
    if (p.vec) {
        int64_t chunks = ceil_div(Nf, 64);
        int64_t cap = p.grid_x;            // the workspace was sized for p.grid_x partial rows
        if (chunks > cap) chunks = cap;
        q.faces_per_chunk = ceil_div(Nf, chunks);
        q.grid_x = (int)ceil_div(Nf, q.faces_per_chunk);
    }
    int gi = persistent_blocks(Nv * C, 256, 16);
    PB_LAUNCH("v2f_bwd_input_generic", v2f_bwd_input_generic_kernel, gi, 256, 0, stream, Nv, C, r, rowptr, entries,
              gradOutput, filter, gradInput);
    dim3 gridf(q.grid_x, (unsigned)ceil_div(Cr, 128));
    PB_LAUNCH("v2f_bwd_filter_generic", v2f_bwd_filter_generic_kernel, gridf, 128, 0, stream, Nf, index_range(Nv), C, r,
              q.faces_per_chunk, face, input, gradOutput, partial);
    return reduce_partials(partial, q.grid_x, 3 * Cr, gradFilter, stream);
}

}  // extern "C"

// ------------------------------------------------------------- allocation-free variant
// Some hosts of this library may not allocate device memory at the moment they call it:
// a plugin invoked inside a region the embedding framework has frozen (its allocator is
// locked or its pool already handed out), a real-time or signal-adjacent callback, or a
// process whose memory budget was fixed at start-up.  For them the filter-gradient
// partials of vertex2facet_backward live in a fixed array that is part of the loaded
// library image on every GPU (it costs PB200_STATIC_SCRATCH_BYTES of device memory per
// GPU from load until exit).
//
// In host code `g_v2f_bwd_static_scratch` is only a handle for the runtime; the device
// address must be asked for with cudaGetSymbolAddress, once per device, with that device
// current.
#define PB200_STATIC_SCRATCH_BYTES (4u << 20)
static __device__ __align__(256) unsigned char g_v2f_bwd_static_scratch[PB200_STATIC_SCRATCH_BYTES];

namespace pb {
static int static_scratch_for_current_device(void** out) {
    static void* cached[64] = {nullptr};
    static std::mutex mu;
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    PB_REQUIRE(dev >= 0 && dev < 64, PB200_EINVAL, "vertex2facet_backward_static: device ordinal %d not supported", dev);
    std::lock_guard<std::mutex> lk(mu);
    if (cached[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_v2f_bwd_static_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_v2f_bwd_static_scratch)");
        PB_REQUIRE(p != nullptr, PB200_ECUDA, "vertex2facet_backward_static: null scratch address");
        cached[dev] = p;
    }
    *out = cached[dev];
    return PB200_OK;
}
}  // namespace pb

extern "C" {

size_t pb200_vertex2facet_backward_static_max_bytes(void) { return PB200_STATIC_SCRATCH_BYTES; }

int pb200_vertex2facet_backward_static(int64_t Nf, int64_t Nv, int C, int r, const float* gradOutput,
                                       const float* input, const float* filter, const int32_t* face,
                                       const int32_t* rowptr, const int32_t* entries, float* gradInput,
                                       float* gradFilter, void* stream_) {
    PB_REQUIRE(Nf >= 0 && Nv >= 0 && C > 0 && r > 0, PB200_EINVAL, "vertex2facet_backward_static: bad sizes");
    size_t need = pb200_vertex2facet_backward_workspace_bytes(Nf, Nv, C, r);
    PB_REQUIRE(need <= PB200_STATIC_SCRATCH_BYTES, PB200_EWORKSPACE,
               "vertex2facet_backward_static: this shape needs %zu bytes of scratch, the built-in array holds %u; "
               "use pb200_vertex2facet_backward with a caller-provided workspace",
               need, (unsigned)PB200_STATIC_SCRATCH_BYTES);
    // argument checks before the first-call set-up, so that a bad call never triggers it
    PB_REQUIRE(gradFilter && (Nf == 0 || (gradOutput && input && filter && face && rowptr && entries && gradInput)),
               PB200_EINVAL, "vertex2facet_backward_static: null pointer");
    void* scratch = nullptr;
    int rc = static_scratch_for_current_device(&scratch);
    if (rc != PB200_OK) return rc;
    // Every partial the second stage reads is written by the first stage of the same call,
    // so nothing in the array has to start at zero.
    return pb200_vertex2facet_backward(Nf, Nv, C, r, gradOutput, input, filter, face, rowptr, entries, gradInput,
                                       gradFilter, scratch, PB200_STATIC_SCRATCH_BYTES, stream_);
}

}  // extern "C"
