// facet2vertex: forward as a vertex-centred pull over the CSR (segmented sum in a fixed
// order, no atomics); backward as a face-centred gather that yields the input gradient
// and per-thread filter-gradient partials in one pass.
#include <type_traits>
#include "common.cuh"
#include "row_walk.cuh"

namespace pb {

// -------------------------------------------------------------------- forward, vectorised
// r == 1, C % 4 == 0, K <= 64.  Two kernels:
//   f2v_fwd_face    item = (face, float4 channel group): wx[f] = (sum_k coeff[f,k]*filter[k]) * input[f],
//                   once per face (a vertex-centred pull would evaluate the K-term sum three
//                   times per face), filter and the tile's coeff rows in shared memory;
//   f2v_fwd_gather  team per output vertex: sum of the wx rows of its CSR entries in ascending
//                   order, times 1/nfCount.  No atomics: deterministic.
constexpr int F2VF_TF = 64;

__global__ void __launch_bounds__(256)
f2v_fwd_face_kernel(int64_t Nf, int CV, int K, const float* __restrict__ coeff, const float4* __restrict__ in,
                    const float4* __restrict__ filt, float4* __restrict__ wx) {
    extern __shared__ float4 smem[];
    const int KP = (K + 3) / 4 * 4 + 4;
    float4* sfilt = smem;                                          // [K][32]
    float* scoef = reinterpret_cast<float*>(smem + K * 32);       // [TF][KP]
    const int cg0 = blockIdx.y * 32;
    const int CVc = CV - cg0 < 32 ? CV - cg0 : 32;
    for (int i = threadIdx.x; i < K * 32; i += blockDim.x) {
        int k = i >> 5, l = i & 31;
        sfilt[i] = l < CVc ? filt[k * CV + cg0 + l] : zero4();
    }
    const int64_t ntiles = (Nf + F2VF_TF - 1) / F2VF_TF;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t f0 = tile * F2VF_TF;
        const int nf_tile = Nf - f0 < F2VF_TF ? (int)(Nf - f0) : F2VF_TF;
        __syncthreads();
        for (int i = threadIdx.x; i < nf_tile * K; i += blockDim.x) {
            int fl = i / K;
            scoef[fl * KP + (i - fl * K)] = __ldg(coeff + f0 * K + i);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nf_tile * CVc; i += blockDim.x) {
            const int fl = i / CVc, c = i - fl * CVc;
            const int64_t f = f0 + fl;
            const float4 x = ldg4(in + f * CV + cg0 + c);
            const float* cf = scoef + fl * KP;
            float4 w = zero4();
            int k = 0;
            for (; k + 4 <= K; k += 4) {
                const float4 c4 = *reinterpret_cast<const float4*>(cf + k);
                fma4s(w, c4.x, sfilt[k * 32 + c]);
                fma4s(w, c4.y, sfilt[(k + 1) * 32 + c]);
                fma4s(w, c4.z, sfilt[(k + 2) * 32 + c]);
                fma4s(w, c4.w, sfilt[(k + 3) * 32 + c]);
            }
            for (; k < K; ++k) fma4s(w, cf[k], sfilt[k * 32 + c]);
            wx[f * CV + cg0 + c] = mul4(w, x);
        }
    }
}

// The same register-blocked, for K <= 32: a face's channels lie on LPF lanes (float4 each; LPF = 4, 8, 16, 32, chunks of 128
// channels behind that), a warp has 32 / LPF faces side by side, and a filter row read from shared memory is used for all FB such
// passes of the warp.  The coefficient rows of the next tile arrive by 4-byte asynchronous copies while this one is
// computed.  (The kernel above took 389 us for 1 758 000 faces of 64 channels, K = 16, bound by its shared-memory reads; this one takes
// 183.  Measured and left: packed multiply-adds with the coefficients paired in registers, 202, or stored in pairs, 224.)
template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst_smem, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src), "n"(BYTES)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int LPF> constexpr int F2VF_PASSES = LPF >= 16 ? 8 : 4;
template <int LPF> constexpr int F2VF_FACES = 8 * F2VF_PASSES<LPF> * (32 / LPF);         // faces of a tile
// floats of a coefficient row; a pad keeps the rows of faces side by side in a warp off one another's banks
template <int LPF> __host__ __device__ constexpr int f2v_pitch(int K) { return (K + 3) / 4 * 4 + (LPF < 32 ? 4 : 0); }

template <int LPF>
__global__ void __launch_bounds__(256)
f2v_fwd_face_blocked_kernel(int64_t Nf, int CV, int K, const float* __restrict__ coeff, const float4* __restrict__ in,
                            const float4* __restrict__ filt, float4* __restrict__ wx) {
    extern __shared__ float4 smem[];
    constexpr int FB = F2VF_PASSES<LPF>, FPW = 32 / LPF, TF = F2VF_FACES<LPF>;
    const int KG = (K + 3) / 4, CP = f2v_pitch<LPF>(K);
    float4* sfilt = smem;                                      // [4 KG][LPF], rows K.. zero
    float* scoef0 = reinterpret_cast<float*>(smem + 4 * KG * LPF);     // [2][TF][CP], double-buffered, pad columns zero
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int l = lane % LPF, fs = lane / LPF;                 // channel group, face among the warp's
    const int cg = blockIdx.y * LPF + l;
    const bool on = cg < CV;
    for (int i = threadIdx.x; i < 4 * KG * LPF; i += blockDim.x) {
        const int k = i / LPF, c = blockIdx.y * LPF + i % LPF;
        sfilt[i] = k < K && c < CV ? filt[k * CV + c] : zero4();
    }
    for (int i = threadIdx.x; i < 2 * TF * CP; i += blockDim.x) scoef0[i] = 0.f;
    __syncthreads();
    const int64_t ntiles = (Nf + TF - 1) / TF;
    auto fetch_coef = [&](int64_t tile, int buf) {             // a lane per coefficient
        if (tile < ntiles && lane < K) {
            const int64_t f0 = tile * TF;
            const int nf_tile = Nf - f0 < TF ? (int)(Nf - f0) : TF;
            const float* src = coeff + f0 * K + lane;
            float* sc = scoef0 + buf * TF * CP + lane;
            for (int fl = warp; fl < nf_tile; fl += 8) cp_async<4>(sc + fl * CP, src + fl * K);
        }
        cp_async_commit();
    };
    fetch_coef(blockIdx.x, 0);
    int buf = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, buf ^= 1) {
        const int64_t f0 = tile * TF;
        const int nf_tile = Nf - f0 < TF ? (int)(Nf - f0) : TF;
        fetch_coef(tile + gridDim.x, buf ^ 1);                 // its readers finished behind the barrier below
        cp_async_wait<1>();                                    // this tile's rows have landed (own copies) ...
        __syncthreads();                                       // ... and everybody else's
        const float* scoef = scoef0 + buf * TF * CP + (warp * FPW + fs) * CP;
        float4 x[FB], w[FB];
#pragma unroll
        for (int i = 0; i < FB; ++i) {
            const int fl = (warp + 8 * i) * FPW + fs;
            w[i] = zero4();
            x[i] = on && fl < nf_tile ? ldg4(in + (f0 + fl) * CV + cg) : zero4();
        }
        for (int g = 0; g < KG; ++g) {
            const float4 fa = sfilt[4 * g * LPF + l], fb = sfilt[(4 * g + 1) * LPF + l];
            const float4 fc = sfilt[(4 * g + 2) * LPF + l], fd = sfilt[(4 * g + 3) * LPF + l];
#pragma unroll
            for (int i = 0; i < FB; ++i) {                     // rows past the tile are stale or zero: unused
                const float4 cf = *reinterpret_cast<const float4*>(scoef + 8 * i * FPW * CP + 4 * g);
                fma4s(w[i], cf.x, fa); fma4s(w[i], cf.y, fb); fma4s(w[i], cf.z, fc); fma4s(w[i], cf.w, fd);
            }
        }
#pragma unroll
        for (int i = 0; i < FB; ++i) {
            const int fl = (warp + 8 * i) * FPW + fs;
            if (on && fl < nf_tile) wx[(f0 + fl) * CV + cg] = mul4(w[i], x[i]);
        }
        __syncthreads();                                       // this tile's buffer may be refilled now
    }
    cp_async_wait<0>();
}

template <int TL>
__global__ void __launch_bounds__(256, 4)
f2v_fwd_gather_kernel(int64_t NvOut, int CV, const int32_t* __restrict__ rowptr, const int32_t* __restrict__ entries,
                      const int32_t* __restrict__ nfCount, const float4* __restrict__ wx, float4* __restrict__ out) {
    const int lane = threadIdx.x % TL;
    const int team = threadIdx.x / TL;
    const int teams = blockDim.x / TL;
    const int cg = blockIdx.y * 32 + lane;
    const bool active = cg < CV;
    // Rows in flight: six where a team is a warp (7.4 M faces, 128 channels: 1.49 ms; eight 1.57; one at a time 1.94), else eight (1.76
    // M faces, 64 channels: 166 us; six 184; one at a time 171).
    constexpr int B = TL == 32 ? 6 : 8;
    // inactive lanes stay in the loop: the team shares its CSR entries through shuffles
    RowWalk<TL, B> walk(rowptr, entries, (int64_t)blockIdx.x * teams + team, (int64_t)gridDim.x * teams, NvOut);
    for (; walk.v < NvOut; walk.step()) {
        const bool some = walk.end > walk.beg;
        const int count = some ? __ldg(nfCount + walk.v) : 1;
        F4x2 acc{0, 0};
        walk.rows([&](const int (&ent)[B]) {
            F4x2 g[B];
#pragma unroll
            for (int u = 0; u < B; ++u) g[u] = active && ent[u] >= 0 ? ldg4x2(wx + (int64_t)(ent[u] >> 2) * CV + cg) : F4x2{0, 0};
#pragma unroll
            for (int u = 0; u < B; ++u) add2(acc, g[u]);
        });
        if (active) {
            float4 o = unpair4(acc);
            if (some) o = scale4(o, 1.f / (float)count);
            __stcs(out + walk.v * CV + cg, o);
        }
    }
}

// ----------------------------------------------------------------------- forward, generic
__global__ void f2v_fwd_generic_kernel(int64_t NvOut, int C, int r, int K, const int32_t* __restrict__ rowptr,
                                       const int32_t* __restrict__ entries, const int32_t* __restrict__ nfCount,
                                       const float* __restrict__ coeff, const float* __restrict__ in,
                                       const float* __restrict__ filt, float* __restrict__ out) {
    const int Cr = C * r;
    int64_t total = NvOut * Cr;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t v = i / Cr;
        int co = (int)(i - v * Cr);
        int c = co / r;
        int beg = rowptr[v], end = rowptr[v + 1];
        float acc = 0.f;
        for (int e = beg; e < end; ++e) {
            int64_t f = entries[e] >> 2;
            float w = 0.f;
            for (int k = 0; k < K; ++k) w = fmaf(__ldg(coeff + f * K + k), __ldg(filt + k * Cr + co), w);
            acc = fmaf(w, __ldg(in + f * C + c), acc);
        }
        out[i] = end > beg ? acc / (float)nfCount[v] : 0.f;
    }
}

// What the backward kernels know of the index arrays: a corner whose vertex, or its output vertex, is outside its range has none and
// nothing is read for it, as in the adjacency.  (With deferred validation they run on indices that nobody has looked at yet.)
struct OutVertex {
    const int32_t* vtMap;                // null: the same vertex
    uint32_t NvIn, NvOut;
    __device__ __forceinline__ int mapped(int vi) const {      // not yet looked at: whoever waits for it does (one of the next hops)
        if ((uint32_t)vi >= NvIn) return -1;
        return vtMap ? __ldg(vtMap + vi) : vi;
    }
    __device__ __forceinline__ int within(int vo) const { return (uint32_t)vo < NvOut ? vo : -1; }
    __device__ __forceinline__ int operator()(int vi) const { return within(mapped(vi)); }
};


// ------------------------------------------------------------------- backward, vectorised
// r == 1, C % 4 == 0, any K <= 64.  A block walks tiles of 32 faces; per tile
//   phase 1  item = (face, float4 channel group): gt = sum over the three corners of
//            gradOutput[vo] * (1/nfCount[vo]);  w = sum_k coeff[f,k]*filter[k];
//            gradInput[f] = gt*w;  t[f] = input[f]*gt is parked in shared memory;
//   phase 2  item = (k, channel group), up to NACC per thread, kept in registers for the whole
//            kernel: gradFilter[k] += coeff[f,k] * t[f] over the tile's faces in face order.
// Phase 1 needs few registers (full occupancy hides the gather latency), phase 2 has no
// global traffic.  Per-block accumulators go to partial[block][K][C]; a second kernel adds
// the blocks in order, so the result is deterministic.
constexpr int F2VB_TF = 32;

template <int NACC>
__global__ void __launch_bounds__(256)
f2v_bwd_tile_kernel(int64_t Nf, int CV, int K, const int32_t* __restrict__ face, OutVertex out_vertex,
                    const int32_t* __restrict__ nfCount, const float* __restrict__ coeff,
                    const float4* __restrict__ in, const float4* __restrict__ filt, const float4* __restrict__ gout,
                    float4* __restrict__ gin, float4* __restrict__ partial) {
    extern __shared__ float4 smem[];
    const int KP = (K + 3) / 4 * 4 + 4;                       // coeff row pitch (floats): 16-byte rows, spread banks
    float4* sfilt = smem;                                      // [K][32]
    float4* st = smem + K * 32;                                // [TF][32]   t = input * gt
    float* scoef = reinterpret_cast<float*>(st + F2VB_TF * 32);    // [TF][KP]
    const int cg0 = blockIdx.y * 32;
    const int CVc = CV - cg0 < 32 ? CV - cg0 : 32;             // channel groups of this chunk
    for (int i = threadIdx.x; i < K * 32; i += blockDim.x) {
        int k = i >> 5, l = i & 31;
        sfilt[i] = l < CVc ? filt[k * CV + cg0 + l] : zero4();
    }
    // this thread's accumulator items (k, c): j = tid + 256 n
    float4 acc[NACC];
    int ak[NACC], ac[NACC];
#pragma unroll
    for (int n = 0; n < NACC; ++n) {
        int j = threadIdx.x + 256 * n;
        ak[n] = j / CVc; ac[n] = j - ak[n] * CVc;
        if (ak[n] >= K) { ak[n] = -1; ac[n] = 0; }
        acc[n] = zero4();
    }
    const int64_t ntiles = (Nf + F2VB_TF - 1) / F2VB_TF;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t f0 = tile * F2VB_TF;
        const int nf_tile = Nf - f0 < F2VB_TF ? (int)(Nf - f0) : F2VB_TF;
        __syncthreads();                                       // previous tile fully consumed
        for (int i = threadIdx.x; i < nf_tile * K; i += blockDim.x) {
            int fl = i / K;
            scoef[fl * KP + (i - fl * K)] = __ldg(coeff + f0 * K + i);
        }
        __syncthreads();
        // ---- phase 1
        for (int i = threadIdx.x; i < nf_tile * CVc; i += blockDim.x) {
            const int fl = i / CVc, c = i - fl * CVc;
            const int64_t f = f0 + fl;
            const int cg = cg0 + c;
            float4 gt = zero4();
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int vo = out_vertex(__ldg(face + 3 * f + j));
                if (vo >= 0) {
                    float rn = __frcp_rn((float)__ldg(nfCount + vo));
                    fma4s(gt, rn, ldg4(gout + (int64_t)vo * CV + cg));
                }
            }
            const float4 x = ldg4(in + f * CV + cg);
            const float* cf = scoef + fl * KP;
            float4 w = zero4();
            int k = 0;
            for (; k + 4 <= K; k += 4) {
                const float4 c4 = *reinterpret_cast<const float4*>(cf + k);
                fma4s(w, c4.x, sfilt[k * 32 + c]);
                fma4s(w, c4.y, sfilt[(k + 1) * 32 + c]);
                fma4s(w, c4.z, sfilt[(k + 2) * 32 + c]);
                fma4s(w, c4.w, sfilt[(k + 3) * 32 + c]);
            }
            for (; k < K; ++k) fma4s(w, cf[k], sfilt[k * 32 + c]);
            __stcs(gin + f * CV + cg, mul4(gt, w));
            st[fl * 32 + c] = mul4(x, gt);
        }
        __syncthreads();
        // ---- phase 2
#pragma unroll
        for (int n = 0; n < NACC; ++n) {
            if (ak[n] >= 0) {
                const float* cf = scoef + ak[n];
                const float4* tp = st + ac[n];
                float4 a = acc[n];
                for (int fl = 0; fl < nf_tile; ++fl) fma4s(a, cf[fl * KP], tp[fl * 32]);
                acc[n] = a;
            }
        }
    }
#pragma unroll
    for (int n = 0; n < NACC; ++n)
        if (ak[n] >= 0) partial[((int64_t)blockIdx.x * K + ak[n]) * CV + cg0 + ac[n]] = acc[n];
}

// K <= 32: a lane keeps NC channels for the whole kernel, with their K filter values and K filter-gradient sums in registers, and
// walks faces: the only operands of the 2 K multiply-adds of a face and channel that come out of shared memory are the K coefficients,
// read once for both sums and broadcast to the warp.  Coefficients, filter and sums go in pairs (k, k + 1), so that the products are
// packed (fma.rn.f32x2) without an operand kept twice.  A face's channels lie on LPF lanes (4, 8, 16, 32; chunks of one width
// behind that on blockIdx.y), a warp has FPW = 32 / LPF faces side by side and four such passes per stage.  Warps share nothing: each has a ring of
// stages of its own (three gradOutput rows, the input row and the coefficients of every face) that asynchronous copies fill, and
// resolves the index chain face -> vtMap -> nfCount one hop per stage ahead of them.
// What bounds it: instructions (126 per warp and face at 16 coefficients, 64 of them multiply-adds) with 8 to 12 warps per SM.  A kernel
// that read filter, coefficients and products from shared memory for every step (register blocks of 4 faces, three block barriers per
// tile) took, per call with a cold L2: 879 000 faces, 64 channels, K = 16 247 us (now 148, copy floor 98); 464 000 faces, 128 channels,
// K = 25 308 (248, floor 101); 879 000 faces, 48 channels, K = 9 226 (136), 32 channels, K = 25 200 (136), 16 channels, K = 16 118 (60).
template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst_smem, const void* src, bool on) {      // off: zeros
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src),
                 "n"(BYTES), "r"(on ? BYTES : 0) : "memory");
}
// Shape by the number of coefficient pairs P.  Registers decide: filter and sums take 4 P NC of them, so up to 16 coefficients a lane holds
// four channels, above that two (25 coefficients, 4 channels: 269 instead of 257 us, with nothing left to overlap loads).  Two stages:
// a third one, or longer ones, take from the L1 that serves the gradOutput rows which neighbouring faces share (16 coefficients: 148
// us with 2 x 4 passes, 171 with 3 x 4, 179 with 2 x 6).
template <int P> constexpr int F2VL_NC = P <= 8 ? 4 : 2;                              // channels of a lane
template <int P> constexpr int F2VL_BLOCKS = P <= 8 ? 2 : P <= 13 ? 3 : 2;            // blocks per SM
constexpr int F2VL_WARPS = 4, F2VL_PASSES = 4, F2VL_STAGES = 2;
template <int LPF> constexpr int F2VL_FACES = F2VL_PASSES * (32 / LPF);             // faces of a stage
// floats of a coefficient row: quads, and rows of faces side by side on different banks
template <int P> constexpr int F2VL_PITCH = (2 * P + 3) / 4 * 4 % 16 == 0 ? (2 * P + 3) / 4 * 4 + 4 : (2 * P + 3) / 4 * 4;
template <int NC> struct F2VLVec { using type = float2; };
template <> struct F2VLVec<4> { using type = float4; };
template <int P, int LPF> struct F2VLStage {
    typename F2VLVec<F2VL_NC<P>>::type row[F2VL_PASSES][4][32];                            // gradOutput of the corners 0..2, input; a lane's own channels
    alignas(16) float coef[F2VL_FACES<LPF> * F2VL_PITCH<P>];
    int4 vo[F2VL_FACES<LPF>];                                  // output vertices of the corners (-1: none) ...
    float4 rn[F2VL_FACES<LPF>];                                // ... and 1 / nfCount of them
};

template <int P, int LPF>
__global__ void __launch_bounds__(32 * F2VL_WARPS, F2VL_BLOCKS<P>)
f2v_bwd_lane_kernel(int64_t Nf, int C, int K, int width, const int32_t* __restrict__ face, OutVertex out_vertex,
                    const int32_t* __restrict__ nfCount, const float* __restrict__ coeff, const float* __restrict__ in,
                    const float* __restrict__ filt, const float* __restrict__ gout, float* __restrict__ gin,
                    float* __restrict__ partial) {
    extern __shared__ __align__(16) unsigned char f2vl_smem[];
    using Stage = F2VLStage<P, LPF>;
    constexpr int FPW = 32 / LPF, TF = F2VL_FACES<LPF>, NE = 3 * TF, NI = (NE + 31) / 32, CP = F2VL_PITCH<P>, D = F2VL_STAGES;
    constexpr int NC = F2VL_NC<P>;
    using Vec = typename F2VLVec<NC>::type;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int l = lane % LPF, fs = lane / LPF;                 // channel pair, face among the warp's
    const int c0 = blockIdx.y * width, here = C - c0 < width ? C - c0 : width;       // channels of this block
    const bool on = l * NC < here;
    // Lanes without channels follow on zeros of their own: they copy nothing and store nothing.  (When they copied channel 0 as well, one
    // address for several places of shared memory, the memory unit took the copies apart: 879 000 faces, 100 channels, 25 coefficients
    // 615 us, now 473; 136 channels, 16 coefficients, with an even share per chunk besides, 1 050 and 534.)
    const int ch = on ? c0 + l * NC : 0;
    Stage* ring = reinterpret_cast<Stage*>(f2vl_smem) + warp * D;

    uint64_t f2[NC][P], acc[NC][P];
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const float lo = 2 * p < K ? __ldg(filt + (2 * p) * C + ch + c) : 0.f;
            const float hi = 2 * p + 1 < K ? __ldg(filt + (2 * p + 1) * C + ch + c) : 0.f;
            f2[c][p] = pair2(lo, hi);
            acc[c][p] = 0;
        }
    for (int s = 0; s < D; ++s) {                              // columns K.. stay zero
        for (int i = lane; i < TF * CP; i += 32) ring[s].coef[i] = 0.f;
        if (!on)
            for (int i = 0; i < 4 * F2VL_PASSES; ++i) ring[s].row[i / 4][i % 4][lane] = Vec{};
    }
    __syncwarp();

    const int64_t ntiles = (Nf + TF - 1) / TF;
    const int tstep = gridDim.x * F2VL_WARPS;
    const int64_t tile0 = (int64_t)blockIdx.x * F2VL_WARPS + warp;
    const bool quads = K == 2 * P && P % 2 == 0 && (reinterpret_cast<uintptr_t>(coeff) & 15) == 0;
    const int row_bytes = C * 4;
    const char* const gout_lane = reinterpret_cast<const char*>(gout + ch);

    auto hop_face = [&](int64_t tile, int i) -> int {
        const int e = lane + 32 * i;
        const int64_t at = tile * NE + e;
        return (e < NE && at < Nf * 3) ? __ldg(face + at) : -1;
    };
    auto hop_vo = [&](int vi) -> int { return out_vertex(vi); };
    auto hop_n = [&](int vo) -> int { return vo < 0 ? 0 : __ldg(nfCount + vo); };
    auto park = [&](Stage& s, int i, int vo, int n) {
        const int e = lane + 32 * i;
        if (e < NE) {
            reinterpret_cast<int*>(s.vo)[e + e / 3] = vo;
            reinterpret_cast<float*>(s.rn)[e + e / 3] = vo < 0 ? 0.f : __frcp_rn((float)n);
        }
    };
    // The copies of a tile, whose corners are parked.  `whole`: all its faces and corners are there; otherwise zeros stand for
    // what is not.
    auto fetch = [&](Stage& s, int64_t tile, bool whole) {
        const int64_t f0 = tile * TF;
        if (whole && on) {
            const char* in_lane = reinterpret_cast<const char*>(in + (f0 + fs) * C + ch);
#pragma unroll
            for (int p = 0; p < F2VL_PASSES; ++p) {
                const int4 vo = s.vo[p * FPW + fs];
                cp_async<4 * NC>(&s.row[p][0][lane], gout_lane + (int64_t)vo.x * row_bytes);
                cp_async<4 * NC>(&s.row[p][1][lane], gout_lane + (int64_t)vo.y * row_bytes);
                cp_async<4 * NC>(&s.row[p][2][lane], gout_lane + (int64_t)vo.z * row_bytes);
                cp_async<4 * NC>(&s.row[p][3][lane], in_lane);
                in_lane += FPW * row_bytes;
            }
        } else if (tile < ntiles && on) {
#pragma unroll 1
            for (int p = 0; p < F2VL_PASSES; ++p) {
                const int fl = p * FPW + fs;
                const int* vo = reinterpret_cast<const int*>(s.vo + fl);
#pragma unroll 1
                for (int j = 0; j < 3; ++j)
                    cp_async<4 * NC>(&s.row[p][j][lane], vo[j] >= 0 ? gout_lane + (int64_t)vo[j] * row_bytes : gout_lane, vo[j] >= 0);
                const bool there = f0 + fl < Nf;
                cp_async<4 * NC>(&s.row[p][3][lane], there ? in + (f0 + fl) * C + ch : in, there);
            }
        }
        if (tile < ntiles) {
            const int nf_tile = Nf - f0 < TF ? (int)(Nf - f0) : TF;
            if (quads) {
                constexpr int Q = P / 2 > 0 ? P / 2 : 1;       // quads of a row
#pragma unroll
                for (int i0 = 0; i0 < TF * Q; i0 += 32) {
                    const int i = i0 + lane, fl = i / Q, q = i % Q;
                    const bool there = i < nf_tile * Q;
                    if (i < TF * Q) cp_async<16>(s.coef + fl * CP + 4 * q, coeff + (there ? f0 * K + 4 * i : 0), there);
                }
            } else if (lane < K) {
                const float* src = coeff + f0 * K + lane;
                if (whole) {
#pragma unroll
                    for (int fl = 0; fl < TF; ++fl, src += K) cp_async<4>(s.coef + fl * CP + lane, src);
                } else
#pragma unroll 1
                    for (int fl = 0; fl < TF; ++fl, src += K) cp_async<4>(s.coef + fl * CP + lane, fl < nf_tile ? src : coeff, fl < nf_tile);
            }
        }
        cp_async_commit();
    };
    auto all_there = [&](int64_t tile, const int (&vo)[NI]) {
        bool mine = true;
#pragma unroll
        for (int i = 0; i < NI; ++i) mine = mine && (vo[i] >= 0 || lane + 32 * i >= NE);
        return __all_sync(0xffffffffu, mine) && (tile + 1) * TF <= Nf;
    };

    // prologue: the first D - 1 tiles resolved up front, then the chain of the three behind them
    int vo0[NI], n0[NI], vo1[NI], vi2[NI];
    bool whole[D];
#pragma unroll
    for (int s = 0; s < D - 1; ++s) {
        int vo[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            vo[i] = hop_vo(hop_face(tile0 + s * tstep, i));
            park(ring[s], i, vo[i], hop_n(vo[i]));
        }
        whole[s] = all_there(tile0 + s * tstep, vo);
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        vo0[i] = hop_vo(hop_face(tile0 + (D - 1) * tstep, i));
        n0[i] = hop_n(vo0[i]);
        vo1[i] = hop_vo(hop_face(tile0 + D * tstep, i));
        vi2[i] = hop_face(tile0 + (D + 1) * tstep, i);
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < D - 1; ++s) fetch(ring[s], tile0 + s * tstep, whole[s]);

    int now = 0, next = D - 1;                                 // stages: of this tile, of tile + (D - 1) tstep
    for (int64_t tile = tile0; tile < ntiles; tile += tstep) {
        int n_next[NI], vo_next[NI], vi_next[NI];
        const bool next_whole = all_there(tile + (D - 1) * tstep, vo0);
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            park(ring[next], i, vo0[i], n0[i]);
            vo1[i] = out_vertex.within(vo1[i]);
            n_next[i] = hop_n(vo1[i]);
            vo_next[i] = out_vertex.mapped(vi2[i]);
            vi_next[i] = hop_face(tile + (D + 2) * tstep, i);
        }
        cp_async_wait<D - 2>();                                // this tile's copies have landed (own ones) ...
        __syncwarp();                                          // ... and the other lanes'; the next corners are parked
        fetch(ring[next], tile + (D - 1) * tstep, next_whole);
        const Stage& s = ring[now];
        const int64_t f0 = tile * TF;
        const int left = on ? (int)(Nf - f0 < TF ? Nf - f0 : TF) - fs : 0;          // this lane stores while p FPW < left
        char* gin_lane = reinterpret_cast<char*>(gin + (f0 + fs) * C + ch);
#pragma unroll
        for (int p = 0; p < F2VL_PASSES; ++p) {
            const float4 rn = s.rn[p * FPW + fs];
            const Vec g0 = s.row[p][0][lane], g1 = s.row[p][1][lane], g2 = s.row[p][2][lane], x = s.row[p][3][lane];
            float gt[NC];
            uint64_t t[NC], w[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                auto at = [&](const Vec& v) { return reinterpret_cast<const float*>(&v)[c]; };
                gt[c] = fmaf(rn.z, at(g2), fmaf(rn.y, at(g1), rn.x * at(g0)));
                const float tc = at(x) * gt[c];
                t[c] = pair2(tc, tc);
            }
            const float* cf = s.coef + (p * FPW + fs) * CP;
#pragma unroll
            for (int q = 0; q < P; q += 2) {
                const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(cf + 2 * q);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (q == 0) w[c] = mul2(k.x, f2[c][0]);
                    else fma2(w[c], k.x, f2[c][q]);
                    fma2(acc[c][q], k.x, t[c]);
                    if (q + 1 < P) {
                        fma2(w[c], k.y, f2[c][q + 1]);
                        fma2(acc[c][q + 1], k.y, t[c]);
                    }
                }
            }
            Vec g;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float2 a = unpair2(w[c]);
                reinterpret_cast<float*>(&g)[c] = gt[c] * (a.x + a.y);
            }
            if (p * FPW < left) __stcs(reinterpret_cast<Vec*>(gin_lane), g);
            gin_lane += FPW * row_bytes;
        }
        __syncwarp();                                          // this stage may be filled again
        now = now + 1 == D ? 0 : now + 1;
        next = next + 1 == D ? 0 : next + 1;
#pragma unroll
        for (int i = 0; i < NI; ++i) { vo0[i] = vo1[i]; n0[i] = n_next[i]; vo1[i] = vo_next[i]; vi2[i] = vi_next[i]; }
    }
    cp_async_wait<0>();
    __syncthreads();                                           // the sums of the faces side by side, then of the warps, in order
    Vec* sums = reinterpret_cast<Vec*>(f2vl_smem);             // [warp][2 P][32]: a warp's ring is longer
    static_assert(sizeof(Stage) * D >= sizeof(Vec) * 2 * P * 32, "the sums reuse the ring");
#pragma unroll
    for (int p = 0; p < P; ++p) {
        Vec a, b;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const float2 v = unpair2(acc[c][p]);
            reinterpret_cast<float*>(&a)[c] = v.x;
            reinterpret_cast<float*>(&b)[c] = v.y;
        }
        sums[(warp * 2 * P + 2 * p) * 32 + lane] = a;
        sums[(warp * 2 * P + 2 * p + 1) * 32 + lane] = b;
    }
    __syncthreads();
    const float* flat = reinterpret_cast<const float*>(sums);
    for (int i = threadIdx.x; i < K * LPF * NC; i += blockDim.x) {
        const int k = i / (LPF * NC), c = i % (LPF * NC);
        float t = 0.f;
        for (int v = 0; v < F2VL_WARPS; ++v)
#pragma unroll
            for (int q = 0; q < FPW; ++q) t += flat[((v * 2 * P + k) * 32 + q * LPF) * NC + c];
        if (c < here) partial[((int64_t)blockIdx.x * K + k) * C + c0 + c] = t;
    }
}

// ---------------------------------------------------------------------- backward, generic
__device__ __forceinline__ float f2v_gt(const int32_t* __restrict__ face, const OutVertex& out_vertex,
                                        const int32_t* __restrict__ nfCount, const float* __restrict__ gout,
                                        int64_t f, int Cr, int co) {
    float gt = 0.f;
    for (int j = 0; j < 3; ++j) {
        const int vo = out_vertex(face[3 * f + j]);
        if (vo >= 0) gt += __ldg(gout + (int64_t)vo * Cr + co) / (float)nfCount[vo];
    }
    return gt;
}

__global__ void f2v_bwd_input_generic_kernel(int64_t Nf, int C, int r, int K, const int32_t* __restrict__ face,
                                             OutVertex out_vertex, const int32_t* __restrict__ nfCount,
                                             const float* __restrict__ coeff, const float* __restrict__ filt,
                                             const float* __restrict__ gout, float* __restrict__ gin) {
    const int Cr = C * r;
    int64_t total = Nf * C;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t f = i / C;
        int c = (int)(i - f * C);
        float acc = 0.f;
        for (int m = 0; m < r; ++m) {
            int co = c * r + m;
            float w = 0.f;
            for (int k = 0; k < K; ++k) w = fmaf(__ldg(coeff + f * K + k), __ldg(filt + k * Cr + co), w);
            acc = fmaf(f2v_gt(face, out_vertex, nfCount, gout, f, Cr, co), w, acc);
        }
        gin[i] = acc;
    }
}

// thread = output channel co, blockIdx.x = chunk of faces (walked in order), blockIdx.z = k
__global__ void f2v_bwd_filter_generic_kernel(int64_t Nf, int C, int r, int K, int64_t faces_per_chunk,
                                              const int32_t* __restrict__ face, OutVertex out_vertex,
                                              const int32_t* __restrict__ nfCount, const float* __restrict__ coeff,
                                              const float* __restrict__ in, const float* __restrict__ gout,
                                              float* __restrict__ partial) {
    const int Cr = C * r;
    int co = blockIdx.y * blockDim.x + threadIdx.x;
    int k = blockIdx.z;
    if (co >= Cr) return;
    int c = co / r;
    int64_t f0 = (int64_t)blockIdx.x * faces_per_chunk;
    int64_t f1 = f0 + faces_per_chunk < Nf ? f0 + faces_per_chunk : Nf;
    float acc = 0.f;
    for (int64_t f = f0; f < f1; ++f) {
        float gt = f2v_gt(face, out_vertex, nfCount, gout, f, Cr, co);
        acc = fmaf(__ldg(coeff + f * K + k) * __ldg(in + f * C + c), gt, acc);
    }
    partial[((int64_t)blockIdx.x * K + k) * Cr + co] = acc;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
static bool vec_ok(int C, int r) { return r == 1 && C % 4 == 0; }
static bool kt_ok(int K) { return K >= 1 && K <= 64; }

struct F2VBwdPlan { bool vec; int grid_x; int64_t faces_per_chunk; };
static F2VBwdPlan f2v_bwd_plan(int64_t Nf, int C, int r, int K) {
    F2VBwdPlan p;
    p.vec = vec_ok(C, r) && kt_ok(K);
    int64_t n = Nf > 0 ? Nf : 1;
    if (p.vec) {
        p.grid_x = persistent_blocks(n, F2VB_TF, 4);
        p.faces_per_chunk = 0;
    } else {
        int64_t chunks = ceil_div(n, 64);
        int64_t cap = (int64_t)sm_count() * 4;
        if (chunks > cap) chunks = cap;
        p.faces_per_chunk = ceil_div(n, chunks);
        p.grid_x = (int)ceil_div(n, p.faces_per_chunk);
    }
    return p;
}

// The per-face stage of the vectorised forward pass on its own: wx[f, :] = (coeff[f] @ filter) * input[f]
// (r = 1, C % 4 == 0); used by pb200_facet2vertex_forward and by the fused facet2vertex + pointwise entry.
bool f2v_face_products_supported(int C, int K) { return vec_ok(C, 1) && kt_ok(K); }

int f2v_face_products(int64_t Nf, int C, int K, const float* input, const float* filter, const float* coeff, float* wx_,
                      cudaStream_t stream) {
    const int CV = C / 4;
    float4* wx = (float4*)wx_;
    if (Nf <= 0) return PB200_OK;
    if (K <= 32) {
        auto run = [&](auto lpf) {
            constexpr int LPF = decltype(lpf)::value, TF = F2VF_FACES<LPF>;
            const size_t smemb = sizeof(float4) * (size_t)((K + 3) / 4 * 4) * LPF + sizeof(float) * 2 * TF * f2v_pitch<LPF>(K);
            PB_CUDA(cudaFuncSetAttribute(f2v_fwd_face_blocked_kernel<LPF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemb));
            PB_LAUNCH("f2v_fwd_face", f2v_fwd_face_blocked_kernel<LPF>, dim3(persistent_blocks(Nf, TF, 4), (unsigned)ceil_div(CV, LPF)),
                      256, smemb, stream, Nf, CV, K, coeff, (const float4*)input, (const float4*)filter, wx);
            return PB200_OK;
        };
        if (CV <= 4) return run(std::integral_constant<int, 4>{});
        if (CV <= 8) return run(std::integral_constant<int, 8>{});
        if (CV <= 16) return run(std::integral_constant<int, 16>{});
        return run(std::integral_constant<int, 32>{});
    } else {
        const int KP = (K + 3) / 4 * 4 + 4;
        size_t smem = sizeof(float4) * 32 * (size_t)K + sizeof(float) * F2VF_TF * KP;
        dim3 gridf(persistent_blocks(Nf, F2VF_TF, 6), (unsigned)ceil_div(CV, 32));
        if (smem > 48 * 1024)
            PB_CUDA(cudaFuncSetAttribute(f2v_fwd_face_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        PB_LAUNCH("f2v_fwd_face", f2v_fwd_face_kernel, gridf, 256, smem, stream, Nf, CV, K, coeff,
                  (const float4*)input, (const float4*)filter, wx);
    }
    return PB200_OK;
}

// The vertex stage on its own: sums of the faces' products, over nfCount (C % 4 == 0, 16-byte aligned rows).
int f2v_gather(int64_t NvOut, int C, const int32_t* rowptr, const int32_t* entries, const int32_t* nfCount, const float* wx, float* output,
               cudaStream_t stream) {
    const TeamGeom g = team_geom(C / 4);
    const dim3 grid(persistent_blocks(NvOut, g.teams, 4), g.chunks);
    PB_DISPATCH_TL(g.TL, PB_LAUNCH("f2v_fwd_gather", f2v_fwd_gather_kernel<TL>, grid, 256, 0, stream, NvOut, C / 4, rowptr, entries, nfCount,
                                   (const float4*)wx, (float4*)output));
    return PB200_OK;
}

}  // namespace pb

using namespace pb;

extern "C" {

size_t pb200_facet2vertex_forward_workspace_bytes(int64_t Nf, int C, int r, int K) {
    if (Nf < 0 || C <= 0 || r <= 0 || K <= 0) return 0;
    if (vec_ok(C, r) && kt_ok(K)) return align_up(sizeof(float) * (size_t)(Nf > 0 ? Nf : 1) * C, 256);
    return 0;
}

int pb200_facet2vertex_forward(int64_t Nf, int64_t NvOut, int C, int r, int K, const float* input,
                               const float* filter, const float* coeff, const int32_t* nfCount,
                               const int32_t* rowptr, const int32_t* entries, float* output,
                               void* workspace, size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(Nf >= 0 && NvOut >= 0 && C > 0 && r > 0 && K > 0, PB200_EINVAL, "facet2vertex_forward: bad sizes");
    if (NvOut == 0) return PB200_OK;
    PB_REQUIRE(output && rowptr && nfCount, PB200_EINVAL, "facet2vertex_forward: null pointer");
    PB_REQUIRE(Nf == 0 || (input && filter && coeff && entries), PB200_EINVAL, "facet2vertex_forward: null pointer");
    const bool vec = vec_ok(C, r) && kt_ok(K) && aligned16(input) && aligned16(filter) && aligned16(output) &&
                     workspace && aligned16(workspace) &&
                     workspace_bytes >= pb200_facet2vertex_forward_workspace_bytes(Nf, C, r, K);
    if (vec_ok(C, r) && kt_ok(K) && aligned16(input) && aligned16(filter) && aligned16(output))
        PB_REQUIRE(vec, PB200_EWORKSPACE, "facet2vertex_forward: workspace missing, misaligned or too small");
    if (vec) {
        float* wx = (float*)workspace;
        int rc = f2v_face_products(Nf, C, K, input, filter, coeff, wx, stream);
        if (rc) return rc;
        return f2v_gather(NvOut, C, rowptr, entries, nfCount, wx, output, stream);
    } else {
        int grid = persistent_blocks(NvOut * C * r, 256, 16);
        PB_LAUNCH("f2v_fwd_generic", f2v_fwd_generic_kernel, grid, 256, 0, stream, NvOut, C, r, K, rowptr, entries,
                  nfCount, coeff, input, filter, output);
    }
    return PB200_OK;
}

size_t pb200_facet2vertex_backward_workspace_bytes(int64_t Nf, int C, int r, int K) {
    if (Nf < 0 || C <= 0 || r <= 0 || K <= 0) return 0;
    F2VBwdPlan p = f2v_bwd_plan(Nf, C, r, K);
    return align_up(sizeof(float) * (size_t)p.grid_x * K * C * r, 256);
}

int pb200_facet2vertex_backward(int64_t Nf, int64_t NvIn, int64_t NvOut, int C, int r, int K,
                                const float* gradOutput, const float* input, const float* filter,
                                const float* coeff, const int32_t* face, const int32_t* nfCount,
                                const int32_t* vtMap, float* gradInput, float* gradFilter, void* workspace,
                                size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(Nf >= 0 && NvIn >= 0 && NvOut >= 0 && C > 0 && r > 0 && K > 0, PB200_EINVAL,
               "facet2vertex_backward: bad sizes");
    PB_REQUIRE(gradFilter, PB200_EINVAL, "facet2vertex_backward: null pointer");
    const int Cr = C * r;
    if (Nf == 0) {
        PB_CUDA(cudaMemsetAsync(gradFilter, 0, sizeof(float) * K * Cr, stream));
        return PB200_OK;
    }
    PB_REQUIRE(gradOutput && input && filter && coeff && face && nfCount && gradInput, PB200_EINVAL,
               "facet2vertex_backward: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_facet2vertex_backward_workspace_bytes(Nf, C, r, K),
               PB200_EWORKSPACE, "facet2vertex_backward: workspace too small");
    const OutVertex out_vertex{vtMap, index_range(vtMap ? NvIn : NvOut), index_range(NvOut)};
    F2VBwdPlan p = f2v_bwd_plan(Nf, C, r, K);
    float* partial = (float*)workspace;
    bool vec = p.vec && aligned16(gradOutput) && aligned16(input) && aligned16(filter) && aligned16(gradInput);
    if (vec) {
        int CV = C / 4;
        if (K <= 32) {
            auto run = [&](auto pairs, auto lpf) {
                constexpr int P = decltype(pairs)::value, LPF = decltype(lpf)::value;
                const int chunks = (int)ceil_div(C, F2VL_NC<P> * LPF), width = (int)ceil_div(C, F2VL_NC<P> * chunks) * F2VL_NC<P>;
                const size_t smemb = sizeof(F2VLStage<P, LPF>) * F2VL_STAGES * F2VL_WARPS;
                const int fit = (int)(228 * 1024 / (smemb + 1024));                // blocks that an SM's shared memory holds
                int64_t gx = (int64_t)(fit < F2VL_BLOCKS<P> ? fit : F2VL_BLOCKS<P>) * sm_count() / chunks;
                if (gx < 1) gx = 1;
                if (gx > ceil_div(Nf, F2VL_WARPS * F2VL_FACES<LPF>)) gx = ceil_div(Nf, F2VL_WARPS * F2VL_FACES<LPF>);
                if (gx > p.grid_x) gx = p.grid_x;
                PB_CUDA(cudaFuncSetAttribute(f2v_bwd_lane_kernel<P, LPF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemb));
                PB_LAUNCH("f2v_bwd", (f2v_bwd_lane_kernel<P, LPF>), dim3((unsigned)gx, chunks), 32 * F2VL_WARPS, smemb, stream, Nf, C, K, width,
                          face, out_vertex, nfCount, coeff, input, filter, gradOutput, gradInput, partial);
                return reduce_partials(partial, (int)gx, (int64_t)K * Cr, gradFilter, stream, FEW_PARTIALS);
            };
            auto width = [&](auto pairs) {
                constexpr int NC = F2VL_NC<decltype(pairs)::value>;
                if (C <= 4 * NC) return run(pairs, std::integral_constant<int, 4>{});
                if (C <= 8 * NC) return run(pairs, std::integral_constant<int, 8>{});
                if (C <= 16 * NC) return run(pairs, std::integral_constant<int, 16>{});
                return run(pairs, std::integral_constant<int, 32>{});
            };
            if (K <= 4) return width(std::integral_constant<int, 2>{});
            if (K <= 10) return width(std::integral_constant<int, 5>{});
            if (K <= 16) return width(std::integral_constant<int, 8>{});
            if (K <= 26) return width(std::integral_constant<int, 13>{});
            return width(std::integral_constant<int, 16>{});
        }
        dim3 grid(p.grid_x, (unsigned)ceil_div(CV, 32));
        const int KP = (K + 3) / 4 * 4 + 4;
        size_t smem = sizeof(float4) * (32 * (size_t)K + F2VB_TF * 32) + sizeof(float) * F2VB_TF * KP;
        const int cvc = CV < 32 ? CV : 32;
        const int nacc = (int)ceil_div((int64_t)K * cvc, 256);
#define PB_F2VB_LAUNCH(N)                                                                                        \
        PB_LAUNCH("f2v_bwd", f2v_bwd_tile_kernel<N>, grid, 256, smem, stream, Nf, CV, K, face, out_vertex, nfCount,   \
                  coeff, (const float4*)input, (const float4*)filter, (const float4*)gradOutput,                \
                  (float4*)gradInput, (float4*)partial)
        if (smem > 48 * 1024) {
            PB_CUDA(cudaFuncSetAttribute(f2v_bwd_tile_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            PB_F2VB_LAUNCH(8);
        } else if (nacc <= 1) { PB_F2VB_LAUNCH(1); }
        else if (nacc <= 2) { PB_F2VB_LAUNCH(2); }
        else if (nacc <= 4) { PB_F2VB_LAUNCH(4); }
        else { PB_F2VB_LAUNCH(8); }
#undef PB_F2VB_LAUNCH
        return reduce_partials(partial, p.grid_x, (int64_t)K * Cr, gradFilter, stream);
    }
    F2VBwdPlan q = p;
    if (p.vec) {      // alignment fell through: reuse the workspace rows that were sized for p
        int64_t chunks = ceil_div(Nf, 64);
        if (chunks > p.grid_x) chunks = p.grid_x;
        q.faces_per_chunk = ceil_div(Nf, chunks);
        q.grid_x = (int)ceil_div(Nf, q.faces_per_chunk);
    }
    int gi = persistent_blocks(Nf * C, 256, 16);
    PB_LAUNCH("f2v_bwd_input_generic", f2v_bwd_input_generic_kernel, gi, 256, 0, stream, Nf, C, r, K, face, out_vertex,
              nfCount, coeff, filter, gradOutput, gradInput);
    PB_REQUIRE(K <= 65535, PB200_EINVAL, "facet2vertex_backward: K too large");
    dim3 gridf(q.grid_x, (unsigned)ceil_div(Cr, 128), K);
    PB_LAUNCH("f2v_bwd_filter_generic", f2v_bwd_filter_generic_kernel, gridf, 128, 0, stream, Nf, C, r, K,
              q.faces_per_chunk, face, out_vertex, nfCount, coeff, input, gradOutput, partial);
    return reduce_partials(partial, q.grid_x, (int64_t)K * Cr, gradFilter, stream);
}

}  // extern "C"
