// facet2vertex: forward as a vertex-centred pull over the CSR (segmented sum in a fixed
// order, no atomics); backward as a face-centred gather that yields the input gradient
// and per-thread filter-gradient partials in one pass.
#include <type_traits>
#include "common.cuh"

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
// computed.  (The kernel above took 389 us for 1 758 000 faces of 64 channels, K = 16, bound by its shared-memory reads.)
__device__ __forceinline__ void cp_async4(void* dst_smem, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src)
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
            for (int fl = warp; fl < nf_tile; fl += 8) cp_async4(sc + fl * CP, src + fl * K);
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
__global__ void __launch_bounds__(256)
f2v_fwd_gather_kernel(int64_t NvOut, int CV, const int32_t* __restrict__ rowptr, const int32_t* __restrict__ entries,
                      const int32_t* __restrict__ nfCount, const float4* __restrict__ wx, float4* __restrict__ out) {
    const int lane = threadIdx.x % TL;
    const int team = threadIdx.x / TL;
    const int teams = blockDim.x / TL;
    const int cg = blockIdx.y * 32 + lane;
    const bool active = cg < CV;
    // inactive lanes stay in the loop: the team shares its CSR entries through shuffles
    const unsigned tmask = TL == 32 ? 0xffffffffu : (((1u << TL) - 1u) << ((threadIdx.x & 31) / TL * TL));
    for (int64_t v = (int64_t)blockIdx.x * teams + team; v < NvOut; v += (int64_t)gridDim.x * teams) {
        const int beg = __ldg(rowptr + v), end = __ldg(rowptr + v + 1);
        float4 acc = zero4();
        for (int base = beg; base < end; base += TL) {
            const int mine = base + lane < end ? __ldg(entries + base + lane) : 0;
            const int cnt = end - base < TL ? end - base : TL;
            for (int i = 0; i < cnt; ++i) {
                const int64_t f = __shfl_sync(tmask, mine, i, TL) >> 2;
                if (active) add4(acc, ldg4(wx + f * CV + cg));
            }
        }
        if (active) {
            if (end > beg) acc = scale4(acc, 1.f / (float)__ldg(nfCount + v));
            __stcs(out + v * CV + cg, acc);
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
f2v_bwd_tile_kernel(int64_t Nf, int CV, int K, const int32_t* __restrict__ face, const int32_t* __restrict__ vtMap,
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
                int vi = __ldg(face + 3 * f + j);
                int vo = vtMap ? __ldg(vtMap + vi) : vi;
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

// The same two phases register-blocked, for K <= 32: a face's channels lie on LPF lanes (float4 each; LPF = 4, 8, 16, 32, chunks of
// 32 behind that), a warp has 32 / LPF faces side by side and four such passes per tile.
//   phase 1  a filter row read from shared memory is used for the four passes' faces;
//   phase 2  a warp owns four coefficients and, while K leaves warps over, a share of the tile's faces: a row of t read from shared
//            memory feeds four accumulators.
// What bounds it: shared memory (70 % busy at 128 channels) and the three barriers of a tile; packed multiply-adds on coefficients
// kept twice changed nothing.  A kernel without register blocking served all widths that are no multiple of 128 before:
// 1 954 000 faces, 64 channels, K = 16 960 -> 606 us; 977 000 faces, 48 channels, K = 9 408 -> 286 us, 100 channels 817 -> 561.
// The index chain of the gather (face -> vtMap -> nfCount) is resolved one hop per tile for the block's next three tiles, so that
// phase 1 finds output vertex and 1/nfCount of every corner in shared memory and issues its twelve gradOutput row loads at once.
template <int LPF> constexpr int F2VB_FACES = 32 * (32 / LPF);         // faces of a tile
template <int LPF>
static size_t f2vb_smem(int K) {
    return sizeof(float4) * ((size_t)(K + 3) / 4 * 4 * LPF + F2VB_FACES<LPF> * LPF) + sizeof(float) * 2 * F2VB_FACES<LPF> * f2v_pitch<LPF>(K) +
           2 * F2VB_FACES<LPF> * 3 * 8;
}

template <int LPF>
__global__ void __launch_bounds__(256, 2)
f2v_bwd_blocked_kernel(int64_t Nf, int CV, int K, const int32_t* __restrict__ face, const int32_t* __restrict__ vtMap,
                       const int32_t* __restrict__ nfCount, const float* __restrict__ coeff,
                       const float4* __restrict__ in, const float4* __restrict__ filt, const float4* __restrict__ gout,
                       float4* __restrict__ gin, float4* __restrict__ partial) {
    extern __shared__ float4 smem[];
    constexpr int FPW = 32 / LPF, TF = F2VB_FACES<LPF>, NE = TF * 3, NI = (NE + 255) / 256;
    const int KG = (K + 3) / 4, CP = f2v_pitch<LPF>(K);            // groups of 4 coefficients (<= 8)
    float4* sfilt = smem;                                      // [4 KG][LPF], rows K.. zero
    float4* st = smem + 4 * KG * LPF;                          // [TF][LPF]   t = input * gt
    float* scoef0 = reinterpret_cast<float*>(st + TF * LPF);   // [2][TF][CP], double-buffered (asynchronous copies)
    int* svo = reinterpret_cast<int*>(scoef0 + 2 * TF * CP);   // [2][NE] output vertex of (face, corner), -1 = none
    float* srn = reinterpret_cast<float*>(svo + 2 * NE);       // [2][NE] 1 / nfCount of that vertex
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int l = lane % LPF, fs = lane / LPF;                 // channel group, face among the warp's
    const int cg = blockIdx.y * LPF + l;
    const bool on = cg < CV;
    for (int i = threadIdx.x; i < 4 * KG * LPF; i += blockDim.x) {
        const int k = i / LPF, c = blockIdx.y * LPF + i % LPF;
        sfilt[i] = k < K && c < CV ? filt[k * CV + c] : zero4();
    }
    for (int i = threadIdx.x; i < 2 * TF * CP; i += blockDim.x) scoef0[i] = 0.f;
    // phase 2: coefficients 4g..4g+3, faces fs + FPW * (slice + slices * i)
    const int slices = 8 / KG, g2 = warp % KG, slice = warp / KG;
    float4 acc[4] = {zero4(), zero4(), zero4(), zero4()};
    const int64_t ntiles = (Nf + TF - 1) / TF;
    // index pipeline (entry e = 3*face + corner of a tile): vertex id of the tile three steps ahead, output vertex two steps
    // ahead, 1/nfCount one step ahead
    auto hop_face = [&](int64_t tile, int i) -> int {
        const int e = threadIdx.x + 256 * i;
        const int64_t at = tile * NE + e;
        return (e < NE && tile < ntiles && at < Nf * 3) ? __ldg(face + at) : -1;
    };
    auto hop_vo = [&](int vi) -> int { return vi < 0 ? -1 : (vtMap ? __ldg(vtMap + vi) : vi); };
    auto hop_rn = [&](int vo) -> float { return vo < 0 ? 0.f : __frcp_rn((float)__ldg(nfCount + vo)); };
    auto park = [&](int b, int i, int vo, float rn) {
        const int e = threadIdx.x + 256 * i;
        if (e < NE) { svo[b * NE + e] = vo; srn[b * NE + e] = rn; }
    };
    const int64_t tstep = gridDim.x;
    int vo1[NI], vi2[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int vo = hop_vo(hop_face(blockIdx.x, i));        // first tile: resolved up front
        park(0, i, vo, hop_rn(vo));
        vo1[i] = hop_vo(hop_face(blockIdx.x + tstep, i));      // second tile
        vi2[i] = hop_face(blockIdx.x + 2 * tstep, i);          // third tile
    }
    auto fetch_coef = [&](int64_t tile, int b) {               // a lane per coefficient; the pad columns stay zero
        if (tile < ntiles && lane < K) {
            const int64_t f0 = tile * TF;
            const int nf_tile = Nf - f0 < TF ? (int)(Nf - f0) : TF;
            const float* src = coeff + f0 * K + lane;
            float* sc = scoef0 + b * TF * CP + lane;
            for (int fl = warp; fl < nf_tile; fl += 8) cp_async4(sc + fl * CP, src + fl * K);
        }
        cp_async_commit();
    };
    __syncthreads();                                           // the zero fill above is complete
    fetch_coef(blockIdx.x, 0);
    int buf = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += tstep, buf ^= 1) {
        const int64_t f0 = tile * TF;
        const int nf_tile = Nf - f0 < TF ? (int)(Nf - f0) : TF;
        // one hop for each of the next three tiles (results are used in the next iteration)
        float rn_next[NI];
        int vo_next[NI], vi_next[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            rn_next[i] = hop_rn(vo1[i]);
            vo_next[i] = hop_vo(vi2[i]);
            vi_next[i] = hop_face(tile + 3 * tstep, i);
        }
        __syncthreads();                                       // previous tile fully consumed
        fetch_coef(tile + tstep, buf ^ 1);                     // the next tile's coefficient rows, asynchronously
        cp_async_wait<1>();                                    // this tile's rows have landed (own copies) ...
        __syncthreads();                                       // ... and everybody else's
        const float* scoef = scoef0 + buf * TF * CP;
        // ---- phase 1: faces (warp + 8 i) * FPW + fs
        // all sixteen row loads of the thread are issued first; the filter sums below need only the coefficients and run
        // while the rows are on their way
        float4 x[4], w[4], gr[4][3];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int fl = (warp + 8 * i) * FPW + fs;
            x[i] = zero4(); w[i] = zero4();
#pragma unroll
            for (int j = 0; j < 3; ++j) gr[i][j] = zero4();
            if (on && fl < nf_tile) {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const int vo = svo[buf * NE + fl * 3 + j];
                    if (vo >= 0) gr[i][j] = ldg4(gout + (int64_t)vo * CV + cg);
                }
                x[i] = ldg4(in + (f0 + fl) * CV + cg);
            }
        }
        for (int g = 0; g < KG; ++g) {                         // rows past the tile are stale or zero: unused
            const float4 fa = sfilt[4 * g * LPF + l], fb = sfilt[(4 * g + 1) * LPF + l];
            const float4 fc = sfilt[(4 * g + 2) * LPF + l], fd = sfilt[(4 * g + 3) * LPF + l];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 cf = *reinterpret_cast<const float4*>(scoef + ((warp + 8 * i) * FPW + fs) * CP + 4 * g);
                fma4s(w[i], cf.x, fa); fma4s(w[i], cf.y, fb); fma4s(w[i], cf.z, fc); fma4s(w[i], cf.w, fd);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int fl = (warp + 8 * i) * FPW + fs;
            float4 gt = zero4();
#pragma unroll
            for (int j = 0; j < 3; ++j) fma4s(gt, srn[buf * NE + fl * 3 + j], gr[i][j]);
            if (on && fl < nf_tile) __stcs(gin + (f0 + fl) * CV + cg, mul4(gt, w[i]));
            if (fl < nf_tile) st[fl * LPF + l] = mul4(x[i], gt);
        }
        __syncthreads();
        // the next tile's corners go to the other index buffer (its readers are behind the barrier above)
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            park(buf ^ 1, i, vo1[i], rn_next[i]);
            vo1[i] = vo_next[i]; vi2[i] = vi_next[i];
        }
        // ---- phase 2, faces in order
        if (slice < slices) {
            const int first = slice * FPW + fs, step = slices * FPW;
            const float* cp = scoef + first * CP + 4 * g2;
            const float4* tp = st + first * LPF + l;
#pragma unroll 4
            for (int fl = first; fl < nf_tile; fl += step, cp += step * CP, tp += step * LPF) {
                const float4 c = *reinterpret_cast<const float4*>(cp), t = *tp;
                fma4s(acc[0], c.x, t); fma4s(acc[1], c.y, t); fma4s(acc[2], c.z, t); fma4s(acc[3], c.w, t);
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();                                           // the sums of the slices, in slice order, and of the side-by-side faces
    float4* sums = st;                                         // [slices * KG][4][32]: st has as many
    if (slice < slices)
#pragma unroll
        for (int j = 0; j < 4; ++j) sums[(warp * 4 + j) * 32 + lane] = acc[j];
    __syncthreads();
    for (int i = threadIdx.x; i < K * LPF; i += blockDim.x) {
        const int k = i / LPF, c = i % LPF;
        float4 s = zero4();
        for (int v = 0; v < slices; ++v)
#pragma unroll
            for (int q = 0; q < FPW; ++q) add4(s, sums[((v * KG + k / 4) * 4 + k % 4) * 32 + q * LPF + c]);
        if (blockIdx.y * LPF + c < CV) partial[((int64_t)blockIdx.x * K + k) * CV + blockIdx.y * LPF + c] = s;
    }
}

// ---------------------------------------------------------------------- backward, generic
__device__ __forceinline__ float f2v_gt(const int32_t* __restrict__ face, const int32_t* __restrict__ vtMap,
                                        const int32_t* __restrict__ nfCount, const float* __restrict__ gout,
                                        int64_t f, int Cr, int co) {
    float gt = 0.f;
    for (int j = 0; j < 3; ++j) {
        int vi = face[3 * f + j];
        int vo = vtMap ? vtMap[vi] : vi;
        if (vo >= 0) gt += __ldg(gout + (int64_t)vo * Cr + co) / (float)nfCount[vo];
    }
    return gt;
}

__global__ void f2v_bwd_input_generic_kernel(int64_t Nf, int C, int r, int K, const int32_t* __restrict__ face,
                                             const int32_t* __restrict__ vtMap, const int32_t* __restrict__ nfCount,
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
            acc = fmaf(f2v_gt(face, vtMap, nfCount, gout, f, Cr, co), w, acc);
        }
        gin[i] = acc;
    }
}

// thread = output channel co, blockIdx.x = chunk of faces (walked in order), blockIdx.z = k
__global__ void f2v_bwd_filter_generic_kernel(int64_t Nf, int C, int r, int K, int64_t faces_per_chunk,
                                              const int32_t* __restrict__ face, const int32_t* __restrict__ vtMap,
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
        float gt = f2v_gt(face, vtMap, nfCount, gout, f, Cr, co);
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
        int CV = C / 4;
        float4* wx = (float4*)workspace;
        int rc = f2v_face_products(Nf, C, K, input, filter, coeff, (float*)wx, stream);
        if (rc) return rc;
        TeamGeom g = team_geom(CV);
        dim3 grid(persistent_blocks(NvOut, g.teams, 8), g.chunks);
        PB_DISPATCH_TL(g.TL, PB_LAUNCH("f2v_fwd_gather", f2v_fwd_gather_kernel<TL>, grid, 256, 0, stream, NvOut, CV,
                                       rowptr, entries, nfCount, (const float4*)wx, (float4*)output));
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
    F2VBwdPlan p = f2v_bwd_plan(Nf, C, r, K);
    float* partial = (float*)workspace;
    bool vec = p.vec && aligned16(gradOutput) && aligned16(input) && aligned16(filter) && aligned16(gradInput);
    if (vec) {
        int CV = C / 4;
        // K <= 32: lanes of a face as many as hold its channels.  Behind 128 channels chunks of 128 on blockIdx.y
        if (K <= 32) {
            auto run = [&](auto lpf) {
                constexpr int LPF = decltype(lpf)::value;
                const int chunks = (int)ceil_div(CV, LPF);
                int64_t gx = ceil_div(2 * (int64_t)sm_count(), chunks);              // two blocks per SM
                if (gx > ceil_div(Nf, F2VB_FACES<LPF>)) gx = ceil_div(Nf, F2VB_FACES<LPF>);
                if (gx > p.grid_x) gx = p.grid_x;
                const size_t smemb = f2vb_smem<LPF>(K);
                PB_CUDA(cudaFuncSetAttribute(f2v_bwd_blocked_kernel<LPF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemb));
                PB_LAUNCH("f2v_bwd", f2v_bwd_blocked_kernel<LPF>, dim3((unsigned)gx, chunks), 256, smemb, stream, Nf, CV, K, face, vtMap,
                          nfCount, coeff, (const float4*)input, (const float4*)filter, (const float4*)gradOutput, (float4*)gradInput,
                          (float4*)partial);
                return reduce_partials(partial, (int)gx, (int64_t)K * Cr, gradFilter, stream);
            };
            if (CV <= 4) return run(std::integral_constant<int, 4>{});
            if (CV <= 8) return run(std::integral_constant<int, 8>{});
            if (CV <= 16) return run(std::integral_constant<int, 16>{});
            return run(std::integral_constant<int, 32>{});
        }
        dim3 grid(p.grid_x, (unsigned)ceil_div(CV, 32));
        const int KP = (K + 3) / 4 * 4 + 4;
        size_t smem = sizeof(float4) * (32 * (size_t)K + F2VB_TF * 32) + sizeof(float) * F2VB_TF * KP;
        const int cvc = CV < 32 ? CV : 32;
        const int nacc = (int)ceil_div((int64_t)K * cvc, 256);
#define PB_F2VB_LAUNCH(N)                                                                                        \
        PB_LAUNCH("f2v_bwd", f2v_bwd_tile_kernel<N>, grid, 256, smem, stream, Nf, CV, K, face, vtMap, nfCount,   \
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
    PB_LAUNCH("f2v_bwd_input_generic", f2v_bwd_input_generic_kernel, gi, 256, 0, stream, Nf, C, r, K, face, vtMap,
              nfCount, coeff, filter, gradOutput, gradInput);
    PB_REQUIRE(K <= 65535, PB200_EINVAL, "facet2vertex_backward: K too large");
    dim3 gridf(q.grid_x, (unsigned)ceil_div(Cr, 128), K);
    PB_LAUNCH("f2v_bwd_filter_generic", f2v_bwd_filter_generic_kernel, gridf, 128, 0, stream, Nf, C, r, K,
              q.faces_per_chunk, face, vtMap, nfCount, coeff, input, gradOutput, partial);
    return reduce_partials(partial, q.grid_x, (int64_t)K * Cr, gradFilter, stream);
}

}  // extern "C"
