// facet2facet for inputs of at most four channels (colours, coordinates), forward and filter gradient, in fp32:
//
//   A[f, (d, ci)]          = (1/T_f) sum_k bary[k, d] * in[k, ci]              over the T_f samples k of face f
//   out[f, co]             = sum_(d, ci) A[f, (d, ci)] * filter[co, ci, d]
//   gradFilter[co, ci, d]  = sum_f gradOutput[f, co] * A[f, (d, ci)]
//
// The tensor-core kernels pad the channels to 16 and the outputs to 128: with three channels, 16 bases and 32 outputs 14 of 15
// products are of zeros, besides a padded copy of the input (1 758 000 faces, 4.4 million samples: copy 165 us, forward 734,
// filter gradient 698).  Here a block takes TF faces at a time, puts their A rows into shared memory (a thread = a face and
// four bases, so that a sample's weights are read in whole sectors) and contracts them with plain multiply-adds on register
// tiles: eight faces x four outputs per thread forward, four (d, ci) x four outputs per item backward, whose running sums stay
// in registers over all tiles of the block.  What bounds it: the multiply-adds and the shared-memory reads that feed them, then
// the samples' weights from memory.  Several blocks per SM overlap the two phases.
#include "common.cuh"

namespace pb {
namespace small {

constexpr int NT = 256;
constexpr int MAX_C = 4, MAX_F = 32;
// Samples whose rows are loaded together (1 758 000 faces, 16 bases, 32 outputs, one at a time: forward 279 us, filter gradient 358; two:
// 244 and 329; four take the filter gradient a block per SM in registers: 249 and 426)
constexpr int AT = 2;

// floats of an A row: a multiple of four, and 4 (mod 8), so that rows read side by side lie on different banks
__host__ __device__ __forceinline__ int a_pitch(int F, int C) { return ((F + 3) / 4 * 4 * C) | 4; }

struct Params {
    int64_t Nf;
    int F, Cout;
    const float* in;
    const float* bary;
    const int32_t* cum;
    const float* filter;                 // forward
    const float* gout;                   // backward
    float* out;                          // forward: output; backward: partial[block][Cout * C * F]
};

// A rows of faces f0 .. f0 + TF - 1 into sa (rows past Nf zero, (d, ci) past F zero)
template <int C, int TF>
__device__ __forceinline__ void face_rows(const Params& p, int64_t f0, float* sa) {
    const int F = p.F, quads = (F + 3) / 4, AP = a_pitch(F, C);
    const bool vec = F % 4 == 0 && (reinterpret_cast<uintptr_t>(p.bary) & 15) == 0;
    for (int i = threadIdx.x; i < TF * quads; i += NT) {
        const int fl = i / quads, q = i - fl * quads;
        const int64_t f = f0 + fl;
        float a[4][C];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int c = 0; c < C; ++c) a[j][c] = 0.f;
        if (f < p.Nf) {
            const int k0 = f > 0 ? __ldg(p.cum + f - 1) : 0, k1 = __ldg(p.cum + f);
            for (int k = k0; k < k1; k += AT) {                    // the rows of AT samples are on their way together
                float b[AT][4], x[AT][C];
#pragma unroll
                for (int t = 0; t < AT; ++t) {
                    const bool on = k + t < k1;
                    const float* src = p.bary + (int64_t)(k + t) * F + 4 * q;
                    if (vec) {
                        const float4 v = on ? ldg4(reinterpret_cast<const float4*>(src)) : zero4();
                        b[t][0] = v.x; b[t][1] = v.y; b[t][2] = v.z; b[t][3] = v.w;
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j) b[t][j] = on && 4 * q + j < F ? __ldg(src + j) : 0.f;
                    }
#pragma unroll
                    for (int c = 0; c < C; ++c) x[t][c] = on ? __ldg(p.in + (int64_t)(k + t) * C + c) : 0.f;
                }
#pragma unroll
                for (int t = 0; t < AT; ++t)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int c = 0; c < C; ++c) a[j][c] = fmaf(b[t][j], x[t][c], a[j][c]);
            }
            const float w = k1 > k0 ? 1.f / (float)(k1 - k0) : 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int c = 0; c < C; ++c) a[j][c] *= w;
        }
        float4* dst = reinterpret_cast<float4*>(sa + fl * AP + 4 * q * C);
        const float* v = &a[0][0];
#pragma unroll
        for (int c = 0; c < C; ++c) dst[c] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    }
}

// CG: groups of four outputs of a block column (4, 8 or 16)
template <int C, int CG>
__global__ void __launch_bounds__(NT) f2f_small_fwd_kernel(Params p) {
    constexpr int FPT = 8, FG = NT / CG, TF = CG == 4 ? FG * 4 : CG == 8 ? FG * 4 : FG * FPT, FT = TF / FG;
    extern __shared__ float4 smem4[];
    const int M = p.F * C, M4 = (p.F + 3) / 4 * 4 * C, AP = a_pitch(p.F, C);
    float4* sw = smem4;                                        // [M4][CG] filter, rows M.. and outputs behind Cout zero
    float* sa = reinterpret_cast<float*>(smem4 + M4 * CG);     // [TF][AP]
    const int co0 = blockIdx.y * 4 * CG;
    for (int i = threadIdx.x; i < M4 * CG * 4; i += NT) {
        const int m = i / (CG * 4), co = co0 + i % (CG * 4);
        reinterpret_cast<float*>(sw)[i] = m < M && co < p.Cout ? __ldg(p.filter + ((int64_t)co * C + m % C) * p.F + m / C) : 0.f;
    }
    const int cg = threadIdx.x % CG, fg = threadIdx.x / CG;
    const int co = co0 + 4 * cg;
    const bool vec = p.Cout % 4 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
    const int64_t ntiles = (p.Nf + TF - 1) / TF;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t f0 = tile * TF;
        __syncthreads();
        face_rows<C, TF>(p, f0, sa);
        __syncthreads();
        float4 acc[FT];
#pragma unroll
        for (int i = 0; i < FT; ++i) acc[i] = zero4();
        const float* row = sa + fg * AP;                       // faces fg + FG * i
        for (int m = 0; m < M4; m += 4) {
            const float4 w0 = sw[m * CG + cg], w1 = sw[(m + 1) * CG + cg], w2 = sw[(m + 2) * CG + cg], w3 = sw[(m + 3) * CG + cg];
#pragma unroll
            for (int i = 0; i < FT; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(row + i * FG * AP + m);
                fma4s(acc[i], a.x, w0); fma4s(acc[i], a.y, w1); fma4s(acc[i], a.z, w2); fma4s(acc[i], a.w, w3);
            }
        }
#pragma unroll
        for (int i = 0; i < FT; ++i) {
            const int64_t f = f0 + fg + i * FG;
            if (f >= p.Nf || co >= p.Cout) continue;
            float* o = p.out + f * p.Cout + co;
            if (vec) {
                *reinterpret_cast<float4*>(o) = acc[i];
            } else {
                const float v[4] = {acc[i].x, acc[i].y, acc[i].z, acc[i].w};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (co + j < p.Cout) o[j] = v[j];
            }
        }
    }
}

// Items = (four (d, ci), four outputs); a thread has NI of them, or, with few, the block's threads share the tile's faces
template <int C, int NI>
__global__ void __launch_bounds__(NT) f2f_small_gfilter_kernel(Params p) {
    constexpr int TF = 64;
    extern __shared__ float4 smem4[];
    const int M = p.F * C, MG = (p.F + 3) / 4 * C, AP = a_pitch(p.F, C);           // groups of four (d, ci)
    const int co0 = blockIdx.y * 64, cw = p.Cout - co0 < 64 ? p.Cout - co0 : 64;   // this block column's outputs
    const int CG = (cw + 3) / 4, items = MG * CG, GP = CG + 1;                      // float4 of a gradOutput row in shared memory
    float4* sg = smem4;                                        // [TF][GP]
    float* sa = reinterpret_cast<float*>(smem4 + TF * GP);     // [TF][AP]
    const int shares = NI == 1 ? NT / items : 1;               // threads that share the faces of an item
    const int share = NI == 1 ? threadIdx.x / items : 0;
    float4 acc[NI][4];
#pragma unroll
    for (int n = 0; n < NI; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[n][j] = zero4();
    int mg[NI], cg[NI];
#pragma unroll
    for (int n = 0; n < NI; ++n) {
        const int item = NI == 1 ? threadIdx.x % items : threadIdx.x + n * NT;
        mg[n] = item < items ? item / CG : 0;
        cg[n] = item < items ? item % CG : 0;
    }
    const bool vec = p.Cout % 4 == 0 && (reinterpret_cast<uintptr_t>(p.gout) & 15) == 0;
    const int64_t ntiles = (p.Nf + TF - 1) / TF;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t f0 = tile * TF;
        __syncthreads();
        for (int i = threadIdx.x; i < TF * CG; i += NT) {
            const int fl = i / CG, c = i - fl * CG;
            float4 v = zero4();
            if (f0 + fl < p.Nf) {
                const float* src = p.gout + (f0 + fl) * p.Cout + co0 + 4 * c;
                if (vec) {
                    v = ldg4(reinterpret_cast<const float4*>(src));
                } else {
                    v.x = __ldg(src);
                    if (4 * c + 1 < cw) v.y = __ldg(src + 1);
                    if (4 * c + 2 < cw) v.z = __ldg(src + 2);
                    if (4 * c + 3 < cw) v.w = __ldg(src + 3);
                }
            }
            sg[fl * GP + c] = v;
        }
        face_rows<C, TF>(p, f0, sa);
        __syncthreads();
        if (share < shares) {
#pragma unroll 4
            for (int fl = share; fl < TF; fl += shares) {
#pragma unroll
                for (int n = 0; n < NI; ++n) {
                    const float4 a = *reinterpret_cast<const float4*>(sa + fl * AP + 4 * mg[n]);
                    const float4 g = sg[fl * GP + cg[n]];
                    fma4s(acc[n][0], a.x, g); fma4s(acc[n][1], a.y, g); fma4s(acc[n][2], a.z, g); fma4s(acc[n][3], a.w, g);
                }
            }
        }
    }
    // shares of an item are added in order
    float4* sums = smem4;                                      // [NT][4]
    if (NI == 1) {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 4; ++j) sums[threadIdx.x * 4 + j] = acc[0][j];
        __syncthreads();
        if (threadIdx.x < items)
            for (int s = 1; s < shares; ++s)
#pragma unroll
                for (int j = 0; j < 4; ++j) add4(acc[0][j], sums[(s * items + threadIdx.x) * 4 + j]);
    }
    float* out = p.out + (int64_t)blockIdx.x * p.Cout * C * p.F;
#pragma unroll
    for (int n = 0; n < NI; ++n) {
        if ((int)threadIdx.x + n * NT >= items) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = 4 * mg[n] + j;
            if (m >= M) continue;
            const float v[4] = {acc[n][j].x, acc[n][j].y, acc[n][j].z, acc[n][j].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int co = 4 * cg[n] + e;
                if (co < cw) out[((int64_t)(co0 + co) * C + m % C) * p.F + m / C] = v[e];
            }
        }
    }
}

// ---------------------------------------------------------------------------- host side
// The line lies where the padding to 16 channels wastes three quarters of the products of the tensor-core kernels.
bool supported(int Cin, int Cout, int F) { return Cin >= 1 && Cin <= MAX_C && Cout >= 1 && F >= 1 && F <= MAX_F; }

template <int C, int CG>
static int launch_fwd(const Params& p, cudaStream_t stream) {
    constexpr int FG = NT / CG, TF = CG == 16 ? FG * 8 : FG * 4;
    const size_t smem = sizeof(float4) * (size_t)((p.F + 3) / 4 * 4 * C) * CG + sizeof(float) * (size_t)TF * a_pitch(p.F, C);
    PB_CUDA(cudaFuncSetAttribute(f2f_small_fwd_kernel<C, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PB_LAUNCH("f2f_fwd_small", (f2f_small_fwd_kernel<C, CG>), dim3(persistent_blocks(p.Nf, TF, 4), (unsigned)ceil_div(p.Cout, 4 * CG)), NT,
              smem, stream, p);
    return PB200_OK;
}

template <int C>
static int forward_c(const Params& p, cudaStream_t stream) {
    if (p.Cout <= 16) return launch_fwd<C, 4>(p, stream);
    if (p.Cout <= 32) return launch_fwd<C, 8>(p, stream);
    return launch_fwd<C, 16>(p, stream);
}

int forward(int64_t Nf, int Cin, int Cout, int F, const float* input, const float* filter, const float* bary, const int32_t* cum,
            float* output, cudaStream_t stream) {
    Params p = {};
    p.Nf = Nf; p.F = F; p.Cout = Cout; p.in = input; p.bary = bary; p.cum = cum; p.filter = filter; p.out = output;
    switch (Cin) {
        case 1: return forward_c<1>(p, stream);
        case 2: return forward_c<2>(p, stream);
        case 3: return forward_c<3>(p, stream);
        default: return forward_c<4>(p, stream);
    }
}

static int gf_blocks(int64_t Nf) { return persistent_blocks(Nf, 64, 4); }
size_t workspace_bytes(int64_t Nf, int Cin, int Cout, int F) {
    return align_up(sizeof(float) * (size_t)gf_blocks(Nf > 0 ? Nf : 1) * Cin * Cout * F, 256);
}

template <int C, int NI>
static int launch_gf(const Params& p, int blocks, cudaStream_t stream) {
    size_t smem = sizeof(float4) * 64 * 17 + sizeof(float) * 64 * (size_t)a_pitch(p.F, C);
    if (smem < NT * 4 * sizeof(float4)) smem = NT * 4 * sizeof(float4);
    PB_CUDA(cudaFuncSetAttribute(f2f_small_gfilter_kernel<C, NI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PB_LAUNCH("f2f_bwd_gfilter_small", (f2f_small_gfilter_kernel<C, NI>), dim3(blocks, (unsigned)ceil_div(p.Cout, 64)), NT, smem, stream, p);
    return PB200_OK;
}

template <int C>
static int gfilter_c(const Params& p, int blocks, cudaStream_t stream) {
    const int cw = p.Cout < 64 ? p.Cout : 64, items = (p.F + 3) / 4 * C * ((cw + 3) / 4);
    if (items <= NT) return launch_gf<C, 1>(p, blocks, stream);
    return launch_gf<C, 2>(p, blocks, stream);
}

int backward_filter(int64_t Nf, int Cin, int Cout, int F, const float* gout, const float* input, const float* bary, const int32_t* cum,
                    float* gfilter, void* ws, cudaStream_t stream) {
    Params p = {};
    p.Nf = Nf; p.F = F; p.Cout = Cout; p.in = input; p.bary = bary; p.cum = cum; p.gout = gout; p.out = (float*)ws;
    const int blocks = gf_blocks(Nf);
    int rc;
    switch (Cin) {
        case 1: rc = gfilter_c<1>(p, blocks, stream); break;
        case 2: rc = gfilter_c<2>(p, blocks, stream); break;
        case 3: rc = gfilter_c<3>(p, blocks, stream); break;
        default: rc = gfilter_c<4>(p, blocks, stream); break;
    }
    if (rc) return rc;
    return reduce_partials((const float*)ws, blocks, (int64_t)Cout * Cin * F, gfilter, stream);
}

}  // namespace small
}  // namespace pb
