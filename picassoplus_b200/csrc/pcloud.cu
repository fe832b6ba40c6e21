// Point-cloud depthwise convolution with hard or fuzzy filter-bin assignment (the SPH3D kernel of
// the dual point/mesh blocks): forward, input gradient and filter gradient.  The reference scatters
// every neighbour pair with float atomics; here the forward pass is a pull over the pairs grouped
// by output point, the input gradient a pull over the pairs grouped by input point (both groupings:
// pb200_build_key_csr on the two columns of nnIndex, pair ids ascending), and the filter gradient
// a fixed-order reduction (a thread owns one output channel, walks its block's pairs in order,
// blocks are added in order).  No floating-point atomics: results do not depend on scheduling.
#include "common.cuh"

namespace pb {
namespace pcloud {

// weight of pair p for output channel co: filter[bin[p], co] (hard assignment) or
// sum_t coeff[p,t] * filter[bin[p,t], co] (fuzzy).  A bin index outside [0, F) contributes 0.
__device__ __forceinline__ float pair_weight(int64_t p, int co, int Cr, int F, int T, const int32_t* __restrict__ bin,
                                             const float* __restrict__ coeff, const float* __restrict__ filter) {
    if (!coeff) {
        const int f = bin[p];
        return (f >= 0 && f < F) ? __ldg(filter + (int64_t)f * Cr + co) : 0.f;
    }
    float w = 0.f;
    for (int t = 0; t < T; ++t) {
        const int f = bin[p * T + t];
        if (f >= 0 && f < F) w = fmaf(coeff[p * T + t], __ldg(filter + (int64_t)f * Cr + co), w);
    }
    return w;
}

// output[o, co] = sum over the pairs p of output point o of input[in_p, co / r] * w_p[co] / nnCount[o]
// (reference: depthwise_conv3d_forward / fuzzy_depthwise_conv3d_forward, pcloud_conv3d_gpu.cu:8-27,94-118:
// each term is divided before it is added)
__global__ void conv_fwd_kernel(int64_t Np, int64_t Mp, int F, int C, int r, int T, const float* __restrict__ input,
                                const float* __restrict__ filter, const int32_t* __restrict__ nnCount,
                                const int32_t* __restrict__ nnIndex, const int32_t* __restrict__ bin,
                                const float* __restrict__ coeff, const int32_t* __restrict__ rowptr,
                                const int32_t* __restrict__ members, float* __restrict__ output) {
    const int Cr = C * r;
    const int64_t total = Mp * Cr;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = i / Cr;
        const int co = (int)(i - o * Cr), cin = co / r;
        const float nn = (float)nnCount[o];
        float acc = 0.f;
        for (int e = rowptr[o]; e < rowptr[o + 1]; ++e) {
            const int64_t p = members[e];
            const int in = nnIndex[2 * p + 1];
            if (in < 0 || in >= Np) continue;
            acc += __ldg(input + (int64_t)in * C + cin) * pair_weight(p, co, Cr, F, T, bin, coeff, filter) / nn;
        }
        output[i] = acc;
    }
}

// gradInput[n, c] = sum over the pairs p of input point n, over m < r, of
// gradOutput[out_p, c*r+m] * w_p[c*r+m] / nnCount[out_p]
// (reference: depthwise_input_backward / fuzzy_depthwise_input_backward, pcloud_conv3d_gpu.cu:30-48,121-147)
__global__ void conv_bwd_input_kernel(int64_t Np, int64_t Mp, int F, int C, int r, int T, const float* __restrict__ gout,
                                      const float* __restrict__ filter, const int32_t* __restrict__ nnCount,
                                      const int32_t* __restrict__ nnIndex, const int32_t* __restrict__ bin,
                                      const float* __restrict__ coeff, const int32_t* __restrict__ rowptr,
                                      const int32_t* __restrict__ members, float* __restrict__ gin) {
    const int Cr = C * r;
    const int64_t total = Np * C;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = i / C;
        const int c = (int)(i - n * C);
        float acc = 0.f;
        for (int e = rowptr[n]; e < rowptr[n + 1]; ++e) {
            const int64_t p = members[e];
            const int o = nnIndex[2 * p];
            if (o < 0 || o >= Mp) continue;
            const float nn = (float)nnCount[o];
            for (int m = 0; m < r; ++m) {
                const int co = c * r + m;
                acc += __ldg(gout + (int64_t)o * Cr + co) * pair_weight(p, co, Cr, F, T, bin, coeff, filter) / nn;
            }
        }
        gin[i] = acc;
    }
}

// partial[block][f, co] = sum over the block's pairs (ascending) of coeff * gradOutput[out_p, co] *
// input[in_p, co / r] / nnCount[out_p] (reference: depthwise_filter_backward /
// fuzzy_depthwise_filter_backward, pcloud_conv3d_gpu.cu:51-88,150-193).  Thread = output channel:
// it alone touches column co of the block's accumulator in shared memory.
__global__ void conv_bwd_filter_kernel(int64_t Np, int64_t Mp, int64_t Nout, int64_t pairs_per_block, int F, int C, int r,
                                       int T, const float* __restrict__ input, const float* __restrict__ gout,
                                       const int32_t* __restrict__ nnCount, const int32_t* __restrict__ nnIndex,
                                       const int32_t* __restrict__ bin, const float* __restrict__ coeff,
                                       float* __restrict__ partial) {
    extern __shared__ float acc[];                   // [F][Cr]
    const int Cr = C * r;
    for (int i = threadIdx.x; i < F * Cr; i += blockDim.x) acc[i] = 0.f;
    __syncthreads();
    const int64_t p0 = (int64_t)blockIdx.x * pairs_per_block;
    int64_t p1 = p0 + pairs_per_block;
    if (p1 > Nout) p1 = Nout;
    for (int co = threadIdx.x; co < Cr; co += blockDim.x) {
        const int cin = co / r;
        for (int64_t p = p0; p < p1; ++p) {
            const int o = nnIndex[2 * p], in = nnIndex[2 * p + 1];
            if (o < 0 || o >= Mp || in < 0 || in >= Np) continue;
            const float d = __ldg(gout + (int64_t)o * Cr + co) * __ldg(input + (int64_t)in * C + cin) / (float)nnCount[o];
            if (!coeff) {
                const int f = bin[p];
                if (f >= 0 && f < F) acc[f * Cr + co] += d;
            } else {
                for (int t = 0; t < T; ++t) {
                    const int f = bin[p * T + t];
                    if (f >= 0 && f < F) acc[f * Cr + co] += coeff[p * T + t] * d;
                }
            }
        }
    }
    __syncthreads();
    float* out = partial + (int64_t)blockIdx.x * F * Cr;
    for (int i = threadIdx.x; i < F * Cr; i += blockDim.x) out[i] = acc[i];
}

// ------------------------------------------------------------------------ vector kernels
// Depth multiplier 1 and C a multiple of 4 (every layer of the reference's networks): a thread owns four
// channels of a point, the filter table lives in shared memory, a term is x * w * (1 / nnCount).
__device__ __forceinline__ float4 pair_weight4(int64_t p, int cg, int CV, int F, int T, const int32_t* __restrict__ bin,
                                               const float* __restrict__ coeff, const float4* __restrict__ sfilt) {
    if (!coeff) {
        const int f = __ldg(bin + p);
        return (f >= 0 && f < F) ? sfilt[f * CV + cg] : zero4();
    }
    float4 w = zero4();
    for (int t = 0; t < T; ++t) {
        const int f = __ldg(bin + p * T + t);
        if (f >= 0 && f < F) fma4s(w, __ldg(coeff + p * T + t), sfilt[f * CV + cg]);
    }
    return w;
}

__global__ void conv_fwd_vec_kernel(int64_t Np, int64_t Mp, int F, int CV, int T, const float4* __restrict__ input,
                                    const float4* __restrict__ filter, const int32_t* __restrict__ nnCount,
                                    const int32_t* __restrict__ nnIndex, const int32_t* __restrict__ bin,
                                    const float* __restrict__ coeff, const int32_t* __restrict__ rowptr,
                                    const int32_t* __restrict__ members, float4* __restrict__ output) {
    extern __shared__ float4 sfilt[];                // [F][CV]
    for (int i = threadIdx.x; i < F * CV; i += blockDim.x) sfilt[i] = filter[i];
    __syncthreads();
    const int64_t total = Mp * CV;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = i / CV;
        const int cg = (int)(i - o * CV);
        const float rn = 1.f / (float)__ldg(nnCount + o);
        float4 acc = zero4();
        for (int e = __ldg(rowptr + o); e < __ldg(rowptr + o + 1); ++e) {
            const int64_t p = __ldg(members + e);
            const int in = __ldg(nnIndex + 2 * p + 1);
            if (in < 0 || in >= Np) continue;
            const float4 w = pair_weight4(p, cg, CV, F, T, bin, coeff, sfilt);
            fma4(acc, scale4(ldg4(input + (int64_t)in * CV + cg), rn), w);
        }
        output[i] = acc;
    }
}

// An input point that many output points name (a padded neighbour list names point 0 over and over) would keep one group of
// lanes walking long after the others are done: 800 pairs took 300 us of a 370 us launch.  Rows longer than this get a block
// each.
constexpr int LONG_ROW = 64;

// The long rows of the input gradient, a role of the launch's first blocks so that they run beside the others.  A block looks
// through LONG_SCAN rows.  For a long one, all threads fetch the next STAGE pairs (index, 1 / count, bins, weights) into shared
// memory, then the block's groups of CV lanes walk equal consecutive parts of them, four row gathers in flight; the groups'
// sums are added in group order.
constexpr int LONG_SCAN = 1024, STAGE = 256, STAGED_BINS = 3;
// beside the 17 KB that they are staged in, a filter table above this needs more than the default 48 KB
constexpr size_t UNASKED_TABLE = 30 * 1024;
static inline int long_blocks(int64_t Np) { return (int)ceil_div(Np, LONG_SCAN); }

__device__ __noinline__ void bwd_input_long_rows(int64_t first, int64_t Np, int64_t Mp, int F, int CV, int T,
                                                    const float4* __restrict__ gout, const float4* __restrict__ filter,
                                                    const int32_t* __restrict__ nnCount, const int32_t* __restrict__ nnIndex,
                                                    const int32_t* __restrict__ bin, const float* __restrict__ coeff,
                                                    const int32_t* __restrict__ rowptr, const int32_t* __restrict__ members,
                                                    float4* __restrict__ gin, float4* sfilt) {
    __shared__ float4 red[256];
    __shared__ int rows[LONG_SCAN], nrows;
    __shared__ int sp[STAGE], so[STAGE], sb[STAGE][STAGED_BINS];
    __shared__ float srn[STAGE], sc[STAGE][STAGED_BINS];
    if (threadIdx.x == 0) nrows = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < LONG_SCAN; i += blockDim.x) {
        const int64_t n = first + i;
        if (n < Np && __ldg(rowptr + n + 1) - __ldg(rowptr + n) > LONG_ROW) rows[atomicAdd(&nrows, 1)] = i;
    }
    __syncthreads();
    const int total = nrows;
    if (total == 0) return;
    for (int i = threadIdx.x; i < F * CV; i += blockDim.x) sfilt[i] = filter[i];
    const int G = blockDim.x / CV, g = threadIdx.x / CV, cg = threadIdx.x - g * CV;
    const bool staged = T <= STAGED_BINS;
    for (int k = 0; k < total; ++k) {
        const int64_t n = first + rows[k];
        const int e0 = __ldg(rowptr + n), e1 = __ldg(rowptr + n + 1);
        float4 acc = zero4();
        for (int s0 = e0; s0 < e1; s0 += STAGE) {
            const int cnt = e1 - s0 < STAGE ? e1 - s0 : STAGE;
            __syncthreads();
            for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
                const int p = __ldg(members + s0 + i);
                const int o = __ldg(nnIndex + 2 * (int64_t)p);
                const bool ok = o >= 0 && o < Mp;
                sp[i] = p;
                so[i] = ok ? o : -1;
                srn[i] = ok ? 1.f / (float)__ldg(nnCount + o) : 0.f;
                if (staged)
                    for (int t = 0; t < T; ++t) {
                        const int f = __ldg(bin + (int64_t)p * T + t);
                        const bool in = f >= 0 && f < F;
                        sb[i][t] = in ? f : 0;
                        sc[i][t] = in ? (coeff ? __ldg(coeff + (int64_t)p * T + t) : 1.f) : 0.f;
                    }
            }
            __syncthreads();
            const int per = (cnt + G - 1) / G, b = g * per;
            const int e = g < G ? (b + per < cnt ? b + per : cnt) : 0;
            for (int q = b; q < e; q += 4) {
                float4 x[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) x[u] = q + u < e && so[q + u] >= 0 ? ldg4(gout + (int64_t)so[q + u] * CV + cg) : zero4();
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (q + u >= e) break;
                    float4 w = zero4();
                    if (staged) for (int t = 0; t < T; ++t) fma4s(w, sc[q + u][t], sfilt[sb[q + u][t] * CV + cg]);
                    else w = pair_weight4(sp[q + u], cg, CV, F, T, bin, coeff, sfilt);
                    fma4(acc, scale4(x[u], srn[q + u]), w);
                }
            }
        }
        red[threadIdx.x] = acc;
        __syncthreads();
        if (g == 0) {
            for (int t = 1; t < G; ++t) add4(acc, red[t * CV + cg]);
            gin[n * CV + cg] = acc;
        }
        __syncthreads();
    }
}

__global__ void conv_bwd_input_vec_kernel(int64_t Np, int64_t Mp, int F, int CV, int T, const float4* __restrict__ gout,
                                          const float4* __restrict__ filter, const int32_t* __restrict__ nnCount,
                                          const int32_t* __restrict__ nnIndex, const int32_t* __restrict__ bin,
                                          const float* __restrict__ coeff, const int32_t* __restrict__ rowptr,
                                          const int32_t* __restrict__ members, int nlong, float4* __restrict__ gin) {
    extern __shared__ float4 sfilt[];
    if ((int)blockIdx.x < nlong) {
        bwd_input_long_rows((int64_t)blockIdx.x * LONG_SCAN, Np, Mp, F, CV, T, gout, filter, nnCount, nnIndex, bin, coeff, rowptr, members,
                            gin, sfilt);
        return;
    }
    for (int i = threadIdx.x; i < F * CV; i += blockDim.x) sfilt[i] = filter[i];
    __syncthreads();
    const int64_t total = Np * CV, nblocks = gridDim.x - nlong;
    for (int64_t i = (int64_t)(blockIdx.x - nlong) * blockDim.x + threadIdx.x; i < total; i += nblocks * blockDim.x) {
        const int64_t n = i / CV;
        const int cg = (int)(i - n * CV);
        float4 acc = zero4();
        const int e0 = __ldg(rowptr + n), e1 = __ldg(rowptr + n + 1);
        if (e1 - e0 > LONG_ROW) continue;
        for (int e = e0; e < e1; ++e) {
            const int64_t p = __ldg(members + e);
            const int o = __ldg(nnIndex + 2 * p);
            if (o < 0 || o >= Mp) continue;
            const float rn = 1.f / (float)__ldg(nnCount + o);
            const float4 w = pair_weight4(p, cg, CV, F, T, bin, coeff, sfilt);
            fma4(acc, scale4(ldg4(gout + (int64_t)o * CV + cg), rn), w);
        }
        gin[i] = acc;
    }
}

// Filter gradient: a block takes a contiguous run of pairs; its 256 threads are SUB groups of CV lanes, group g
// walks every SUB-th pair of the run in order and adds into its own copy of the [F][C] accumulator in shared
// memory (a lane alone touches its four columns of its copy); the copies are added in group order, the blocks in
// block order: fixed order throughout.
__global__ void conv_bwd_filter_vec_kernel(int64_t Np, int64_t Mp, int64_t Nout, int pairs_per_block, int F, int CV, int T,
                                           int SUB, const float4* __restrict__ input, const float4* __restrict__ gout,
                                           const int32_t* __restrict__ nnCount, const int32_t* __restrict__ nnIndex,
                                           const int32_t* __restrict__ bin, const float* __restrict__ coeff,
                                           float4* __restrict__ partial) {
    extern __shared__ float4 acc4[];                 // [SUB][F][CV]
    for (int i = threadIdx.x; i < SUB * F * CV; i += blockDim.x) acc4[i] = zero4();
    __syncthreads();
    const int g = threadIdx.x / CV, cg = threadIdx.x - g * CV;
    const int64_t p0 = (int64_t)blockIdx.x * pairs_per_block;
    int64_t p1 = p0 + pairs_per_block;
    if (p1 > Nout) p1 = Nout;
    if (g < SUB) {
        float4* mine = acc4 + (size_t)g * F * CV;
        for (int64_t p = p0 + g; p < p1; p += SUB) {
            const int o = __ldg(nnIndex + 2 * p), in = __ldg(nnIndex + 2 * p + 1);
            if (o < 0 || o >= Mp || in < 0 || in >= Np) continue;
            const float rn = 1.f / (float)__ldg(nnCount + o);
            const float4 d = mul4(scale4(ldg4(gout + (int64_t)o * CV + cg), rn), ldg4(input + (int64_t)in * CV + cg));
            if (!coeff) {
                const int f = __ldg(bin + p);
                if (f >= 0 && f < F) add4(mine[f * CV + cg], d);
            } else {
                for (int t = 0; t < T; ++t) {
                    const int f = __ldg(bin + p * T + t);
                    if (f >= 0 && f < F) fma4s(mine[f * CV + cg], __ldg(coeff + p * T + t), d);
                }
            }
        }
    }
    __syncthreads();
    float4* out = partial + (int64_t)blockIdx.x * F * CV;
    for (int i = threadIdx.x; i < F * CV; i += blockDim.x) {
        float4 s4 = acc4[i];
        for (int q = 1; q < SUB; ++q) add4(s4, acc4[(size_t)q * F * CV + i]);
        out[i] = s4;
    }
}

static bool sizes_ok(int64_t Np, int64_t Mp, int64_t Nout, int F, int C, int r, int T) {
    return Np >= 0 && Mp >= 0 && Nout >= 0 && F > 0 && C > 0 && r > 0 && T > 0 && Np < (1LL << 31) && Mp < (1LL << 31) &&
           Nout < (1LL << 31) && (int64_t)F * C * r * 4 <= 200 * 1024;
}
// ------------------------------------------------------------------------ cooperative kernels
// C of 32, 64 or 128: the lanes of a point sit in one warp, so lane j fetches the indices of the j-th
// pair of a run and the run is walked with shuffles, a few pairs at a time: the row gathers of a step are in
// flight together. TT: 1 = one bin per pair, 3 = three weighted bins, 0 = any T.
// Same order of additions as the vector kernels.
template <int CV>
__device__ __forceinline__ unsigned group_mask(int gbase) {
    return CV == 32 ? 0xffffffffu : (((1u << (CV & 31)) - 1u) << gbase);
}

// A lane owns VPL float4 of the row, LN lanes a point: with two per lane (64 and 128 channels) the index fetches, shuffles and
// bin look-ups of a pair are shared by twice the channels, which is what these kernels are short of (the load/store pipe), and
// U = 2 pairs per step keep as many row gathers in flight per warp as four with one float4.
template <int CV> struct Lanes {
    static constexpr int VPL = CV >= 16 ? 2 : 1, LN = CV / VPL, U = VPL == 2 ? 2 : 4;
};

// The bins and weights of the pair a lane fetched (TT of 1 or 3), handed to the group's lanes by shuffles.  A bin outside
// [0, F) becomes `none` with weight 0: bin 0 where filter rows are read, -1 where gradients are added with weights (a weight of 0
// in a real bin is added there like any other: 0 x NaN is NaN; without weights the 0 alone tells, 1 % faster).
template <int TT>
struct LaneBins {
    int f[TT == 3 ? 3 : 1];
    float c[TT == 3 ? 3 : 1];
};

template <int TT>
__device__ __forceinline__ void load_bins(LaneBins<TT>& b, bool have, int64_t p, int F, int none, const int32_t* __restrict__ bin,
                                          const float* __restrict__ coeff) {
#pragma unroll
    for (int t = 0; t < (TT == 3 ? 3 : 1); ++t) {
        b.f[t] = have ? __ldg(bin + p * (TT == 3 ? 3 : 1) + t) : -1;
        b.c[t] = TT == 3 ? (have ? __ldg(coeff + p * 3 + t) : 0.f) : 1.f;
        if ((unsigned)b.f[t] >= (unsigned)F) { b.f[t] = none; b.c[t] = 0.f; }
    }
}

// out += x * rn * weight of the pair, for the lane's float4
template <int TT, int CV>
__device__ __forceinline__ void add_pair(float4 (&acc)[Lanes<CV>::VPL], const float4 (&x)[Lanes<CV>::VPL], float rn, const LaneBins<TT>& b, int64_t p,
                                         unsigned mask, int src, int ln, bool ok, int F, int T, const int32_t* __restrict__ bin,
                                         const float* __restrict__ coeff, const float4* __restrict__ sfilt) {
    constexpr int VPL = Lanes<CV>::VPL, LN = Lanes<CV>::LN;
    float4 w[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i) w[i] = zero4();
    if constexpr (TT == 0) {
        if (ok)
#pragma unroll
            for (int i = 0; i < VPL; ++i) w[i] = pair_weight4(p, ln + i * LN, CV, F, T, bin, coeff, sfilt);
    } else {
#pragma unroll
        for (int t = 0; t < TT; ++t) {
            const int f = __shfl_sync(mask, b.f[t], src);            // out of range: bin 0 with weight 0
            const float c = __shfl_sync(mask, b.c[t], src);
#pragma unroll
            for (int i = 0; i < VPL; ++i) fma4s(w[i], c, sfilt[f * CV + ln + i * LN]);
        }
    }
    if (ok)
#pragma unroll
        for (int i = 0; i < VPL; ++i) fma4(acc[i], scale4(x[i], rn), w[i]);
}

template <int TT, int CV>
__global__ void __launch_bounds__(256, 4)
conv_fwd_coop_kernel(int64_t Np, int64_t Mp, int F, int T, const float4* __restrict__ input,
                     const float4* __restrict__ filter, const int32_t* __restrict__ nnCount,
                     const int32_t* __restrict__ nnIndex, const int32_t* __restrict__ bin, const float* __restrict__ coeff,
                     const int32_t* __restrict__ rowptr, const int32_t* __restrict__ members, float4* __restrict__ output) {
    constexpr int VPL = Lanes<CV>::VPL, LN = Lanes<CV>::LN, U = Lanes<CV>::U;
    extern __shared__ float4 sfilt[];
    for (int i = threadIdx.x; i < F * CV; i += blockDim.x) sfilt[i] = filter[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, ln = lane % LN, gbase = lane - ln;
    const unsigned mask = group_mask<LN>(gbase);
    const int64_t stride = (int64_t)gridDim.x * (blockDim.x / LN);
    for (int64_t o = (int64_t)blockIdx.x * (blockDim.x / LN) + threadIdx.x / LN; o < Mp; o += stride) {
        const int e0 = __ldg(rowptr + o), e1 = __ldg(rowptr + o + 1);
        const float rn = 1.f / (float)__ldg(nnCount + o);
        float4 acc[VPL];
#pragma unroll
        for (int i = 0; i < VPL; ++i) acc[i] = zero4();
        for (int e = e0; e < e1; e += LN) {
            int p_mine = 0, in_mine = -1;
            LaneBins<TT> mybins;
            const bool have = e + ln < e1;
            if (have) {
                p_mine = __ldg(members + e + ln);
                in_mine = __ldg(nnIndex + 2 * (int64_t)p_mine + 1);
            }
            if constexpr (TT != 0) load_bins<TT>(mybins, have, p_mine, F, 0, bin, coeff);
            const int n = e1 - e < LN ? e1 - e : LN;
            for (int j = 0; j < n; j += U) {
                float4 x[U][VPL];
                int pp[U];
                bool ok[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int src = gbase + ((j + u) & (LN - 1));
                    pp[u] = TT == 0 ? __shfl_sync(mask, p_mine, src) : 0;
                    const int in = __shfl_sync(mask, in_mine, src);
                    ok[u] = j + u < n && in >= 0 && in < Np;
#pragma unroll
                    for (int i = 0; i < VPL; ++i) x[u][i] = ok[u] ? ldg4(input + (int64_t)in * CV + ln + i * LN) : zero4();
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    add_pair<TT, CV>(acc, x[u], rn, mybins, pp[u], mask, gbase + ((j + u) & (LN - 1)), ln, ok[u], F, T, bin, coeff, sfilt);
            }
        }
#pragma unroll
        for (int i = 0; i < VPL; ++i) output[o * CV + ln + i * LN] = acc[i];
    }
}

// A group takes W = LN / 4 consecutive input points per step: their pairs are one contiguous run of the grouping,
// and when it fits the group's lanes (the usual case: an input point is the neighbour of a few output points) one
// fetch of the indices serves all W points.
template <int TT, int CV>
__global__ void __launch_bounds__(256, 3)
conv_bwd_input_coop_kernel(int64_t Np, int64_t Mp, int F, int T, const float4* __restrict__ gout,
                           const float4* __restrict__ filter, const int32_t* __restrict__ nnCount,
                           const int32_t* __restrict__ nnIndex, const int32_t* __restrict__ bin,
                           const float* __restrict__ coeff, const int32_t* __restrict__ rowptr,
                           const int32_t* __restrict__ members, int nlong, float4* __restrict__ gin) {
    constexpr int VPL = Lanes<CV>::VPL, LN = Lanes<CV>::LN, U = Lanes<CV>::U, W = LN / 4;
    extern __shared__ float4 sfilt[];
    if ((int)blockIdx.x < nlong) {
        bwd_input_long_rows((int64_t)blockIdx.x * LONG_SCAN, Np, Mp, F, CV, T, gout, filter, nnCount, nnIndex, bin, coeff, rowptr, members,
                            gin, sfilt);
        return;
    }
    for (int i = threadIdx.x; i < F * CV; i += blockDim.x) sfilt[i] = filter[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, ln = lane % LN, gbase = lane - ln;
    const unsigned mask = group_mask<LN>(gbase);
    const int64_t stride = (int64_t)(gridDim.x - nlong) * (blockDim.x / LN) * W;
    for (int64_t base = ((int64_t)(blockIdx.x - nlong) * (blockDim.x / LN) + threadIdx.x / LN) * W; base < Np; base += stride) {
        int rp_mine = 0;
        if (ln <= W) rp_mine = __ldg(rowptr + (base + ln < Np ? base + ln : Np));
        const int E0 = __shfl_sync(mask, rp_mine, gbase), EW = __shfl_sync(mask, rp_mine, gbase + W);
        const bool together = EW - E0 <= LN;
        int p_mine = 0, o_mine = -1;
        float rn_mine = 0.f;
        LaneBins<TT> mybins;
        auto fetch = [&](int e, bool have) {
            p_mine = 0, o_mine = -1, rn_mine = 0.f;
            if (have) p_mine = __ldg(members + e);
            if (have) o_mine = __ldg(nnIndex + 2 * (int64_t)p_mine);
            if constexpr (TT != 0) load_bins<TT>(mybins, have, p_mine, F, 0, bin, coeff);
            if (o_mine >= Mp) o_mine = -1;
            if (o_mine >= 0) rn_mine = 1.f / (float)__ldg(nnCount + o_mine);
        };
        float4 acc[VPL];
        // pairs of the fetched run, slots [j, end)
        auto walk = [&](int j, int end) {
            for (; j < end; j += U) {
                float4 x[U][VPL];
                int pp[U];
                float rn[U];
                bool ok[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int src = gbase + ((j + u) & (LN - 1));
                    pp[u] = TT == 0 ? __shfl_sync(mask, p_mine, src) : 0;
                    const int o = __shfl_sync(mask, o_mine, src);
                    rn[u] = __shfl_sync(mask, rn_mine, src);
                    ok[u] = j + u < end && o >= 0;
#pragma unroll
                    for (int i = 0; i < VPL; ++i) x[u][i] = ok[u] ? ldg4(gout + (int64_t)o * CV + ln + i * LN) : zero4();
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    add_pair<TT, CV>(acc, x[u], rn[u], mybins, pp[u], mask, gbase + ((j + u) & (LN - 1)), ln, ok[u], F, T, bin, coeff, sfilt);
            }
        };
        if (together) fetch(E0 + ln, E0 + ln < EW);
#pragma unroll 1
        for (int k = 0; k < W; ++k) {
            const int e0 = __shfl_sync(mask, rp_mine, gbase + k), e1 = __shfl_sync(mask, rp_mine, gbase + k + 1);
            if (e1 - e0 > LONG_ROW) continue;
#pragma unroll
            for (int i = 0; i < VPL; ++i) acc[i] = zero4();
            if (together) {
                walk(e0 - E0, e1 - E0);
            } else {
                for (int e = e0; e < e1; e += LN) {
                    fetch(e + ln, e + ln < e1);
                    walk(0, e1 - e < LN ? e1 - e : LN);
                }
            }
            if (base + k < Np)
#pragma unroll
                for (int i = 0; i < VPL; ++i) gin[(base + k) * CV + ln + i * LN] = acc[i];
        }
    }
}

// Filter gradient: a block of SUB groups of CV lanes takes a contiguous run of pairs, group g the g-th equal part
// of it, walked in order into the group's own copy of the [F][C] accumulator in shared memory; copies are added in
// group order, blocks in block order.
template <int TT, int CV>
__global__ void __launch_bounds__(256)
conv_bwd_filter_coop_kernel(int64_t Np, int64_t Mp, int64_t Nout, int pairs_per_block, int SUB, int F, int T,
                            const float4* __restrict__ input, const float4* __restrict__ gout,
                            const int32_t* __restrict__ nnCount, const int32_t* __restrict__ nnIndex,
                            const int32_t* __restrict__ bin, const float* __restrict__ coeff, float4* __restrict__ partial) {
    extern __shared__ float4 acc4[];                 // [SUB][F][CV]
    for (int i = threadIdx.x; i < SUB * F * CV; i += blockDim.x) acc4[i] = zero4();
    __syncthreads();
    const int lane = threadIdx.x & 31, cg = lane % CV, gbase = lane - cg, g = threadIdx.x / CV;
    const unsigned mask = group_mask<CV>(gbase);
    const int per_group = (pairs_per_block + SUB - 1) / SUB;
    const int64_t b0 = (int64_t)blockIdx.x * pairs_per_block;
    int64_t b1 = b0 + pairs_per_block;
    if (b1 > Nout) b1 = Nout;
    const int64_t q0 = b0 + (int64_t)g * per_group;
    int64_t q1 = q0 + per_group;
    if (q1 > b1) q1 = b1;
    float4* mine = acc4 + (size_t)g * F * CV;
    for (int64_t q = q0; q < q1; q += CV) {
        int o_mine = -1, in_mine = -1;
        float rn_mine = 0.f;
        LaneBins<TT> mybins;
        const bool have = q + cg < q1;
        if (have) {
            o_mine = __ldg(nnIndex + 2 * (q + cg));
            in_mine = __ldg(nnIndex + 2 * (q + cg) + 1);
        }
        if constexpr (TT != 0) load_bins<TT>(mybins, have, q + cg, F, TT == 3 ? -1 : 0, bin, coeff);
        if (o_mine >= 0 && o_mine < Mp) rn_mine = 1.f / (float)__ldg(nnCount + o_mine);
        const int n = q1 - q < CV ? (int)(q1 - q) : CV;
        for (int j = 0; j < n; j += 4) {
            float4 gr[4], xr[4];
            float rn[4];
            bool ok[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int src = gbase + ((j + u) & (CV - 1));
                const int o = __shfl_sync(mask, o_mine, src);
                const int in = __shfl_sync(mask, in_mine, src);
                rn[u] = __shfl_sync(mask, rn_mine, src);
                ok[u] = j + u < n && o >= 0 && o < Mp && in >= 0 && in < Np;
                gr[u] = ok[u] ? ldg4(gout + (int64_t)o * CV + cg) : zero4();
                xr[u] = ok[u] ? ldg4(input + (int64_t)in * CV + cg) : zero4();
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 d = mul4(scale4(gr[u], rn[u]), xr[u]);
                if constexpr (TT != 0) {
                    const int src = gbase + ((j + u) & (CV - 1));
#pragma unroll
                    for (int t = 0; t < (TT == 3 ? 3 : 1); ++t) {
                        const int f = __shfl_sync(mask, mybins.f[t], src);
                        const float c = __shfl_sync(mask, mybins.c[t], src);
                        if (ok[u] && (TT == 3 ? f >= 0 : c != 0.f)) fma4s(mine[f * CV + cg], c, d);
                    }
                } else if (ok[u]) {
                    const int64_t p = q + j + u;
                    if (!coeff) {
                        const int fb = __ldg(bin + p);
                        if (fb >= 0 && fb < F) add4(mine[fb * CV + cg], d);
                    } else {
                        for (int t = 0; t < T; ++t) {
                            const int fb = __ldg(bin + p * T + t);
                            if (fb >= 0 && fb < F) fma4s(mine[fb * CV + cg], __ldg(coeff + p * T + t), d);
                        }
                    }
                }
            }
        }
    }
    __syncthreads();
    float4* out = partial + (int64_t)blockIdx.x * F * CV;
    for (int i = threadIdx.x; i < F * CV; i += blockDim.x) {
        float4 s4 = acc4[i];
        for (int k = 1; k < SUB; ++k) add4(s4, acc4[(size_t)k * F * CV + i]);
        out[i] = s4;
    }
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
// the vector kernels: depth multiplier 1, channels a multiple of 4 and at most 1024 (one group of lanes per point),
// and a filter table that leaves room in shared memory for at least one accumulator copy
static bool vec_ok(int F, int C, int r) { return r == 1 && C % 4 == 0 && C <= 1024 && (size_t)F * C * 4 <= 48 * 1024; }
// pairs of a filter-gradient block: 2048 (partial tables stay small against the gathers), fewer where that would leave less
// than six blocks per SM to hide the gathers' latency, 256 at least
static int vec_pairs_per_block(int64_t Nout) {
    int64_t n = ceil_div(ceil_div(Nout > 0 ? Nout : 1, 6 * (int64_t)sm_count()), 32) * 32;
    return (int)(n < 256 ? 256 : n > 2048 ? 2048 : n);
}
static int vec_filter_blocks(int64_t Nout) { return (int)ceil_div(Nout > 0 ? Nout : 1, vec_pairs_per_block(Nout)); }
static int vec_sub_groups(int F, int C) {
    int sub = 256 / (C / 4);
    if (sub < 1) sub = 1;
    while (sub > 1 && (size_t)sub * F * C * 4 > 96 * 1024) --sub;
    return sub;
}

// groups of a filter-gradient block: as many accumulator copies as fit 56 KB (four blocks on an SM), whole warps
static int coop_sub_groups(int F, int C) {
    const int CV = C / 4, step = 32 / CV, most = 256 / CV;
    int sub = (int)((56 * 1024) / ((size_t)F * C * 4)) / step * step;
    return sub < step ? step : sub > most ? most : sub;
}
static bool coop_ok(int F, int C) {
    return (C == 32 || C == 64 || C == 128) && (size_t)coop_sub_groups(F, C) * F * C * 4 <= 200 * 1024;
}

template <int TT, int CV>
static int launch_fwd_coop(int64_t Np, int64_t Mp, int F, int T, const float* input, const float* filter, const int32_t* nnCount,
                           const int32_t* nnIndex, const int32_t* bin, const float* coeff, const int32_t* rowptr,
                           const int32_t* members, float* output, cudaStream_t stream) {
    PB_LAUNCH("pcloud_conv_fwd", (conv_fwd_coop_kernel<TT, CV>), persistent_blocks(Mp * Lanes<CV>::LN, 256, 8), 256, sizeof(float4) * F * CV,
              stream, Np, Mp, F, T, (const float4*)input, (const float4*)filter, nnCount, nnIndex, bin, coeff, rowptr, members,
              (float4*)output);
    return PB200_OK;
}

template <int TT, int CV>
static int launch_bwd_coop(int64_t Np, int64_t Mp, int64_t Nout, int nb, int F, int T, const float* input, const float* filter,
                           const float* gout, const int32_t* nnCount, const int32_t* nnIndex, const int32_t* bin,
                           const float* coeff, const int32_t* rowptr, const int32_t* members, float* gin, float* partial,
                           cudaStream_t stream) {
    if (Np > 0) {
        const int nlong = Nout > LONG_ROW ? long_blocks(Np) : 0;
        if (sizeof(float4) * F * CV > UNASKED_TABLE)
            PB_CUDA(cudaFuncSetAttribute(conv_bwd_input_coop_kernel<TT, CV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(sizeof(float4) * F * CV)));
        PB_LAUNCH("pcloud_conv_bwd_input", (conv_bwd_input_coop_kernel<TT, CV>), nlong + persistent_blocks(Np * Lanes<CV>::LN, 256, 8), 256,
                  sizeof(float4) * F * CV, stream, Np, Mp, F, T, (const float4*)gout, (const float4*)filter, nnCount, nnIndex, bin,
                  coeff, rowptr, members, nlong, (float4*)gin);
    }
    const int sub = coop_sub_groups(F, 4 * CV);
    const size_t smem = sizeof(float4) * (size_t)sub * F * CV;
    PB_CUDA(cudaFuncSetAttribute(conv_bwd_filter_coop_kernel<TT, CV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PB_LAUNCH("pcloud_conv_bwd_filter", (conv_bwd_filter_coop_kernel<TT, CV>), nb, sub * CV, smem, stream, Np, Mp, Nout,
              vec_pairs_per_block(Nout), sub, F, T, (const float4*)input, (const float4*)gout, nnCount, nnIndex, bin, coeff,
              (float4*)partial);
    return PB200_OK;
}

// the kernels are built for CV of 8, 16, 32 and for one bin per pair, three weighted bins, or any T
#define PB_COOP_DISPATCH(FN, ...)                                                                                  \
    (tt == 1 ? (CV == 8 ? FN<1, 8>(__VA_ARGS__) : CV == 16 ? FN<1, 16>(__VA_ARGS__) : FN<1, 32>(__VA_ARGS__))      \
     : tt == 3 ? (CV == 8 ? FN<3, 8>(__VA_ARGS__) : CV == 16 ? FN<3, 16>(__VA_ARGS__) : FN<3, 32>(__VA_ARGS__))    \
               : (CV == 8 ? FN<0, 8>(__VA_ARGS__) : CV == 16 ? FN<0, 16>(__VA_ARGS__) : FN<0, 32>(__VA_ARGS__)))

static int filter_blocks(int64_t Nout) {
    int64_t b = ceil_div(Nout > 0 ? Nout : 1, 256);         // at least 256 pairs per block
    const int cap = 4 * sm_count();
    return (int)(b < cap ? b : cap);
}

}  // namespace pcloud
}  // namespace pb

using namespace pb;
using namespace pb::pcloud;

extern "C" {

int pb200_pcloud_conv3d_forward(int64_t Np, int64_t Mp, int64_t Nout, int F, int C, int r, int T, const float* input,
                                const float* filter, const int32_t* nnCount, const int32_t* nnIndex,
                                const int32_t* binIndex, const float* binCoeff, const int32_t* rowptr_out,
                                const int32_t* members_out, float* output, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(sizes_ok(Np, Mp, Nout, F, C, r, T), PB200_EINVAL, "pcloud_conv3d_forward: bad sizes");
    if (Mp == 0) return PB200_OK;
    PB_REQUIRE(filter && nnCount && rowptr_out && output && (Nout == 0 || (input && nnIndex && binIndex && members_out)),
               PB200_EINVAL, "pcloud_conv3d_forward: null pointer");
    if (vec_ok(F, C, r) && aligned16(input) && aligned16(filter) && aligned16(output)) {
        const int CV = C / 4;
        if (coop_ok(F, C)) {
            const int tt = !binCoeff ? 1 : T == 3 ? 3 : 0;
            return PB_COOP_DISPATCH(launch_fwd_coop, Np, Mp, F, T, input, filter, nnCount, nnIndex, binIndex, binCoeff, rowptr_out,
                                    members_out, output, stream);
        }
        PB_LAUNCH("pcloud_conv_fwd", conv_fwd_vec_kernel, persistent_blocks(Mp * CV, 256, 8), 256, sizeof(float) * F * C, stream,
                  Np, Mp, F, CV, T, (const float4*)input, (const float4*)filter, nnCount, nnIndex, binIndex, binCoeff, rowptr_out,
                  members_out, (float4*)output);
        return PB200_OK;
    }
    PB_LAUNCH("pcloud_conv_fwd", conv_fwd_kernel, persistent_blocks(Mp * C * r, 256, 16), 256, 0, stream, Np, Mp, F, C, r, T,
              input, filter, nnCount, nnIndex, binIndex, binCoeff, rowptr_out, members_out, output);
    return PB200_OK;
}

size_t pb200_pcloud_conv3d_backward_workspace_bytes(int64_t Nout, int F, int C, int r) {
    if (Nout < 0 || F <= 0 || C <= 0 || r <= 0) return 0;
    const size_t nb = vec_ok(F, C, r) && vec_filter_blocks(Nout) > filter_blocks(Nout) ? vec_filter_blocks(Nout) : filter_blocks(Nout);
    return align_up(nb * F * C * r * sizeof(float), 256);
}

int pb200_pcloud_conv3d_backward(int64_t Np, int64_t Mp, int64_t Nout, int F, int C, int r, int T, const float* gradOutput,
                                 const float* input, const float* filter, const int32_t* nnCount, const int32_t* nnIndex,
                                 const int32_t* binIndex, const float* binCoeff, const int32_t* rowptr_in,
                                 const int32_t* members_in, float* gradInput, float* gradFilter, void* workspace,
                                 size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(sizes_ok(Np, Mp, Nout, F, C, r, T), PB200_EINVAL, "pcloud_conv3d_backward: bad sizes");
    PB_REQUIRE(gradFilter && filter && (Np == 0 || (gradInput && rowptr_in)), PB200_EINVAL,
               "pcloud_conv3d_backward: null pointer");
    PB_REQUIRE(Nout == 0 || (gradOutput && input && nnCount && nnIndex && binIndex && members_in), PB200_EINVAL,
               "pcloud_conv3d_backward: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_pcloud_conv3d_backward_workspace_bytes(Nout, F, C, r), PB200_EWORKSPACE,
               "pcloud_conv3d_backward: workspace too small");
    if (vec_ok(F, C, r) && aligned16(input) && aligned16(filter) && aligned16(gradOutput) && aligned16(gradInput) &&
        aligned16(workspace)) {
        const int CV = C / 4;
        if (coop_ok(F, C)) {
            const int nbc = vec_filter_blocks(Nout);
            const int tt = !binCoeff ? 1 : T == 3 ? 3 : 0;
            const int rc = PB_COOP_DISPATCH(launch_bwd_coop, Np, Mp, Nout, nbc, F, T, input, filter, gradOutput, nnCount, nnIndex,
                                            binIndex, binCoeff, rowptr_in, members_in, gradInput, (float*)workspace, stream);
            if (rc != PB200_OK) return rc;
            return reduce_partials((const float*)workspace, nbc, (int64_t)F * C, gradFilter, stream);
        }
        if (Np > 0) {
            const int nlong = Nout > LONG_ROW ? long_blocks(Np) : 0;
            if (sizeof(float) * F * C > UNASKED_TABLE)
                PB_CUDA(cudaFuncSetAttribute(conv_bwd_input_vec_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(sizeof(float) * F * C)));
            PB_LAUNCH("pcloud_conv_bwd_input", conv_bwd_input_vec_kernel, nlong + persistent_blocks(Np * CV, 256, 8), 256,
                      sizeof(float) * F * C, stream, Np, Mp, F, CV, T, (const float4*)gradOutput, (const float4*)filter, nnCount,
                      nnIndex, binIndex, binCoeff, rowptr_in, members_in, nlong, (float4*)gradInput);
        }
        const int nbv = vec_filter_blocks(Nout), sub = vec_sub_groups(F, C);
        const size_t smemv = sizeof(float) * (size_t)sub * F * C;
        const int threads = sub * CV < 32 ? 32 : ((sub * CV + 31) / 32) * 32;
        PB_CUDA(cudaFuncSetAttribute(conv_bwd_filter_vec_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemv));
        PB_LAUNCH("pcloud_conv_bwd_filter", conv_bwd_filter_vec_kernel, nbv, threads, smemv, stream, Np, Mp, Nout,
                  vec_pairs_per_block(Nout), F, CV, T, sub, (const float4*)input, (const float4*)gradOutput, nnCount, nnIndex, binIndex,
                  binCoeff, (float4*)workspace);
        return reduce_partials((const float*)workspace, nbv, (int64_t)F * C, gradFilter, stream);
    }
    if (Np > 0)
        PB_LAUNCH("pcloud_conv_bwd_input", conv_bwd_input_kernel, persistent_blocks(Np * C, 256, 16), 256, 0, stream, Np, Mp,
                  F, C, r, T, gradOutput, filter, nnCount, nnIndex, binIndex, binCoeff, rowptr_in, members_in, gradInput);
    const int nb = filter_blocks(Nout);
    const int Cr = C * r;
    const int threads = Cr >= 256 ? 256 : ((Cr + 31) / 32) * 32;
    const size_t smem = sizeof(float) * (size_t)F * Cr;
    PB_CUDA(cudaFuncSetAttribute(conv_bwd_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PB_LAUNCH("pcloud_conv_bwd_filter", conv_bwd_filter_kernel, nb, threads, smem, stream, Np, Mp, Nout,
              ceil_div(Nout > 0 ? Nout : 1, nb), F, C, r, T, input, gradOutput, nnCount, nnIndex, binIndex, binCoeff,
              (float*)workspace);
    return reduce_partials((const float*)workspace, nb, (int64_t)F * Cr, gradFilter, stream);
}

}  // extern "C"
