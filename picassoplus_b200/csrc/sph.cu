// Spherical-harmonic basis of (N,3) cartesian points: projection to the unit sphere,
// azimuth / polar angles, and the (L+1)^2 real components in the reference's column
// order (per degree l: cos(m*phi) terms m = l..1, the m = 0 term, sin(m*phi) terms
// m = l..1), L <= 5.  One thread per point; the K outputs are staged through shared
// memory so the global store is coalesced.
#include "common.cuh"
#include "sph_core.cuh"

namespace pb {

template <int L>
__global__ void __launch_bounds__(SPH_BLOCK)
sph_harm_kernel(int64_t N, const float* __restrict__ xyz, SphConst cst, float* __restrict__ out, bool vec) {
    constexpr int K = (L + 1) * (L + 1);
    __shared__ __align__(16) float stage[SPH_BLOCK * sph_pitch<K>];
    const int64_t base = (int64_t)blockIdx.x * SPH_BLOCK;
    const int64_t i = base + threadIdx.x;
    if (i < N) {
        float o[K];
        sph_eval(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], L, cst.c, o);
        put_row<K>(stage, o);
    }
    __syncthreads();
    write_rows<K>(stage, (int)(N - base < SPH_BLOCK ? N - base : SPH_BLOCK), out + base * K, vec);
}

// out[f] = mean over the samples k of face f of the components of xyz[k] (0 for a face without samples): the two
// steps sph_harm + per-face mean of the rows in one pass, without the (samples, K) array in between.  A thread walks
// its face's samples in ascending order and adds each evaluation to its sums, so the result has the
// bits of the two-step path.
template <int L>
__global__ void __launch_bounds__(SPH_BLOCK)
face_mean_sph_harm_kernel(int64_t Nf, int64_t NiK, const float* __restrict__ xyz, const int32_t* __restrict__ cum,
                          SphConst cst, float* __restrict__ out, bool vec) {
    constexpr int K = (L + 1) * (L + 1);
    __shared__ __align__(16) float stage[SPH_BLOCK * sph_pitch<K>];
    const int64_t base = (int64_t)blockIdx.x * SPH_BLOCK;
    const int64_t f = base + threadIdx.x;
    if (f < Nf) {
        int64_t k0 = f > 0 ? cum[f - 1] : 0, k1 = cum[f];
        if (k0 < 0) k0 = 0;
        if (k1 > NiK) k1 = NiK;
        float acc[K];
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] = 0.f;
        for (int64_t i = k0; i < k1; ++i) {
            float one[K];
            sph_eval(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], L, cst.c, one);
#pragma unroll
            for (int k = 0; k < K; ++k) acc[k] = __fadd_rn(acc[k], one[k]);        // not contracted with a component's last product
        }
        const float inv = k1 > k0 ? 1.f / (float)(k1 - k0) : 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k) acc[k] *= inv;
        put_row<K>(stage, acc);
    }
    __syncthreads();
    write_rows<K>(stage, (int)(Nf - base < SPH_BLOCK ? Nf - base : SPH_BLOCK), out + base * K, vec);
}

// The three-row vertex2facet filter of a layer, corners (3,K) @ weights (K,C), and its gradient corners^T @ gradFilter:
// K <= 36 terms, a few thousand results.  Both are one short launch; as library GEMMs they were two of the step's
// larger host costs.
__global__ void corner_filter_kernel(int K, int C, const float* __restrict__ corners, const float* __restrict__ weights,
                                     float* __restrict__ filter) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * C) return;
    const int j = i / C, c = i - j * C;
    float acc = 0.f;
    for (int k = 0; k < K; ++k) acc = fmaf(__ldg(corners + j * K + k), __ldg(weights + (int64_t)k * C + c), acc);
    filter[i] = acc;
}

__global__ void corner_filter_bwd_kernel(int K, int C, const float* __restrict__ corners, const float* __restrict__ gfilter,
                                         float* __restrict__ gweights) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= K * C) return;
    const int k = i / C, c = i - k * C;
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 3; ++j) acc = fmaf(__ldg(corners + j * K + k), __ldg(gfilter + j * C + c), acc);
    gweights[i] = acc;
}

}  // namespace pb

using namespace pb;

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

extern "C" int pb200_corner_filter(int K, int C, const float* corners, const float* weights, float* filter, void* stream) {
    PB_REQUIRE(K > 0 && C > 0 && K <= (1 << 15) && C <= (1 << 15), PB200_EINVAL, "corner_filter: bad sizes");
    PB_REQUIRE(corners && weights && filter, PB200_EINVAL, "corner_filter: null pointer");
    PB_LAUNCH("corner_filter", corner_filter_kernel, (unsigned)ceil_div(3 * C, 128), 128, 0, (cudaStream_t)stream, K, C, corners,
              weights, filter);
    return PB200_OK;
}

extern "C" int pb200_corner_filter_backward(int K, int C, const float* corners, const float* gradFilter, float* gradWeights,
                                            void* stream) {
    PB_REQUIRE(K > 0 && C > 0 && K <= (1 << 15) && C <= (1 << 15), PB200_EINVAL, "corner_filter_backward: bad sizes");
    PB_REQUIRE(corners && gradFilter && gradWeights, PB200_EINVAL, "corner_filter_backward: null pointer");
    PB_LAUNCH("corner_filter_bwd", corner_filter_bwd_kernel, (unsigned)ceil_div(K * C, 128), 128, 0, (cudaStream_t)stream, K, C,
              corners, gradFilter, gradWeights);
    return PB200_OK;
}

extern "C" int pb200_face_mean_sph_harm(int64_t Nf, int64_t NiK, int L, const float* xyz, const int32_t* numInterior,
                                        float* out, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(Nf >= 0 && NiK >= 0, PB200_EINVAL, "face_mean_sph_harm: bad size");
    PB_REQUIRE(L >= 0 && L <= 5, PB200_EINVAL, "face_mean_sph_harm: degree L=%d not supported (0..5)", L);
    if (Nf == 0) return PB200_OK;
    PB_REQUIRE(numInterior && out && (NiK == 0 || xyz), PB200_EINVAL, "face_mean_sph_harm: null pointer");
    static const SphConst cst = make_sph_const();
    PB_DISPATCH_DEGREE(L, PB_LAUNCH("face_mean_sph_harm", face_mean_sph_harm_kernel<DEG>, (unsigned)ceil_div(Nf, SPH_BLOCK), SPH_BLOCK, 0,
                                    stream, Nf, NiK, xyz, numInterior, cst, out, aligned16(out)));
    return PB200_OK;
}

extern "C" int pb200_sph_harm_coeff(int64_t N, int L, const float* xyz, float* out, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(N >= 0, PB200_EINVAL, "sph_harm_coeff: bad size");
    PB_REQUIRE(L >= 0 && L <= 5, PB200_EINVAL, "sph_harm_coeff: degree L=%d not supported (0..5)", L);
    if (N == 0) return PB200_OK;
    PB_REQUIRE(xyz && out, PB200_EINVAL, "sph_harm_coeff: null pointer");
    static const SphConst cst = make_sph_const();
    PB_DISPATCH_DEGREE(L, PB_LAUNCH("sph_harm", sph_harm_kernel<DEG>, (unsigned)ceil_div(N, SPH_BLOCK), SPH_BLOCK, 0, stream, N, xyz, cst,
                                    out, aligned16(out)));
    return PB200_OK;
}
