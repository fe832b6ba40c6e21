// out (M, N) = A^T (M, rows) @ B (rows, N) in fp32 FFMA: the weight gradient of a product whose operands may not be rounded
// (the point-cloud layer).  The library's fp32 GEMM gives this shape (a contraction over 10^4..10^6 rows into a matrix of at
// most a few 64 x 64 tiles) to a handful of blocks: 141 us for 65 537 rows, 64 x 64, where the operands' bytes take 5 us and the
// multiply-adds 8.  Here the rows are split over enough blocks for two per SM; a block keeps its 64 x 64 tile in registers
// (4 x 4 per thread) and stages 16 rows at a time in shared memory, the next 16 on their way in registers; the partial tiles are
// added in block order.
#include "common.cuh"

namespace pb {
namespace rcf {

constexpr int TM = 64, TN = 64, RK = 16;
constexpr int MIN_ROWS = 128;                    // fewer rows per block cost more in partial tiles than they gain

static int splits(int64_t rows, int M, int N) {
    const int64_t tiles = ceil_div(M, TM) * ceil_div(N, TN);
    int64_t s = ceil_div(2 * (int64_t)sm_count(), tiles);
    const int64_t most = ceil_div(rows > 0 ? rows : 1, MIN_ROWS);
    return (int)(s < most ? s : most);
}

template <bool VEC>
__global__ void __launch_bounds__(256)
contract_kernel(int64_t rows, int M, int N, int64_t per, const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ partial) {
    __shared__ float4 sa[2][RK][TM / 4], sb[2][RK][TN / 4];
    const int m0 = blockIdx.y * TM, n0 = blockIdx.z * TN;
    const int64_t r0 = (int64_t)blockIdx.x * per, r1 = r0 + per < rows ? r0 + per : rows;
    const int lr = threadIdx.x >> 4, lc = threadIdx.x & 15;              // staged row and group of four columns
    const int tm = threadIdx.x >> 4, tn = threadIdx.x & 15;              // this thread's four rows / columns of the tile
    auto fetch = [&](const float* X, int W, int c0, int64_t r) -> float4 {
        const int c = c0 + 4 * lc;
        if (r >= r1 || c >= W) return zero4();
        const float* p = X + r * W + c;
        if (VEC) return ldg4(reinterpret_cast<const float4*>(p));
        return make_float4(__ldg(p), c + 1 < W ? __ldg(p + 1) : 0.f, c + 2 < W ? __ldg(p + 2) : 0.f, c + 3 < W ? __ldg(p + 3) : 0.f);
    };
    float4 acc[4] = {zero4(), zero4(), zero4(), zero4()};
    float4 a = fetch(A, M, m0, r0 + lr), b = fetch(B, N, n0, r0 + lr);
    int buf = 0;
    for (int64_t r = r0; r < r1; r += RK, buf ^= 1) {
        sa[buf][lr][lc] = a;
        sb[buf][lr][lc] = b;
        __syncthreads();
        a = fetch(A, M, m0, r + RK + lr);
        b = fetch(B, N, n0, r + RK + lr);
#pragma unroll
        for (int k = 0; k < RK; ++k) {
            const float4 x = sa[buf][k][tm], y = sb[buf][k][tn];
            fma4s(acc[0], x.x, y); fma4s(acc[1], x.y, y); fma4s(acc[2], x.z, y); fma4s(acc[3], x.w, y);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + 4 * tm + i;
        if (m >= M) continue;
        float* o = partial + ((int64_t)blockIdx.x * M + m) * N + n0 + 4 * tn;
        const float v[4] = {acc[i].x, acc[i].y, acc[i].z, acc[i].w};
        for (int j = 0; j < 4; ++j)
            if (n0 + 4 * tn + j < N) o[j] = v[j];
    }
}

}  // namespace rcf
}  // namespace pb

using namespace pb;

extern "C" {

size_t pb200_rows_contract_f32_workspace_bytes(int64_t rows, int M, int N) {
    if (rows < 0 || M <= 0 || N <= 0) return 0;
    return align_up(sizeof(float) * (size_t)rcf::splits(rows, M, N) * M * N, 256);
}

int pb200_rows_contract_f32(int64_t rows, int M, int N, const float* A, const float* B, float* out, void* workspace, size_t workspace_bytes,
                            void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(rows >= 0 && M > 0 && N > 0 && M <= 65535 * rcf::TM && N <= 65535 * rcf::TN, PB200_EINVAL, "rows_contract_f32: bad sizes");
    PB_REQUIRE(out && (rows == 0 || (A && B)), PB200_EINVAL, "rows_contract_f32: null pointer");
    if (rows == 0) {
        PB_CUDA(cudaMemsetAsync(out, 0, sizeof(float) * (size_t)M * N, stream));
        return PB200_OK;
    }
    PB_REQUIRE(workspace && workspace_bytes >= pb200_rows_contract_f32_workspace_bytes(rows, M, N), PB200_EWORKSPACE,
               "rows_contract_f32: workspace too small");
    const int s = rcf::splits(rows, M, N);
    const int64_t per = ceil_div(ceil_div(rows, s), rcf::RK) * rcf::RK;
    const int used = (int)ceil_div(rows, per);
    const bool vec = M % 4 == 0 && N % 4 == 0 && ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) == 0;
    const dim3 grid(used, (unsigned)ceil_div(M, rcf::TM), (unsigned)ceil_div(N, rcf::TN));
    float* partial = (float*)workspace;
    if (vec) PB_LAUNCH("rows_contract_f32", rcf::contract_kernel<true>, grid, 256, 0, stream, rows, M, N, per, A, B, partial);
    else PB_LAUNCH("rows_contract_f32", rcf::contract_kernel<false>, grid, 256, 0, stream, rows, M, N, per, A, B, partial);
    return reduce_partials(partial, used, (int64_t)M * N, out, stream);
}

}  // extern "C"
