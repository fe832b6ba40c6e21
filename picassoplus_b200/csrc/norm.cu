// Batch normalisation of feature rows (N, C) behind the pointwise stage of the layers (activation first, then
// normalisation, as the reference's modules order them: picasso/mesh/layers.py:117-120), forward and backward, and the
// mean over the rows of every sample of a batch.
//
// All of it is memory traffic: a row array is 4*N*C bytes and nothing is computed per value beyond a few FMAs.  What
// counts is how often the rows are read and written.  As separate passes (statistics, transform; reduction, element-wise
// gradient) a layer moves 8 row arrays; here the element-wise gradient is formed by its consumer while it loads
// (pointwise_tc.cu, MODE 2: 3 arrays less), and behind facet2facet, bias, activation and statistics are one pass (4 less).
//
// Behind the vertex layers the statistics come from torch (at::batch_norm_update_stats), and norm_apply repeats torch's
// rounding, so that a stack of layers reproduces nn.BatchNorm1d's activations bit for bit.  Statistics taken in the
// producing kernel's epilogue were correct to 1e-7 and saved another 9 % of a scene encoder's step, but the next layer's
// operands keep 16 bits and ReLU and max pooling decide on the sign of what results: after three levels the gradients
// differed by 1e-2 from those of the separate modules.  Left out for that.
//
// Statistics made here are (count, mean, sum of squared deviations) triples, merged pairwise in a fixed order: no cancellation
// however large the mean is against the deviation, and the same bits on every run.
//
// Layout: a team of TL = min(32, C/V) threads takes a row, a thread V = 4 (16-byte loads, C % 4 == 0 and aligned rows)
// or 1 channels of it; four rows of a thread are in flight; gridDim.y walks chunks of 32 thread columns.
#include "common.cuh"
#include "moments.cuh"

namespace pb {
namespace norm {

template <int V> struct Vec { float v[V]; };
template <int V> __device__ __forceinline__ Vec<V> load(const float* p) {
    Vec<V> r;
    if (V == 4) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        r.v[0] = t.x; r.v[1 % V] = t.y; r.v[2 % V] = t.z; r.v[3 % V] = t.w;
    } else {
        r.v[0] = *p;
    }
    return r;
}
template <int V> __device__ __forceinline__ void store(float* p, const Vec<V>& x) {
    if (V == 4) *reinterpret_cast<float4*>(p) = make_float4(x.v[0], x.v[1 % V], x.v[2 % V], x.v[3 % V]);
    else *p = x.v[0];
}

constexpr int THREADS = 256;
constexpr int UNROLL = 4;

// rows <- act(rows + bias) in place; partial[block][3][C] = (count, mean, M2) of the block's results
template <int V, int TL>
__global__ void __launch_bounds__(THREADS)
stats_kernel(int64_t N, int C, float* __restrict__ rows, const float* __restrict__ bias, int relu, float* __restrict__ partial) {
    constexpr int TEAMS = THREADS / TL;
    __shared__ Moments red[TEAMS][TL][V];
    const int lane = threadIdx.x % TL, team = threadIdx.x / TL;
    const int c = (blockIdx.y * 32 + lane) * V;
    const bool active = c < C;
    float shift[V], s1[V], s2[V], b[V];
    int64_t n = 0;
#pragma unroll
    for (int j = 0; j < V; ++j) { shift[j] = s1[j] = s2[j] = 0.f; b[j] = active && bias ? bias[c + j] : 0.f; }
    if (active) {
        const int64_t step = (int64_t)gridDim.x * TEAMS;
        auto take = [&](Vec<V> x, int64_t r) {
#pragma unroll
            for (int j = 0; j < V; ++j) { x.v[j] += b[j]; if (relu) x.v[j] = relu_of(x.v[j]); }
            store<V>(rows + r * C + c, x);
            if (n == 0)
#pragma unroll
                for (int j = 0; j < V; ++j) shift[j] = x.v[j];
            ++n;
#pragma unroll
            for (int j = 0; j < V; ++j) { const float d = x.v[j] - shift[j]; s1[j] += d; s2[j] = fmaf(d, d, s2[j]); }
        };
        int64_t r = (int64_t)blockIdx.x * TEAMS + team;
        for (; r + (UNROLL - 1) * step < N; r += UNROLL * step) {
            Vec<V> x[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) x[u] = load<V>(rows + (r + u * step) * C + c);
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) take(x[u], r + u * step);
        }
        for (; r < N; r += step) take(load<V>(rows + r * C + c), r);
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
        red[team][lane][j] = moments((float)n, shift[j], s1[j], s2[j]);
    }
    __syncthreads();
    if (team == 0 && active) {
#pragma unroll
        for (int j = 0; j < V; ++j) {
            Moments m = red[0][lane][j];
#pragma unroll 1
            for (int t = 1; t < TEAMS; ++t) merge(m, red[t][lane][j]);
            float* p = partial + (int64_t)blockIdx.x * 3 * C + c + j;
            p[0] = m.n; p[C] = m.mean; p[2 * C] = m.m2;
        }
    }
}

// Merges the partials of every channel: 32 slices side by side, then the slices pairwise.  Writes what the transform and
// the backward pass need and moves the running statistics (unbiased variance, as torch's batch norm does).
constexpr int FS = 32;
__global__ void __launch_bounds__(32 * FS)
finalize_kernel(int nparts, int C, const float* __restrict__ partial, float eps, float momentum,
                float* __restrict__ running_mean, float* __restrict__ running_var, int64_t* __restrict__ batches,
                float* __restrict__ mean, float* __restrict__ invstd) {
    __shared__ Moments red[FS][32];
    const int c = blockIdx.x * 32 + threadIdx.x, y = threadIdx.y;
    const int per = (nparts + FS - 1) / FS;
    Moments m{0.f, 0.f, 0.f};
    if (c < C) {
        const int end = nparts < (y + 1) * per ? nparts : (y + 1) * per;
#pragma unroll 4
        for (int b = y * per; b < end; ++b) {
            const float* p = partial + (int64_t)b * 3 * C + c;
            merge(m, Moments{p[0], p[C], p[2 * C]});
        }
    }
    red[y][threadIdx.x] = m;
#pragma unroll
    for (int h = FS / 2; h > 0; h >>= 1) {
        __syncthreads();
        if (y < h) { merge(m, red[y + h][threadIdx.x]); red[y][threadIdx.x] = m; }
    }
    if (y == 0 && c < C) {
        const float var = m.m2 / m.n;
        mean[c] = m.mean;
        invstd[c] = rsqrtf(var + eps);
        if (running_mean) {
            running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * m.mean;
            running_var[c] = (1.f - momentum) * running_var[c] + momentum * (m.m2 / (m.n - 1.f));
        }
        if (c == 0 && batches) *batches += 1;
    }
}

__global__ void invstd_kernel(int C, const float* __restrict__ var, float eps, int64_t* __restrict__ batches, float* __restrict__ invstd) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < C) invstd[c] = rsqrtf(var[c] + eps);
    if (c == 0 && batches) *batches += 1;
}

template <int V, int TL>
__global__ void __launch_bounds__(THREADS)
apply_kernel(int64_t N, int C, const float* __restrict__ act, const float* __restrict__ mean, const float* __restrict__ invstd,
             const float* __restrict__ gamma, const float* __restrict__ beta, float* __restrict__ out) {
    constexpr int TEAMS = THREADS / TL;
    const int lane = threadIdx.x % TL, team = threadIdx.x / TL;
    const int c = (blockIdx.y * 32 + lane) * V;
    if (c >= C) return;
    float m[V], w[V], k[V], b[V];
#pragma unroll
    for (int j = 0; j < V; ++j) {
        m[j] = mean[c + j]; k[j] = invstd[c + j]; w[j] = gamma ? gamma[c + j] : 1.f; b[j] = beta ? beta[c + j] : 0.f;
    }
    const int64_t step = (int64_t)gridDim.x * TEAMS;
    auto put = [&](Vec<V> x, int64_t r) {
#pragma unroll
        for (int j = 0; j < V; ++j) x.v[j] = fmaf(w[j] * (x.v[j] - m[j]), k[j], b[j]);
        store<V>(out + r * C + c, x);
    };
    int64_t r = (int64_t)blockIdx.x * TEAMS + team;
    for (; r + (UNROLL - 1) * step < N; r += UNROLL * step) {
        Vec<V> x[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) x[u] = load<V>(act + (r + u * step) * C + c);
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) put(x[u], r + u * step);
    }
    for (; r < N; r += step) put(load<V>(act + r * C + c), r);
}

// partial[block][2][C] = sums of g and of g * (act - mean) over the block's rows
template <int V, int TL>
__global__ void __launch_bounds__(THREADS)
bwd_reduce_kernel(int64_t N, int C, const float* __restrict__ g, const float* __restrict__ act, const float* __restrict__ mean,
                  float* __restrict__ partial) {
    constexpr int TEAMS = THREADS / TL;
    __shared__ float red[2][TEAMS][TL][V];
    const int lane = threadIdx.x % TL, team = threadIdx.x / TL;
    const int c = (blockIdx.y * 32 + lane) * V;
    const bool active = c < C;
    float sg[V], sx[V], m[V];
#pragma unroll
    for (int j = 0; j < V; ++j) { sg[j] = sx[j] = 0.f; m[j] = active ? mean[c + j] : 0.f; }
    if (active) {
        const int64_t step = (int64_t)gridDim.x * TEAMS;
        auto take = [&](const Vec<V>& a, const Vec<V>& x) {
#pragma unroll
            for (int j = 0; j < V; ++j) { sg[j] += a.v[j]; sx[j] = fmaf(a.v[j], x.v[j] - m[j], sx[j]); }
        };
        int64_t r = (int64_t)blockIdx.x * TEAMS + team;
        for (; r + (UNROLL - 1) * step < N; r += UNROLL * step) {
            Vec<V> a[UNROLL], x[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) { a[u] = load<V>(g + (r + u * step) * C + c); x[u] = load<V>(act + (r + u * step) * C + c); }
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) take(a[u], x[u]);
        }
        for (; r < N; r += step) take(load<V>(g + r * C + c), load<V>(act + r * C + c));
    }
#pragma unroll
    for (int j = 0; j < V; ++j) { red[0][team][lane][j] = sg[j]; red[1][team][lane][j] = sx[j]; }
    __syncthreads();
    if (team == 0 && active) {
#pragma unroll
        for (int j = 0; j < V; ++j) {
            float a = sg[j], x = sx[j];
#pragma unroll 1
            for (int t = 1; t < TEAMS; ++t) { a += red[0][t][lane][j]; x += red[1][t][lane][j]; }
            float* p = partial + (int64_t)blockIdx.x * 2 * C + c + j;
            p[0] = a; p[C] = x;
        }
    }
}

// gradAct = scale * g + k2 * (act - mean) + k1, with k1 = -scale * sum(g) / N, k2 = -scale * invstd^2 * sum(g (act - mean)) / N
__global__ void __launch_bounds__(32 * FS)
bwd_finalize_kernel(int nparts, int64_t N, int C, const float* __restrict__ partial, const float* __restrict__ invstd,
                    const float* __restrict__ gamma, float* __restrict__ ggamma, float* __restrict__ gbeta,
                    float* __restrict__ scale, float* __restrict__ k1, float* __restrict__ k2) {
    __shared__ float red[2][FS][32];
    const int c = blockIdx.x * 32 + threadIdx.x, y = threadIdx.y;
    const int per = (nparts + FS - 1) / FS;
    float a = 0.f, x = 0.f;
    if (c < C)
        for (int b = y * per; b < nparts && b < (y + 1) * per; ++b) {
            const float* p = partial + (int64_t)b * 2 * C + c;
            a += p[0]; x += p[C];
        }
    red[0][y][threadIdx.x] = a;
    red[1][y][threadIdx.x] = x;
    __syncthreads();
    if (y == 0 && c < C) {
        for (int k = 1; k < FS; ++k) { a += red[0][k][threadIdx.x]; x += red[1][k][threadIdx.x]; }
        const float is = invstd[c], s = gamma ? gamma[c] * is : is, inv = 1.f / (float)N;
        if (ggamma) ggamma[c] = x * is;
        if (gbeta) gbeta[c] = a;
        scale[c] = s;
        k1[c] = -s * a * inv;
        k2[c] = -s * is * is * x * inv;
    }
}

// gm = gradAct (as above; without statistics: g) where the activation let the value through, and partial[block][C] = its
// column sums (the bias gradient).  For layers whose consumer cannot form gm on the fly.
template <int V, int TL, bool BN>
__global__ void __launch_bounds__(THREADS)
bwd_apply_kernel(int64_t N, int C, const float* __restrict__ g, const float* __restrict__ act, const float* __restrict__ mean,
                 const float* __restrict__ scale, const float* __restrict__ k1, const float* __restrict__ k2, int relu,
                 float* __restrict__ gm, float* __restrict__ partial) {
    constexpr int TEAMS = THREADS / TL;
    __shared__ float red[TEAMS][TL][V];
    const int lane = threadIdx.x % TL, team = threadIdx.x / TL;
    const int c = (blockIdx.y * 32 + lane) * V;
    const bool active = c < C;
    float m[V], s[V], a1[V], a2[V], sum[V];
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const bool on = BN && active;
        m[j] = on ? mean[c + j] : 0.f; s[j] = on ? scale[c + j] : 1.f; a1[j] = on ? k1[c + j] : 0.f; a2[j] = on ? k2[c + j] : 0.f;
        sum[j] = 0.f;
    }
    if (active) {
        const int64_t step = (int64_t)gridDim.x * TEAMS;
        auto put = [&](Vec<V> d, const Vec<V>& x, int64_t r) {
#pragma unroll
            for (int j = 0; j < V; ++j) {
                if (BN) d.v[j] = fmaf(s[j], d.v[j], fmaf(a2[j], x.v[j] - m[j], a1[j]));
                if (relu) d.v[j] = relu_grad(d.v[j], x.v[j]);
                sum[j] += d.v[j];
            }
            store<V>(gm + r * C + c, d);
        };
        int64_t r = (int64_t)blockIdx.x * TEAMS + team;
        for (; r + (UNROLL - 1) * step < N; r += UNROLL * step) {
            Vec<V> d[UNROLL], x[UNROLL];
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) { d[u] = load<V>(g + (r + u * step) * C + c); x[u] = load<V>(act + (r + u * step) * C + c); }
#pragma unroll
            for (int u = 0; u < UNROLL; ++u) put(d[u], x[u], r + u * step);
        }
        for (; r < N; r += step) put(load<V>(g + r * C + c), load<V>(act + r * C + c), r);
    }
#pragma unroll
    for (int j = 0; j < V; ++j) red[team][lane][j] = sum[j];
    __syncthreads();
    if (team == 0 && active) {
#pragma unroll
        for (int j = 0; j < V; ++j) {
            float a = sum[j];
#pragma unroll 1
            for (int t = 1; t < TEAMS; ++t) a += red[t][lane][j];
            partial[(int64_t)blockIdx.x * C + c + j] = a;
        }
    }
}

struct Geom { int V, TL, grid, chunks; };
static Geom geom(int64_t N, int C, bool vec) {
    Geom g;
    g.V = vec ? 4 : 1;
    const int cols = C / g.V;
    g.TL = pow2_ceil(cols < 32 ? cols : 32);
    g.chunks = (int)ceil_div(cols, 32);
    g.grid = persistent_blocks(N > 0 ? N : 1, (THREADS / g.TL) * 8, 4);        // at least eight rows per thread, four blocks per SM
    return g;
}
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

#define NORM_DISPATCH(g, ...)                                                            \
    if ((g).V == 4) { constexpr int V = 4; PB_DISPATCH_TL((g).TL, __VA_ARGS__) }         \
    else { constexpr int V = 1; PB_DISPATCH_TL((g).TL, __VA_ARGS__) }

// ---- mean over the rows of every sample (rows of a sample are consecutive) --------------------------------------
// Two stages so that one sample of a million rows fills the chip as well as a thousand samples of a hundred: blocks own
// equal runs of rows, add up the piece of each sample inside their run, and a block per (sample, 128 channels) adds the
// pieces in order.  A piece is named by its first block, so the second stage finds it by division.
constexpr int SEG_ROWS = 512;

__global__ void __launch_bounds__(256)
segment_pieces_kernel(int64_t N, int C, int B, const int64_t* __restrict__ ends, const float* __restrict__ rows,
                      float* __restrict__ pieces) {
    // piece (block, sample): at row block + sample, which no other pair with a common row shares (both only grow)
    const int64_t r0 = (int64_t)blockIdx.x * SEG_ROWS, r1 = r0 + SEG_ROWS < N ? r0 + SEG_ROWS : N;
    __shared__ float red[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int lo = 0, hi = B;                                        // first sample that ends behind r0
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (ends[mid] > r0) hi = mid; else lo = mid + 1; }
    const int c = blockIdx.y * 32 + lane;
    int64_t r = r0;
    for (int s = lo; s < B && r < r1; ++s) {
        const int64_t e = ends[s] < r1 ? ends[s] : r1;
        float a = 0.f;
        if (c < C) {
            int64_t i = r + warp;
            for (; i + 24 < e; i += 32) {
                const float v0 = rows[i * C + c], v1 = rows[(i + 8) * C + c], v2 = rows[(i + 16) * C + c], v3 = rows[(i + 24) * C + c];
                a += v0; a += v1; a += v2; a += v3;
            }
            for (; i < e; i += 8) a += rows[i * C + c];
        }
        red[warp][lane] = a;
        __syncthreads();
        if (warp == 0 && c < C && e > r) {
            for (int w = 1; w < 8; ++w) a += red[w][lane];
            pieces[((int64_t)blockIdx.x + s) * C + c] = a;
        }
        __syncthreads();
        if (e > r) r = e;
    }
}

__global__ void __launch_bounds__(32 * 8)
segment_finish_kernel(int64_t N, int C, int B, const int64_t* __restrict__ ends, const float* __restrict__ pieces, float* __restrict__ out) {
    __shared__ float red[8][32];
    const int s = blockIdx.x, c = blockIdx.y * 32 + threadIdx.x;
    // with deferred validation the ends may be anything yet: pieces exist for rows 0 .. N - 1 only
    const int64_t before = s > 0 ? ends[s - 1] : 0, end = ends[s];
    const int64_t b = before < 0 ? 0 : before < N ? before : N, e = end < 0 ? 0 : end < N ? end : N;
    float a = 0.f;
    if (c < C && e > b)
        for (int64_t k = b / SEG_ROWS + threadIdx.y; k <= (e - 1) / SEG_ROWS; k += 8) a += pieces[(k + s) * C + c];
    red[threadIdx.y][threadIdx.x] = a;
    __syncthreads();
    if (threadIdx.y == 0 && c < C) {
        for (int w = 1; w < 8; ++w) a += red[w][threadIdx.x];
        out[(int64_t)s * C + c] = a / (float)(end - before);           // a sample without rows: 0 / 0, as the mean of nothing is
    }
}

__global__ void __launch_bounds__(256)
segment_mean_bwd_kernel(int64_t N, int C, int B, const int64_t* __restrict__ ends, const float* __restrict__ g,
                        float* __restrict__ gin) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t r = (int64_t)blockIdx.x * 8 + warp; r < N; r += (int64_t)gridDim.x * 8) {
        int lo = 0, hi = B;
        while (lo < hi) { const int mid = (lo + hi) >> 1; if (ends[mid] > r) hi = mid; else lo = mid + 1; }
        const float inv = lo < B ? 1.f / (float)(ends[lo] - (lo > 0 ? ends[lo - 1] : 0)) : 0.f;
        for (int c = lane; c < C; c += 32) gin[r * C + c] = lo < B ? g[(int64_t)lo * C + c] * inv : 0.f;
    }
}

}  // namespace norm
}  // namespace pb

using namespace pb;
using namespace pb::norm;

extern "C" {

int pb200_norm_parts(int64_t N, int C) {
    if (N < 0 || C <= 0) return 0;
    const int a = geom(N, C, false).grid;
    const int b = C % 4 == 0 ? geom(N, C, true).grid : 0;
    return a > b ? a : b;
}

int pb200_bias_act_stats(int64_t N, int C, float* rows, const float* bias, int relu, float* partial, int* nparts, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(N > 0 && C > 0, PB200_EINVAL, "bias_act_stats: bad sizes");
    PB_REQUIRE(rows && partial && nparts, PB200_EINVAL, "bias_act_stats: null pointer");
    const Geom g = geom(N, C, C % 4 == 0 && aligned16(rows));
    const dim3 grid(g.grid, g.chunks);
    NORM_DISPATCH(g, PB_LAUNCH("bias_act_stats", (stats_kernel<V, TL>), grid, THREADS, 0, stream, N, C, rows, bias, relu, partial))
    *nparts = g.grid;
    return PB200_OK;
}

int pb200_norm_finalize(int nparts, int C, const float* partial, float eps, float momentum, float* runningMean, float* runningVar,
                        int64_t* batches, float* mean, float* invstd, void* stream) {
    PB_REQUIRE(nparts > 0 && C > 0, PB200_EINVAL, "norm_finalize: bad sizes");
    PB_REQUIRE(partial && mean && invstd && (!runningMean == !runningVar), PB200_EINVAL, "norm_finalize: null pointer");
    PB_LAUNCH("norm_finalize", finalize_kernel, (unsigned)ceil_div(C, 32), dim3(32, FS), 0, (cudaStream_t)stream, nparts, C, partial, eps,
              momentum, runningMean, runningVar, batches, mean, invstd);
    return PB200_OK;
}

int pb200_norm_invstd(int C, const float* var, float eps, int64_t* batches, float* invstd, void* stream) {
    PB_REQUIRE(C > 0 && var && invstd, PB200_EINVAL, "norm_invstd: bad size or null pointer");
    PB_LAUNCH("norm_invstd", invstd_kernel, (unsigned)ceil_div(C, 128), 128, 0, (cudaStream_t)stream, C, var, eps, batches, invstd);
    return PB200_OK;
}

int pb200_norm_apply(int64_t N, int C, const float* act, const float* mean, const float* invstd, const float* gamma, const float* beta,
                     float* out, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(N >= 0 && C > 0, PB200_EINVAL, "norm_apply: bad sizes");
    if (N == 0) return PB200_OK;
    PB_REQUIRE(act && mean && invstd && out, PB200_EINVAL, "norm_apply: null pointer");
    const Geom g = geom(N, C, C % 4 == 0 && aligned16(act) && aligned16(out));
    const dim3 grid(g.grid * 2, g.chunks);
    NORM_DISPATCH(g, PB_LAUNCH("norm_apply", (apply_kernel<V, TL>), grid, THREADS, 0, stream, N, C, act, mean, invstd, gamma, beta, out))
    return PB200_OK;
}

int pb200_norm_backward_reduce(int64_t N, int C, const float* gradOutput, const float* act, const float* mean, const float* invstd,
                               const float* gamma, float* partial, float* gradGamma, float* gradBeta, float* scale, float* k1, float* k2,
                               void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(N > 0 && C > 0, PB200_EINVAL, "norm_backward_reduce: bad sizes");
    PB_REQUIRE(gradOutput && act && mean && invstd && partial && scale && k1 && k2, PB200_EINVAL, "norm_backward_reduce: null pointer");
    const Geom g = geom(N, C, C % 4 == 0 && aligned16(gradOutput) && aligned16(act));
    const dim3 grid(g.grid, g.chunks);
    NORM_DISPATCH(g, PB_LAUNCH("norm_bwd_reduce", (bwd_reduce_kernel<V, TL>), grid, THREADS, 0, stream, N, C, gradOutput, act, mean, partial))
    PB_LAUNCH("norm_bwd_finalize", bwd_finalize_kernel, (unsigned)ceil_div(C, 32), dim3(32, FS), 0, stream, g.grid, N, C, partial, invstd,
              gamma, gradGamma, gradBeta, scale, k1, k2);
    return PB200_OK;
}

int pb200_norm_backward_apply(int64_t N, int C, const float* gradOutput, const float* act, const float* mean, const float* scale,
                              const float* k1, const float* k2, int relu, float* masked, float* partial, float* gradBias,
                              void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(N > 0 && C > 0, PB200_EINVAL, "norm_backward_apply: bad sizes");
    PB_REQUIRE(gradOutput && act && masked && partial && gradBias && (!mean || (scale && k1 && k2)), PB200_EINVAL,
               "norm_backward_apply: null pointer");
    const Geom g = geom(N, C, C % 4 == 0 && aligned16(gradOutput) && aligned16(act) && aligned16(masked));
    const dim3 grid(g.grid, g.chunks);
    if (mean) {
        NORM_DISPATCH(g, PB_LAUNCH("norm_bwd_apply", (bwd_apply_kernel<V, TL, true>), grid, THREADS, 0, stream, N, C, gradOutput, act, mean,
                                   scale, k1, k2, relu, masked, partial))
    } else {
        NORM_DISPATCH(g, PB_LAUNCH("norm_bwd_apply", (bwd_apply_kernel<V, TL, false>), grid, THREADS, 0, stream, N, C, gradOutput, act, mean,
                                   scale, k1, k2, relu, masked, partial))
    }
    return reduce_partials(partial, g.grid, C, gradBias, stream);
}

size_t pb200_segment_mean_workspace_bytes(int64_t N, int B, int C) {
    if (N < 0 || B < 0 || C <= 0) return 0;
    return align_up(sizeof(float) * (size_t)(ceil_div(N, SEG_ROWS) + B) * C, 256);
}

int pb200_segment_mean(int64_t N, int B, int C, const float* rows, const int64_t* ends, float* out, void* workspace,
                       size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(N >= 0 && B >= 0 && C > 0, PB200_EINVAL, "segment_mean: bad sizes");
    if (B == 0) return PB200_OK;
    PB_REQUIRE(ends && out && (N == 0 || rows), PB200_EINVAL, "segment_mean: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_segment_mean_workspace_bytes(N, B, C), PB200_EWORKSPACE,
               "segment_mean: workspace too small");
    float* pieces = (float*)workspace;
    if (N > 0)
        PB_LAUNCH("segment_pieces", segment_pieces_kernel, dim3((unsigned)ceil_div(N, SEG_ROWS), (unsigned)ceil_div(C, 32)), 256, 0, stream,
                  N, C, B, ends, rows, pieces);
    PB_LAUNCH("segment_finish", segment_finish_kernel, dim3((unsigned)B, (unsigned)ceil_div(C, 32)), dim3(32, 8), 0, stream, N, C, B, ends,
              pieces, out);
    return PB200_OK;
}

int pb200_segment_mean_backward(int64_t N, int B, int C, const float* gradOutput, const int64_t* ends, float* gradInput, void* stream) {
    PB_REQUIRE(N >= 0 && B >= 0 && C > 0, PB200_EINVAL, "segment_mean_backward: bad sizes");
    if (N == 0) return PB200_OK;
    PB_REQUIRE(gradInput && (B == 0 || (gradOutput && ends)), PB200_EINVAL, "segment_mean_backward: null pointer");
    PB_LAUNCH("segment_mean_bwd", segment_mean_bwd_kernel, persistent_blocks(N, 32, 8), 256, 0, (cudaStream_t)stream, N, C, B, ends,
              gradOutput, gradInput);
    return PB200_OK;
}

}  // extern "C"
