// facet2facet for colours: three input channels and 4 or 16 bases (one or four quads, rows of 16-byte multiples), forward and filter
// gradient, in fp32, with the layer around them.  f2f_small.cu has the formulas and serves the other sizes.
//
// A warp works by itself through batches of eight faces:
//   * a lane makes the A values of one face and quad of bases, so that a sample's weights are read in whole sectors; the samples
//     of the next batch are on their way while this one is contracted;
//   * the batch's A rows lie in shared memory, where the whole warp reads them (one broadcast for four values); a lane owns one or
//     two outputs and keeps their filter column (forward) or their sums (filter gradient) in registers, in pairs of (d, ci) so that
//     the multiply-adds are packed.
// Bias, activation and the statistics of the result are the forward kernel's epilogue, the way back through normalisation and
// activation is the gradient kernel's prologue: a lane is a channel, its factors and sums are registers.
// What bounds it: instructions (about 100 per face and warp, 24 of them multiply-adds at 16 bases and 32 outputs) with 12 warps per SM.
// 1 758 000 faces, 4.4 million samples, 16 bases, 32 outputs: forward 255 us with bias, ReLU and statistics (247 without, and 77 for
// those, before), gradient 288 us with normalisation, ReLU and bias gradient (325 and 96); a layer's training step 1 064 -> 826 us,
// with 64 outputs 1 700 -> 1 330, with 16 738 -> 587.  Measured and left: 9 and 25 bases, whose rows have to be read in single floats
// (956 -> 1 019, 1 499 -> 2 362 us); 8 and 12, whose rows leave quads of the warp idle (800 000 faces, 33 outputs, forward 97 -> 173 us and
// 136 -> 173, gradient 136 -> 235 and 159 -> 237); samples through shared memory by asynchronous copies (350, 384 us), five blocks per SM
// (spills: 490, 410), two outputs per lane at 32 outputs (348, 556).
#include <type_traits>
#include "common.cuh"
#include "moments.cuh"

namespace pb {
namespace rgb {

constexpr int WARPS = 4, NT = 32 * WARPS;
constexpr int C = 3;
constexpr int AHEAD = 4;                 // samples of a face that are loaded a batch ahead; further ones when their turn comes

constexpr int BF = 8;                    // faces of a batch: what a warp makes rows of at once with four quads

struct Params {
    int64_t Nf;
    int Cout;
    int lpf;                             // lanes of a face: 16 (two faces side by side) or 32
    const float* in;
    const float* bary;
    const int32_t* cum;
    const float* filter;                 // forward
    const float* bias;                   // forward, may be null
    int relu;
    float* out;                          // forward: result; gradient: partial[block][Cout * C * F]
    float* stats;                        // forward, may be null: partial[block][3][Cout] moments of the result
    const float* gout;                   // gradient
    const float* act;                    // gradient: activated rows, null: gout is taken as it is
    pb200_norm_gradient norm;            // gradient: mean null: no normalisation
    float* sums;                         // gradient, may be null: partial[block][Cout] column sums (bias gradient)
};

// The A values of a warp's batches: lane = (face, quad of bases)
template <int Q>
struct Rows {
    static constexpr int F = 4 * Q, M = F * C, AP = M | 4;    // bases, floats of a row and its pitch
    const Params& p;
    int step, fl, q;                                           // batches from one of the warp's to the next
    uint64_t b[AHEAD][2];                                      // the first samples of this batch's face: weights, channels
    float x[AHEAD][C];
    int k0, k1, n0, n1;                                        // samples of this batch's face, of the next one's

    __device__ __forceinline__ Rows(const Params& p_, int batch, int step_) : p(p_), step(step_) {
        const int lane = threadIdx.x & 31;
        fl = lane / Q; q = lane - fl * Q;
        range(batch, k0, k1);
        range(batch + step, n0, n1);
        ask(k0, k1);
    }
    __device__ __forceinline__ void range(int64_t batch, int& a, int& e) const {
        const int64_t f = batch * BF + fl;
        a = e = 0;
        if (fl < BF && f < p.Nf) {
            if (f > 0) a = __ldg(p.cum + f - 1);
            e = __ldg(p.cum + f);
        }
    }
    __device__ __forceinline__ void ask(int a, int e) {
        const float* src = p.bary + (int64_t)a * F + 4 * q;
        const float* in = p.in + (int64_t)a * C;
#pragma unroll
        for (int t = 0; t < AHEAD; ++t, src += F, in += C) {
            const bool on = a + t < e;
            b[t][0] = b[t][1] = 0;
#pragma unroll
            for (int c = 0; c < C; ++c) x[t][c] = 0.f;
            if (on) {
                const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(src));
                b[t][0] = v.x; b[t][1] = v.y;
#pragma unroll
                for (int c = 0; c < C; ++c) x[t][c] = __ldg(in + c);
            }
        }
    }
    // this batch's rows into sa, and the next batch's samples on their way
    __device__ __forceinline__ void put(int batch, float* sa) {
        uint64_t a[C][2];
#pragma unroll
        for (int c = 0; c < C; ++c) a[c][0] = a[c][1] = 0;
        auto add = [&] {
#pragma unroll
            for (int t = 0; t < AHEAD; ++t)
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const uint64_t xx = pair2(x[t][c], x[t][c]);
                    fma2(a[c][0], b[t][0], xx);
                    fma2(a[c][1], b[t][1], xx);
                }
        };
        add();
        for (int k = k0 + AHEAD; k < k1; k += AHEAD) { ask(k, k1); add(); }
        const float w = k1 > k0 ? __frcp_rn((float)(k1 - k0)) : 0.f;
        __syncwarp();                                          // the rows of the batch before are read
        if (fl < BF) {
            float v[4 * C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const float2 lo = unpair2(a[c][0]), hi = unpair2(a[c][1]);
                v[c] = lo.x * w; v[C + c] = lo.y * w; v[2 * C + c] = hi.x * w; v[3 * C + c] = hi.y * w;
            }
            float4* dst = reinterpret_cast<float4*>(sa + fl * AP + 4 * q * C);
#pragma unroll
            for (int c = 0; c < C; ++c) dst[c] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
        }
        k0 = n0; k1 = n1;
        ask(k0, k1);
        range((int64_t)batch + 2 * step, n0, n1);
        __syncwarp();
    }
};

// NO: outputs of a lane, lpf apart
template <int Q, int NO>
__global__ void __launch_bounds__(NT, 4 * Q * C * NO <= 48 ? 3 : 2) f2f_rgb_fwd_kernel(Params p) {
    using R = Rows<Q>;
    constexpr int F = R::F, PAIRS = R::M / 2;
    __shared__ __align__(16) float rows[WARPS][BF * R::AP];
    __shared__ norm::Moments red[WARPS * 2][32 * NO];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = lane % p.lpf, fs = lane / p.lpf, fpw = 32 / p.lpf;
    uint64_t w[NO][PAIRS];
    float bias[NO], shift[NO], s1[NO], s2[NO];
    int co[NO];
    int64_t n = 0;
#pragma unroll
    for (int o = 0; o < NO; ++o) {
        co[o] = (blockIdx.y * NO + o) * p.lpf + l;
        const bool on = co[o] < p.Cout;
        auto value = [&](int m) { return on ? __ldg(p.filter + ((int64_t)co[o] * C + m % C) * F + m / C) : 0.f; };
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) w[o][i] = pair2(value(2 * i), value(2 * i + 1));
        bias[o] = on && p.bias ? __ldg(p.bias + co[o]) : 0.f;
        shift[o] = s1[o] = s2[o] = 0.f;
    }
    const int nbatches = (int)((p.Nf + BF - 1) / BF), step = gridDim.x * WARPS;
    int batch = blockIdx.x * WARPS + warp;
    float* const sa = rows[warp];
    R r(p, batch, step);
    for (; batch < nbatches; batch += step) {
        r.put(batch, sa);
        const int64_t f0 = (int64_t)batch * BF, left = p.Nf - f0;
        const int here = left < BF ? (int)left : BF;           // faces of the batch
        float* dst = p.out + (f0 + fs) * p.Cout;
#pragma unroll 2
        for (int i = fs; i < here; i += fpw, dst += fpw * p.Cout) {
            const ulonglong2* a = reinterpret_cast<const ulonglong2*>(sa + i * R::AP);
            uint64_t even[NO], odd[NO];
#pragma unroll
            for (int m = 0; m < PAIRS / 2; ++m) {
                const ulonglong2 v = a[m];
#pragma unroll
                for (int o = 0; o < NO; ++o) {
                    if (m == 0) { even[o] = mul2(v.x, w[o][0]); odd[o] = mul2(v.y, w[o][1]); }
                    else { fma2(even[o], v.x, w[o][2 * m]); fma2(odd[o], v.y, w[o][2 * m + 1]); }
                }
            }
#pragma unroll
            for (int o = 0; o < NO; ++o) {
                add2(even[o], odd[o]);
                const float2 e = unpair2(even[o]);
                float y = (e.x + e.y) + bias[o];
                if (p.relu) y = norm::relu_of(y);
                if (co[o] < p.Cout) dst[co[o]] = y;
                if (n == 0) shift[o] = y;
                const float d = y - shift[o];
                s1[o] += d;
                s2[o] = fmaf(d, d, s2[o]);
            }
            ++n;
        }
    }
    if (!p.stats) return;
#pragma unroll
    for (int o = 0; o < NO; ++o) red[warp * fpw + fs][o * p.lpf + l] = norm::moments((float)n, shift[o], s1[o], s2[o]);
    __syncthreads();
    for (int i = threadIdx.x; i < NO * p.lpf; i += NT) {
        const int c = blockIdx.y * NO * p.lpf + i;
        norm::Moments m = red[0][i];
        for (int t = 1; t < WARPS * fpw; ++t) norm::merge(m, red[t][i]);
        float* dst = p.stats + (int64_t)blockIdx.x * 3 * p.Cout + c;
        if (c < p.Cout) { dst[0] = m.n; dst[p.Cout] = m.mean; dst[2 * p.Cout] = m.m2; }
    }
}

template <int Q, int NO>
__global__ void __launch_bounds__(NT, 4 * Q * C * NO <= 48 ? 3 : 2) f2f_rgb_gfilter_kernel(Params p) {
    using R = Rows<Q>;
    constexpr int F = R::F, M = R::M, PAIRS = M / 2;
    __shared__ __align__(16) float rows[WARPS][BF * R::AP];
    constexpr int MS = 8;
    __shared__ float red[MS * NT * NO];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = lane % p.lpf, fs = lane / p.lpf, fpw = 32 / p.lpf;
    uint64_t acc[NO][PAIRS];
    float sum[NO], mean[NO], scale[NO], k1[NO], k2[NO];
    int co[NO];
#pragma unroll
    for (int o = 0; o < NO; ++o) {
        const int c = (blockIdx.y * NO + o) * p.lpf + l;
        co[o] = c < p.Cout ? c : p.Cout - 1;                   // lanes without an output follow one and store nothing
        sum[o] = 0.f; scale[o] = 1.f; mean[o] = k1[o] = k2[o] = 0.f;
        if (p.norm.mean) {
            mean[o] = __ldg(p.norm.mean + co[o]); scale[o] = __ldg(p.norm.scale + co[o]);
            k1[o] = __ldg(p.norm.k1 + co[o]); k2[o] = __ldg(p.norm.k2 + co[o]);
        }
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) acc[o][i] = 0;
    }
    const int nbatches = (int)((p.Nf + BF - 1) / BF), step = gridDim.x * WARPS;
    int batch = blockIdx.x * WARPS + warp;
    float* const sa = rows[warp];
    R r(p, batch, step);
    for (; batch < nbatches; batch += step) {
        const int64_t f0 = (int64_t)batch * BF, left = p.Nf - f0;
        const int here = left < BF ? (int)left : BF;           // faces of the batch
        float g[BF][NO], y[BF][NO];
        const float *src = p.gout + (f0 + fs) * p.Cout, *srca = p.act + (f0 + fs) * p.Cout;
#pragma unroll
        for (int i = 0; i < BF; ++i, src += fpw * p.Cout, srca += fpw * p.Cout) {
            const bool on = i * fpw + fs < here;
#pragma unroll
            for (int o = 0; o < NO; ++o) {
                g[i][o] = on ? __ldg(src + co[o]) : 0.f;
                y[i][o] = on && p.act ? __ldg(srca + co[o]) : 0.f;
            }
        }
        r.put(batch, sa);
#pragma unroll
        for (int i = 0; i < BF; ++i) {
            const int fi = i * fpw + fs;
            if (fi >= here) break;
            uint64_t gg[NO];
#pragma unroll
            for (int o = 0; o < NO; ++o) {
                float v = g[i][o];
                if (p.norm.mean) v = fmaf(scale[o], v, fmaf(k2[o], y[i][o] - mean[o], k1[o]));
                if (p.act && p.relu) v = norm::relu_grad(v, y[i][o]);
                sum[o] += v;
                gg[o] = pair2(v, v);
            }
            const ulonglong2* a = reinterpret_cast<const ulonglong2*>(sa + fi * R::AP);
#pragma unroll
            for (int m = 0; m < PAIRS / 2; ++m) {
                const ulonglong2 v = a[m];
#pragma unroll
                for (int o = 0; o < NO; ++o) { fma2(acc[o][2 * m], v.x, gg[o]); fma2(acc[o][2 * m + 1], v.y, gg[o]); }
            }
        }
    }
    // the sums of the warps, in order, MS values of (d, ci) at a time; the column sums are the value behind the last
    float* const out = p.out + (int64_t)blockIdx.x * p.Cout * M;
    const int width = NO * p.lpf, mine = (warp * fpw + fs) * width + l;
#pragma unroll
    for (int m0 = 0; m0 <= M; m0 += MS) {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < MS; ++j) {
            const int m = m0 + j;
            if (m > M) break;
#pragma unroll
            for (int o = 0; o < NO; ++o) {
                float v = sum[o];
                if (m < M) { const float2 e = unpair2(acc[o][m < M ? m / 2 : 0]); v = m % 2 ? e.y : e.x; }
                red[j * NT * NO + mine + o * p.lpf] = v;
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < MS * width; i += NT) {
            const int j = i / width, c = i - j * width, at = blockIdx.y * width + c, m = m0 + j;
            if (at >= p.Cout || m > M) continue;
            float t = red[j * NT * NO + c];
            for (int k = 1; k < WARPS * fpw; ++k) t += red[j * NT * NO + k * width + c];
            if (m < M) out[((int64_t)at * C + m % C) * F + m / C] = t;
            else if (p.sums) p.sums[(int64_t)blockIdx.x * p.Cout + at] = t;
        }
    }
}

// ---------------------------------------------------------------------------- host side
bool supported(int Cin, int F, const float* bary) {
    return Cin == C && (F == 4 || F == 16) && (reinterpret_cast<uintptr_t>(bary) & 15) == 0;
}
// Where these kernels are the faster ones, over 4 096 to 1 000 000 faces and 1 to 400 outputs (f2f_small.cu -> these, 400 000 faces):
//   the operator alone: forward with 16 bases and up to 16 outputs (55 -> 45 us; 24 outputs 64 -> 68; 4 bases 20 -> 31), gradient with 12 to 32
//     outputs (4 bases 62 -> 56, 16 bases 95 -> 81; 40 outputs 73 -> 81 and 108 -> 134, 3 outputs and 16 bases 58 -> 62);
//   the layer forward from 4 outputs on (8 outputs 95 -> 58; with less the statistics' few rows hold the grid down: 50 -> 71);
//   the layer's gradients too, except where a second column of 64 outputs is nearly empty and f2f_small.cu reads rows in 16-byte
//     pieces (80 outputs, 4 bases 262 -> 296; 75 outputs 361 -> 318, 128 341 -> 313).
bool forward_alone(int Cout, int F) { return F == 16 && Cout <= 16; }
bool gradient_alone(int Cout) { return Cout >= 12 && Cout <= 32; }
bool layer_forward(int Cout) { return Cout >= 4; }
bool layer_gradient(int Cout) { return Cout >= 4 && (Cout <= 64 || Cout > 100 || Cout % 4 != 0); }

// Calls go(Q, NO): quads of a row, two outputs per lane where there are more than a warp's
template <typename Go>
static int with_shape(int F, int Cout, Go&& go) {
    const std::integral_constant<int, 1> one{};
    const std::integral_constant<int, 2> two{};
    const std::integral_constant<int, 4> four{};
    if (F == 4) return Cout > 32 ? go(one, two) : go(one, one);
    return Cout > 32 ? go(four, two) : go(four, one);
}

template <typename Kernel>
static int blocks_per_sm(Kernel k) {
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, NT, 0) == cudaSuccess && n > 0 ? n : 1;
}

// `most`: rows of statistics that the caller has room for
int forward(int64_t Nf, int Cout, int F, const float* input, const float* filter, const float* bary, const int32_t* cum, const float* bias,
            int relu, float* output, float* stats, int most, int* nparts, cudaStream_t stream) {
    Params p = {};
    p.Nf = Nf; p.Cout = Cout; p.lpf = Cout <= 16 ? 16 : 32;
    p.in = input; p.bary = bary; p.cum = cum; p.filter = filter; p.bias = bias; p.relu = relu; p.out = output; p.stats = stats;
    return with_shape(F, Cout, [&](auto q, auto no) {
        constexpr int Q = decltype(q)::value, NO = decltype(no)::value;
        static const int per_sm = blocks_per_sm(f2f_rgb_fwd_kernel<Q, NO>);
        const int columns = (int)ceil_div(Cout, NO * p.lpf);
        int gx = persistent_blocks(Nf, WARPS * BF, (int)ceil_div(per_sm, columns));
        if (stats && gx > most) gx = most;
        if (nparts) *nparts = gx;
        PB_LAUNCH("f2f_fwd_small", (f2f_rgb_fwd_kernel<Q, NO>), dim3(gx, columns), NT, 0, stream, p);
        return (int)PB200_OK;
    });
}

static int gf_blocks(int64_t Nf) { return persistent_blocks(Nf, 64, 4); }
size_t workspace_bytes(int64_t Nf, int Cout, int F) {
    return align_up(sizeof(float) * (size_t)gf_blocks(Nf > 0 ? Nf : 1) * (C * F + 1) * Cout, 256);
}

int backward_filter(int64_t Nf, int Cout, int F, const float* gout, const float* act, int relu, const pb200_norm_gradient* norm,
                    const float* input, const float* bary, const int32_t* cum, float* gfilter, float* gbias, void* ws, cudaStream_t stream) {
    Params p = {};
    p.Nf = Nf; p.Cout = Cout; p.lpf = Cout <= 16 ? 16 : 32;
    p.in = input; p.bary = bary; p.cum = cum; p.gout = gout; p.act = act; p.relu = relu; p.out = (float*)ws;
    if (norm) p.norm = *norm;
    return with_shape(F, Cout, [&](auto q, auto no) {
        constexpr int Q = decltype(q)::value, NO = decltype(no)::value;
        static const int per_sm = blocks_per_sm(f2f_rgb_gfilter_kernel<Q, NO>);
        const int columns = (int)ceil_div(Cout, NO * p.lpf), room = gf_blocks(Nf);
        int gx = persistent_blocks(Nf, WARPS * BF, (int)ceil_div(per_sm, columns));
        if (gx > room) gx = room;
        const int64_t n = (int64_t)Cout * C * F;
        Params now = p;
        now.sums = gbias ? now.out + gx * n : nullptr;
        PB_LAUNCH("f2f_bwd_gfilter_small", (f2f_rgb_gfilter_kernel<Q, NO>), dim3(gx, columns), NT, 0, stream, now);
        int rc = reduce_partials(now.out, gx, n, gfilter, stream);
        if (rc == PB200_OK && gbias) rc = reduce_partials(now.sums, gx, Cout, gbias, stream);
        return rc;
    });
}

}  // namespace rgb
}  // namespace pb
