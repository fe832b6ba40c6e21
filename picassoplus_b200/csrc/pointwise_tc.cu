// Module-level fusion of the two HBM-bound mesh operators with the pointwise stage that follows
// them in the layer modules (picasso/mesh/layers.py:109-120 V2FConv3d.forward, :166-175
// F2VConv3d.forward: operator -> matmul(depth_weights) -> + bias -> ReLU):
//
//   out^T[co, row] = act( sum_c  Wd[c, co] * feat[row, c]  + bias[co] )
//
// The rows of `feat` are produced on the fly and go to HBM only where the backward pass wants them (many rows with room for them take
// two kernels instead, see GATHER_ALONE):
//   vertex2facet:  feat[f, c] = sum_{k<3} filter[k, c] * input[face[f, k], c]        (r = 1)
//   facet2vertex:  feat[v, c] = (sum over the CSR entries (f, corner) of v of wx[f, c]) / nfCount[v]
//                  (wx = the per-face products of the facet2vertex forward pass)
// Per CTA (persistent) and per tile of 256 rows:
//   * 16 producer warps gather and combine the operand rows (whole 128-byte lines per load, four rows per warp at a time) and write
//     them as 64-byte swizzled K-major bf16 rows (one stage = 32 channels);
//   * one thread streams the pre-swizzled weight blocks with 1-D bulk copies, one issues tcgen05.mma (M = 128 output channels,
//     N = 256 rows, K = 16 per instruction, fp32 accumulation in TMEM, two accumulators);
//   * 8 epilogue warps drain the other accumulator meanwhile, add the bias, apply the activation and store out[row, co] coalesced.
// What bounds it: memory, and the epilogue's instructions per value.  978 000 rows 64 -> 64 in fp32 mode: 240 us with the
// producers doing the epilogue, 235 with four warps of its own, 107 with eight and no per-value predicates (no epilogue at
// all: 75); gradient rows 128 -> 128 with mask and masked copy 397 -> 330 us (5.9 TB/s).
// Precision modes: bf16 operands (one product per term) or bf16 hi + lo operands (three products,
// about 1e-5 relative: the fp32 mode).  All waits are bounded (tc_ptx.cuh).
#include "common.cuh"
#include "tc_ptx.cuh"
#include "tc_runtime.cuh"

namespace pb {

// per-face products of the facet2vertex forward pass (f2v.cu): wx[f, :] = (coeff[f] @ filter) * input[f]
int f2v_face_products(int64_t Nf, int C, int K, const float* input, const float* filter, const float* coeff, float* wx,
                      cudaStream_t stream);
int f2v_gather(int64_t NvOut, int C, const int32_t* rowptr, const int32_t* entries, const int32_t* nfCount, const float* wx, float* output,
               cudaStream_t stream);
bool f2v_face_products_supported(int C, int K);

namespace pw {

using namespace ptx;

constexpr int TILE_R = 256;                 // rows per tile (UMMA N)
constexpr int UM = 128;                     // output channels per launch (UMMA M), zero-padded
constexpr int PWARPS = 16;
// epilogue warps: two per TMEM quadrant; one for facet2vertex rows, whose gathers need the registers
template <int MODE> constexpr int EWARPS_OF = MODE == 1 ? 4 : 8;
template <int MODE> constexpr int NTHREADS = (PWARPS + EWARPS_OF<MODE> + 2) * 32;
constexpr int ROW_TILE_BYTES = TILE_R * 64;
constexpr int W_TILE_BYTES = UM * 64;
constexpr int KB = 32;                      // channels per stage (one 64-byte bf16 operand row)
constexpr int IDS = 8;                      // entries of a facet2vertex row that are kept in registers

// weight image: Wimg[kb][split][co 0..127][32 bf16, 64B-swizzled], element (co, k) = Wd[kb*32 + k][co0 + co]
// at wd[k * sk + n * sn]: (sk, sn) = (Cout, 1) for the layer's weights as they are, (1, Cin) for their transpose
__global__ void pw_prep_weights_kernel(int Cmid, int64_t sk, int64_t sn, int co0, int cchunk, int nkb, int nsplit,
                                       const float* __restrict__ wd, uint8_t* __restrict__ wimg) {
    const int64_t total = (int64_t)nkb * UM * 4;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i & 3);                   // 16-byte chunk = 8 channels
        const int co = (int)((i >> 2) % UM);
        const int kb = (int)(i / (4 * UM));
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float v[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int ci = kb * KB + c * 8 + 2 * j + e;
                v[e] = (co < cchunk && ci < Cmid) ? __ldg(wd + ci * sk + (co0 + co) * sn) : 0.f;
            }
            if (nsplit == 1) { hi[j] = pack_bf16x2(v[0], v[1]); lo[j] = 0u; }
            else split_bf16x2(v[0], v[1], hi[j], lo[j]);
        }
        uint8_t* base = wimg + (int64_t)kb * nsplit * W_TILE_BYTES;
        const uint32_t off = swz64_offset((uint32_t)co, (uint32_t)c);
        *reinterpret_cast<uint4*>(base + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        if (nsplit == 2) *reinterpret_cast<uint4*>(base + W_TILE_BYTES + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
}

struct Params {
    int64_t Nrows;            // faces (vertex2facet) or output vertices (facet2vertex)
    int C;                    // channels of the gathered rows (a multiple of 8)
    int Cout;                 // output channels of this launch's chunk (<= 128)
    int out_stride;           // floats per output row
    int nkb;                  // 32-channel stages per tile
    int nstages;
    int relu;
    // vertex2facet rows
    const float* vin;         // (Nv, C)
    const float* vfilt;       // (3, C)
    const int32_t* face;      // (Nrows, 3)
    int64_t Nv;
    // facet2vertex rows
    const float* wx;          // (Nf, C) per-face products
    const int32_t* rowptr;
    const int32_t* entries;
    const int32_t* nfCount;
    // masked rows (backward of the pointwise stage)
    const float* rows;        // (Nrows, C) upstream gradient
    const float* mask;        // (Nrows, C) activated output; NULL = neither mask nor normalisation
    int relu_mask;            // the gradient passes where the activated output is > 0
    float* masked_out;        // (Nrows, C) the masked gradient, written as a by-product; NULL = not wanted
    // gradient through a batch normalisation behind the activation: rows <- scale * rows + k2 * (mask - mean) + k1, per channel,
    // before the mask is applied (norm.cu); NULL = none
    const float *bn_mean, *bn_scale, *bn_k1, *bn_k2;
    float* feat_out;          // (Nrows, C) the gathered rows, written as a by-product for the backward pass; NULL = not wanted
    const uint8_t* wimg;
    const float* bias;        // (Cout chunk) or NULL
    float* out;               // first output channel of the chunk
    // inference: outputs are normalised with the running statistics (first channel of the chunk); ev_var NULL = not
    const float *ev_mean, *ev_var, *ev_gamma, *ev_beta;
    float ev_eps;
    int* async_err;
    int wait_budget;
};

__host__ __device__ inline size_t stage_bytes(int nsplit) { return (size_t)nsplit * (ROW_TILE_BYTES + W_TILE_BYTES); }

// MODE 0: vertex2facet rows, MODE 1: facet2vertex rows, MODE 2: rows that are there already, a gradient's masked by an activation
template <int NSPLIT, int MODE>
__global__ void __launch_bounds__(NTHREADS<MODE>, 1) rows_pointwise_tc_kernel(Params p) {
    constexpr int EWARPS = EWARPS_OF<MODE>, W_WARP = PWARPS + EWARPS;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = p.nstages, C = p.C, Cout = p.Cout;
    const size_t sbytes = stage_bytes(NSPLIT);
    uint8_t* stages = smem;                       // stage: [rows hi][rows lo?][weights hi][weights lo?]
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)S * sbytes);
    uint64_t* full = bars;                        // [S] producers (16 warps) + weight bytes
    uint64_t* empty = bars + S;                   // [S] MMA done with the stage
    uint64_t* acc_full = bars + 2 * S;            // [2] accumulator of a tile complete
    uint64_t* acc_free = bars + 2 * S + 2;        // [2] and read out
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    if (tid == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(&full[s], PWARPS + 1); mbar_init(&empty[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_free[a], EWARPS); }
        abort_flag[0] = 0;
        abort_flag[1] = p.wait_budget;
        fence_barrier_init();
    }
    if (warp == W_WARP) { tmem_alloc(tmem_slot, 2 * TILE_R); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int64_t ntiles = (p.Nrows + TILE_R - 1) / TILE_R;

    if (warp < PWARPS) {
        // ===================================== producers =====================================
        // A warp has 16 rows of the tile, four at a time: lane = row rg of the four, channels 4j..4j+3 of the stage's 32.  A warp's
        // load then reads whole 128-byte lines (two lanes of 32 bytes per row met 16 lines per load, and the L1 was what the
        // kernel waited for).
        // facet2vertex rows keep the two lanes: their gathers come from L2, a line is wanted by three vertices, and what the small
        // L1 can hold meanwhile is 64 bytes of every row of the tile, not 128 (128 channels: 499 against 574 us).
        const int rg = lane >> 3, j = lane & 7, m0 = MODE == 1 ? warp * 16 + (lane >> 1) : warp * 16 + rg;
        const uint32_t stages32 = smem_u32(stages);
        int st_i = 0;
        uint32_t st_ph = 0;

        // what the rows are made of: vertex2facet a row of the warp per lane, facet2vertex the thread's own row; the next tile's is
        // loaded while this one's rows are
        struct Source { int v[3]; int beg, n; float inv_n; };
        auto source = [&](int64_t tile, Source& s) {
            const int64_t row = tile * TILE_R + (MODE == 1 ? m0 : warp * 16 + lane);
            const bool valid = (MODE == 1 || lane < 16) && row < p.Nrows;
            if (MODE == 0) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    s.v[k] = valid ? __ldg(p.face + 3 * row + k) : -1;
                    if (s.v[k] < 0 || s.v[k] >= p.Nv) s.v[k] = -1;            // a bad index contributes nothing
                }
            } else if (MODE == 1) {
                s.beg = valid ? __ldg(p.rowptr + row) : 0;
                s.n = valid ? __ldg(p.rowptr + row + 1) - s.beg : 0;
                s.inv_n = s.n > 0 ? 1.f / (float)__ldg(p.nfCount + row) : 0.f;
            }
        };
        Source cur, nxt;
        source(blockIdx.x, nxt);
        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const int64_t row0 = tile * TILE_R + m0;             // rows row0 + 4k; facet2vertex: row0
            cur = nxt;
            source(tile + gridDim.x, nxt);
            int id[MODE == 1 ? IDS : 1];
            if (MODE == 1) {
#pragma unroll
                for (int e = 0; e < IDS; ++e) id[e] = e < cur.n ? __ldg(p.entries + cur.beg + e) >> 2 : 0;
            }
            for (int kb = 0; kb < p.nkb; ++kb) {
                float4 a[4];
                const int c = kb * KB + 4 * j;
                const bool in = c < C;
#pragma unroll
                for (int k = 0; k < 4; ++k) a[k] = zero4();
                if (MODE == 0) {
                    // the k-ascending FMA chain of the stand-alone vertex2facet kernel, the loads of two rows ahead of it
                    float4 fl[3];
#pragma unroll
                    for (int t = 0; t < 3; ++t) fl[t] = in ? ldg4(reinterpret_cast<const float4*>(p.vfilt + (int64_t)t * C + c)) : zero4();
#pragma unroll
                    for (int k0 = 0; k0 < 4; k0 += 2) {
                        int v[2][3];
                        float4 x[2][3];
#pragma unroll
                        for (int k = 0; k < 2; ++k)
#pragma unroll
                            for (int t = 0; t < 3; ++t) {
                                v[k][t] = __shfl_sync(0xffffffffu, cur.v[t], 4 * (k0 + k) + rg);
                                if (!in) v[k][t] = -1;
                                if (v[k][t] >= 0) x[k][t] = ldg4(reinterpret_cast<const float4*>(p.vin + (int64_t)v[k][t] * C + c));
                            }
#pragma unroll
                        for (int k = 0; k < 2; ++k)
#pragma unroll
                            for (int t = 0; t < 3; ++t)
                                if (v[k][t] >= 0) fma4(a[k0 + k], fl[t], x[k][t]);
                    }
                } else if (MODE == 1) {
                    // ascending CSR entries, then one scaling: the arithmetic of the stand-alone gather kernel.  The rows of four
                    // entries are on their way at a time; a[2i], a[2i + 1] = channels kb*32 + 16i + 8h ..+7
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int ci = kb * KB + 16 * i + 8 * (lane & 1);
                        if (ci >= C) continue;
                        const float* base = p.wx + ci;
#pragma unroll
                        for (int e0 = 0; e0 < IDS; e0 += 4) {
                            if (e0 >= cur.n) break;
                            float4 x[4][2];
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (e0 + e < cur.n) {
                                    const float4* src = reinterpret_cast<const float4*>(base + (int64_t)id[e0 + e] * C);
                                    x[e][0] = ldg4(src); x[e][1] = ldg4(src + 1);
                                }
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (e0 + e < cur.n) { add4(a[2 * i], x[e][0]); add4(a[2 * i + 1], x[e][1]); }
                        }
                        for (int e = IDS; e < cur.n; ++e) {
                            const float4* src = reinterpret_cast<const float4*>(base + (int64_t)(__ldg(p.entries + cur.beg + e) >> 2) * C);
                            add4(a[2 * i], ldg4(src));
                            add4(a[2 * i + 1], ldg4(src + 1));
                        }
                        if (cur.n > 0) { a[2 * i] = scale4(a[2 * i], cur.inv_n); a[2 * i + 1] = scale4(a[2 * i + 1], cur.inv_n); }
                    }
                } else {
                    float4 mk[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        mk[k] = zero4();
                        if (!in || row0 + 4 * k >= p.Nrows) continue;
                        a[k] = ldg4(reinterpret_cast<const float4*>(p.rows + (row0 + 4 * k) * C + c));
                        if (p.mask) mk[k] = ldg4(reinterpret_cast<const float4*>(p.mask + (row0 + 4 * k) * C + c));
                    }
                    if (p.bn_mean && in) {
                        const float4 mu = ldg4(reinterpret_cast<const float4*>(p.bn_mean + c)), sc = ldg4(reinterpret_cast<const float4*>(p.bn_scale + c));
                        const float4 k1 = ldg4(reinterpret_cast<const float4*>(p.bn_k1 + c)), k2 = ldg4(reinterpret_cast<const float4*>(p.bn_k2 + c));
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            a[k].x = fmaf(sc.x, a[k].x, fmaf(k2.x, mk[k].x - mu.x, k1.x));
                            a[k].y = fmaf(sc.y, a[k].y, fmaf(k2.y, mk[k].y - mu.y, k1.y));
                            a[k].z = fmaf(sc.z, a[k].z, fmaf(k2.z, mk[k].z - mu.z, k1.z));
                            a[k].w = fmaf(sc.w, a[k].w, fmaf(k2.w, mk[k].w - mu.w, k1.w));
                        }
                    }
                    if (p.mask && p.relu_mask) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            a[k] = make_float4(mk[k].x > 0.f ? a[k].x : 0.f, mk[k].y > 0.f ? a[k].y : 0.f, mk[k].z > 0.f ? a[k].z : 0.f,
                                               mk[k].w > 0.f ? a[k].w : 0.f);
                    }
                }
                float* const side = MODE == 2 ? p.masked_out : p.feat_out;
                if (MODE == 1) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int ci = kb * KB + 16 * (k >> 1) + 8 * (lane & 1) + 4 * (k & 1);
                        if (side && ci < C && row0 < p.Nrows) *reinterpret_cast<float4*>(side + row0 * C + ci) = a[k];
                    }
                } else if (side && in) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (row0 + 4 * k < p.Nrows) *reinterpret_cast<float4*>(side + (row0 + 4 * k) * C + c) = a[k];
                }
                if (!warp_wait(&empty[st_i], st_ph ^ 1u, abort_flag, lane)) { tile = ntiles; break; }
                const uint32_t st = stages32 + (uint32_t)st_i * (uint32_t)sbytes;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t at = MODE == 1 ? st + swz64_offset((uint32_t)m0, (uint32_t)(2 * (k >> 1) + (lane & 1))) + (uint32_t)(k & 1) * 8u
                                                  : st + swz64_offset((uint32_t)(m0 + 4 * k), (uint32_t)(j >> 1)) + (uint32_t)(j & 1) * 8u;
                    uint32_t h0, h1, l0, l1;
                    if (NSPLIT == 1) {
                        h0 = pack_bf16x2(a[k].x, a[k].y); h1 = pack_bf16x2(a[k].z, a[k].w);
                    } else {
                        split_bf16x2(a[k].x, a[k].y, h0, l0); split_bf16x2(a[k].z, a[k].w, h1, l1);
                        sts_u2(at + ROW_TILE_BYTES, l0, l1);
                    }
                    sts_u2(at, h0, h1);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[st_i]);
                if (++st_i == S) { st_i = 0; st_ph ^= 1u; }
            }
        }
    } else if (warp < W_WARP) {
        // ========== epilogue: accumulator rows = output channels, columns = rows of the tile ==========
        const int q = warp & 3;
        const int co = q * 32 + lane;
        const float bv = (p.bias && co < Cout) ? __ldg(p.bias + co) : 0.f;
        float ev_m = 0.f, ev_s = 1.f, ev_b = 0.f;
        if (p.ev_var && co < Cout) {
            ev_m = __ldg(p.ev_mean + co);
            ev_s = 1.f / sqrtf(__ldg(p.ev_var + co) + p.ev_eps);
            if (p.ev_gamma) ev_s *= __ldg(p.ev_gamma + co);
            if (p.ev_beta) ev_b = __ldg(p.ev_beta + co);
        }
        uint32_t tcount = 0;
        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++tcount) {
            const int64_t r0 = tile * TILE_R;
            const uint32_t b = tcount & 1u;
            if (!warp_wait(&acc_full[b], (tcount >> 1) & 1u, abort_flag, lane)) break;
            tc_fence_after();
            if (q * 32 < Cout) {
#pragma unroll 1
                for (int col = ((warp - PWARPS) >> 2) * 32; col < TILE_R; col += EWARPS / 4 * 32) {
                    uint32_t r[32];
                    tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + b * TILE_R + (uint32_t)col, r);
                    tmem_ld_wait();
                    const int64_t left = p.Nrows - (r0 + col);               // rows of this group that exist
                    float* const o = p.out + (r0 + col) * p.out_stride + co;
                    if (co >= Cout || left <= 0) continue;
                    auto value = [&](int j) {
                        float v = __uint_as_float(r[j]) + bv;
                        return p.relu ? fmaxf(v, 0.f) : v;
                    };
                    // a warp's instructions per value are what an epilogue takes its time for: the whole group without predicates
                    if (left >= 32 && !p.ev_var) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[(uint32_t)(j * p.out_stride)] = value(j);
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (j < left) o[(uint32_t)(j * p.out_stride)] = fmaf(value(j) - ev_m, ev_s, ev_b);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_free[b]);
        }
    } else if (warp == W_WARP) {
        // ================================ weight loader (TMA engine) ==========================
        if (elect_one()) {
            const uint32_t bytes = (uint32_t)(NSPLIT * W_TILE_BYTES);
            int s = 0;
            uint32_t ph = 0;
            bool alive = true;
            for (int64_t tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
                for (int kb = 0; kb < p.nkb; ++kb) {
                    if (!mbar_wait(&empty[s], ph ^ 1u, abort_flag)) { alive = false; break; }
                    mbar_arrive_expect_tx(&full[s], bytes);
                    bulk_g2s(stages + (size_t)s * sbytes + (size_t)NSPLIT * ROW_TILE_BYTES, p.wimg + (size_t)kb * bytes, bytes,
                             &full[s]);
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
            }
            if (!alive) {                       // let copies in flight land before shared memory is released
                long long t0 = clock64();
                while (clock64() - t0 < 2000000) { }
            }
        }
    } else {
        // ================================ MMA issuer =========================================
        if (elect_one()) {
            constexpr uint32_t idesc = instr_desc(FMT_BF16, UM, TILE_R);
            const uint64_t dbase = smem_desc_kmajor(smem_u32(stages), 64, SWZ_64B);
            int s = 0;
            uint32_t ph = 0, tcount = 0;
            bool alive = true;
            for (int64_t tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x, ++tcount) {
                const uint32_t acc = tmem_base + (tcount & 1u) * TILE_R;
                if (!mbar_wait(&acc_free[tcount & 1u], ((tcount >> 1) & 1u) ^ 1u, abort_flag)) break;
                tc_fence_after();
                for (int kb = 0; kb < p.nkb; ++kb) {
                    if (!mbar_wait(&full[s], ph, abort_flag)) { alive = false; break; }
                    tc_fence_after();
                    const uint64_t rows_hi = dbase + (uint64_t)(((uint32_t)s * (uint32_t)sbytes) >> 4);
                    const uint64_t w_hi = rows_hi + (uint64_t)((NSPLIT * ROW_TILE_BYTES) >> 4);
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) {          // 2 x 32 bytes of K (16 bf16 each)
                        const uint64_t adv = (uint64_t)(ks * 2);
                        const uint32_t first = (kb | ks) != 0;
                        if (NSPLIT == 1) {
                            mma_f16(acc, w_hi + adv, rows_hi + adv, idesc, first);
                        } else {
                            const uint64_t rows_lo = rows_hi + (uint64_t)(ROW_TILE_BYTES >> 4);
                            const uint64_t w_lo = w_hi + (uint64_t)(W_TILE_BYTES >> 4);
                            mma_f16(acc, w_lo + adv, rows_hi + adv, idesc, first);
                            mma_f16(acc, w_hi + adv, rows_lo + adv, idesc, 1u);
                            mma_f16(acc, w_hi + adv, rows_hi + adv, idesc, 1u);
                        }
                    }
                    tc_commit(&empty[s]);
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
                if (alive) tc_commit(&acc_full[tcount & 1u]);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == W_WARP) tmem_dealloc(tmem_base, 2 * TILE_R);
    if (tid == 0 && abort_flag[0] && p.async_err) {
        *p.async_err = 4;
        __threadfence_system();
    }
}

// ---------------------------------------------------------------------------- host side
// From this many rows on, a call that is given room for its gathered rows (`features`) runs the operator's own kernel into it and the
// product on those rows: same sums, same bits, one launch more.  The fused producers keep 512 threads' gathers in flight per SM beside
// 130 KB of operand buffers, the operator's kernel 2048 with all of L1.  980 000 vertices 128 -> 128: 805 us fused, 335 + 160 apart;
// 1.76 M faces 64 -> 128: 519 against 122 + 230.  Below, the launch costs what it saves: a scene of 2 x 120^2 with its backward pass
// 1 209 us fused, 1 278 with every gather apart, 1 222 with those from 100 000 rows on (spread of a side 20).
// The line is one of rows for facet2vertex at 8 to 384 channels and as many outputs (122 500 rows 0.54 to 0.93 of the fused time, 108 900
// up to 1.0), and for vertex2facet where the backward pass wants the rows (195 000 rows at most 1.01).
constexpr int64_t GATHER_ALONE = 100000;
// vertex2facet that would write its rows for the product alone: the fused kernel reads three rows of a face that its neighbours read too
// and writes none, so the other way pays where the outputs are many or take more than one launch, and for wide rows where the vertices
// outgrow L2.  Layers with their running statistics, fused -> apart: 195 000 faces 64 -> 64 channels 55 -> 64 us, 128 -> 16 75 -> 88, 64 -> 128
// 73 -> 66, 102 800 128 -> 128 53 -> 61, 128 -> 256 108 -> 96; 448 000 32 -> 16 69 -> 83, 64 -> 64 122 -> 109; 879 000 32 -> 16 137 -> 146, 16 -> 32
// 128 -> 131, 32 -> 64 152 -> 148; 1.76 M 16 -> 64 270 -> 241.
static bool rows_for_product_alone(int64_t rows, int C, int Cout) {
    if (C < 64) return rows * Cout >= 50000000;
    return rows * Cout >= 17000000 || rows >= 600000;
}
struct Plan { int nsplit, nkb, nstages; size_t smem, wimg_bytes; };

static Plan plan(int C, int precision) {
    Plan pl;
    pl.nsplit = precision == PB200_PREC_BF16 ? 1 : 2;
    pl.nkb = (C + KB - 1) / KB;
    pl.nstages = pl.nsplit == 2 ? 4 : 6;
    pl.smem = (size_t)pl.nstages * stage_bytes(pl.nsplit) + 1024 + 256;
    pl.wimg_bytes = (size_t)pl.nkb * pl.nsplit * W_TILE_BYTES;
    return pl;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// What a layer adds around the product: normalisation of the outputs, the by-product (pb200_pointwise_extra).
static int set_extra(Params& p, const pb200_pointwise_extra* x, const char* where) {
    if (!x) return PB200_OK;
    PB_REQUIRE(!x->features || aligned16(x->features), PB200_EINVAL, "%s: features must be 16-byte aligned", where);
    PB_REQUIRE(!x->var || x->mean, PB200_EINVAL, "%s: variance without mean", where);
    p.feat_out = x->features;
    p.ev_mean = x->mean; p.ev_var = x->var; p.ev_gamma = x->gamma; p.ev_beta = x->beta; p.ev_eps = x->eps;
    return PB200_OK;
}

template <int MODE>
static int launch(const char* label, const Params& p, const Plan& pl, int grid, cudaStream_t stream) {
    if (pl.nsplit == 2) {
        PB_CUDA(cudaFuncSetAttribute(rows_pointwise_tc_kernel<2, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
        PB_LAUNCH(label, (rows_pointwise_tc_kernel<2, MODE>), grid, NTHREADS<MODE>, pl.smem, stream, p);
    } else {
        PB_CUDA(cudaFuncSetAttribute(rows_pointwise_tc_kernel<1, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
        PB_LAUNCH(label, (rows_pointwise_tc_kernel<1, MODE>), grid, NTHREADS<MODE>, pl.smem, stream, p);
    }
    return PB200_OK;
}

template <int MODE>
static int run(Params p, int Cout, const float* wd, const float* bias, float* out, int precision, void* ws,
               cudaStream_t stream, bool transposed = false) {
    int rc = tc::check_async_error("pointwise fusion");
    if (rc) return rc;
    const Plan pl = plan(p.C, precision);
    uint8_t* wimg = (uint8_t*)ws;
    p.nkb = pl.nkb; p.nstages = pl.nstages; p.out_stride = Cout;
    p.async_err = tc::async_error_word();
    p.wait_budget = tc::wait_budget_kclocks();
    const int64_t ntiles = ceil_div(p.Nrows, TILE_R);
    const int grid = (int)(ntiles < sm_count() ? ntiles : sm_count());
    const Params all = p;
    for (int co0 = 0; co0 < Cout; co0 += UM) {
        const int cchunk = Cout - co0 < UM ? Cout - co0 : UM;
        PB_LAUNCH("pw_prep_weights", pw_prep_weights_kernel, persistent_blocks((int64_t)pl.nkb * UM * 4, 256, 8), 256, 0, stream,
                  p.C, (int64_t)(transposed ? 1 : Cout), (int64_t)(transposed ? p.C : 1), co0, cchunk, pl.nkb, pl.nsplit, wd, wimg);
        p.Cout = cchunk; p.wimg = wimg; p.bias = bias ? bias + co0 : nullptr; p.out = out + co0;
        p.ev_mean = all.ev_var ? all.ev_mean + co0 : nullptr; p.ev_var = all.ev_var ? all.ev_var + co0 : nullptr;
        p.ev_gamma = all.ev_gamma ? all.ev_gamma + co0 : nullptr; p.ev_beta = all.ev_beta ? all.ev_beta + co0 : nullptr;
        const char* label = MODE == 0 ? "v2f_pointwise_tc" : (MODE == 1 ? "f2v_pointwise_tc" : "masked_rows_tc");
        if (co0 > 0 && MODE != 2 && p.feat_out) {
            // the first chunk's launch has written the gathered rows: the others read them (978 000 faces, 256 output
            // channels from 128: 99 us per chunk instead of 176)
            p.rows = p.feat_out; p.mask = nullptr; p.feat_out = nullptr;
            int rc2 = launch<2>(label, p, pl, grid, stream);
            if (rc2) return rc2;
            p.feat_out = all.feat_out;
            continue;
        }
        if (co0 > 0) p.masked_out = nullptr;                                // by-products are written by the first chunk's launch
        rc = launch<MODE>(label, p, pl, grid, stream);
        if (rc) return rc;
    }
    return PB200_OK;
}

}  // namespace pw
}  // namespace pb

using namespace pb;

extern "C" {

int pb200_layer_wants_features(int64_t rows) { return rows >= pw::GATHER_ALONE; }
int pb200_vertex2facet_layer_wants_features(int64_t rows, int C, int Cout) {
    return rows >= pw::GATHER_ALONE && pw::rows_for_product_alone(rows, C, Cout);
}

size_t pb200_vertex2facet_pointwise_workspace_bytes(int C, int precision) {
    if (C <= 0) return 0;
    return align_up(pw::plan(C, precision).wimg_bytes, 256);
}

int pb200_vertex2facet_pointwise_forward(int64_t Nf, int64_t Nv, int C, int Cout, const float* input, const float* filter,
                                         const int32_t* face, const float* depthWeights, const float* bias, int relu,
                                         float* output, int precision, void* workspace, size_t workspace_bytes, void* stream) {
    return pb200_vertex2facet_layer_forward(Nf, Nv, C, Cout, input, filter, face, depthWeights, bias, relu, output, precision, nullptr,
                                            workspace, workspace_bytes, stream);
}

int pb200_vertex2facet_layer_forward(int64_t Nf, int64_t Nv, int C, int Cout, const float* input, const float* filter,
                                         const int32_t* face, const float* depthWeights, const float* bias, int relu,
                                         float* output, int precision, const pb200_pointwise_extra* extra, void* workspace,
                                         size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(Nf >= 0 && Nv >= 0 && C > 0 && Cout > 0 && C % 8 == 0 && Nf < (1LL << 31) && Nv < (1LL << 31), PB200_EINVAL,
               "vertex2facet_pointwise_forward: bad sizes (channels must be a multiple of 8)");
    PB_REQUIRE(precision == PB200_PREC_FP32 || precision == PB200_PREC_BF16, PB200_EINVAL,
               "vertex2facet_pointwise_forward: precision must be PB200_PREC_FP32 or PB200_PREC_BF16");
    if (Nf == 0) return PB200_OK;
    PB_REQUIRE(input && filter && face && depthWeights && output, PB200_EINVAL, "vertex2facet_pointwise_forward: null pointer");
    PB_REQUIRE(pw::aligned16(input) && pw::aligned16(filter) && pw::aligned16(workspace), PB200_EINVAL,
               "vertex2facet_pointwise_forward: input, filter and workspace must be 16-byte aligned");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_vertex2facet_pointwise_workspace_bytes(C, precision), PB200_EWORKSPACE,
               "vertex2facet_pointwise_forward: workspace too small");
    pw::Params p = {};
    p.Nrows = Nf; p.C = C; p.relu = relu;
    p.vin = input; p.vfilt = filter; p.face = face; p.Nv = Nv;
    if (int rc = pw::set_extra(p, extra, "vertex2facet_pointwise_forward")) return rc;
    if (p.feat_out && Nf >= pw::GATHER_ALONE) {
        if (int rc = pb200_vertex2facet_forward(Nf, Nv, C, 1, input, filter, face, p.feat_out, stream)) return rc;
        p.rows = p.feat_out; p.feat_out = nullptr;
        return pw::run<2>(p, Cout, depthWeights, bias, output, precision, workspace, stream);
    }
    return pw::run<0>(p, Cout, depthWeights, bias, output, precision, workspace, stream);
}

size_t pb200_facet2vertex_pointwise_workspace_bytes(int64_t Nf, int C, int precision) {
    if (C <= 0 || Nf < 0) return 0;
    return align_up(pw::plan(C, precision).wimg_bytes, 256) + align_up(sizeof(float) * (size_t)(Nf > 0 ? Nf : 1) * C, 256);
}

int pb200_facet2vertex_pointwise_forward(int64_t Nf, int64_t NvOut, int C, int K, int Cout, const float* input,
                                         const float* filter, const float* coeff, const int32_t* nfCount, const int32_t* rowptr,
                                         const int32_t* entries, const float* depthWeights, const float* bias, int relu,
                                         float* output, int precision, void* workspace, size_t workspace_bytes, void* stream) {
    return pb200_facet2vertex_layer_forward(Nf, NvOut, C, K, Cout, input, filter, coeff, nfCount, rowptr, entries, depthWeights, bias,
                                            relu, output, precision, nullptr, workspace, workspace_bytes, stream);
}

int pb200_facet2vertex_layer_forward(int64_t Nf, int64_t NvOut, int C, int K, int Cout, const float* input,
                                         const float* filter, const float* coeff, const int32_t* nfCount,
                                         const int32_t* rowptr, const int32_t* entries, const float* depthWeights,
                                         const float* bias, int relu, float* output, int precision,
                                         const pb200_pointwise_extra* extra, void* workspace, size_t workspace_bytes,
                                         void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(Nf >= 0 && NvOut >= 0 && C > 0 && K > 0 && Cout > 0 && C % 8 == 0 && f2v_face_products_supported(C, K) &&
                   Nf < (1LL << 29) && NvOut < (1LL << 31),
               PB200_EINVAL, "facet2vertex_pointwise_forward: bad sizes (channels must be a multiple of 8)");
    PB_REQUIRE(precision == PB200_PREC_FP32 || precision == PB200_PREC_BF16, PB200_EINVAL,
               "facet2vertex_pointwise_forward: precision must be PB200_PREC_FP32 or PB200_PREC_BF16");
    if (NvOut == 0) return PB200_OK;
    PB_REQUIRE(rowptr && nfCount && depthWeights && output && (Nf == 0 || (input && filter && coeff && entries)), PB200_EINVAL,
               "facet2vertex_pointwise_forward: null pointer");
    PB_REQUIRE(workspace && pw::aligned16(workspace) &&
                   workspace_bytes >= pb200_facet2vertex_pointwise_workspace_bytes(Nf, C, precision),
               PB200_EWORKSPACE, "facet2vertex_pointwise_forward: workspace missing, misaligned or too small");
    PB_REQUIRE(Nf == 0 || (pw::aligned16(input) && pw::aligned16(filter)), PB200_EINVAL,
               "facet2vertex_pointwise_forward: input and filter must be 16-byte aligned");
    float* wx = (float*)((char*)workspace + align_up(pw::plan(C, precision).wimg_bytes, 256));
    if (Nf > 0) {
        int rc = f2v_face_products(Nf, C, K, input, filter, coeff, wx, stream);
        if (rc) return rc;
    }
    pw::Params p = {};
    p.Nrows = NvOut; p.C = C; p.relu = relu;
    p.wx = wx; p.rowptr = rowptr; p.entries = entries; p.nfCount = nfCount;
    if (int rc = pw::set_extra(p, extra, "facet2vertex_pointwise_forward")) return rc;
    if (p.feat_out && NvOut >= pw::GATHER_ALONE) {
        if (int rc = f2v_gather(NvOut, C, rowptr, entries, nfCount, wx, p.feat_out, stream)) return rc;
        p.rows = p.feat_out; p.feat_out = nullptr;
        return pw::run<2>(p, Cout, depthWeights, bias, output, precision, workspace, stream);
    }
    return pw::run<1>(p, Cout, depthWeights, bias, output, precision, workspace, stream);
}

size_t pb200_masked_rows_matmul_workspace_bytes(int C, int precision) {
    if (C <= 0) return 0;
    return align_up(pw::plan(C, precision).wimg_bytes, 256);
}

int pb200_rows_pointwise_forward(int64_t Nrows, int C, int Cout, const float* rows, const float* weights, const float* bias,
                                 int relu, float* output, int precision, void* workspace, size_t workspace_bytes, void* stream) {
    return pb200_rows_layer_forward(Nrows, C, Cout, rows, weights, bias, relu, output, precision, nullptr, workspace, workspace_bytes,
                                    stream);
}

int pb200_rows_layer_forward(int64_t Nrows, int C, int Cout, const float* rows, const float* weights, const float* bias,
                                 int relu, float* output, int precision, const pb200_pointwise_extra* extra, void* workspace,
                                 size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(Nrows >= 0 && C > 0 && Cout > 0 && C % 8 == 0 && Nrows < (1LL << 31), PB200_EINVAL,
               "rows_pointwise_forward: bad sizes (the row width must be a multiple of 8)");
    PB_REQUIRE(precision == PB200_PREC_FP32 || precision == PB200_PREC_BF16, PB200_EINVAL,
               "rows_pointwise_forward: precision must be PB200_PREC_FP32 or PB200_PREC_BF16");
    if (Nrows == 0) return PB200_OK;
    PB_REQUIRE(rows && weights && output, PB200_EINVAL, "rows_pointwise_forward: null pointer");
    PB_REQUIRE(pw::aligned16(rows) && pw::aligned16(workspace), PB200_EINVAL,
               "rows_pointwise_forward: rows and workspace must be 16-byte aligned");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_masked_rows_matmul_workspace_bytes(C, precision), PB200_EWORKSPACE,
               "rows_pointwise_forward: workspace too small");
    pw::Params p = {};
    p.Nrows = Nrows; p.C = C; p.relu = relu;
    p.rows = rows;
    if (int rc = pw::set_extra(p, extra, "rows_pointwise_forward")) return rc;
    return pw::run<2>(p, Cout, weights, bias, output, precision, workspace, stream);
}

int pb200_masked_rows_matmul(int64_t Nrows, int C, int Cout, const float* rows, const float* mask, const float* weights,
                             float* output, float* maskedRows, int precision, void* workspace, size_t workspace_bytes,
                             void* stream) {
    return pb200_gradient_rows_matmul(Nrows, C, Cout, rows, mask, 1, nullptr, weights, 0, output, maskedRows, precision, workspace,
                                      workspace_bytes, stream);
}

int pb200_gradient_rows_matmul(int64_t Nrows, int C, int Cout, const float* rows, const float* mask, int relu,
                               const pb200_norm_gradient* norm, const float* weights, int transposed, float* output, float* maskedRows,
                               int precision, void* workspace, size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(Nrows >= 0 && C > 0 && Cout > 0 && C % 8 == 0 && Nrows < (1LL << 31), PB200_EINVAL,
               "masked_rows_matmul: bad sizes (the row width must be a multiple of 8)");
    PB_REQUIRE(precision == PB200_PREC_FP32 || precision == PB200_PREC_BF16, PB200_EINVAL,
               "masked_rows_matmul: precision must be PB200_PREC_FP32 or PB200_PREC_BF16");
    if (Nrows == 0) return PB200_OK;
    PB_REQUIRE(rows && weights && output, PB200_EINVAL, "masked_rows_matmul: null pointer");
    PB_REQUIRE(pw::aligned16(rows) && pw::aligned16(mask) && pw::aligned16(maskedRows) && pw::aligned16(workspace), PB200_EINVAL,
               "masked_rows_matmul: rows, mask, maskedRows and workspace must be 16-byte aligned");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_masked_rows_matmul_workspace_bytes(C, precision), PB200_EWORKSPACE,
               "masked_rows_matmul: workspace too small");
    pw::Params p = {};
    p.Nrows = Nrows; p.C = C; p.relu = 0;
    p.rows = rows; p.mask = mask; p.masked_out = maskedRows; p.relu_mask = relu;
    if (norm) {
        PB_REQUIRE(mask && norm->mean && norm->scale && norm->k1 && norm->k2 && pw::aligned16(norm->mean) && pw::aligned16(norm->scale) &&
                       pw::aligned16(norm->k1) && pw::aligned16(norm->k2),
                   PB200_EINVAL, "masked_rows_matmul: normalisation needs the activated rows and 16-byte aligned per-channel arrays");
        p.bn_mean = norm->mean; p.bn_scale = norm->scale; p.bn_k1 = norm->k1; p.bn_k2 = norm->k2;
    }
    return pw::run<2>(p, Cout, weights, nullptr, output, precision, workspace, stream, transposed != 0);
}

}  // extern "C"
