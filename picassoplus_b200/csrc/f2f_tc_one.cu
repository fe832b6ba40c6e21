// facet2facet for faces with exactly one sample each, forward and input gradient, on tcgen05 + TMEM:
//
//   out[f, cn] = sum_d w[f, d] * sum_ck rows[f, ck] * W[ck, cn, d]
//
// (forward: rows = input, ck counts input channels, cn output channels; input gradient: rows = gradOutput, the roles
// exchanged).  The inner sum is a product on the tensor cores, the outer one an epilogue over the accumulator: the scheme
// of f2f_tc_gin.cu, whose kernel serves faces with several samples.  There the two warps of a TMEM quadrant share the
// SAMPLES of a face; with one sample half of them did nothing but read the same columns again, and the other half's chain of
// TMEM loads and sums per slice was three times as long as the slice's products at 64 channels (two scenes of 880 000 faces,
// 64 -> 64, 16 bases: 924 us, products alone 300 us).  Here
//   * 16 epilogue warps (thread = face) drain one of two accumulators together: the four warps of a TMEM quadrant take the slice's
//     channel quadruples in turn, load a quadruple's columns together, hand the accumulator back as soon as their last columns
//     are in registers, and store 16 bytes per quadruple (eight warps per accumulator: 316 instead of 288 us for 880 000 faces, 64 ->
//     64, 16 bases, and 5 % more on most other shapes);
//   * a slice holds as many channels as fill the accumulator (NQ; drained in groups of G), its filter image exactly the rows the
//     product reads, and a filter stage as many K-blocks as fit twice (a hand-over per K-block cost the bf16 mode a third);
//   * a tile's rows arrive by tiled bulk copies of 16 channels x 128 rows, swizzled as the operand wants it, in the operand buffer
//     itself: the 32 floats of a row's K-block take the two 64-byte slots that its bf16 hi and lo go to, and one warp converts them in
//     place.  (Two warps that loaded rows into registers were slower than a tile's products: 64 meshes, 64 -> 128 channels, both
//     directions 179 -> 124 us; 1.76 M faces, 64 -> 64: 1 620 -> 1 246.)  The registers of the block are dealt out by role;
//   * with many products per slice CTAs work in pairs (cta_group::2): each keeps its own tile and accumulators and half of every
//     filter block, the CTA of rank 0 issues, and its peer's filter stream, converter and epilogue report to its barriers;
//   * a work item is a tile of 128 faces (a pair of them) and a run of slices: few tiles are spread over the chip by splitting
//     their slices;
//   * the next item's rows and weights are asked towards L2 while this one's are copied.
// Per call with a cold L2, before (register loaders, no pairs) and now: 464 000 faces, 128 -> 128, 25 bases 832 -> 763 us, 16 bases 544 ->
// 468, 9 bases 413 -> 314; 880 000 faces, 64 -> 64, 16 bases 380 -> 288; 464 000 faces, 32 -> 32, 16 bases 130 -> 75; bf16, 128 -> 128, 25
// bases 441 -> 400.  What bounds it: the three products per term at 128 channels (0.91 of the burst rate), below that the round
// trips between issue and epilogue, some 1 300 clocks per slice.  Measured and left: one commit per slice for both its last
// filter stage and its accumulator (1 313 -> 1 242 us at 64 channels, 29.6 -> 31.1 ms at 128, 25 bases); 16-byte stores at 25 bases (the
// second sum does not fit the registers: 755 -> 789 us); probing the barriers without sleeping (nothing).  All waits are bounded.
#include <cuda.h>
#include <type_traits>
#include "common.cuh"
#include "tc_ptx.cuh"
#include "tc_runtime.cuh"

namespace pb {
namespace tc {

namespace gin {
int prep_filter_bf16(int F, int Cin, int co0, int Cout, int nq, int nslices, int kst, int nsplit, int rows, int64_t s_co, int64_t s_ci,
                     const float* filter, uint8_t* wimg, cudaStream_t stream);
}

namespace one {

using namespace ptx;

constexpr int TILE_M = 128;
constexpr int NCOLS = 256;                       // accumulator columns
constexpr int EWARPS = 16;                       // epilogue warps: four per TMEM quadrant
constexpr int GWARPS = 1;                        // row converters
constexpr int NTHREADS = (EWARPS + 3 + GWARPS) * 32;
// Registers per thread: at launch, of the epilogue's four warpgroups, of the two that hold filter stream, issue, row stream and converters
constexpr int REGS_LAUNCH = 96, REGS_EPILOGUE = 104, REGS_OTHER = 64;
static_assert(NTHREADS % 128 == 0 && EWARPS * 32 * REGS_EPILOGUE + (NTHREADS - EWARPS * 32) * REGS_OTHER == NTHREADS * REGS_LAUNCH,
              "the shares are what the block is launched with");
constexpr int KTILE_BYTES = TILE_M * 64;         // 32 channels of the tile's rows
constexpr int MAX_CK = 256;                      // contracted channels per launch
constexpr int MAX_GBUFS = 3;                     // tile buffers
constexpr int RAW_STAGES = 2, RAW_BYTES = 2 * KTILE_BYTES;       // where rows are not converted in place: K-blocks on their way

struct Params {
    int64_t Nf;
    int nitems;                      // pairs of tiles x slice groups
    int Cn, Ck;
    int nslices, kst, nmma;
    int nstages, kb, gbufs;          // filter stages, K-blocks of 32 channels in one stage (divides kst), tile buffers
    int staged;                      // one operand: rows come through stages of one K-block (see plan)
    int groups, per_group;           // slice groups of a tile, slices of a group
    const float* rows;
    int stride;                      // floats per row
    int accumulate;                  // later chunks of contracted channels add to out
    const float* w;                  // weight rows padded to Fp floats
    int Fp;
    const uint8_t* wimg;
    float* out;
    int* async_err;
    int wait_budget;
};

template <int F> constexpr int NQ = F == 4 ? 64 : F == 9 ? 28 : F == 16 ? 16 : 10;      // channels of a slice
template <int F> constexpr int G = F == 25 ? 2 : 4;                                     // channels of a step

// sum over the F columns in v with the weights b: packed pairs, two chains
template <int F>
__device__ __forceinline__ float weighted(const float* v, const float (&b)[(F + 3) / 4 * 4]) {
    float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll
    for (int i = 0; i < F / 2; ++i) {
        const float2 x = make_float2(v[2 * i], v[2 * i + 1]), y = make_float2(b[2 * i], b[2 * i + 1]);
        if (i & 1) s1 = __ffma2_rn(y, x, s1);
        else s0 = __ffma2_rn(y, x, s0);
    }
    float s = (s0.x + s1.x) + (s0.y + s1.y);
    if (F & 1) s = fmaf(b[F - 1], v[F - 1], s);
    return s;
}

// The barriers that the issuing thread waits on lie in the CTA of rank 0 and are arrived at from both
template <bool PAIR>
__device__ __forceinline__ void arrive_first(uint64_t* bar) {
    if constexpr (PAIR) mbar_arrive_at(at_rank(bar, 0));
    else mbar_arrive(bar);
}
template <bool PAIR>
__device__ __forceinline__ bool wait_first(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    if constexpr (PAIR) return mbar_wait_cluster(bar, parity, abort_flag);
    else return mbar_wait(bar, parity, abort_flag);
}
template <bool PAIR>
__device__ __forceinline__ void multiply(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (PAIR) mma_f16_pair(d_tmem, a_desc, b_desc, idesc, accumulate);
    else mma_f16(d_tmem, a_desc, b_desc, idesc, accumulate);
}
template <bool PAIR>
__device__ __forceinline__ void commit(uint64_t* bar) {
    if constexpr (PAIR) tc_commit_pair(bar);
    else tc_commit(bar);
}

template <int NSPLIT, int F, bool PAIR>
__global__ void __launch_bounds__(NTHREADS, 1) f2f_one_sample_tc_kernel(Params p, const __grid_constant__ CUtensorMap rows_map) {
    constexpr int nq = NQ<F>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = p.nstages, KST = p.kst;
    const bool staged = NSPLIT == 1 && p.staged;
    const uint32_t gtile_bytes = (staged ? 1u : 2u) * KST * KTILE_BYTES;
    constexpr int NB = PAIR ? 2 : 1;          // CTAs of a product: each has its own tile and its share of a filter block's rows
    const uint32_t w_bytes = (uint32_t)p.nmma * 64 / NB, wblk_bytes = NSPLIT * w_bytes, wstage_bytes = wblk_bytes * p.kb;
    const uint32_t rank = PAIR ? cluster_rank() : 0;
    uint8_t* gtile = smem;
    uint8_t* raw = smem + (size_t)p.gbufs * gtile_bytes;
    uint8_t* wst = raw + (staged ? RAW_STAGES * RAW_BYTES : 0);
    uint64_t* bars = reinterpret_cast<uint64_t*>(wst + (size_t)S * wstage_bytes);
    uint64_t* w_full = bars;                  // [S]
    uint64_t* w_empty = bars + S;             // [S]
    uint64_t* w_peer = bars + 2 * S;          // [S] rank 0: the peer's half has landed
    uint64_t* acc_full = bars + 3 * S;        // [2]
    uint64_t* acc_empty = bars + 3 * S + 2;   // [2] rank 0: both blocks' epilogues
    uint64_t* raw_full = bars + 3 * S + 4;    // [MAX_GBUFS] rows in the tile buffer (a K-block of them in a stage) as they are in memory
    uint64_t* g_full = raw_full + MAX_GBUFS;  // [MAX_GBUFS] converted; rank 0: in both blocks
    uint64_t* g_empty = g_full + MAX_GBUFS;   // [MAX_GBUFS] all products of the item done with the buffer
    uint64_t* raw_empty = g_empty + MAX_GBUFS;   // [RAW_STAGES] a stage's rows are in the tile buffer
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(raw_empty + RAW_STAGES);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    if (tid == 0) {
        for (int s = 0; s < S; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], 1); mbar_init(&w_peer[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], NB * EWARPS); }
        for (int b = 0; b < MAX_GBUFS; ++b) { mbar_init(&raw_full[b], 1); mbar_init(&g_full[b], NB * GWARPS); mbar_init(&g_empty[b], 1); }
        for (int b = 0; b < RAW_STAGES; ++b) mbar_init(&raw_empty[b], GWARPS);
        abort_flag[0] = 0;
        abort_flag[1] = p.wait_budget;
        fence_barrier_init();
    }
    if constexpr (PAIR) { __syncthreads(); cluster_sync(); }      // the peer's barriers are there
    if (warp == EWARPS) {
        if constexpr (PAIR) tmem_alloc_pair(tmem_slot, 512);
        else { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int nitems = p.nitems, item0 = blockIdx.x / NB, item_step = gridDim.x / NB;
    if (warp < EWARPS) registers_take<REGS_EPILOGUE>();
    else registers_keep<REGS_OTHER>();

    if (warp < EWARPS) {
        // ===================== epilogue (thread = face) =====================
        const int q = warp & 3, sub = warp >> 2;
        const int r = q * 32 + lane;
        const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16);
        const bool vec = p.Cn % G<F> == 0 && (reinterpret_cast<uintptr_t>(p.out) & (4 * G<F> - 1)) == 0;
        uint32_t sc = 0;
        bool alive = true;
        for (int item = item0; item < nitems && alive; item += item_step) {
            const int64_t f = (int64_t)(item / p.groups * NB + rank) * TILE_M + r;
            const int s0 = item % p.groups * p.per_group;
            const int s1 = s0 + p.per_group < p.nslices ? s0 + p.per_group : p.nslices;
            const bool valid = f < p.Nf;
            float b[(F + 3) / 4 * 4];
            {
                const float4* src = reinterpret_cast<const float4*>(p.w + (valid ? f : 0) * p.Fp);
#pragma unroll
                for (int i = 0; i < (F + 3) / 4; ++i) {
                    const float4 v = valid ? ldg4(src + i) : zero4();
                    b[4 * i] = v.x; b[4 * i + 1] = v.y; b[4 * i + 2] = v.z; b[4 * i + 3] = v.w;
                }
            }
            float* const row = p.out + f * p.Cn;
            // old: what the chunks of contracted channels before have left there, when the caller has it already
            auto store = [&](int c, const float (&s)[G<F>], const float4* old) {
                if (!valid || c >= p.Cn) return;
                if (vec) {
                    if constexpr (G<F> == 4) {
                        float4 v = make_float4(s[0], s[1], s[2], s[3]);
                        float4* dst = reinterpret_cast<float4*>(row + c);
                        if (p.accumulate) add4(v, old ? *old : *dst);
                        *dst = v;
                    } else {
                        float2 v = make_float2(s[0], s[1]);
                        float2* dst = reinterpret_cast<float2*>(row + c);
                        if (p.accumulate) { v.x += dst->x; v.y += dst->y; }
                        *dst = v;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < G<F>; ++j)
                        if (c + j < p.Cn) row[c + j] = p.accumulate ? row[c + j] + s[j] : s[j];
                }
            };
            for (int slice = s0; slice < s1; ++slice, ++sc) {
                const uint32_t a = sc & 1u;
                const int c0 = slice * nq;
                int left = (p.Cn - c0 + G<F> - 1) / G<F>;         // steps of the slice that exist
                if (left > nq / G<F>) left = nq / G<F>;
                // With few bases a quadruple is little work, and the loads of what is there already, one behind another, were what a
                // slice took (4 bases, 320 -> 256 channels, 300 000 faces: bf16 1 025 us, 563 with the slice's loads ahead of the wait)
                constexpr int AHEAD = F == 4 ? nq / G<F> / (EWARPS / 4) : 1;
                float4 old[AHEAD];
                if constexpr (F == 4) {
#pragma unroll
                    for (int i = 0; i < AHEAD; ++i) {
                        const int c = c0 + G<F> * (sub + i * (EWARPS / 4));
                        old[i] = p.accumulate && vec && valid && c < p.Cn ? *reinterpret_cast<const float4*>(row + c) : zero4();
                    }
                }
                int ok = 1;
                if (lane == 0) ok = mbar_wait(&acc_full[a], (sc >> 1) & 1u, abort_flag) ? 1 : 0;
                if (!__shfl_sync(0xffffffffu, ok, 0)) { alive = false; break; }
                tc_fence_after();
                auto hand_back = [&](int k) {                     // after the loads of this warp's last quadruple
                    if (k + EWARPS / 4 < left) return;
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) arrive_first<PAIR>(&acc_empty[a]);
                };
                if (sub >= left) hand_back(left);                 // nothing of this slice for this warp
                auto step = [&](int k, const float4* have) {
                    float s[G<F>], v[G<F> * F];
                    const uint32_t t = tbase + a * NCOLS + (uint32_t)(k * G<F> * F);
                    if constexpr (F == 16) { tmem_ld32f(t, v); tmem_ld32f(t + 32, v + 32); }
                    else tmem_ld_row<G<F> * F>(t, v);
                    tmem_ld_wait();
                    hand_back(k);
#pragma unroll
                    for (int j = 0; j < G<F>; ++j) s[j] = weighted<F>(v + j * F, b);
                    store(c0 + G<F> * k, s, have);
                };
                if constexpr (F == 4) {
#pragma unroll
                    for (int i = 0; i < AHEAD; ++i)
                        if (sub + i * (EWARPS / 4) < left) step(sub + i * (EWARPS / 4), &old[i]);
                } else {
                    for (int k = sub; k < left; k += EWARPS / 4) step(k, nullptr);
                }
            }
        }
    } else if (warp >= EWARPS + 3) {
        // ===================== row converters =====================
        // a task is 32 channels of 32 rows: a lane turns its row's 32 floats, which lie in the two 64-byte slots of that row
        // (channels 0..15 and 16..31), into bf16 hi and lo in the same two slots, or from a stage into the tile buffer's one
        const int gw = warp - (EWARPS + 3);
        auto convert = [&](uint32_t rr, uint32_t from, uint32_t from2, uint32_t to, uint32_t to2) {
            const uint32_t sw = rr >> 1 & 3u;
            float4 v[8];
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) { v[c] = lds_f4(from + ((c ^ sw) << 4)); v[4 + c] = lds_f4(from2 + ((c ^ sw) << 4)); }
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) {
                const float4 a = v[2 * c], b = v[2 * c + 1];
                uint32_t hi[4], lo[4];
                if (NSPLIT == 1) {
                    hi[0] = pack_bf16x2(a.x, a.y); hi[1] = pack_bf16x2(a.z, a.w);
                    hi[2] = pack_bf16x2(b.x, b.y); hi[3] = pack_bf16x2(b.z, b.w);
                } else {
                    split_bf16x2(a.x, a.y, hi[0], lo[0]); split_bf16x2(a.z, a.w, hi[1], lo[1]);
                    split_bf16x2(b.x, b.y, hi[2], lo[2]); split_bf16x2(b.z, b.w, hi[3], lo[3]);
                    sts_u4(to2 + ((c ^ sw) << 4), lo[0], lo[1], lo[2], lo[3]);
                }
                sts_u4(to + ((c ^ sw) << 4), hi[0], hi[1], hi[2], hi[3]);
            }
        };
        uint32_t icount = 0, blocks = 0;
        bool alive = true;
        for (int item = item0; item < nitems && alive; item += item_step, ++icount) {
            const uint32_t gb = icount % p.gbufs, gph = icount / p.gbufs & 1u;
            const uint32_t tile = smem_u32(gtile) + gb * gtile_bytes;
            if (staged) {
                if (!warp_wait(&g_empty[gb], gph ^ 1u, abort_flag, lane)) break;
                for (int ks = 0; ks < KST; ++ks, ++blocks) {
                    const uint32_t st = blocks % RAW_STAGES;
                    if (!warp_wait(&raw_full[st], blocks / RAW_STAGES & 1u, abort_flag, lane)) { alive = false; break; }
                    for (uint32_t part = gw; part < 4; part += GWARPS) {
                        const uint32_t rr = part * 32 + lane, from = smem_u32(raw) + st * RAW_BYTES + rr * 64;
                        const uint32_t to = tile + (uint32_t)ks * KTILE_BYTES + rr * 64;
                        convert(rr, from, from + KTILE_BYTES, to, to);
                    }
                    fence_proxy_async();                          // these reads before the next copy, these writes before the products
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&raw_empty[st]);
                }
                if (!alive) break;
            } else {
                if (!warp_wait(&raw_full[gb], gph, abort_flag, lane)) break;
                for (int task = gw; task < 4 * KST; task += GWARPS) {
                    const uint32_t rr = (uint32_t)(task & 3) * 32 + lane;
                    const uint32_t first = tile + (uint32_t)(task >> 2) * KTILE_BYTES + rr * 64, second = first + (uint32_t)KST * KTILE_BYTES;
                    convert(rr, first, second, first, second);
                }
                fence_proxy_async();
                __syncwarp();
            }
            if (lane == 0) arrive_first<PAIR>(&g_full[gb]);
        }
    } else if (warp == EWARPS + 2) {
        // ===================== row stream (TMA engine) =====================
        if (elect_one()) {
            uint32_t icount = 0, blocks = 0;
            bool alive = true;
            for (int item = item0; item < nitems && alive; item += item_step, ++icount) {
                const int64_t f0 = (int64_t)(item / p.groups * NB + rank) * TILE_M;
                const uint32_t gb = icount % p.gbufs, gph = icount / p.gbufs & 1u;
                const int64_t n0 = (int64_t)((item + item_step) / p.groups * NB + rank) * TILE_M;
                if (n0 < p.Nf && n0 != f0) {                      // the next item's rows and weights, on their way to L2
                    const int64_t n = p.Nf - n0 < TILE_M ? p.Nf - n0 : TILE_M;
                    if (p.stride == p.Ck) prefetch_l2(p.rows + n0 * p.stride, (uint32_t)(n * p.stride * 4));
                    prefetch_l2(p.w + n0 * p.Fp, (uint32_t)(n * p.Fp * 4));
                }
                if (staged) {
                    for (int ks = 0; ks < KST; ++ks, ++blocks) {
                        const uint32_t st = blocks % RAW_STAGES;
                        if (!mbar_wait(&raw_empty[st], (blocks / RAW_STAGES & 1u) ^ 1u, abort_flag)) { alive = false; break; }
                        mbar_arrive_expect_tx(&raw_full[st], RAW_BYTES);
                        tile_g2s(raw + st * RAW_BYTES, &rows_map, ks * 32, (int)f0, &raw_full[st]);
                        tile_g2s(raw + st * RAW_BYTES + KTILE_BYTES, &rows_map, ks * 32 + 16, (int)f0, &raw_full[st]);
                    }
                    continue;
                }
                if (!mbar_wait(&g_empty[gb], gph ^ 1u, abort_flag)) { alive = false; break; }
                mbar_arrive_expect_tx(&raw_full[gb], gtile_bytes);
                uint8_t* const dst = gtile + (size_t)gb * gtile_bytes;
                for (int ks = 0; ks < KST; ++ks) {
                    tile_g2s(dst + (size_t)ks * KTILE_BYTES, &rows_map, ks * 32, (int)f0, &raw_full[gb]);
                    tile_g2s(dst + (size_t)(KST + ks) * KTILE_BYTES, &rows_map, ks * 32 + 16, (int)f0, &raw_full[gb]);
                }
            }
            // The commits behind the last accumulator are waited for by nobody else, and in a pair they arrive in both CTAs: none leaves
            // its shared memory to another block while one is on its way.  A buffer that was never used is free from the start.
            for (int i = 0; i < p.gbufs && alive; ++i, ++icount)
                alive = mbar_wait(&g_empty[icount % p.gbufs], (icount / p.gbufs & 1u) ^ 1u, abort_flag);
            if (!alive) {                                         // let copies in flight land before shared memory is released
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000) { }
            }
        }
    } else if (warp == EWARPS) {
        // ===================== filter stream (TMA engine) =====================
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            bool alive = true;
            for (int item = item0; item < nitems && alive; item += item_step) {
                const int s0 = item % p.groups * p.per_group;
                const int s1 = s0 + p.per_group < p.nslices ? s0 + p.per_group : p.nslices;
                for (int blk = s0 * KST; blk < s1 * KST; blk += p.kb) {
                    if (!mbar_wait(&w_empty[s], ph ^ 1u, abort_flag)) { alive = false; break; }
                    mbar_arrive_expect_tx(&w_full[s], wstage_bytes);
                    const uint8_t* src = p.wimg + (size_t)blk * NB * wblk_bytes + (size_t)rank * w_bytes;
                    if (!PAIR) bulk_g2s(wst + (size_t)s * wstage_bytes, src, wstage_bytes, &w_full[s]);
                    else for (int i = 0; i < p.kb * NSPLIT; ++i)  // [K-block][hi, lo][rows]: this CTA's half of the rows
                        bulk_g2s(wst + (size_t)s * wstage_bytes + (size_t)i * w_bytes, src + (size_t)i * NB * w_bytes, w_bytes, &w_full[s]);
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
            }
            for (int i = 0; i < S && alive; ++i) {                // the last commits of every stage, as above
                alive = mbar_wait(&w_empty[s], ph ^ 1u, abort_flag);
                if (++s == S) { s = 0; ph ^= 1u; }
            }
            if (!alive) {                                         // let copies in flight land before shared memory is released
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000) { }
            }
        }
    } else {
        // ===================== MMA issue (rank 0), word that the filter has landed (rank 1) =====================
        if (PAIR && rank != 0) {
            if (elect_one()) {
                int s = 0;
                uint32_t ph = 0;
                bool alive = true;
                for (int item = item0; item < nitems && alive; item += item_step) {
                    const int s0 = item % p.groups * p.per_group;
                    const int s1 = s0 + p.per_group < p.nslices ? s0 + p.per_group : p.nslices;
                    for (int blk = s0 * KST; blk < s1 * KST; blk += p.kb) {
                        if (!mbar_wait(&w_full[s], ph, abort_flag)) { alive = false; break; }
                        arrive_first<PAIR>(&w_peer[s]);
                        if (++s == S) { s = 0; ph ^= 1u; }
                    }
                }
            }
        } else if (elect_one()) {
            const uint32_t idesc = instr_desc(FMT_BF16, NB * TILE_M, (uint32_t)p.nmma);
            const uint64_t dg_base = smem_desc_kmajor(smem_u32(gtile), 64, SWZ_64B);
            const uint64_t dw_base = smem_desc_kmajor(smem_u32(wst), 64, SWZ_64B);
            int s = 0;
            uint32_t ph = 0, icount = 0, sc = 0;
            bool alive = true;
            for (int item = item0; item < nitems && alive; item += item_step, ++icount) {
                const int s0 = item % p.groups * p.per_group;
                const int s1 = s0 + p.per_group < p.nslices ? s0 + p.per_group : p.nslices;
                const uint32_t gb = icount % p.gbufs, gph = icount / p.gbufs & 1u;
                const uint64_t dg_tile = dg_base + (uint64_t)((gb * gtile_bytes) >> 4);
                if (!wait_first<PAIR>(&g_full[gb], gph, abort_flag)) break;
                for (int slice = s0; slice < s1 && alive; ++slice, ++sc) {
                    const uint32_t a = sc & 1u;
                    if (!wait_first<PAIR>(&acc_empty[a], ((sc >> 1) & 1u) ^ 1u, abort_flag)) { alive = false; break; }
                    tc_fence_after();
                    const uint32_t d_tmem = tmem_base + a * NCOLS;
                    for (int ks0 = 0; ks0 < KST; ks0 += p.kb) {
                        if (!mbar_wait(&w_full[s], ph, abort_flag) || (PAIR && !mbar_wait_cluster(&w_peer[s], ph, abort_flag))) { alive = false; break; }
                        tc_fence_after();
                        for (int kk = 0; kk < p.kb; ++kk) {
                            const int ks = ks0 + kk;
                            const uint64_t dg_hi = dg_tile + (uint64_t)(((uint32_t)ks * KTILE_BYTES) >> 4);
                            const uint64_t dw_hi = dw_base + (uint64_t)(((uint32_t)s * wstage_bytes + kk * wblk_bytes) >> 4);
#pragma unroll
                            for (int k2 = 0; k2 < 2; ++k2) {
                                const uint64_t adv = (uint64_t)(k2 * 2);
                                const uint32_t first = (ks | k2) != 0;
                                if (NSPLIT == 1) {
                                    multiply<PAIR>(d_tmem, dg_hi + adv, dw_hi + adv, idesc, first);
                                } else {
                                    const uint64_t dg_lo = dg_hi + (uint64_t)(((uint32_t)KST * KTILE_BYTES) >> 4);
                                    const uint64_t dw_lo = dw_hi + (uint64_t)(w_bytes >> 4);
                                    multiply<PAIR>(d_tmem, dg_lo + adv, dw_hi + adv, idesc, first);
                                    multiply<PAIR>(d_tmem, dg_hi + adv, dw_lo + adv, idesc, 1u);
                                    multiply<PAIR>(d_tmem, dg_hi + adv, dw_hi + adv, idesc, 1u);
                                }
                            }
                        }
                        commit<PAIR>(&w_empty[s]);
                        if (++s == S) { s = 0; ph ^= 1u; }
                    }
                    if (alive) commit<PAIR>(&acc_full[a]);
                }
                if (alive) commit<PAIR>(&g_empty[gb]);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_sync();                           // both have drained their barriers: nothing of this CTA is used any more
    tc_fence_after();
    if (warp == EWARPS) {
        if constexpr (PAIR) tmem_dealloc_pair(tmem_base, 512);
        else tmem_dealloc(tmem_base, 512);
    }
    if (tid == 0 && *abort_flag && p.async_err) {
        *p.async_err = 2;
        __threadfence_system();
    }
}

// ---------------------------------------------------------------------------- host side
struct Plan { bool pair, staged; int nsplit, nq, nslices, kst, nmma, nblocks, gbufs; size_t smem, wimg_bytes; };

// K-blocks of 32 contracted channels from which CTAs work in pairs, three products per term.  A pair halves the traffic of the filter
// blocks, from L2 and from shared memory, and pays with a round trip between two SMs per slice: worth it where a slice is 24
// products long (464 000 faces, 128 -> 128: 25 bases 851 -> 761 us, 16 bases 529 -> 466, 9 bases 343 -> 312; 3 000 faces 27.6 -> 25.6),
// not at 18 (96 -> 96, 16 bases: 294 -> 306), 12 (880 000 faces, 64 -> 64: 288 -> 331) or 8 (bf16, 128 -> 128, 25 bases: 400 -> 542).
constexpr int PAIR_FROM = 4;
// Five and seven blocks make a round trip each, as no larger filter stage divides them.  Five still pair where CTAs have several tiles,
// because only a pair's smaller filter blocks leave room for a second tile buffer (160 -> 128, 16 bases, alone -> in pairs: 40 000 faces 135 ->
// 89 us, 10 000 34 -> 45); seven never (224 -> 128, 16 bases: 40 000 faces 179 -> 194, 10 000 44 -> 54).
static bool in_pairs(int kst, bool several_tiles) { return kst >= PAIR_FROM && kst != 7 && (kst != 5 || several_tiles); }

static int nq_of(int F) { return F == 4 ? NQ<4> : F == 9 ? NQ<9> : F == 16 ? NQ<16> : NQ<25>; }

static Plan plan(int Cn, int CkAll, int F, int precision, bool several_tiles) {
    Plan pl;
    const int Ck = CkAll < MAX_CK ? CkAll : MAX_CK;
    pl.nsplit = operand_mode(precision).nsplit;
    pl.nq = nq_of(F);
    const int g = F == 25 ? G<25> : G<4>, cn = (Cn + g - 1) / g * g;
    pl.kst = (Ck + 31) / 32;
    pl.pair = pl.nsplit == 2 && in_pairs(pl.kst, several_tiles);
    const int step = pl.pair ? 32 : 16;                           // columns of a product
    pl.nmma = ((pl.nq > cn ? cn : pl.nq) * F + step - 1) / step * step;
    pl.nslices = (Cn + pl.nq - 1) / pl.nq;
    const size_t budget = 226 * 1024;
    const size_t gt = (size_t)2 * pl.kst * KTILE_BYTES, wblk = (size_t)pl.nsplit * pl.nmma * 64, ws = pl.pair ? wblk / 2 : wblk;
    // a second tile buffer takes the row copy off the critical path, when at least three filter blocks still fit beside it
    pl.gbufs = (2 * gt + 1024 + 640 + 3 * ws <= budget) ? 2 : 1;
    if (3 * gt + 1024 + 640 + 2 * pl.kst * ws <= budget) pl.gbufs = 3;
    size_t fixed = pl.gbufs * gt + 1024 + 640;
    // One operand fills half of what its rows take on the way.  Where that leaves a single buffer, rows come through stages of one K-block
    // instead of in place, and two buffers of the operand alone fit (bf16, 256 -> 256, 25 bases, 40 000 faces: 198 us in place, 169
    // so; 192 -> 64, 9 bases, 300 000 faces 214 and 140).
    pl.staged = pl.nsplit == 1 && pl.gbufs == 1;
    if (pl.staged) {
        pl.gbufs = 2;
        fixed = (size_t)2 * pl.kst * KTILE_BYTES + RAW_STAGES * RAW_BYTES + 1024 + 640;
    }
    pl.nblocks = (int)((budget - fixed) / ws);
    if (pl.nblocks > 16) pl.nblocks = 16;
    pl.smem = fixed + pl.nblocks * ws;
    pl.wimg_bytes = (size_t)pl.nslices * pl.kst * wblk;
    return pl;
}

// bf16 operands (hi + lo or single), rows readable 16 bytes at a time
bool supported(int Cn, int Ck, int F, int precision) {
    if (precision != PB200_PREC_FP32 && precision != PB200_PREC_BF16) return false;
    if (!(F == 4 || F == 9 || F == 16 || F == 25) || Cn < 1 || Ck < 4 || Ck % 4 != 0) return false;
    for (const bool several : {false, true}) {
        const Plan pl = plan(Cn, Ck, F, precision, several);
        if (pl.nblocks < 2 || pl.smem > 227 * 1024) return false;
    }
    return true;
}

// the image of a pair, whose columns are rounded further up, is no smaller than the other
size_t workspace_bytes(int Cn, int Ck, int F, int precision) { return align_up(plan(Cn, Ck, F, precision, true).wimg_bytes, 256); }

// Tensor map of (Nf, channels) floats with `stride` floats between rows: boxes of 16 channels x 128 rows, laid down as 64-byte rows with
// the 64-byte swizzle, the layout of the product's operand
static int map_rows(CUtensorMap* map, const float* rows, int64_t Nf, int channels, int stride, const char* label) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            fn = nullptr;
        return (Encode)fn;
    }();
    PB_REQUIRE(encode, PB200_ECUDA, "%s: the driver has no cuTensorMapEncodeTiled", label);
    const cuuint64_t dims[2] = {(cuuint64_t)channels, (cuuint64_t)Nf}, strides[1] = {(cuuint64_t)stride * 4};
    const cuuint32_t box[2] = {16, TILE_M}, step[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(rows), dims, strides, box, step,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    PB_REQUIRE(r == CUDA_SUCCESS, PB200_ECUDA, "%s: cuTensorMapEncodeTiled failed (%d) for %lld rows of %d floats", label, (int)r,
               (long long)Nf, channels);
    return PB200_OK;
}

template <int NSPLIT, int F, bool PAIR>
static int launch(const char* label, const Params& p, const CUtensorMap& map, int grid, size_t smem, cudaStream_t stream) {
    PB_CUDA(cudaFuncSetAttribute(f2f_one_sample_tc_kernel<NSPLIT, F, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    static const int regs = [] {                                  // built with fewer it would wait for registers that are not there (build.py refuses to)
        cudaFuncAttributes a;
        return cudaFuncGetAttributes(&a, f2f_one_sample_tc_kernel<NSPLIT, F, PAIR>) == cudaSuccess ? a.numRegs : 0;
    }();
    PB_REQUIRE(regs == REGS_LAUNCH, PB200_ECUDA, "%s: built with %d registers per thread instead of %d", label, regs, REGS_LAUNCH);
    cudaLaunchAttribute two;
    two.id = cudaLaunchAttributeClusterDimension;
    two.val.clusterDim.x = 2; two.val.clusterDim.y = two.val.clusterDim.z = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid); c.blockDim = dim3(NTHREADS); c.dynamicSmemBytes = smem; c.stream = stream;
    c.attrs = &two; c.numAttrs = PAIR ? 1 : 0;
    LaunchScope scope(label, stream);
    PB_CUDA(cudaLaunchKernelEx(&c, f2f_one_sample_tc_kernel<NSPLIT, F, PAIR>, p, map));
    return PB200_OK;
}

// forward = true: the operator's forward pass (filter (Cn, Ck, F)); false: its input gradient (filter (Ck, Cn, F))
int run(int64_t Nf, int Cn, int Ck, int F, const float* rows, const float* filter, const float* w, int Fp, float* out, int precision,
        void* ws, cudaStream_t stream, bool forward) {
    const char* label = forward ? "f2f_fwd_one_tc" : "f2f_bwd_gin_one_tc";
    int rc = check_async_error(forward ? "facet2facet_forward" : "facet2facet_backward");
    if (rc) return rc;
    const int64_t s_ck = forward ? (int64_t)F : (int64_t)Cn * F, s_cn = forward ? (int64_t)Ck * F : (int64_t)F;
    for (int k0 = 0; k0 < Ck; k0 += MAX_CK) {
        const int chunk = Ck - k0 < MAX_CK ? Ck - k0 : MAX_CK;
        // a plan of its own for every chunk: the last one may be short
        const Plan pl = plan(Cn, chunk, F, precision, ceil_div(Nf, TILE_M) > sm_count());
        const int kst = pl.kst;
        const int nb = pl.pair ? 2 : 1, sms = sm_count() / nb;        // CTAs, and those that work on items of their own
        const int64_t ntiles = ceil_div(Nf, nb * TILE_M);
        // Slice groups of a tile.  With fewer tiles than SMs a tile's slices go to as many CTAs as there are.  With a few tiles per
        // SM the last wave is short of tiles: groups are halved while that evens it out, but a group keeps enough products (two
        // slices of three, four of one) for the copy of the next item's rows to hide behind.
        int groups = 1;
        if (ntiles < sms) {
            groups = (int)(sms / ntiles);
            if (groups > pl.nslices) groups = pl.nslices;
        } else {
            const int keep = pl.nsplit == 2 ? 2 : 4;
            while (ntiles * groups < 8LL * sms && pl.nslices >= 2 * groups * keep) groups *= 2;
        }
        const int per_group = (int)ceil_div(pl.nslices, groups);
        groups = (int)ceil_div(pl.nslices, per_group);
        const int64_t items = ntiles * groups;
        PB_REQUIRE(items < 0x7fffffff / 2, PB200_EINVAL, "%s: %lld faces are too many", label, (long long)Nf);
        const int grid = nb * (int)(items < sms ? items : sms);
        rc = gin::prep_filter_bf16(F, Cn, k0, chunk, pl.nq, pl.nslices, kst, pl.nsplit, pl.nmma, s_ck, s_cn, filter, (uint8_t*)ws, stream);
        if (rc) return rc;
        Params p;
        p.Nf = Nf; p.nitems = (int)items; p.Cn = Cn; p.Ck = chunk;
        p.nslices = pl.nslices; p.kst = kst; p.nmma = pl.nmma; p.gbufs = pl.gbufs; p.staged = pl.staged;
        p.kb = kst;
        while (p.kb > 1 && (kst % p.kb != 0 || pl.nblocks < 2 * p.kb)) --p.kb;
        p.nstages = pl.nblocks / p.kb;
        p.groups = groups; p.per_group = per_group;
        p.rows = rows + k0; p.stride = Ck; p.accumulate = k0 > 0 ? 1 : 0;
        p.w = w; p.Fp = Fp; p.wimg = (const uint8_t*)ws; p.out = out;
        p.async_err = async_error_word();
        p.wait_budget = wait_budget_kclocks();
        CUtensorMap map;
        rc = map_rows(&map, p.rows, Nf, chunk, Ck, label);
        if (rc) return rc;
        const bool two = pl.nsplit == 2;
        auto go = [&](auto f) {
            constexpr int FF = decltype(f)::value;
            if (pl.pair) return launch<2, FF, true>(label, p, map, grid, pl.smem, stream);
            return two ? launch<2, FF, false>(label, p, map, grid, pl.smem, stream) : launch<1, FF, false>(label, p, map, grid, pl.smem, stream);
        };
        switch (F) {
            case 4: rc = go(std::integral_constant<int, 4>{}); break;
            case 9: rc = go(std::integral_constant<int, 9>{}); break;
            case 16: rc = go(std::integral_constant<int, 16>{}); break;
            default: rc = go(std::integral_constant<int, 25>{}); break;
        }
        if (rc) return rc;
    }
    return PB200_OK;
}

}  // namespace one
}  // namespace tc
}  // namespace pb
