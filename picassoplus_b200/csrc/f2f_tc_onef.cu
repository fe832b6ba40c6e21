// facet2facet filter gradient for faces with exactly one sample each, on tcgen05 + TMEM:
//
//   gradFilter[co, ci, d] = sum_f w[f, d] * input[f, ci] * gradOutput[f, co]
//
// Faces are the contracted dimension of a product whose rows are (basis, channel of one tensor) pairs and whose columns are
// channels of the other.  One tensor has to be multiplied by the weights ("expanded", F operand elements per element); the
// other is a plain operand.  f2f_tc_gfilter.cu, which serves faces with several samples, writes the expanded operand to shared
// memory, pads the output channels to 128, and works through stages of 16 faces whose loads, records and hand-overs form one
// chain: with all its loads, all its arithmetic and two of three products taken out a stage still took 1030 of its 1300 clocks
// (1 758 000 faces, 64 -> 64, 16 bases: 2037 us, products alone 300).  Here
//   * the expanded operand lives in TMEM, as the A side: lane = (basis, channel), columns = faces.  A thread keeps one channel's
//     values of the stage's faces in registers, multiplies them by one basis' weights per tile of 128 rows, splits and
//     stores 16 columns; shared memory holds only the plain operand and the weights;
//   * rows and columns are as wide as the channels need: 64 channels give tiles of two bases, 32 of four, and the columns are
//     the other tensor's channels rounded up to 16.  Either tensor can be the expanded one;
//   * every role has several stages under way: one warp starts the bulk copies of a whole ring of stages, four groups of four
//     warps build the expanded operand of every fourth stage each (one warp per TMEM quadrant), four warps the plain
//     operand and the transposed weights of every fourth stage each, and the thread that issues the products goes round the tiles.
// A CTA owns a block of channels of both tensors, a run of tiles (as many as fit in TMEM beside the ring of expanded
// operands) and a chunk of faces; the runs of one chunk work side by side, so that their common rows come from L2.
// The accumulators are added to the CTA's sums in global memory every 4096 faces (the tensor core's adder truncates, see
// f2f_tc_gfilter.cu) with reductions that nothing waits for; each address has one thread that adds, so the order is fixed.
// A second kernel adds the chunks in order.  All waits are bounded.
// Now 685 us for the case above (bf16 1964 -> 372), 2074 for 930 000 faces, 128 -> 128, 25 bases (2524 before; bf16 2335 -> 1490).
// What bounds it: hand-overs -- a stage without any work takes 490 clocks, with 64 channels 880 of which 384 are products, with
// 128 channels 1090 (576 products; two operand buffers are what fits beside three accumulators).  Two or four groups on one
// stage are slower (697 -> 814, 1196 us), two bulk-copy warps the same.
#include <math.h>
#include <string.h>
#include <type_traits>
#include "common.cuh"
#include "tc_ptx.cuh"
#include "tc_runtime.cuh"

namespace pb {
namespace tc {
namespace onef {

using namespace ptx;

constexpr int EG = 4;                         // groups of four warps (TMEM quadrants) that build the expanded operand
constexpr int EWARPS = 4 * EG;
constexpr int GWARPS = 4;                     // warps that write the plain operand and the weights
constexpr int MMA_WARP = EWARPS + GWARPS;
constexpr int LOAD_WARP = MMA_WARP + 1;
constexpr int NTHREADS = (LOAD_WARP + 1) * 32;
constexpr int ROWS = 128;                     // rows of a tile (TMEM lanes)
constexpr int MAX_N = 128;                    // columns of a tile
constexpr int TMEM_COLS = 512;
constexpr int ACOLS = 16;                     // columns of one tile's operand in a stage
constexpr int MAX_SLOTS = 8;                  // stages of the plain operand in shared memory
constexpr int MAX_F = 32;
constexpr int MAX_NT = 5;                      // tiles of a CTA
constexpr int MAX_RAW = 8;                    // stages of raw rows in shared memory
constexpr int FLUSH_FACES = 4096;             // as in f2f_tc_gfilter.cu

// faces of a stage: 16 columns of TMEM per tile in both modes (hi + lo of 16 faces, or 32 faces)
template <int NSPLIT> constexpr int FACES = NSPLIT == 2 ? 16 : 32;

struct Params {
    int64_t Nf;
    const float* x;                  // expanded tensor, rows of C1 floats
    const float* g;                  // plain tensor, rows of C2 floats
    const float* w;                  // weight rows of Fp floats
    int C1, C2, F, Fp;
    int R, dpt;                      // channels of x per block, bases per tile (dpt * R <= 128)
    int nb1, nb2, N;                 // channel blocks of x and of g, columns of a tile (multiple of 16)
    int gpitch;                      // floats per staged row of g
    int nbuf, a_col;                 // operand ring: buffers, first TMEM column
    int tiles, groups, nt;           // tiles of a channel block, runs of them, longest run
    int chunks, nraw, slots;         // face chunks, raw ring depth, plain operand ring depth (4 or 8 each)
    int64_t nstages;
    float* sums;                     // [CTA][nt * N rounded up to 32][128]
    int swap;                        // x is gradOutput
    float* out;                      // (Cout, Cin, F)
    int* async_err;
    int wait_budget;
};

__host__ __device__ __forceinline__ int sum_cols(const Params& p) { return (p.nt * p.N + 31) / 32 * 32; }
__host__ __device__ __forceinline__ int raw_floats(const Params& p, int faces) { return faces * (p.R + p.gpitch + p.Fp); }
__device__ __forceinline__ int run_start(const Params& p, int group) { return group * p.tiles / p.groups; }

// position in a ring, and the parity of its pass
struct Ring {
    int i = 0;
    uint32_t ph = 0;
    __device__ __forceinline__ void step(int by, int n) { for (i += by; i >= n; i -= n) ph ^= 1u; }
};

__device__ __forceinline__ void red_add(float* p, float v) { asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory"); }

// One warp's share of a flush: its TMEM quadrant, every EG-th group of 32 columns, stored to or added to the CTA's sums
__device__ __noinline__ void flush(uint32_t tmem_quadrant, float* sums, int first, int ngroups, bool add) {
    for (int gi = first; gi < ngroups; gi += EG) {
        uint32_t r[32];
        tmem_ld32(tmem_quadrant + (uint32_t)(gi * 32), r);
        tmem_ld_wait();
        float* dst = sums + (size_t)(gi * 32) * ROWS;
        if (add) {
#pragma unroll
            for (int j = 0; j < 32; ++j) red_add(dst + j * ROWS, __uint_as_float(r[j]));
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) dst[j * ROWS] = __uint_as_float(r[j]);
        }
    }
}

template <int NSPLIT>
__global__ void __launch_bounds__(NTHREADS, 1) f2f_one_sample_gfilter_kernel(Params p) {
    constexpr int FS = FACES<NSPLIT>;
    constexpr int FLUSH = FLUSH_FACES / FS;
    constexpr int W_BYTES = MAX_F * FS * 4;                       // weights of a stage, [basis][face]
    // A wait tells a barrier's phase from the one before, not from the one two before or behind.  A warp that takes every
    // fourth stage therefore has rings of 4 or 8 slots, where it has itself seen a slot's last phase; what it waits for of the
    // products is the end of a stage 2 to 8 stages back, on barriers that come round every 8 stages.
    static_assert(EG == 4 && GWARPS == 4, "see the ring depths");
    const int SLOTS = p.slots;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int blocks = (p.N + 63) / 64;                           // 64-column blocks of the plain operand
    const uint32_t sbo = (uint32_t)blocks * 1024u;                // next 8 faces
    const uint32_t g_split = (FS / 8) * sbo, slot_bytes = NSPLIT * g_split;
    const uint32_t raw_bytes = (uint32_t)raw_floats(p, FS) * 4u;  // rows of x, of g, weights
    const uint32_t raw_g = (uint32_t)(FS * p.R) * 4u, raw_w = raw_g + (uint32_t)(FS * p.gpitch) * 4u;
    uint8_t* const gring = smem;
    uint8_t* const wring = smem + SLOTS * (size_t)slot_bytes;
    uint8_t* const raw = wring + SLOTS * W_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(raw + p.nraw * (size_t)raw_bytes);
    uint64_t* g_full = bars;                      // [SLOTS]   plain operand and weights of a stage written
    uint64_t* a_full = bars + MAX_SLOTS;          // [4]       expanded operand of a stage (mod 4) written
    uint64_t* done = a_full + 4;                  // [8]       products of a stage (mod 8) done
    uint64_t* raw_full = done + 8;                // [MAX_RAW] rows of a stage have arrived
    uint64_t* raw_free = raw_full + MAX_RAW;      // [MAX_RAW] and have been read
    uint64_t* acc_done = raw_free + MAX_RAW;      // all products issued so far complete
    uint64_t* acc_free = acc_done + 1;            // accumulators read out
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    if (tid == 0) {
        for (int s = 0; s < SLOTS; ++s) mbar_init(&g_full[s], 1);
        for (int b = 0; b < 4; ++b) mbar_init(&a_full[b], 4);
        for (int b = 0; b < 8; ++b) mbar_init(&done[b], 1);
        for (int r = 0; r < p.nraw; ++r) { mbar_init(&raw_full[r], 1); mbar_init(&raw_free[r], 5); }
        mbar_init(acc_done, 1);
        mbar_init(acc_free, EWARPS);
        abort_flag[0] = 0;
        abort_flag[1] = p.wait_budget;
        fence_barrier_init();
    }
    // rows and channels that a last stage or a last block does not have are read (and multiplied by zero, or never looked at)
    for (uint32_t i = tid; i < p.nraw * raw_bytes / 4; i += NTHREADS) reinterpret_cast<float*>(raw)[i] = 0.f;
    fence_proxy_async();
    if (warp == MMA_WARP) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // this CTA's channel blocks, run of tiles and chunk of faces
    const int kinds = p.nb1 * p.nb2 * p.groups;
    const int chunk = blockIdx.x / kinds, kind = blockIdx.x - chunk * kinds;
    const int pair = kind / p.groups, group = kind - pair * p.groups;
    const int b1 = pair % p.nb1, b2 = pair / p.nb1;
    const int t0 = run_start(p, group), nt = run_start(p, group + 1) - t0;
    const int64_t st0 = p.nstages * chunk / p.chunks;
    const int nst = (int)(p.nstages * (chunk + 1) / p.chunks - st0);

    if (warp < EWARPS) {
        // ===================== expanded operand (thread = row of a tile) =====================
        const int q = warp & 3, eg = warp >> 2, r = q * 32 + lane;
        const int dl = r / p.R, c = r - dl * p.R;                  // basis inside the tile, channel inside the block
        const int d0 = t0 * p.dpt + dl;
        const uint32_t quadrant = tmem_base + ((uint32_t)(q * 32) << 16);
        const uint32_t w32 = smem_u32(wring), x32 = smem_u32(raw) + (uint32_t)c * 4u;
        const int ngroups = (nt * p.N + 31) / 32;
        float* const sums = p.sums + (size_t)blockIdx.x * sum_cols(p) * ROWS + r;
        Ring rr, ar, gr;
        rr.step(eg, p.nraw); ar.step(eg, p.nbuf); gr.step(eg, SLOTS);
        uint32_t aph = 0;
        bool alive = true, flushed = false;
        int boundary = FLUSH - 1;                                  // last stage before the next flush
        for (int st = eg; st < nst; st += EG) {
            // stage st needs a product behind the boundary to be done, and that one needs the accumulators read out; a
            // boundary without such a stage for every group is left to the end
            if (st > boundary + p.nbuf && boundary + p.nbuf + EG < nst) {
                if (!warp_wait(acc_done, aph, abort_flag, lane)) { alive = false; break; }
                aph ^= 1u;
                tc_fence_after();
                flush(quadrant, sums, eg, ngroups, flushed);
                flushed = true;
                boundary += FLUSH;
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_free);
            }
            // (the warp that reports the weights has seen the rows arrive)
            const int slot = gr.i;
            if (!warp_wait(&g_full[slot], gr.ph, abort_flag, lane)) { alive = false; break; }
            float x[FS];
            {
                const uint32_t a = x32 + (uint32_t)rr.i * raw_bytes, pitch = (uint32_t)p.R * 4u;
#pragma unroll
                for (int k = 0; k < FS; ++k) x[k] = lds_f32(a + k * pitch);
            }
            if (st >= p.nbuf && !warp_wait(&done[(st - p.nbuf) & 7], (uint32_t)((st - p.nbuf) >> 3) & 1u, abort_flag, lane)) {
                alive = false;
                break;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_free[rr.i]);
            tc_fence_after();
            const uint32_t dst = quadrant + (uint32_t)(p.a_col + ar.i * p.nt * ACOLS), ws = w32 + (uint32_t)slot * W_BYTES;
            for (int t = 0; t < nt; ++t) {
                const int d = d0 + t * p.dpt;                      // rows without a basis or a channel are never read
                const uint32_t wd = ws + (uint32_t)((d < p.F ? d : 0) * FS) * 4u;
                uint32_t o[16];
#pragma unroll
                for (int k = 0; k < FS; k += 4) {
                    const float4 wv = lds_f4(wd + k * 4);
                    const float2 u = __fmul2_rn(make_float2(x[k], x[k + 1]), make_float2(wv.x, wv.y));
                    const float2 v = __fmul2_rn(make_float2(x[k + 2], x[k + 3]), make_float2(wv.z, wv.w));
                    if (NSPLIT == 2) {
                        split_bf16x2(u.x, u.y, o[k / 2], o[8 + (k / 2) % 8]);
                        split_bf16x2(v.x, v.y, o[k / 2 + 1], o[8 + (k / 2 + 1) % 8]);
                    } else {
                        o[k / 2] = pack_bf16x2(u.x, u.y);
                        o[k / 2 + 1] = pack_bf16x2(v.x, v.y);
                    }
                }
                tmem_st16(dst + (uint32_t)(t * ACOLS), o);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[st & 3]);
            rr.step(EG, p.nraw); ar.step(EG, p.nbuf); gr.step(EG, SLOTS);
        }
        if (alive && warp_wait(acc_done, aph, abort_flag, lane)) {
            tc_fence_after();
            flush(quadrant, sums, eg, ngroups, flushed);
            tc_fence_before();
        }
    } else if (warp < MMA_WARP) {
        // ===================== plain operand and weights (warp = every GWARPS-th stage) =====================
        const int gw = warp - EWARPS;
        const uint32_t g32 = smem_u32(gring), w32 = smem_u32(wring), raw32 = smem_u32(raw);
        const int fl = lane % FS;
        // `n` rows of g at `src` as the operand at `dst`; LPR lanes of a row hold 4 channels each
        auto put_rows = [&](auto lprc, uint32_t src, uint32_t dst, int n) {
            constexpr int LPR = decltype(lprc)::value, RPP = 32 / LPR;
            const int l = lane % LPR, rsub = lane / LPR;
            if (4 * l >= p.N) return;
            const bool live = b2 * p.N + 4 * l < p.C2;
            // 8-byte half l&1 of 16-byte chunk (l&15)/2 ^ (f&7) of row f&7; rows of a pass differ in bits that rsub does not have
            dst += (uint32_t)(l >> 4) * 1024u + (uint32_t)(l & 1) * 8u + (uint32_t)rsub * 128u
                   + ((((uint32_t)(l & 15) >> 1) ^ (uint32_t)rsub) << 4);
            src += (uint32_t)(rsub * p.gpitch + 4 * l) * 4u;
#pragma unroll
            for (int k = 0; k < FS; k += RPP) {
                float4 v = lds_f4(src + (uint32_t)(k * p.gpitch) * 4u);
                if (!live || k + rsub >= n) v = zero4();
                const uint32_t a = (dst ^ ((uint32_t)(k & 7) << 4)) + (uint32_t)(k >> 3) * sbo + (uint32_t)(k & 7) * 128u;
                uint32_t h0, h1, l0, l1;
                if (NSPLIT == 2) {
                    split_bf16x2(v.x, v.y, h0, l0);
                    split_bf16x2(v.z, v.w, h1, l1);
                    sts_u2(a + g_split, l0, l1);
                } else {
                    h0 = pack_bf16x2(v.x, v.y);
                    h1 = pack_bf16x2(v.z, v.w);
                }
                sts_u2(a, h0, h1);
            }
        };
        Ring rr, gr;
        rr.step(gw, p.nraw); gr.step(gw, SLOTS);
        for (int st = gw; st < nst; st += GWARPS) {
            const int64_t left = p.Nf - (st0 + st) * FS;
            const int n = left < FS ? (int)left : FS;              // faces of the stage
            if ((st >= SLOTS && !warp_wait(&done[(st - SLOTS) & 7], (uint32_t)((st - SLOTS) >> 3) & 1u, abort_flag, lane)) ||
                !warp_wait(&raw_full[rr.i], rr.ph, abort_flag, lane)) break;
            const uint32_t rb = raw32 + (uint32_t)rr.i * raw_bytes, gdst = g32 + (uint32_t)gr.i * slot_bytes;
            if (p.N <= 32) put_rows(std::integral_constant<int, 8>{}, rb + raw_g, gdst, n);
            else if (p.N <= 64) put_rows(std::integral_constant<int, 16>{}, rb + raw_g, gdst, n);
            else put_rows(std::integral_constant<int, 32>{}, rb + raw_g, gdst, n);
            const uint32_t wdst = w32 + (uint32_t)gr.i * W_BYTES + (uint32_t)fl * 4u;
#pragma unroll
            for (int i = 0; i < MAX_F / 4 * FS / 32; ++i) {
                const int quad = lane / FS + i * (32 / FS);
                if (4 * quad >= p.Fp) continue;
                float4 v = lds_f4(rb + raw_w + (uint32_t)(fl * p.Fp + 4 * quad) * 4u);
                if (fl >= n) v = zero4();
                const uint32_t a = wdst + (uint32_t)(4 * quad * FS) * 4u;
                sts_f32(a, v.x); sts_f32(a + FS * 4, v.y); sts_f32(a + 2 * FS * 4, v.z); sts_f32(a + 3 * FS * 4, v.w);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&g_full[gr.i]); mbar_arrive(&raw_free[rr.i]); }
            gr.step(GWARPS, SLOTS);
            rr.step(GWARPS, p.nraw);
        }
    } else if (warp == LOAD_WARP) {
        // ===================== bulk copies of the rows =====================
        const int xw = p.C1 - b1 * p.R < p.R ? p.C1 - b1 * p.R : p.R, gwid = p.C2 - b2 * p.N < p.gpitch ? p.C2 - b2 * p.N : p.gpitch;
        Ring rr;
        bool alive = true;
        if (elect_one()) {
            for (int st = 0; st < nst; ++st) {
                const int64_t f0 = (st0 + st) * FS, left = p.Nf - f0;
                const int n = left < FS ? (int)left : FS;
                if (!mbar_wait(&raw_free[rr.i], rr.ph ^ 1u, abort_flag)) { alive = false; break; }
                uint8_t* const dst = raw + (size_t)rr.i * raw_bytes;
                uint64_t* bar = &raw_full[rr.i];
                mbar_arrive_expect_tx(bar, (uint32_t)(n * (xw + gwid + p.Fp)) * 4u);
                if (p.nb1 == 1) bulk_g2s(dst, p.x + f0 * p.C1, (uint32_t)(n * p.C1) * 4u, bar);
                else for (int k = 0; k < n; ++k) bulk_g2s(dst + (size_t)k * p.R * 4, p.x + (f0 + k) * p.C1 + b1 * p.R, (uint32_t)xw * 4u, bar);
                if (p.nb2 == 1) bulk_g2s(dst + raw_g, p.g + f0 * p.C2, (uint32_t)(n * p.C2) * 4u, bar);
                else for (int k = 0; k < n; ++k) bulk_g2s(dst + raw_g + (size_t)k * p.gpitch * 4, p.g + (f0 + k) * p.C2 + b2 * p.N, (uint32_t)gwid * 4u, bar);
                bulk_g2s(dst + raw_w, p.w + f0 * p.Fp, (uint32_t)(n * p.Fp) * 4u, bar);
                rr.step(1, p.nraw);
            }
        }
        if (!alive) {                                              // let copies in flight land before shared memory is released
            const long long t = clock64();
            while (clock64() - t < 2000000) { }
        }
    } else if (elect_one()) {
        // ===================== products =====================
        const uint32_t idesc = instr_desc(FMT_BF16, ROWS, (uint32_t)p.N) | (1u << 16);      // B is MN-major
        const uint64_t dg = smem_desc_mnmajor_b16(smem_u32(gring), 1024, sbo);
        const uint32_t a_first = tmem_base + (uint32_t)p.a_col, a_step = (uint32_t)(p.nt * ACOLS), a_end = a_first + p.nbuf * a_step;
        const uint64_t g_step = slot_bytes >> 4, g_end = dg + SLOTS * g_step, lo = g_split >> 4;
        // every instruction of this thread is on the way from one stage to the next: the number of tiles is a constant in it
        auto products = [&](auto ntc) {
            constexpr int NT = decltype(ntc)::value;
            uint32_t d[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) d[t] = tmem_base + (uint32_t)(t * p.N);
            bool wait_free = false;
            uint32_t fph = 0, accumulate = 0, a = a_first;
            uint64_t g_hi = dg;
            int left = FLUSH;                                      // stages until the next flush
            for (int st = 0; st < nst; ++st) {
                // (the warps that report the expanded operand have seen the plain one)
                if (!mbar_wait(&a_full[st & 3], (uint32_t)(st >> 2) & 1u, abort_flag)) return;
                if (wait_free) {
                    wait_free = false;
                    if (!mbar_wait(acc_free, fph, abort_flag)) return;
                    fph ^= 1u;
                    accumulate = 0;
                }
                tc_fence_after();
                auto round = [&](uint32_t acol, uint64_t b, uint32_t acc) {
#pragma unroll
                    for (int t = 0; t < NT; ++t) mma_f16_ta(d[t], a + (uint32_t)(t * ACOLS) + acol, b, idesc, acc);
                };
                if (NSPLIT == 2) {
                    round(8, g_hi, accumulate);
                    round(0, g_hi + lo, 1u);
                    round(0, g_hi, 1u);
                } else {
                    round(0, g_hi, accumulate);
                    round(8, g_hi + (uint64_t)((2 * sbo) >> 4), 1u);
                }
                tc_commit(&done[st & 7]);
                accumulate = 1;
                if (--left == 0) {
                    left = FLUSH;
                    if (st + p.nbuf + EG < nst) { tc_commit(acc_done); wait_free = true; }
                }
                if ((a += a_step) == a_end) a = a_first;
                if ((g_hi += g_step) == g_end) g_hi = dg;
            }
            tc_commit(acc_done);
        };
        switch (nt) {
            case 1: products(std::integral_constant<int, 1>{}); break;
            case 2: products(std::integral_constant<int, 2>{}); break;
            case 3: products(std::integral_constant<int, 3>{}); break;
            case 4: products(std::integral_constant<int, 4>{}); break;
            default: products(std::integral_constant<int, 5>{}); break;
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == MMA_WARP) tmem_dealloc(tmem_base, TMEM_COLS);
    if (tid == 0 && *abort_flag && p.async_err) {
        *p.async_err = 3;
        __threadfence_system();
    }
}

// gradFilter = the chunks' sums in order; a block takes 64 rows of one column, a quarter of it every fourth chunk
__global__ void __launch_bounds__(256) f2f_one_sample_gfilter_reduce_kernel(Params p) {
    __shared__ float part[4][64];
    const int e = threadIdx.x & 63, sub = threadIdx.x >> 6;
    const int64_t total = (int64_t)p.nb1 * p.nb2 * p.tiles * p.N * 2;
    const int kinds = p.nb1 * p.nb2 * p.groups;
    const size_t cta = (size_t)sum_cols(p) * ROWS;
    for (int64_t i = blockIdx.x; i < total; i += gridDim.x) {
        const int r = (int)(i & 1) * 64 + e;
        int64_t u = i >> 1;
        const int n = (int)(u % p.N); u /= p.N;
        const int t = (int)(u % p.tiles), pair = (int)(u / p.tiles);
        int group = 0;
        while (run_start(p, group + 1) <= t) ++group;
        const int col = (t - run_start(p, group)) * p.N + n;
        const int dl = r / p.R, c1 = pair % p.nb1 * p.R + r - dl * p.R, c2 = pair / p.nb1 * p.N + n, d = t * p.dpt + dl;
        const bool live = dl < p.dpt && d < p.F && c1 < p.C1 && c2 < p.C2;
        const float* src = p.sums + (size_t)(pair * p.groups + group) * cta + (size_t)col * ROWS + r;
        float s = 0.f;
        if (live)
#pragma unroll 4
            for (int k = sub; k < p.chunks; k += 4) s += __ldg(src + (size_t)k * kinds * cta);
        part[sub][e] = s;
        __syncthreads();
        if (sub == 0 && live) {
            const int ci = p.swap ? c2 : c1, co = p.swap ? c1 : c2, Cin = p.swap ? p.C2 : p.C1;
            p.out[((int64_t)co * Cin + ci) * p.F + d] = (part[0][e] + part[1][e]) + (part[2][e] + part[3][e]);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------- host side
static size_t smem_bytes(const Params& p, int nsplit, int faces) {
    return 1024 + p.slots * ((size_t)nsplit * (faces / 8) * ((p.N + 63) / 64) * 1024 + (size_t)MAX_F * faces * 4) +
           (size_t)p.nraw * raw_floats(p, faces) * 4 + 512;
}

// The split of the work, everything but the pointers: the way (which tensor is expanded, its channel blocks, tiles per CTA) with
// the least estimated time.  A stage of a CTA takes the longest of its products (half a clock per column), the building of the
// expanded operand (about 100 clocks per tile and 250 besides) and its rows (about 24 bytes per clock from L2).
static void make_plan(int64_t Nf, int Cin, int Cout, int F, int precision, Params& p) {
    const int nsplit = operand_mode(precision).nsplit, fs = nsplit == 2 ? FACES<2> : FACES<1>, products = nsplit == 2 ? 3 : 2;
    const int sms = sm_count(), Fp = (F + 3) / 4 * 4;
    p = Params();
    double best = 0.;
    for (int swap = 0; swap < 2; ++swap) {
        const int C1 = swap ? Cout : Cin, C2 = swap ? Cin : Cout;
        int nb2 = (C2 + MAX_N - 1) / MAX_N;
        const int N = ((C2 + nb2 - 1) / nb2 + 15) / 16 * 16;
        nb2 = (C2 + N - 1) / N;
        const int gpitch = nb2 == 1 ? C2 : N;
        const int least = (C1 + ROWS - 1) / ROWS;
        for (int want = least; want <= 8 * least && (want == least || C1 / want >= 16); ++want) {
            const int R = ((C1 + want - 1) / want + 3) / 4 * 4, nb1 = (C1 + R - 1) / R;
            int dpt = ROWS / R < F ? ROWS / R : F;
            const int tiles = (F + dpt - 1) / dpt;
            dpt = (F + tiles - 1) / tiles;
            const int fit = TMEM_COLS / (N + 2 * ACOLS);
            for (int longest = 1; longest <= fit && longest <= tiles && longest <= MAX_NT; ++longest) {
                const int groups = (tiles + longest - 1) / longest, nt = (tiles + groups - 1) / groups, kinds = nb1 * nb2 * groups;
                double t = nt * products * (N > 64 ? N / 2. : 32.) + 200.;
                const double build = (nt * 300. + 350.) / EG, rows = fs * (R + gpitch + Fp) * 4. / 24.;
                const double copies = 350. + 35. * fs * ((nb1 > 1) + (nb2 > 1));
                if (build > t) t = build;
                if (rows > t) t = rows;
                if (copies > t) t = copies;
                const double cost = kinds <= sms ? t / (sms / kinds) : t * ((kinds + sms - 1) / sms);
                if (best == 0. || cost < best) {
                    best = cost;
                    p.swap = swap; p.C1 = C1; p.C2 = C2; p.R = R; p.dpt = dpt; p.nb1 = nb1; p.nb2 = nb2; p.N = N; p.gpitch = gpitch;
                    p.tiles = tiles; p.groups = groups; p.nt = nt;
                }
            }
        }
    }
    p.Nf = Nf; p.F = F; p.Fp = Fp;
    p.a_col = p.nt * p.N;
    p.nbuf = (TMEM_COLS - p.a_col) / (p.nt * ACOLS);
    if (p.nbuf > 4) p.nbuf = 4;
    p.nraw = MAX_RAW;
    p.slots = MAX_SLOTS;
    if (smem_bytes(p, nsplit, fs) > 227 * 1024) p.slots = 4;
    if (smem_bytes(p, nsplit, fs) > 227 * 1024) p.nraw = 4;
    p.nstages = ceil_div(Nf > 0 ? Nf : 1, fs);
    // chunks of faces: as many as the chip has room for, but with few faces no more than pay: a chunk's sums cost a write and a
    // read (about 4 TB/s), a stage about 0.3 us
    int64_t chunks = sms / (p.nb1 * p.nb2 * p.groups);
    const int64_t pay = (int64_t)sqrt((double)p.nstages * 0.3e-6 / (2. * 4. * Cin * Cout * F / 4e12));
    if (chunks > pay) chunks = pay;
    if (chunks > p.nstages) chunks = p.nstages;
    p.chunks = chunks < 1 ? 1 : (int)chunks;
}

// A call wants its plan several times (workspace, checks, launch), and a training loop the same one every step
static const Params& plan(int64_t Nf, int Cin, int Cout, int F, int precision) {
    static thread_local int64_t key[6] = {-1, 0, 0, 0, 0, 0};
    static thread_local Params last;
    const int64_t now[6] = {Nf, Cin, Cout, F, precision, sm_count()};
    if (memcmp(key, now, sizeof(key)) != 0) {
        make_plan(Nf, Cin, Cout, F, precision, last);
        memcpy(key, now, sizeof(key));
    }
    return last;
}

// bf16 operands (hi + lo or single); rows of both tensors in pieces of 16 bytes
bool supported(int Cin, int Cout, int F, int precision) {
    if (precision != PB200_PREC_FP32 && precision != PB200_PREC_BF16) return false;
    // (blocks of 128 channels, 32 bases and rings of four fit into shared memory)
    return Cin >= 4 && Cout >= 4 && Cin % 4 == 0 && Cout % 4 == 0 && F >= 1 && F <= MAX_F;
}

size_t workspace_bytes(int64_t Nf, int Cin, int Cout, int F, int precision) {
    const Params& p = plan(Nf, Cin, Cout, F, precision);
    return align_up((size_t)p.nb1 * p.nb2 * p.groups * p.chunks * sum_cols(p) * ROWS * sizeof(float), 256);
}

template <int NSPLIT>
static int launch(const Params& p, cudaStream_t stream) {
    const size_t smem = smem_bytes(p, NSPLIT, FACES<NSPLIT>);
    PB_CUDA(cudaFuncSetAttribute(f2f_one_sample_gfilter_kernel<NSPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PB_LAUNCH("f2f_bwd_gfilter_one_tc", (f2f_one_sample_gfilter_kernel<NSPLIT>), p.nb1 * p.nb2 * p.groups * p.chunks, NTHREADS, smem, stream, p);
    return PB200_OK;
}

// w: weight rows of F rounded up to 4 floats, pad columns zero; all pointers 16-byte aligned
int backward_filter(int64_t Nf, int Cin, int Cout, int F, const float* gout, const float* input, const float* w, float* gfilter,
                    int precision, void* ws, cudaStream_t stream) {
    int rc = check_async_error("facet2facet_backward");
    if (rc) return rc;
    Params p = plan(Nf, Cin, Cout, F, precision);
    p.x = p.swap ? gout : input;
    p.g = p.swap ? input : gout;
    p.w = w; p.sums = (float*)ws; p.out = gfilter;
    p.async_err = async_error_word();
    p.wait_budget = wait_budget_kclocks();
    rc = operand_mode(precision).nsplit == 2 ? launch<2>(p, stream) : launch<1>(p, stream);
    if (rc) return rc;
    const int64_t items = (int64_t)p.nb1 * p.nb2 * p.tiles * p.N * 2;
    PB_LAUNCH("f2f_bwd_gfilter_one_reduce", f2f_one_sample_gfilter_reduce_kernel, persistent_blocks(items, 1, 16), 256, 0, stream, p);
    return PB200_OK;
}

}  // namespace onef
}  // namespace tc
}  // namespace pb
