// Quadric-error mesh decimation, one pass (the reference's `meshDecimationLauncher`,
// picasso/mesh/pi_modules/source/decimate_gpu.cu:618-747) and the cluster merge
// (`combineClustersLauncher`, decimate_gpu.cu:750-812), entirely on the device.
//
// The reference sorts edge indices with a comparator sort, loops over the samples of the batch
// on the host (unique / cost / sort per sample), copies the sorted candidates to the host and
// clusters vertices there in two sequential sweeps.  Here one pass is, for the whole batch at once:
//   1. the vertex CSR of the faces; a thread per vertex sorts its row, collects the other ends of the
//      edges it owns (an edge belongs to its lower vertex), sorts those and so knows its distinct
//      candidate edges and, by their multiplicity, the boundary edges (seen once): candidates come out
//      in (lower, higher) order after one prefix sum, without sorting the edges of the batch;
//   2. vertex quadrics pulled through the CSR in ascending (face, corner) order (no float atomics:
//      run-to-run deterministic), boundary quadrics in the same walk; candidate costs.  A candidate's
//      place in the cost order is the 64-bit key (cost, candidate): nothing is sorted by cost;
//   3. the first sequential sweep (an edge is taken when neither end is covered) is the greedy
//      matching in key order.  It equals the fixed point of "take every edge whose key is the
//      smallest among the live edges at both of its ends", computed in parallel rounds
//      (atomicMin per vertex).  The sweep's early stop keeps the first want[s] matched edges in key
//      order: their last key is found by radix selection among the matched edges;
//   4. the second sweep attaches every still-uncovered vertex through its lowest-keyed
//      edge: after a complete first sweep no edge joins two uncovered vertices, so these
//      choices are independent; its early stop is the same selection;
//   5. cluster positions (members added in ascending vertex id), relabelled faces, degenerate
//      flags, vertex map and the per-sample output sizes.
// Results equal the sequential procedure's for any input.
//
// A pass is a chain of dependent steps over small arrays: what it costs is launches, grid-wide
// synchronisations and latency far more than bytes.  Radix sorts of the edges and of the costs took 70 of
// its 170 launches; steps 3 and 4, thirty-odd steps of their own, are ONE kernel: a block per sample where
// samples are small (steps separated by block barriers), a cooperative grid with a bounded barrier
// otherwise.  Two scenes of 490 000 vertices, three levels of 1/4: 9.2 -> 4.6 ms; 64 shapes of 642
// vertices, two levels: 4.6 -> 1.26 ms (host loop and level preparation included).
//
// This file is compiled with --fmad=false: every float operation is rounded on its own, so the
// costs (and therefore the clustering) can be reproduced exactly by a plain C restatement.
#include "common.cuh"
#include "scan.cuh"
#include "warp_sort.cuh"

namespace pb {
namespace dec {

typedef unsigned long long u64;
constexpr u64 NO_KEY = ~0ull;

// ------------------------------------------------------------------------ small helpers
// sample that owns vertex (or face) id x: first s with x < cum[s]; B when none
__device__ __forceinline__ int sample_of(int x, const int32_t* __restrict__ cum, int B) {
    int lo = 0, hi = B;
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (x < cum[mid]) hi = mid; else lo = mid + 1; }
    return lo;
}

// appends the elements whose `pred` holds to list[*counter...]; called by whole warps
__device__ __forceinline__ void warp_append(bool pred, uint32_t value, uint32_t* __restrict__ list, int32_t* counter) {
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (m == 0) return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    int32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pred) list[base + __popc(m & ((1u << lane) - 1u))] = value;
}

// SWEEP values per lane, those with what[j] == wanted, with one addition to the counter
constexpr int SWEEP = 4;
__device__ __forceinline__ void warp_append_all(const int (&what)[SWEEP], int wanted, const uint32_t (&value)[SWEEP],
                                                uint32_t* __restrict__ list, int32_t* counter) {
    const int lane = threadIdx.x & 31;
    unsigned m[SWEEP];
    int total = 0;
#pragma unroll
    for (int j = 0; j < SWEEP; ++j) { m[j] = __ballot_sync(0xffffffffu, what[j] == wanted); total += __popc(m[j]); }
    if (total == 0) return;
    int32_t base = 0;
    if (lane == 0) base = atomicAdd(counter, total);
    base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
    for (int j = 0; j < SWEEP; ++j) {
        if (what[j] == wanted) list[base + __popc(m[j] & ((1u << lane) - 1u))] = value[j];
        base += __popc(m[j]);
    }
}

// counter[key] += 1 for the lanes with key >= 0, one atomic per distinct key of the warp; called by whole warps
__device__ __forceinline__ void warp_count(int key, int32_t* counter) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __match_any_sync(0xffffffffu, key >= 0 ? key : -1 - lane);
    if (key >= 0 && lane == __ffs(m) - 1) atomicAdd(&counter[key], __popc(m));
}

// face edge slots as the reference numbers them (decimate_gpu.cu:262-308):
// slot 0 joins corners (0,1), slot 1 corners (0,2), slot 2 corners (1,2)
__device__ __forceinline__ int slot_a(int k) { return k == 2 ? 1 : 0; }
__device__ __forceinline__ int slot_b(int k) { return k == 0 ? 1 : 2; }

// ------------------------------------------------------------------ vertex CSR and edges
// a face with an id outside [0, Nv) is reported and takes part in nothing
__device__ __forceinline__ bool read_face(const int32_t* __restrict__ face, int64_t f, int64_t Nv, int (&v)[3]) {
    v[0] = face[3 * f]; v[1] = face[3 * f + 1]; v[2] = face[3 * f + 2];
    return v[0] >= 0 && v[1] >= 0 && v[2] >= 0 && v[0] < Nv && v[1] < Nv && v[2] < Nv;
}

__global__ void count_corners_kernel(int64_t Nf, int64_t Nv, const int32_t* __restrict__ face, int32_t* __restrict__ cnt,
                                     int32_t* __restrict__ status) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= Nf) return;
    int v[3];
    if (!read_face(face, f, Nv, v)) { *status = PB200_EINDEX; return; }
#pragma unroll
    for (int c = 0; c < 3; ++c) atomicAdd(&cnt[v[c]], 1);
}

__global__ void fill_corners_kernel(int64_t Nf, int64_t Nv, const int32_t* __restrict__ face, int32_t* __restrict__ cursor,
                                    int32_t* __restrict__ entries) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= Nf) return;
    int v[3];
    if (!read_face(face, f, Nv, v)) return;
#pragma unroll
    for (int c = 0; c < 3; ++c) entries[atomicAdd(&cursor[v[c]], 1)] = (int32_t)((f << 2) | c);
}

// The edge of corner (f, c), s-th of two: its slot, the other end, and whether corner c owns the instance (it is the lower
// end; of a degenerate edge the corner that the slot names first)
__device__ __forceinline__ bool corner_edge(const int32_t* __restrict__ face, int32_t entry, int v, int s, int& other, uint32_t& e) {
    const int64_t f = entry >> 2;
    const int c = entry & 3;
    const int k = c == 0 ? s : (c == 1 ? 2 * s : 1 + s);
    const int oc = slot_a(k) == c ? slot_b(k) : slot_a(k);
    other = face[3 * f + oc];
    e = (uint32_t)(3 * f + k);
    return other > v || (other == v && slot_a(k) == c);
}

// Per vertex: row sorted; distinct other ends of its own edges, ascending, to hi[2 * rowptr[v] ...], their number to
// ucnt[v]; boundary flag of every edge instance.  Long rows (more than SHORT corners) are taken by the whole warp,
// which sorts them by radix, with room in tmpA and tmpB (two words per entry of the row each).  Ranks by counting are
// quadratic: a pass over a fan of 3000 triangles took 31.7 ms, now 1.8.
constexpr int SHORT = 16;

__global__ void __launch_bounds__(128)
vertex_edges_kernel(int64_t Nv, const int32_t* __restrict__ face, const int32_t* __restrict__ rowptr, int32_t* entries,
                    int32_t* hi, int32_t* __restrict__ ucnt, uint8_t* __restrict__ bnd, int32_t* tmpA, uint32_t* tmpB,
                    int32_t* __restrict__ tile_sum) {
    __shared__ int32_t hist[128 / 32][WARP_SORT_BINS];
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int beg = 0, end = 0;
    if (v < Nv) { beg = rowptr[v]; end = rowptr[v + 1]; }
    const int deg = end - beg;
    int found = 0;
    if (deg > 0 && deg <= SHORT) {
        int32_t a[SHORT];
        for (int i = 0; i < deg; ++i) {
            const int32_t x = entries[beg + i];
            int j = i - 1;
            while (j >= 0 && a[j] > x) { a[j + 1] = a[j]; --j; }
            a[j + 1] = x;
        }
        int32_t o[2 * SHORT];
        uint32_t id[2 * SHORT];
        int n = 0;
        for (int i = 0; i < deg; ++i) {
            entries[beg + i] = a[i];
            for (int s = 0; s < 2; ++s) {
                int other;
                uint32_t e;
                if (!corner_edge(face, a[i], (int)v, s, other, e)) continue;
                int j = n++ - 1;
                while (j >= 0 && o[j] > other) { o[j + 1] = o[j]; id[j + 1] = id[j]; --j; }
                o[j + 1] = other; id[j + 1] = e;
            }
        }
        for (int i = 0; i < n; ++i) {
            const bool first = i == 0 || o[i - 1] != o[i], last = i + 1 == n || o[i + 1] != o[i];
            bnd[id[i]] = first && last;
            if (first) hi[2 * (int64_t)beg + found++] = o[i];
        }
    }
    unsigned waiting = __ballot_sync(0xffffffffu, deg > SHORT);
    while (waiting) {
        const int owner = __ffs(waiting) - 1;
        waiting &= waiting - 1;
        const int64_t b = __shfl_sync(0xffffffffu, beg, owner);
        const int d = __shfl_sync(0xffffffffu, deg, owner);
        const int vv = (int)(v - lane + owner);
        // the row, sorted (four passes: the result is where it was)
        warp_sort(reinterpret_cast<uint32_t*>(entries + b), reinterpret_cast<uint32_t*>(tmpA + 2 * b), d, 31, hist[threadIdx.x >> 5]);
        // other ends of its own edges to tmpA, sorted
        int n = 0;
        for (int i0 = 0; i0 < 2 * d; i0 += 32) {
            const int i = i0 + lane;
            int other = 0;
            uint32_t e;
            const bool own = i < 2 * d && corner_edge(face, entries[b + (i >> 1)], vv, i & 1, other, e);
            const unsigned m = __ballot_sync(0xffffffffu, own);
            if (own) tmpA[2 * b + n + __popc(m & ((1u << lane) - 1u))] = other;
            n += __popc(m);
        }
        const uint32_t* o = warp_sort(reinterpret_cast<uint32_t*>(tmpA + 2 * b), tmpB + 2 * b, n, 32 - __clz((int)Nv), hist[threadIdx.x >> 5]);
        // an instance is a boundary edge when its other end is there once
        for (int i = lane; i < 2 * d; i += 32) {
            int other;
            uint32_t e;
            if (!corner_edge(face, entries[b + (i >> 1)], vv, i & 1, other, e)) continue;
            int l = 0, r = n;
            while (l < r) { const int mid = (l + r) >> 1; if (o[mid] < (uint32_t)other) l = mid + 1; else r = mid; }
            bnd[e] = l + 1 == n || o[l + 1] != (uint32_t)other;
        }
        int total = 0;
        for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            const bool first = i < n && (i == 0 || o[i - 1] != o[i]);
            const unsigned m = __ballot_sync(0xffffffffu, first);
            if (first) hi[2 * b + total + __popc(m & ((1u << lane) - 1u))] = (int32_t)o[i];
            total += __popc(m);
        }
        if (lane == owner) found = total;
        __syncwarp();
    }
    if (v < Nv) ucnt[v] = found;
    const int sum = __reduce_add_sync(0xffffffffu, found);
    if (lane == 0 && sum > 0) atomicAdd(&tile_sum[v / scan::TILE], sum);
}

// candidates in (lower, higher) order; ustart[v] = first candidate of vertex v, ustart[Nv] = their number.  Samples are
// clustered independently of one another: an edge between two of them is reported and nothing is clustered.
constexpr int32_t ECROSS = 1;

__global__ void __launch_bounds__(scan::THREADS)
candidates_kernel(int64_t Nv, int B, const int32_t* __restrict__ nvIn, int32_t* __restrict__ status, const int32_t* __restrict__ ucnt, const int32_t* __restrict__ tile_sum, const int32_t* __restrict__ rowptr,
                  const int32_t* __restrict__ hi, int32_t* __restrict__ ustart, int32_t* __restrict__ ulo, int32_t* __restrict__ uhi) {
    __shared__ int sh[scan::THREADS / 32];
    const int before = scan::tiles_before(tile_sum, blockIdx.x, sh);
    const int64_t base = (int64_t)blockIdx.x * scan::TILE + (int64_t)threadIdx.x * scan::ITEMS;
    int n[scan::ITEMS], s = 0;
    scan::load_items(ucnt, Nv, base, n);
#pragma unroll
    for (int j = 0; j < scan::ITEMS; ++j) s += n[j];
    int run = before + scan::block_exclusive(s, sh);
    int sample = base < Nv ? sample_of((int)base, nvIn, B) : B;
#pragma unroll
    for (int j = 0; j < scan::ITEMS; ++j) {
        const int64_t v = base + j;
        if (v >= Nv) break;
        ustart[v] = run;
        while (sample < B && nvIn[sample] <= v) ++sample;
        const int end = sample < B ? nvIn[sample] : 0;
        const int64_t src = 2 * (int64_t)rowptr[v];
        for (int i = 0; i < n[j]; ++i) {
            const int other = hi[src + i];
            ulo[run + i] = (int32_t)v;
            uhi[run + i] = other;
            if (other >= end) *status = ECROSS;
        }
        run += n[j];
        if (v + 1 == Nv) ustart[Nv] = run;
    }
}

// ---------------------------------------------------------------------------- quadrics
__device__ __forceinline__ void plane_quadric(const float n0, const float n1, const float n2, const float d, float* Q) {
    Q[0] = n0 * n0; Q[1] = n0 * n1; Q[2] = n0 * n2;
    Q[3] = n1 * n1; Q[4] = n1 * n2; Q[5] = n2 * n2;
    Q[6] = n0 * d;  Q[7] = n1 * d;  Q[8] = n2 * d;
    Q[9] = d * d;
}

// One thread per vertex: the face quadrics of its corners in ascending (face, corner) order
// (decimate_gpu.cu:225-256), then the boundary quadrics of the corners' edges in the same
// order, lower edge slot first (decimate_gpu.cu:311-374).
__global__ void vertex_quadric_kernel(int64_t Nv, int D, int useArea, float wgtBnd, const int32_t* __restrict__ rowptr,
                                      const int32_t* __restrict__ entries, const int32_t* __restrict__ face,
                                      const float* __restrict__ plane, const float* __restrict__ vertex,
                                      const uint8_t* __restrict__ bnd, float* __restrict__ Qout) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= Nv) return;
    float acc[10];
#pragma unroll
    for (int t = 0; t < 10; ++t) acc[t] = 0.f;
    const int beg = rowptr[v], end = rowptr[v + 1];
    for (int p = beg; p < end; ++p) {
        const int64_t f = entries[p] >> 2;
        const float* pl = plane + 5 * f;
        float Q[10];
        plane_quadric(pl[0], pl[1], pl[2], pl[3], Q);
        const float area = pl[4] * 100.0f;
        const float w = useArea ? area / 3 : 1.0f;
#pragma unroll
        for (int t = 0; t < 10; ++t) acc[t] += Q[t] * w;
    }
    if (wgtBnd > 0)
        for (int p = beg; p < end; ++p) {
            const int64_t f = entries[p] >> 2;
            const int c = entries[p] & 3;
            for (int s = 0; s < 2; ++s) {
                const int k = c == 0 ? s : (c == 1 ? 2 * s : 1 + s);
                if (!bnd[3 * f + k]) continue;
                const int a = face[3 * f + slot_a(k)], b = face[3 * f + slot_b(k)];
                const int vi = a <= b ? a : b, vj = a <= b ? b : a;
                const float* pl = plane + 5 * f;
                const float* pi = vertex + (int64_t)vi * D;
                const float* pj = vertex + (int64_t)vj * D;
                const float dx0 = pj[0] - pi[0], dx1 = pj[1] - pi[1], dx2 = pj[2] - pi[2];
                float b0 = pl[1] * dx2 - pl[2] * dx1;
                float b1 = pl[2] * dx0 - pl[0] * dx2;
                float b2 = pl[0] * dx1 - pl[1] * dx0;
                float len = sqrtf(b0 * b0 + b1 * b1 + b2 * b2);
                len = len > 1e-20f ? len : 1e-20f;
                b0 /= len; b1 /= len; b2 /= len;
                const float d = -(b0 * pi[0] + b1 * pi[1] + b2 * pi[2]);
                float wb = (dx0 * dx0 + dx1 * dx1 + dx2 * dx2) * 100.0f;
                if (useArea) wb *= wgtBnd; else wb = wgtBnd;
                float Q[10];
                plane_quadric(b0, b1, b2, d, Q);
#pragma unroll
                for (int t = 0; t < 10; ++t) acc[t] += Q[t] * wb;
            }
        }
#pragma unroll
    for (int t = 0; t < 10; ++t) Qout[10 * v + t] = acc[t];
}

// quadric error x^T A x + 2 b.x + c with the reference's association (decimate_gpu.cu:189-197)
__device__ __forceinline__ float quadric_error(const float* x, const float (*A)[3], const float* b, float c) {
    return ((x[0] * A[0][0] + x[1] * A[1][0] + x[2] * A[2][0]) * x[0]
          + (x[0] * A[0][1] + x[1] * A[1][1] + x[2] * A[2][1]) * x[1]
          + (x[0] * A[0][2] + x[1] * A[1][2] + x[2] * A[2][2]) * x[2])
          + (x[0] * b[0] + x[1] * b[1] + x[2] * b[2]) * 2
          + c;
}

// A column of the reduction below with I pivots found so far: swap, scale and eliminate, or false where it has no pivot.  A pivot column
// of A is not updated, nothing reads it again.
template <int I, int J>
__device__ __forceinline__ bool take_column(float (&M)[3][7], float tol) {
    constexpr int C0 = J < 3 ? J + 1 : J;
    float p = fabsf(M[I][J]);
    int k = I;
#pragma unroll
    for (int r = I + 1; r < 3; ++r) {
        const float q = fabsf(M[r][J]);
        if (p < q) { p = q; k = r; }
    }
    if (p <= tol) {
#pragma unroll
        for (int r = I; r < 3; ++r) M[r][J] = 0.f;
        return false;
    }
#pragma unroll
    for (int r = I + 1; r < 3; ++r)
#pragma unroll
        for (int c = J; c < 7; ++c) {
            const float t = M[I][c];
            M[I][c] = k == r ? M[r][c] : t;
            M[r][c] = k == r ? t : M[r][c];
        }
    const float piv = M[I][J];
#pragma unroll
    for (int c = C0; c < 7; ++c) M[I][c] = M[I][c] / piv;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        if (r == I) continue;
        const float m = M[r][J];
#pragma unroll
        for (int c = C0; c < 7; ++c) M[r][c] -= m * M[I][c];
    }
    return true;
}

// Gauss-Jordan reduction of [A | b | I] with partial pivoting and the reference's column
// tolerance (decimate_gpu.cu:80-187): minimiser -A^-1 b and the reciprocal condition estimate.
// Row and column are constants of every step, so that the matrix stays in registers; a column without a pivot makes them run apart, and
// the steps behind it are picked from all there can be.  With a matrix indexed by variables, in local memory, the costs of a
// scene of 490 000 vertices to a quarter of them took 146 us (64 now), of a plane 126 (90), of a tilted plane 195 (120).
__device__ __forceinline__ float reduce_system(const float (&A)[3][3], const float (&b)[3], float (&xyz)[3]) {
    float M[3][7];
    float normA = 0.f;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        float s = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) { M[r][c] = A[r][c]; M[r][4 + c] = r == c ? 1.f : 0.f; s += fabsf(A[r][c]); }
        M[r][3] = b[r];
        if (normA < s) normA = s;
    }
    const float tol = 2.220446049250313e-16f * 7 * normA;
    int i = 3, j = 3;                                  // pivots found, columns done
    if (!take_column<0, 0>(M, tol)) { i = 0; j = 1; }
    else if (!take_column<1, 1>(M, tol)) { i = 1; j = 2; }
    else if (!take_column<2, 2>(M, tol)) { i = 2; j = 3; }
    for (; i < 3 && j < 7; ++j) {
        bool taken;
        switch (8 * i + j) {
            case 1: taken = take_column<0, 1>(M, tol); break;
            case 2: taken = take_column<0, 2>(M, tol); break;
            case 3: taken = take_column<0, 3>(M, tol); break;
            case 4: taken = take_column<0, 4>(M, tol); break;
            case 5: taken = take_column<0, 5>(M, tol); break;
            case 6: taken = take_column<0, 6>(M, tol); break;
            case 8 + 2: taken = take_column<1, 2>(M, tol); break;
            case 8 + 3: taken = take_column<1, 3>(M, tol); break;
            case 8 + 4: taken = take_column<1, 4>(M, tol); break;
            case 8 + 5: taken = take_column<1, 5>(M, tol); break;
            case 8 + 6: taken = take_column<1, 6>(M, tol); break;
            case 16 + 3: taken = take_column<2, 3>(M, tol); break;
            case 16 + 4: taken = take_column<2, 4>(M, tol); break;
            case 16 + 5: taken = take_column<2, 5>(M, tol); break;
            default: taken = take_column<2, 6>(M, tol); break;
        }
        i += taken;
    }
    xyz[0] = -M[0][3]; xyz[1] = -M[1][3]; xyz[2] = -M[2][3];
    float normInv = 0.f;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float s = fabsf(M[r][4]) + fabsf(M[r][5]) + fabsf(M[r][6]);
        if (normInv < s) normInv = s;
    }
    return 1 / (normA * normInv);
}

// sortable image of a cost: ascending unsigned order = ascending cost, -0 = +0, every NaN last
__device__ __forceinline__ uint32_t cost_key(float c) {
    if (c != c) return 0xffffffffu;
    if (c == 0.f) c = 0.f;
    const uint32_t u = __float_as_uint(c);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// one candidate per thread (decimate_gpu.cu:378-416); order key = (cost, candidate)
__global__ void __launch_bounds__(128)
edge_cost_kernel(int64_t Nv, int D, const int32_t* __restrict__ ustart, const int32_t* __restrict__ ulo, const int32_t* __restrict__ uhi,
                 const float* __restrict__ vertex, const float* __restrict__ Qv, u64* __restrict__ key, float* __restrict__ costOut) {
    const int nu = ustart[Nv];
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < nu; u += gridDim.x * blockDim.x) {
        const int vi = ulo[u], vj = uhi[u];
        float q[10];
#pragma unroll
        for (int t = 0; t < 10; ++t) q[t] = Qv[10 * (int64_t)vi + t] + Qv[10 * (int64_t)vj + t];
        const float A[3][3] = {{q[0], q[1], q[2]}, {q[1], q[3], q[4]}, {q[2], q[4], q[5]}};
        const float b[3] = {q[6], q[7], q[8]};
        float x[3], cost;
        const float rc = reduce_system(A, b, x);
        if (rc > 1e-6f) cost = quadric_error(x, A, b, q[9]);
        else {
            const float ei = quadric_error(vertex + (int64_t)vi * D, A, b, q[9]);
            const float ej = quadric_error(vertex + (int64_t)vj * D, A, b, q[9]);
            cost = ei < ej ? ei : ej;
        }
        key[u] = ((u64)cost_key(cost) << 32) | (u64)(uint32_t)u;
        if (costOut) costOut[u] = cost;
    }
}

// ---------------------------------------------------------------------------- clustering
// All of both sweeps in one kernel.  Arrays that one step writes and a later one reads are read with __ldcg (the steps'
// writers are other threads, in grid mode on other SMs).
struct Cluster {
    int64_t Nv;
    int B;
    const int32_t *nvIn, *want, *ustart, *ulo, *uhi;
    const u64* key;
    uint8_t* covered;
    u64 *vminA, *vminB, *vminC;
    uint32_t *listA, *listB, *taken, *joined;
    int32_t *matched, *attached;          // (B) edges of the first / second sweep per sample
    // grid mode only
    u64* prefix;                          // (B) selection: key digits fixed so far
    int32_t* rest;                        // (B) selection: how many are still to take
    int32_t* hist;                        // (B << digit bits)
    int digit_bits;
    int32_t* counters;                    // 8 ints, zero (the last one is contract_kernel's)
    unsigned* barrier;                    // 2 words, zero: arrivals, give-up flag
    int32_t* rounds;                      // rounds on the grid, live edges handed to the tail
    int32_t* status;
    int32_t *vtReplace, *head, *next;     // clusters as linked lists: head[root], next[member] hold id + 1, 0 = end
};

// The steps of a group of threads: a block over one sample's candidates, or the grid over all of them.
// Live edges below which one block goes on alone: its rounds cost a block barrier, a grid round some 10 us but the whole chip's
// loads (hierarchy of two scenes: 1711 us of clustering with 8192, 1550 with 2048, 1545 with 1024).
constexpr int TAIL = 1024;
constexpr long long BARRIER_CLOCKS = 4000000000ll;       // about two seconds

__device__ __forceinline__ bool grid_barrier(unsigned* bar, int32_t* status) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        __threadfence();
        const unsigned target = (atomicAdd(&bar[0], 1u) / gridDim.x + 1u) * gridDim.x;
        const long long t0 = clock64();
        unsigned seen, gone;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&bar[0]) : "memory");
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(gone) : "l"(&bar[1]) : "memory");
            if (gone || clock64() - t0 > BARRIER_CLOCKS) { ok = 0; break; }
        } while ((int)(seen - target) < 0);
        if (!ok) { atomicExch(&bar[1], 1u); *status = PB200_ECUDA; }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

__device__ __forceinline__ bool is_covered(const uint8_t* c, int v) { return __ldcg(c + v) != 0; }

// a live edge posts its key at both ends
__device__ __forceinline__ void post_edge(const Cluster& p, uint32_t u, u64* vmin) {
    const int lo = p.ulo[u], hi = p.uhi[u];
    if (is_covered(p.covered, lo) || is_covered(p.covered, hi)) return;
    const u64 k = p.key[u];
    atomicMin(&vmin[lo], k);
    atomicMin(&vmin[hi], k);
}
// 2: taken, 1: still live (the slots of the other array are cleared for the next round), 0: dead
__device__ __forceinline__ int take_edge(const Cluster& p, uint32_t u, const u64* vmin, u64* vnext) {
    const int lo = p.ulo[u], hi = p.uhi[u];
    const u64 k = p.key[u];
    if (__ldcg(&vmin[lo]) == k && __ldcg(&vmin[hi]) == k) {
        p.covered[lo] = 1;
        p.covered[hi] = 1;
        return 2;
    }
    if (is_covered(p.covered, lo) || is_covered(p.covered, hi)) return 0;
    vnext[lo] = NO_KEY;
    vnext[hi] = NO_KEY;
    return 1;
}
// second sweep: the uncovered end of an edge with one covered end, or -1
__device__ __forceinline__ int free_end(const Cluster& p, uint32_t u) {
    const int lo = p.ulo[u], hi = p.uhi[u];
    if (lo == hi) return -1;
    const bool cl = is_covered(p.covered, lo), ch = is_covered(p.covered, hi);
    return cl == ch ? -1 : (cl ? hi : lo);
}
__device__ __forceinline__ void join(const Cluster& p, int member, int root) {
    p.vtReplace[member] = -root;
    atomicAdd(&p.vtReplace[root], 1);
    p.next[member] = atomicExch(&p.head[root], member + 1);
}
// first sweep applied (decimate_gpu.cu:568-584): the lower vertex is contracted into the higher one
__device__ __forceinline__ void apply_taken(const Cluster& p, uint32_t u) { join(p, p.ulo[u], p.uhi[u]); }
// second sweep applied (decimate_gpu.cu:586-612)
__device__ __forceinline__ void apply_joined(const Cluster& p, uint32_t u) {
    const int lo = p.ulo[u], hi = p.uhi[u];
    const bool cl = is_covered(p.covered, lo);
    const int seed = cl ? lo : hi, joiner = cl ? hi : lo;
    const int rep = __ldcg(&p.vtReplace[seed]);
    join(p, joiner, rep < 0 ? -rep : seed);
}

// rounds of one block over the live list `from` (n edges; nullptr: the candidates u0 ... u0 + n) until none is left;
// taken edges are appended to `taken`.  Every round takes at least the lowest live edge: n + 1 rounds bound the loop.
template <typename OnTaken>
__device__ void block_rounds(const Cluster& p, uint32_t u0, uint32_t* from, uint32_t* list0, uint32_t* list1, int n, u64* vmin, u64* vnext,
                             OnTaken&& on_taken) {
    __shared__ int32_t live[3];
    if (threadIdx.x < 3) live[threadIdx.x] = 0;
    __syncthreads();
    uint32_t* out = list0;
    uint32_t* other = list1;
    int slot = 0;
    for (int round = 0, limit = n + 1; n > 0 && round < limit; ++round) {
        if (threadIdx.x == 0) live[(slot + 1) % 3] = 0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const uint32_t u = from ? __ldcg(from + i) : u0 + i;
            if (p.ulo[u] != p.uhi[u]) post_edge(p, u, vmin);
        }
        __syncthreads();
        for (int i0 = 0; i0 < n; i0 += blockDim.x) {
            const int i = i0 + threadIdx.x;
            int what = 0;
            uint32_t u = 0;
            if (i < n) {
                u = from ? __ldcg(from + i) : u0 + i;
                if (p.ulo[u] != p.uhi[u]) what = take_edge(p, u, vmin, vnext);
            }
            on_taken(what == 2, u);
            warp_append(what == 1, u, out, &live[slot]);
        }
        __syncthreads();
        n = live[slot];
        slot = (slot + 1) % 3;
        from = out;
        uint32_t* t = out; out = other; other = t;
        u64* tv = vmin; vmin = vnext; vnext = tv;
    }
    __syncthreads();
}

// k-th smallest key (k >= 1) among the n listed candidates, by a block: eight bits at a time from the top
__device__ u64 block_select(const Cluster& p, const uint32_t* list, int n, int k, int ubits) {
    __shared__ int32_t hist[256];
    __shared__ int digit, left;
    u64 prefix = 0;
    for (int shift = 56; shift >= 0; shift -= 8) {
        if (shift < 32 && shift >= ubits) { prefix <<= 8; continue; }          // candidate ids have no such digit
        for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const u64 key = p.key[__ldcg(list + i)];
            if (shift == 56 || (key >> (shift + 8)) == prefix) atomicAdd(&hist[(int)(key >> shift) & 255], 1);
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            int c[8], s = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) { c[j] = hist[threadIdx.x * 8 + j]; s += c[j]; }
            int inc = s;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, inc, o); if ((int)threadIdx.x >= o) inc += t; }
            int run = inc - s;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (run < k && run + c[j] >= k) { digit = threadIdx.x * 8 + j; left = k - run; }
                run += c[j];
            }
        }
        __syncthreads();
        prefix = (prefix << 8) | (u64)digit;
        k = left;
        __syncthreads();
    }
    return prefix;
}

__device__ __forceinline__ int bit_length(int x) { return 32 - __clz(x); }

// A block per sample.
__global__ void __launch_bounds__(1024) cluster_samples_kernel(Cluster p) {
    __shared__ int32_t count;
    if (__ldcg(p.status) != 0) return;
    for (int s = blockIdx.x; s < p.B; s += gridDim.x) {
        const int v0 = s > 0 ? p.nvIn[s - 1] : 0, v1 = p.nvIn[s];
        const int u0 = p.ustart[v0], n = p.ustart[v1] - u0, want = p.want[s];
        const int ubits = bit_length(u0 + n);
        uint32_t* taken = p.taken + v0;                        // at most one edge per two vertices
        uint32_t* joined = p.joined + v0;                      // at most one edge per vertex
        if (threadIdx.x == 0) count = 0;
        __syncthreads();
        if (want <= 0 || n == 0) continue;                     // uniform over the block
        block_rounds(p, (uint32_t)u0, nullptr, p.listA + u0, p.listB + u0, n, p.vminA, p.vminB,
                     [&](bool yes, uint32_t u) { warp_append(yes, u, taken, &count); });
        const int matched = count;
        const u64 last = matched > want ? block_select(p, taken, matched, want, ubits) : NO_KEY;
        for (int i = threadIdx.x; i < matched; i += blockDim.x) {
            const uint32_t u = __ldcg(taken + i);
            if (p.key[u] <= last) apply_taken(p, u);
        }
        __syncthreads();
        if (matched < want) {
            if (threadIdx.x == 0) count = 0;
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                const int v = free_end(p, u0 + i);
                if (v >= 0) atomicMin(&p.vminC[v], p.key[u0 + i]);
            }
            __syncthreads();
            for (int i0 = 0; i0 < n; i0 += blockDim.x) {
                const int i = i0 + threadIdx.x;
                bool yes = false;
                if (i < n) {
                    const int v = free_end(p, u0 + i);
                    yes = v >= 0 && __ldcg(&p.vminC[v]) == p.key[u0 + i];
                }
                warp_append(yes, u0 + i, joined, &count);
            }
            __syncthreads();
            const int found = count;
            const u64 end = found > want - matched ? block_select(p, joined, found, want - matched, ubits) : NO_KEY;
            for (int i = threadIdx.x; i < found; i += blockDim.x) {
                const uint32_t u = __ldcg(joined + i);
                if (p.key[u] <= end) apply_joined(p, u);
            }
        }
        __syncthreads();
    }
}

// The whole grid over the whole batch (cooperative launch).
constexpr int GRID_THREADS = 512;

__device__ __forceinline__ int select_goal(const Cluster& p, int s, bool second) {      // edges to keep, or -1: all of them
    const int m = __ldcg(&p.matched[s]), w = p.want[s];
    if (!second) return m > w ? w : -1;
    const int need = w - m;
    return need > 0 && __ldcg(&p.attached[s]) > need ? need : -1;
}

// prefix[s] = last key to keep of every sample whose list is too long; false: the barrier gave up
__device__ bool grid_select(const Cluster& p, const uint32_t* list, int n, bool second, int ubits, int32_t* flag) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    for (int s = tid; s < p.B; s += nt) {
        const int goal = select_goal(p, s, second);
        p.prefix[s] = 0;
        p.rest[s] = goal;
        if (goal >= 0) *flag = 1;
    }
    if (!grid_barrier(p.barrier, p.status)) return false;
    if (__ldcg(flag) == 0) return true;
    const int bits = p.digit_bits, bins = 1 << bits;
    for (int shift = 64 - bits; shift >= 0; shift -= bits) {
        const bool empty = shift < 32 && shift >= ubits;
        if (!empty) {
            // one atomic per distinct digit of a warp: the upper digits are the costs' exponents, the same for most
            for (int i0 = tid - (int)(threadIdx.x & 31); i0 < n; i0 += nt) {
                const int i = i0 + (int)(threadIdx.x & 31);
                int at = -1;
                if (i < n) {
                    const uint32_t u = __ldcg(list + i);
                    const int s = sample_of(p.ulo[u], p.nvIn, p.B);
                    if (__ldcg(&p.rest[s]) >= 0) {
                        const u64 key = p.key[u];
                        if (shift + bits >= 64 || (key >> (shift + bits)) == __ldcg(&p.prefix[s]))
                            at = (s << bits) + (int)((key >> shift) & (u64)(bins - 1));
                    }
                }
                warp_count(at, p.hist);
            }
            if (!grid_barrier(p.barrier, p.status)) return false;
        }
        const int lane = threadIdx.x & 31;
        for (int s = tid >> 5; s < p.B; s += nt >> 5) {         // a warp per sample
            const int k = __ldcg(&p.rest[s]);
            if (k < 0) continue;
            u64 digit = 0;
            int left = k;
            if (!empty) {
                int before = 0, at = -1, rem = 0;
                for (int b0 = 0; b0 < bins; b0 += 32) {
                    const int64_t h = ((int64_t)s << bits) + b0 + lane;
                    const int c = b0 + lane < bins ? __ldcg(&p.hist[h]) : 0;
                    if (b0 + lane < bins) p.hist[h] = 0;
                    int inc = c;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += t; }
                    if (before + inc - c < k && before + inc >= k) { at = b0 + lane; rem = k - (before + inc - c); }
                    before += __shfl_sync(0xffffffffu, inc, 31);
                }
                const unsigned m = __ballot_sync(0xffffffffu, at >= 0);
                const int src = m ? __ffs(m) - 1 : 0;
                digit = (u64)(unsigned)__shfl_sync(0xffffffffu, at, src);
                left = __shfl_sync(0xffffffffu, rem, src);
            }
            if (lane == 0) { p.prefix[s] = (__ldcg(&p.prefix[s]) << bits) | digit; p.rest[s] = left; }
        }
        if (!grid_barrier(p.barrier, p.status)) return false;
    }
    return true;
}

__global__ void __launch_bounds__(GRID_THREADS, 2) cluster_grid_kernel(Cluster p) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    // the barrier's give-up flag shares the word: nobody raises it before everybody has passed the first barrier
    if (__ldcg(p.status) != 0) return;
    const int lane = threadIdx.x & 31;
    const int nu = p.ustart[p.Nv];
    const int ubits = bit_length(nu);
    int32_t* live = p.counters;             // [3] in turn
    int32_t* ntaken = p.counters + 3;
    int32_t* njoined = p.counters + 4;
    int32_t* flags = p.counters + 5;        // [2]
    // ---- first sweep
    uint32_t *from = nullptr, *out = p.listA, *other = p.listB;
    u64 *vmin = p.vminA, *vnext = p.vminB;
    int n = nu, slot = 0, rounds = 0;
    auto eligible = [&](uint32_t u) {
        const int lo = p.ulo[u];
        if (lo == p.uhi[u]) return false;
        const int s = sample_of(lo, p.nvIn, p.B);
        return s < p.B && p.want[s] > 0;
    };
    auto took = [&](bool yes, uint32_t u) {
        warp_append(yes, u, p.taken, ntaken);
        if (__any_sync(0xffffffffu, yes)) warp_count(yes ? sample_of(p.ulo[u], p.nvIn, p.B) : -1, p.matched);
    };
    while (n > TAIL || (from == nullptr && n > 0)) {
        if (tid == 0) live[(slot + 1) % 3] = 0;
        // SWEEP edges of a thread at a time: their chains of loads overlap, and the lists' counters see one addition per batch of a warp
        for (int i0 = tid; i0 < n; i0 += SWEEP * nt) {
            uint32_t u[SWEEP];
            int lo[SWEEP], hi[SWEEP];
            u64 k[SWEEP];
            bool on[SWEEP];
#pragma unroll
            for (int j = 0; j < SWEEP; ++j) {
                on[j] = i0 + j * nt < n;
                u[j] = !on[j] ? 0u : from ? __ldcg(from + i0 + j * nt) : (uint32_t)(i0 + j * nt);
            }
#pragma unroll
            for (int j = 0; j < SWEEP; ++j) {
                on[j] = on[j] && (from || eligible(u[j]));
                lo[j] = on[j] ? p.ulo[u[j]] : 0; hi[j] = on[j] ? p.uhi[u[j]] : 0; k[j] = on[j] ? p.key[u[j]] : 0;
            }
#pragma unroll
            for (int j = 0; j < SWEEP; ++j) on[j] = on[j] && !is_covered(p.covered, lo[j]) && !is_covered(p.covered, hi[j]);
            u64 a[SWEEP], b[SWEEP];
#pragma unroll
            for (int j = 0; j < SWEEP; ++j) { a[j] = on[j] ? __ldcg(&vmin[lo[j]]) : 0; b[j] = on[j] ? __ldcg(&vmin[hi[j]]) : 0; }
#pragma unroll
            for (int j = 0; j < SWEEP; ++j) {                   // slots only fall: a key above what is there need not be posted
                if (k[j] < a[j]) atomicMin(&vmin[lo[j]], k[j]);
                if (k[j] < b[j]) atomicMin(&vmin[hi[j]], k[j]);
            }
        }
        if (!grid_barrier(p.barrier, p.status)) return;
        for (int i0 = tid - lane; i0 < n; i0 += SWEEP * nt) {
            uint32_t u[SWEEP];
            int what[SWEEP];
#pragma unroll
            for (int j = 0; j < SWEEP; ++j) {
                const int i = i0 + j * nt + lane;
                u[j] = i >= n ? 0u : from ? __ldcg(from + i) : (uint32_t)i;
                what[j] = i < n && (from || eligible(u[j])) ? 1 : 0;
            }
#pragma unroll
            for (int j = 0; j < SWEEP; ++j) what[j] = what[j] ? take_edge(p, u[j], vmin, vnext) : 0;
            warp_append_all(what, 2, u, p.taken, ntaken);
#pragma unroll
            for (int j = 0; j < SWEEP; ++j)
                if (__any_sync(0xffffffffu, what[j] == 2)) warp_count(what[j] == 2 ? sample_of(p.ulo[u[j]], p.nvIn, p.B) : -1, p.matched);
            warp_append_all(what, 1, u, out, &live[slot]);
        }
        if (!grid_barrier(p.barrier, p.status)) return;
        n = __ldcg(&live[slot]);
        slot = (slot + 1) % 3;
        from = out;
        uint32_t* t = out; out = other; other = t;
        u64* tv = vmin; vmin = vnext; vnext = tv;
        ++rounds;
    }
    if (tid == 0 && p.rounds) { p.rounds[0] = rounds; p.rounds[1] = n; }
    if (n > 0 && blockIdx.x == 0) block_rounds(p, 0u, from, out, other, n, vmin, vnext, took);
    if (!grid_barrier(p.barrier, p.status)) return;
    const int matched = __ldcg(ntaken);
    if (!grid_select(p, p.taken, matched, false, ubits, &flags[0])) return;
    for (int i = tid; i < matched; i += nt) {
        const uint32_t u = __ldcg(p.taken + i);
        const int s = sample_of(p.ulo[u], p.nvIn, p.B);
        if (__ldcg(&p.rest[s]) < 0 || p.key[u] <= __ldcg(&p.prefix[s])) apply_taken(p, u);
    }
    // ---- second sweep, in the samples that the first one left short
    auto short_of = [&](uint32_t u) {
        const int s = sample_of(p.ulo[u], p.nvIn, p.B);
        return s < p.B && __ldcg(&p.matched[s]) < p.want[s];
    };
    for (int s = tid; s < p.B; s += nt)
        if (__ldcg(&p.matched[s]) < p.want[s]) flags[1] = 1;
    if (!grid_barrier(p.barrier, p.status)) return;
    if (__ldcg(&flags[1]) == 0) return;
    for (int i = tid; i < nu; i += nt) {
        const int v = free_end(p, i);
        if (v >= 0 && short_of(i)) atomicMin(&p.vminC[v], p.key[i]);
    }
    if (!grid_barrier(p.barrier, p.status)) return;
    for (int i0 = blockIdx.x * blockDim.x; i0 < nu; i0 += nt) {
        const int i = i0 + threadIdx.x;
        bool yes = false;
        if (i < nu) {
            const int v = free_end(p, i);
            yes = v >= 0 && short_of(i) && __ldcg(&p.vminC[v]) == p.key[i];
        }
        warp_append(yes, (uint32_t)i, p.joined, njoined);
        if (__any_sync(0xffffffffu, yes)) warp_count(yes ? sample_of(p.ulo[i], p.nvIn, p.B) : -1, p.attached);
    }
    if (!grid_barrier(p.barrier, p.status)) return;
    const int found = __ldcg(njoined);
    if (tid == 0) flags[0] = 0;
    if (!grid_barrier(p.barrier, p.status)) return;
    if (!grid_select(p, p.joined, found, true, ubits, &flags[0])) return;
    for (int i = tid; i < found; i += nt) {
        const uint32_t u = __ldcg(p.joined + i);
        const int s = sample_of(p.ulo[u], p.nvIn, p.B);
        if (__ldcg(&p.rest[s]) < 0 || p.key[u] <= __ldcg(&p.prefix[s])) apply_joined(p, u);
    }
}

// -------------------------------------------------------------------- contraction, faces
// decimate_gpu.cu:403-441: a representative moves to the mean of its cluster (members added in ascending id), a vertex on its
// own keeps its row, a contracted vertex's row is zero.  map: rows go to map[v] and rows with map[v] < 0 nowhere; NULL: to v.
// A cluster's members come as a list in no particular order.  A thread sorts a few in registers; more than FEW are taken by
// the warp, which copies them to a piece of `a` (handed out by *cursor; `b` as long) and sorts them there.  (A thread that looked for
// the next larger member by a walk over the list is quadratic: a pass that makes one cluster of a thousand took 41.8 ms and
// now takes 1.3; a cluster of 10^5, 140 ms now, would have taken minutes.)
constexpr int FEW = 16;

__global__ void __launch_bounds__(128)
contract_kernel(int64_t Nv, int D, const int32_t* __restrict__ vtReplace, const int32_t* __restrict__ head, const int32_t* __restrict__ next,
                const float* __restrict__ vertexIn, const int32_t* __restrict__ map, float* __restrict__ vertexOut, uint32_t* a, uint32_t* b,
                int32_t* cursor) {
    __shared__ int32_t hist[128 / 32][WARP_SORT_BINS];
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int to = v < Nv ? (map ? map[v] : (int)v) : -1;
    const int rep = to >= 0 ? vtReplace[v] : 0;
    if (to >= 0 && rep <= FEW) {
        const float* own = vertexIn + v * D;
        float* out = vertexOut + (int64_t)to * D;
        if (rep <= 0) {
            for (int t = 0; t < D; ++t) out[t] = rep == 0 ? own[t] : 0.f;
        } else {
            int id[FEW];
            int n = 0;
            for (int m = head[v]; m != 0 && n < rep; m = next[m - 1]) {
                int j = n++ - 1;
                while (j >= 0 && id[j] > m) { id[j + 1] = id[j]; --j; }
                id[j + 1] = m;
            }
            for (int t = 0; t < D; ++t) {
                float acc = 0.f;
                for (int i = 0; i < n; ++i) acc += vertexIn[(int64_t)(id[i] - 1) * D + t];
                out[t] = (acc + own[t]) / (rep + 1);
            }
        }
    }
    unsigned waiting = __ballot_sync(0xffffffffu, rep > FEW);
    while (waiting) {
        const int owner = __ffs(waiting) - 1;
        waiting &= waiting - 1;
        const int size = __shfl_sync(0xffffffffu, rep, owner), dst = __shfl_sync(0xffffffffu, to, owner);
        const int64_t vv = v - lane + owner;
        int base = 0, n = 0;
        if (lane == 0) {
            base = atomicAdd(cursor, size);
            for (int m = head[vv]; m != 0 && n < size; m = next[m - 1]) a[base + n++] = (uint32_t)m;
        }
        base = __shfl_sync(0xffffffffu, base, 0);
        n = __shfl_sync(0xffffffffu, n, 0);
        const uint32_t* id = warp_sort(a + base, b + base, n, 32 - __clz((int)Nv), hist[threadIdx.x >> 5]);
        const float* own = vertexIn + vv * D;
        float* out = vertexOut + (int64_t)dst * D;
        for (int t = lane; t < D; t += 32) {
            float acc = 0.f;
#pragma unroll 8
            for (int i = 0; i < n; ++i) acc += vertexIn[(int64_t)(id[i] - 1) * D + t];
            out[t] = (acc + own[t]) / (size + 1);
        }
    }
}

// decimate_gpu.cu:444-507; a block per scan tile of faces, whose kept ones it also counts
__global__ void __launch_bounds__(scan::THREADS)
face_relabel_kernel(int64_t Nf, int64_t Nv, int B, const int32_t* __restrict__ mfIn, const int32_t* __restrict__ vtReplace,
                    const int32_t* __restrict__ faceIn, int32_t* __restrict__ faceOut, uint8_t* __restrict__ isDegenerate,
                    int32_t* __restrict__ kept, int32_t* __restrict__ mfOut, int32_t* __restrict__ tile_sum) {
    __shared__ int sh[scan::THREADS / 32];
    int mine = 0;
#pragma unroll 1
    for (int j = 0; j < scan::ITEMS; ++j) {
        const int64_t f = (int64_t)blockIdx.x * scan::TILE + j * scan::THREADS + threadIdx.x;
        int s = -1;
        if (f < Nf) {
            int v[3];
            bool deg = !read_face(faceIn, f, Nv, v);
            if (!deg) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int rep = vtReplace[v[c]];
                    if (rep < 0) v[c] = -rep;
                }
                deg = v[0] == v[1] || v[0] == v[2] || v[1] == v[2];
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) faceOut[3 * f + c] = v[c];
            isDegenerate[f] = deg ? 1 : 0;
            if (!deg) {
                kept[v[0]] = 1; kept[v[1]] = 1; kept[v[2]] = 1;
                s = sample_of((int)f, mfIn, B);
                if (s > B - 1) s = B - 1;
                ++mine;
            }
        }
        warp_count(s, mfOut);
    }
    mine = scan::block_sum(mine, sh);
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = mine;
}

// kept vertices of a scan tile and of every sample
__global__ void __launch_bounds__(scan::THREADS)
kept_totals_kernel(int64_t Nv, int B, const int32_t* __restrict__ nvIn, const int32_t* __restrict__ kept, int32_t* __restrict__ tile_sum,
                   int32_t* __restrict__ nvOut) {
    __shared__ int sh[scan::THREADS / 32];
    int mine = 0;
#pragma unroll 1
    for (int j = 0; j < scan::ITEMS; ++j) {
        const int64_t v = (int64_t)blockIdx.x * scan::TILE + j * scan::THREADS + threadIdx.x;
        const bool k = v < Nv && kept[v] != 0;
        const int s = k ? sample_of((int)v, nvIn, B) : -1;
        warp_count(s < B ? s : -1, nvOut);
        mine += k;
    }
    mine = scan::block_sum(mine, sh);
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = mine;
}

// decimate_gpu.cu:509-533: kept vertices are numbered in order, the others map to -1
__global__ void __launch_bounds__(scan::THREADS)
vertex_map_kernel(int64_t Nv, const int32_t* __restrict__ kept, const int32_t* __restrict__ tile_sum, int32_t* __restrict__ vtMap) {
    __shared__ int sh[scan::THREADS / 32];
    const int before = scan::tiles_before(tile_sum, blockIdx.x, sh);
    const int64_t base = (int64_t)blockIdx.x * scan::TILE + (int64_t)threadIdx.x * scan::ITEMS;
    int k[scan::ITEMS], s = 0;
    scan::load_items(kept, Nv, base, k);
#pragma unroll
    for (int j = 0; j < scan::ITEMS; ++j) s += k[j];
    int run = before + scan::block_exclusive(s, sh);
#pragma unroll
    for (int j = 0; j < scan::ITEMS; ++j) {
        if (base + j < Nv) vtMap[base + j] = k[j] ? run : -1;
        run += k[j];
    }
}

__global__ void face_update_kernel(int64_t Nf, const int32_t* __restrict__ vtMap, const uint8_t* __restrict__ isDegenerate,
                                   int32_t* __restrict__ faceOut) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= Nf || isDegenerate[f]) return;
#pragma unroll
    for (int c = 0; c < 3; ++c) faceOut[3 * f + c] = vtMap[faceOut[3 * f + c]];
}

// The kept faces behind one another with the new vertex ids, and their geometry (the arithmetic of
// triangle_geometry_kernel in adjacency.cu)
__global__ void __launch_bounds__(scan::THREADS)
emit_faces_kernel(int64_t Nf, int D, const int32_t* __restrict__ tile_sum, const uint8_t* __restrict__ isDegenerate,
                  const int32_t* __restrict__ relabelled, const int32_t* __restrict__ vtMap, const float* __restrict__ vertex,
                  int32_t* __restrict__ faceOut, float* __restrict__ geom, int32_t* cursor) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *cursor = 0;      // contract_kernel's, for another call on the same pass
    __shared__ int sh[scan::THREADS / 32];
    __shared__ int step[scan::ITEMS + 1][scan::THREADS / 32];
    const int before = scan::tiles_before(tile_sum, blockIdx.x, sh);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * scan::TILE;
    unsigned keeps[scan::ITEMS];
#pragma unroll
    for (int j = 0; j < scan::ITEMS; ++j) {
        const int64_t f = base + j * scan::THREADS + threadIdx.x;
        keeps[j] = __ballot_sync(0xffffffffu, f < Nf && !isDegenerate[f]);
        if (lane == 0) step[j][warp] = __popc(keeps[j]);
    }
    __syncthreads();
    int run = before;
#pragma unroll 1
    for (int j = 0; j < scan::ITEMS; ++j) {
        int at = run;
        for (int w = 0; w < scan::THREADS / 32; ++w) { if (w < warp) at += step[j][w]; run += step[j][w]; }
        if (!((keeps[j] >> lane) & 1u)) continue;
        at += __popc(keeps[j] & ((1u << lane) - 1u));
        const int64_t f = base + j * scan::THREADS + threadIdx.x;
        int v[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) { v[c] = vtMap[relabelled[3 * f + c]]; faceOut[3 * (int64_t)at + c] = v[c]; }
        const float *a = vertex + (int64_t)v[0] * D, *b = vertex + (int64_t)v[1] * D, *c = vertex + (int64_t)v[2] * D;
        const float ax = a[0], ay = a[1], az = a[2];
        const float ux = b[0] - ax, uy = b[1] - ay, uz = b[2] - az;
        const float vx = c[0] - ax, vy = c[1] - ay, vz = c[2] - az;
        float nx = uy * vz - uz * vy, ny = uz * vx - ux * vz, nz = ux * vy - uy * vx;
        const float l2 = sqrtf(nx * nx + ny * ny + nz * nz);
        const float den = l2 + 1e-10f;
        nx = nx / den; ny = ny / den; nz = nz / den;
        float* g = geom + 5 * (int64_t)at;
        g[0] = nx; g[1] = ny; g[2] = nz;
        g[3] = -(nx * ax + ny * ay + nz * az);
        g[4] = l2 / 2.f;
    }
}

// running totals of the samples' sizes and what is to be removed of each
__global__ void __launch_bounds__(1024)
begin_pass_kernel(int B, const int32_t* __restrict__ nv, const int32_t* __restrict__ mf, const int32_t* __restrict__ target,
                  int32_t* __restrict__ nvCum, int32_t* __restrict__ mfCum, int32_t* __restrict__ want) {
    __shared__ int wt[2][32];
    __shared__ int carry[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 2) carry[threadIdx.x] = 0;
    __syncthreads();
    for (int s0 = 0; s0 < B; s0 += 1024) {
        const int s = s0 + threadIdx.x;
        int x[2] = {s < B ? nv[s] : 0, s < B ? mf[s] : 0};
        int inc[2] = {x[0], x[1]};
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
#pragma unroll
            for (int t = 0; t < 2; ++t) { const int y = __shfl_up_sync(0xffffffffu, inc[t], o); if (lane >= o) inc[t] += y; }
        if (lane == 31) { wt[0][warp] = inc[0]; wt[1][warp] = inc[1]; }
        __syncthreads();
        int tot[2] = {carry[0], carry[1]};
        for (int w = 0; w < 32; ++w)
            for (int t = 0; t < 2; ++t) { if (w < warp) inc[t] += wt[t][w]; tot[t] += wt[t][w]; }
        if (s < B) { nvCum[s] = carry[0] + inc[0]; mfCum[s] = carry[1] + inc[1]; want[s] = x[0] - target[s]; }
        __syncthreads();
        if (threadIdx.x < 2) carry[threadIdx.x] = tot[threadIdx.x];
        __syncthreads();
    }
}

// ------------------------------------------------------------------------ cluster merge
// decimate_gpu.cu:750-812.  repB_work[vo] of a vertex B kept becomes its id in A; a vertex of A
// whose representative was contracted in B follows that contraction.
__global__ void merge_back_kernel(int64_t nvA, int64_t nvB, const int32_t* __restrict__ repA, const int32_t* __restrict__ mapA,
                                  int32_t* __restrict__ repB_work, int32_t* __restrict__ repOut) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nvA) return;
    repOut[v] = repA[v];
    const int vo = mapA[v];
    if (vo >= 0 && vo < nvB && repB_work[vo] >= 0) repB_work[vo] = (int32_t)v;
}
__global__ void merge_follow_kernel(int64_t nvA, int64_t nvB, const int32_t* __restrict__ repA, const int32_t* __restrict__ mapA,
                                    const int32_t* __restrict__ repB_work, const int32_t* __restrict__ mapB, int32_t* repOut,
                                    int32_t* __restrict__ mapOut, int32_t* __restrict__ status) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nvA) return;
    const int own = mapA[v];
    mapOut[v] = (own >= 0 && own < nvB) ? mapB[own] : -1;
    int64_t vi = v;
    if (repA[v] < 0) vi = -(int64_t)repA[v];
    if (vi >= nvA) { *status = PB200_EINDEX; return; }
    const int vo = mapA[vi];
    if (vo < 0) return;
    if (vo >= nvB) { *status = PB200_EINDEX; return; }
    const int rb = repB_work[vo];
    if (rb >= 0) return;
    const int64_t root_b = -(int64_t)rb;
    if (root_b >= nvB) { *status = PB200_EINDEX; return; }
    const int root_a = repB_work[root_b];
    if (root_a < 0 || root_a >= nvA) { *status = PB200_EINDEX; return; }
    repOut[v] = -root_a;
    atomicAdd(&repOut[root_a], 1);
}

// ---------------------------------------------------------------------------- workspace
struct Carve {
    char* p;
    size_t used;
    explicit Carve(void* base) : p((char*)base), used(0) {}
    template <typename T> T* take(size_t n) {
        T* r = p ? (T*)(p + used) : nullptr;
        used += align_up(sizeof(T) * (n > 0 ? n : 1), 256);
        return r;
    }
};

struct Work {
    // cleared to 0 / to 0xff by one memset each
    char *zero_begin, *ones_begin;
    size_t zero_bytes, ones_bytes;
    int32_t *cnt, *utile, *head, *kept, *matched, *attached, *hist, *counters, *status, *rounds;
    unsigned* barrier;
    uint8_t* covered;
    u64 *vminA, *vminB, *vminC;
    // written before they are read
    int32_t *nvCum, *mfCum, *want, *rowptr, *entries, *hi, *ucnt, *ustart, *ulo, *uhi, *next, *tile, *ftile, *rest, *relabelled;
    uint32_t *listA, *listB, *taken, *joined;
    u64 *key, *prefix;
    uint8_t *bnd, *degenerate;
    float* Q;
    int digit_bits;
    size_t total;
};

static Work carve(void* base, int64_t B, int64_t Nv, int64_t Nf) {
    Work w;
    Carve c(base);
    const size_t Ne = (size_t)(3 * Nf), V = (size_t)Nv, S = (size_t)B;
    w.digit_bits = B <= 4096 ? 8 : 4;                           // selection histograms of every sample: at most 64 MB
    w.zero_begin = c.p;
    w.cnt = c.take<int32_t>(V + 1);
    w.utile = c.take<int32_t>((size_t)scan::tiles(Nv));
    w.head = c.take<int32_t>(V);  w.kept = c.take<int32_t>(V + 1);  w.covered = c.take<uint8_t>(V);
    w.matched = c.take<int32_t>(S);  w.attached = c.take<int32_t>(S);  w.hist = c.take<int32_t>(S << w.digit_bits);
    w.counters = c.take<int32_t>(8);  w.barrier = c.take<unsigned>(2);  w.rounds = c.take<int32_t>(2);  w.status = c.take<int32_t>(1);
    w.zero_bytes = c.used;
    w.ones_begin = c.p ? c.p + c.used : nullptr;
    w.vminA = c.take<u64>(V);  w.vminB = c.take<u64>(V);  w.vminC = c.take<u64>(V);
    w.ones_bytes = c.used - w.zero_bytes;
    w.nvCum = c.take<int32_t>(S);  w.mfCum = c.take<int32_t>(S);  w.want = c.take<int32_t>(S);
    w.rowptr = c.take<int32_t>(V + 1);  w.entries = c.take<int32_t>(Ne);  w.hi = c.take<int32_t>(2 * Ne);
    w.ucnt = c.take<int32_t>(V);  w.ustart = c.take<int32_t>(V + 1);
    w.ulo = c.take<int32_t>(Ne);  w.uhi = c.take<int32_t>(Ne);
    w.next = c.take<int32_t>(V);
    w.tile = c.take<int32_t>((size_t)scan::tiles(Nv));  w.ftile = c.take<int32_t>((size_t)scan::tiles(Nf));
    w.rest = c.take<int32_t>(S);  w.prefix = c.take<u64>(S);
    w.key = c.take<u64>(Ne);                                    // long rows use it before the costs exist
    w.listA = c.take<uint32_t>(2 * Ne);                         // and this (listA, listB)
    w.listB = w.listA ? w.listA + Ne : nullptr;
    w.taken = c.take<uint32_t>(V);  w.joined = c.take<uint32_t>(V);
    w.relabelled = c.take<int32_t>(Ne);
    w.bnd = c.take<uint8_t>(Ne);  w.degenerate = c.take<uint8_t>((size_t)Nf);
    w.Q = c.take<float>(10 * V);
    w.total = c.used + 256;
    return w;
}

// Samples with at most this many faces go to a block each: their candidates (three per two faces) are some twenty per
// thread, and a step then costs a block barrier instead of a grid barrier.
constexpr int64_t SAMPLE_FACES = 16384;

// Clustering, relabelled faces and vertex map of one pass: everything up to the sizes of its result.
static int cluster_pass(const Work& w, int useArea, float wgtBnd, int64_t B, int64_t D, int64_t Nv, int64_t Nf, int64_t most_faces,
                        const int32_t* nvIn, const int32_t* mfIn, const int32_t* want, const float* vertexIn, const int32_t* faceIn,
                        const float* planeIn, int32_t* nvOut, int32_t* mfOut, int32_t* vtReplace, int32_t* vtMap, int32_t* relabelled,
                        uint8_t* isDegenerate, float* edgeCost, cudaStream_t stream) {
    PB_CUDA(cudaMemsetAsync(w.zero_begin, 0, w.zero_bytes, stream));
    PB_CUDA(cudaMemsetAsync(nvOut, 0, sizeof(int32_t) * B, stream));
    PB_CUDA(cudaMemsetAsync(mfOut, 0, sizeof(int32_t) * B, stream));
    if (Nv == 0) return PB200_OK;
    PB_CUDA(cudaMemsetAsync(vtReplace, 0, sizeof(int32_t) * Nv, stream));
    const int vt = scan::tiles(Nv);
    if (Nf > 0) {
        PB_CUDA(cudaMemsetAsync(w.ones_begin, 0xff, w.ones_bytes, stream));
        const unsigned fgrid = (unsigned)ceil_div(Nf, 256);
        PB_LAUNCH("dec_count_corners", count_corners_kernel, fgrid, 256, 0, stream, Nf, Nv, faceIn, w.cnt, w.status);
        PB_LAUNCH("scan_tile_totals", scan::tile_totals_kernel, vt, scan::THREADS, 0, stream, (const int32_t*)w.cnt, Nv, w.tile);
        PB_LAUNCH("scan_row_starts", scan::row_starts_kernel, vt, scan::THREADS, 0, stream, (const int32_t*)w.cnt, Nv, (const int32_t*)w.tile,
                  w.rowptr, w.cnt, (int32_t*)nullptr);
        PB_LAUNCH("dec_fill_corners", fill_corners_kernel, fgrid, 256, 0, stream, Nf, Nv, faceIn, w.cnt, w.entries);
        PB_LAUNCH("dec_vertex_edges", vertex_edges_kernel, (unsigned)ceil_div(Nv, 128), 128, 0, stream, Nv, faceIn, (const int32_t*)w.rowptr,
                  w.entries, w.hi, w.ucnt, w.bnd, (int32_t*)w.key, w.listA, w.utile);
        PB_LAUNCH("dec_candidates", candidates_kernel, vt, scan::THREADS, 0, stream, Nv, (int)B, nvIn, w.status,
                  (const int32_t*)w.ucnt, (const int32_t*)w.utile,
                  (const int32_t*)w.rowptr, (const int32_t*)w.hi, w.ustart, w.ulo, w.uhi);
        PB_LAUNCH("dec_vertex_quadric", vertex_quadric_kernel, (unsigned)ceil_div(Nv, 128), 128, 0, stream, Nv, (int)D, useArea ? 1 : 0, wgtBnd,
                  (const int32_t*)w.rowptr, (const int32_t*)w.entries, faceIn, planeIn, vertexIn, (const uint8_t*)w.bnd, w.Q);
        PB_LAUNCH("dec_edge_cost", edge_cost_kernel, persistent_blocks(3 * Nf, 128, 16), 128, 0, stream, Nv, (int)D, (const int32_t*)w.ustart,
                  (const int32_t*)w.ulo, (const int32_t*)w.uhi, vertexIn, (const float*)w.Q, w.key, edgeCost);
        Cluster p;
        p.Nv = Nv; p.B = (int)B; p.nvIn = nvIn; p.want = want; p.ustart = w.ustart; p.ulo = w.ulo; p.uhi = w.uhi; p.key = w.key;
        p.covered = w.covered; p.vminA = w.vminA; p.vminB = w.vminB; p.vminC = w.vminC;
        p.listA = w.listA; p.listB = w.listB; p.taken = w.taken; p.joined = w.joined; p.matched = w.matched; p.attached = w.attached;
        p.prefix = w.prefix; p.rest = w.rest; p.hist = w.hist; p.digit_bits = w.digit_bits; p.counters = w.counters; p.barrier = w.barrier;
        p.rounds = w.rounds; p.status = w.status; p.vtReplace = vtReplace; p.head = w.head; p.next = w.next;
        if (most_faces <= SAMPLE_FACES) {
            const int threads = most_faces <= 512 ? 256 : (most_faces <= 2048 ? 512 : 1024);
            PB_LAUNCH("dec_cluster_samples", cluster_samples_kernel, (unsigned)(B < 65535 ? B : 65535), threads, 0, stream, p);
        } else {
            // as many blocks as have work and fit at once
            int64_t blocks = ceil_div(3 * Nf, GRID_THREADS * 4);
            int per_sm = 0;
            PB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cluster_grid_kernel, GRID_THREADS, 0));
            if (blocks > (int64_t)sm_count() * per_sm) blocks = (int64_t)sm_count() * per_sm;
            PB_REQUIRE(blocks > 0, PB200_ECUDA, "mesh_simplify: the clustering kernel does not fit this device");
            void* args[] = {&p};
            LaunchScope scope("dec_cluster_grid", stream);
            PB_CUDA(cudaLaunchCooperativeKernel((void*)cluster_grid_kernel, dim3((unsigned)blocks), dim3(GRID_THREADS), args, 0, stream));
        }
        PB_LAUNCH("dec_face_relabel", face_relabel_kernel, scan::tiles(Nf), scan::THREADS, 0, stream, Nf, Nv, (int)B, mfIn,
                  (const int32_t*)vtReplace, faceIn, relabelled, isDegenerate, w.kept, mfOut, w.ftile);
    }
    PB_LAUNCH("dec_kept_totals", kept_totals_kernel, vt, scan::THREADS, 0, stream, Nv, (int)B, nvIn, (const int32_t*)w.kept, w.tile, nvOut);
    PB_LAUNCH("dec_vertex_map", vertex_map_kernel, vt, scan::THREADS, 0, stream, Nv, (const int32_t*)w.kept, (const int32_t*)w.tile, vtMap);
    return PB200_OK;
}

static bool sizes_ok(int64_t B, int64_t D, int64_t Nv, int64_t Nf) {
    return B >= 1 && B < (1 << 20) && D >= 3 && D <= 4096 && Nv >= 0 && Nf >= 0 && Nf < (1LL << 29) && Nv < (1LL << 30);
}

}  // namespace dec
}  // namespace pb

using namespace pb;
using namespace pb::dec;

extern "C" {

size_t pb200_mesh_simplify_workspace_bytes(int64_t B, int64_t Nv, int64_t Nf) {
    if (B < 0 || Nv < 0 || Nf < 0) return 0;
    return carve(nullptr, B, Nv, Nf).total;
}

int pb200_mesh_simplify(int useArea, float wgtBnd, int64_t B, int64_t D, int64_t Nv, int64_t Nf,
                        const int32_t* nvIn, const int32_t* mfIn, const int32_t* nv2Remove, const float* vertexIn,
                        const int32_t* faceIn, const float* planeIn, int32_t* nvOut, int32_t* mfOut, float* vertexOut,
                        int32_t* faceOut, int32_t* vtReplace, int32_t* vtMap, uint8_t* isDegenerate, float* edgeCost,
                        int64_t* info, void* workspace, size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(sizes_ok(B, D, Nv, Nf), PB200_EINVAL, "mesh_simplify: bad sizes");
    PB_REQUIRE(Nv > 0 || Nf == 0, PB200_EINVAL, "mesh_simplify: faces without vertices");
    PB_REQUIRE(nvIn && mfIn && nv2Remove && nvOut && mfOut, PB200_EINVAL, "mesh_simplify: null pointer");
    PB_REQUIRE(Nv == 0 || (vertexIn && vertexOut && vtReplace && vtMap), PB200_EINVAL, "mesh_simplify: null pointer");
    PB_REQUIRE(Nf == 0 || (faceIn && planeIn && faceOut && isDegenerate), PB200_EINVAL, "mesh_simplify: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_mesh_simplify_workspace_bytes(B, Nv, Nf), PB200_EWORKSPACE,
               "mesh_simplify: workspace too small");
    if (info) info[0] = info[1] = info[2] = info[3] = 0;

    // the per-sample running totals decide the segmentation: check them on the host (B values each)
    int64_t most_faces = 0;
    {
        int32_t* h = (int32_t*)malloc(sizeof(int32_t) * 2 * (size_t)B);
        PB_REQUIRE(h, PB200_EINVAL, "mesh_simplify: out of host memory");
        cudaError_t e = cudaMemcpyAsync(h, nvIn, sizeof(int32_t) * B, cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(h + B, mfIn, sizeof(int32_t) * B, cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        bool ok = e == cudaSuccess;
        for (int64_t s = 0; ok && s < B; ++s) {
            const int32_t pv = s ? h[s - 1] : 0, pf = s ? h[B + s - 1] : 0;
            ok = h[s] >= pv && h[B + s] >= pf;
            if (h[B + s] - pf > most_faces) most_faces = h[B + s] - pf;
        }
        ok = ok && h[B - 1] == Nv && h[2 * B - 1] == Nf;
        free(h);
        if (e != cudaSuccess) return cuda_fail(e, "mesh_simplify: reading the sample sizes");
        PB_REQUIRE(ok, PB200_EINVAL, "mesh_simplify: nvIn / mfIn must be non-decreasing running totals ending at Nv / Nf");
    }
    const Work w = carve(workspace, B, Nv, Nf);
    int rc = cluster_pass(w, useArea, wgtBnd, B, D, Nv, Nf, most_faces, nvIn, mfIn, nv2Remove, vertexIn, faceIn, planeIn, nvOut, mfOut,
                          vtReplace, vtMap, faceOut, isDegenerate, edgeCost, stream);
    if (rc) return rc;
    if (Nv > 0)
        PB_LAUNCH("dec_contract", contract_kernel, (unsigned)ceil_div(Nv, 128), 128, 0, stream, Nv, (int)D, (const int32_t*)vtReplace,
                  (const int32_t*)w.head, (const int32_t*)w.next, vertexIn, (const int32_t*)nullptr, vertexOut, w.listA, w.listB, w.counters + 7);
    if (Nf > 0)
        PB_LAUNCH("dec_face_update", face_update_kernel, (unsigned)ceil_div(Nf, 256), 256, 0, stream, Nf,
                  (const int32_t*)vtMap, (const uint8_t*)isDegenerate, faceOut);
    int32_t status = 0, counts[3] = {0, 0, 0};
    PB_CUDA(cudaMemcpyAsync(&status, w.status, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    if (info && Nf > 0) {
        PB_CUDA(cudaMemcpyAsync(&counts[0], w.ustart + Nv, sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
        PB_CUDA(cudaMemcpyAsync(&counts[1], w.rounds, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
    }
    PB_CUDA(cudaStreamSynchronize(stream));
    PB_REQUIRE(status != PB200_EINDEX, PB200_EINDEX, "mesh_simplify: face holds a vertex id outside [0, Nv)");
    PB_REQUIRE(status != ECROSS, PB200_EINDEX, "mesh_simplify: a face joins vertices of two samples");
    PB_REQUIRE(status == 0, PB200_ECUDA, "mesh_simplify: a wait inside the clustering kernel ran out");
    if (info) { info[0] = counts[0]; info[1] = counts[1]; info[2] = counts[2]; }
    return PB200_OK;
}

int pb200_decimate_begin(int useArea, float wgtBnd, int64_t B, int64_t D, int64_t Nv, int64_t Nf, int64_t mostFaces, const int32_t* nv,
                         const int32_t* mf, const int32_t* target, const float* vertexIn, const int32_t* faceIn, const float* planeIn,
                         int32_t* nvOut, int32_t* mfOut, int32_t* status, int32_t* vtReplace, int32_t* vtMap, void* workspace,
                         size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(sizes_ok(B, D, Nv, Nf) && Nv > 0, PB200_EINVAL, "decimate_begin: bad sizes");
    PB_REQUIRE(nv && mf && target && nvOut && mfOut && status && vertexIn && vtReplace && vtMap && (Nf == 0 || (faceIn && planeIn)),
               PB200_EINVAL, "decimate_begin: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_mesh_simplify_workspace_bytes(B, Nv, Nf), PB200_EWORKSPACE,
               "decimate_begin: workspace too small");
    const Work w = carve(workspace, B, Nv, Nf);
    PB_LAUNCH("dec_begin_pass", begin_pass_kernel, 1, 1024, 0, stream, (int)B, nv, mf, target, w.nvCum, w.mfCum, w.want);
    int rc = cluster_pass(w, useArea, wgtBnd, B, D, Nv, Nf, mostFaces, w.nvCum, w.mfCum, w.want, vertexIn, faceIn, planeIn, nvOut, mfOut,
                          vtReplace, vtMap, w.relabelled, w.degenerate, nullptr, stream);
    if (rc) return rc;
    PB_CUDA(cudaMemcpyAsync(status, w.status, sizeof(int32_t), cudaMemcpyDeviceToDevice, stream));
    return PB200_OK;
}

int pb200_decimate_finish(int64_t B, int64_t D, int64_t Nv, int64_t Nf, const float* vertexIn, const int32_t* vtReplace,
                          const int32_t* vtMap, float* vertexOut, int32_t* faceOut, float* geometryOut, void* workspace,
                          size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(sizes_ok(B, D, Nv, Nf) && Nv > 0, PB200_EINVAL, "decimate_finish: bad sizes");
    PB_REQUIRE(vertexIn && vtReplace && vtMap && vertexOut && (Nf == 0 || (faceOut && geometryOut)), PB200_EINVAL,
               "decimate_finish: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= pb200_mesh_simplify_workspace_bytes(B, Nv, Nf), PB200_EWORKSPACE,
               "decimate_finish: workspace too small");
    const Work w = carve(workspace, B, Nv, Nf);
    PB_LAUNCH("dec_contract", contract_kernel, (unsigned)ceil_div(Nv, 128), 128, 0, stream, Nv, (int)D, vtReplace, (const int32_t*)w.head,
              (const int32_t*)w.next, vertexIn, vtMap, vertexOut, w.listA, w.listB, w.counters + 7);
    if (Nf > 0)
        PB_LAUNCH("dec_emit_faces", emit_faces_kernel, scan::tiles(Nf), scan::THREADS, 0, stream, Nf, (int)D, (const int32_t*)w.ftile,
                  (const uint8_t*)w.degenerate, (const int32_t*)w.relabelled, vtMap, (const float*)vertexOut, faceOut, geometryOut,
                  w.counters + 7);
    return PB200_OK;
}

int pb200_combine_clusters(int64_t nvA, int64_t nvB, const int32_t* repA, const int32_t* mapA, const int32_t* repB,
                           const int32_t* mapB, int32_t* repOut, int32_t* mapOut, int32_t* status, void* workspace,
                           size_t workspace_bytes, void* stream_) {
    cudaStream_t stream = (cudaStream_t)stream_;
    PB_REQUIRE(nvA >= 0 && nvB >= 0 && nvA < (1LL << 31) - 1 && nvB < (1LL << 31) - 1, PB200_EINVAL,
               "combine_clusters: bad sizes");
    PB_REQUIRE(status && (nvA == 0 || (repA && mapA && repOut && mapOut)) && (nvB == 0 || (repB && mapB)), PB200_EINVAL,
               "combine_clusters: null pointer");
    PB_REQUIRE(workspace && workspace_bytes >= sizeof(int32_t) * (size_t)(nvB + 1), PB200_EWORKSPACE,
               "combine_clusters: workspace too small");
    PB_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), stream));
    if (nvA == 0) return PB200_OK;
    int32_t* rb = (int32_t*)workspace;
    if (nvB > 0) PB_CUDA(cudaMemcpyAsync(rb, repB, sizeof(int32_t) * nvB, cudaMemcpyDeviceToDevice, stream));
    const unsigned grid = (unsigned)ceil_div(nvA, 256);
    PB_LAUNCH("dec_merge_back", merge_back_kernel, grid, 256, 0, stream, nvA, nvB, repA, mapA, rb, repOut);
    PB_LAUNCH("dec_merge_follow", merge_follow_kernel, grid, 256, 0, stream, nvA, nvB, repA, mapA, (const int32_t*)rb, mapB, repOut,
              mapOut, status);
    return PB200_OK;
}

}  // extern "C"
