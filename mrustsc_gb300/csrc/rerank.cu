// rerank.cu -- exact finish of every row: candidates from the lists are
// pruned to the final threshold, re-measured in the FP32 difference form on
// the caller's coordinates, sorted by (distance, id), and any group of
// candidates whose FP32 gap is inside the difference form's error bound and
// that reaches the first k positions is adjudicated in FP64.
//
// This is what makes the neighbour lists equal to the FP64 exact kNN with
// lowest-index tie-break (tests/test_neighbors_audit.py:52-61) whatever form
// produced the candidates.  In reference-snap mode the value is instead the
// reference Metal kernel's (crates/scrust-gpu/src/kernels/knn.rs:223-244) and
// the order its (d^2, id) order (knn.rs:179-182), with no adjudication.
//
// One warp per row in the common case; rows whose lists overflowed, or whose
// union exceeds the warp's capacity, go to a block-per-row fallback that
// re-measures the whole row.
#include <cooperative_groups.h>

#include "common.cuh"
#include "internal.h"
#include "lists.cuh"

namespace scrust {

namespace {

constexpr int RR_WARPS = 4;
constexpr int RC = kRerankUnion;  // keys per warp
constexpr int FB_CAP = 4096;  // keys per fallback block
constexpr int FB_THREADS = 256;
constexpr int FB_ROWS = 32;      // rows at a time, a cluster each
constexpr int FB_CLUSTER = 8;
// Solves of up to this many columns: a block a row, three an SM at a time.  (A
// row is then short against the cluster's barriers: 700, 2,100, 4,000, 8,000 and
// 16,000 rows of which every one comes here took 0.99, 2.2, 4.0, 8.6 and 21.5 ms
// by clusters, 0.47, 0.53, 0.73, 1.5 and 3.9 ms so.  More columns would take
// more scratch than the 32 rows of a million do.)
constexpr int64_t FB_BLOCK_COLUMNS = 32768;

struct RerankArgs {
    const float* qx;
    const float* rx;
    const float* qn2;
    const float* rn2;
    CosineRows cosine;
    int raw_stride;  // floats per row of cosine.raw
    int post;  // distances of cosine rows are written by a pass after this one
    const float* qraw;
    const float* rraw;
    RowBounds bounds;
    Lists lists;
    const uint32_t* perm;  // list entry (candidate id) -> input reference row, or null
    const uint32_t* qperm; // list row -> input query row, or null (a self solve: perm)
    const float* xs;       // working rows in list order (ordered solves), or null
    const float* xr_list;  // reference rows indexed by list entry (xs for a self solve)
    int ids_only;          // the lists hold ids only (collected below their thresholds): keep every entry
    int xs_stride;         // floats per row of xs and xr_list
    int xs_v8;             // rows padded with zeros to a multiple of 8 floats, 32-byte aligned
    const uint32_t* row_lo;  // per input row: first row of its solve (a batch of solves), or null
    const uint32_t* row_hi;  // per input row: end of its solve
    const float* theta;    // per list: its threshold when the candidate pass ended, or null
    int64_t nq, nr;
    int d, k, mode, metric, self;
    int64_t self_offset;  // query row q is reference row q + self_offset
    float gamma;
    uint32_t* out_idx;
    float* out_dist;
    uint32_t* fb_rows;
    uint32_t* fb_count;
    uint32_t* fb_next;
    uint32_t* big_rows;   // rows with many survivors, for the second sorted pass
    uint32_t* big_count;
    uint32_t* big_next;
    uint32_t* wide_rows;  // rows for the eight-a-lane pass of a solve of many neighbours
    uint32_t* wide_count;
    uint32_t* wide_next;
    float* fb_scratch;
    int* err;
};

__device__ __forceinline__ float compute_r(const RerankArgs& a, int64_t q, uint32_t j) {
    if (a.mode == SCRUST_MODE_REFERENCE_SNAP)
        return dist2_reference_snap(a.qx + q * a.d, a.rx + (int64_t)j * a.d, a.d, a.qn2[q], a.rn2[j]);
    return dist2_f32(a.qx + q * a.d, a.rx + (int64_t)j * a.d, a.d);
}

// Two sorted FP32 values that the difference form cannot order reliably.
__device__ __forceinline__ bool tied(const RerankArgs& a, float r1, float r2) {
    if (a.mode == SCRUST_MODE_REFERENCE_SNAP) return false;
    float tol = a.gamma * (r1 + r2) + kTieAbs;
    if (a.metric == SCRUST_METRIC_COSINE)
        tol += 2.384185791015625e-07f * (sqrtf(r1) + sqrtf(r2)) + 1e-14f;
    return (r2 - r1) <= tol;
}

__device__ __forceinline__ double adjudicate(const RerankArgs& a, int64_t q, uint32_t j) {
    if (a.metric == SCRUST_METRIC_COSINE)
        return cosine_f64(a.qraw + q * a.d, a.rraw + (int64_t)j * a.d, a.d, a.cosine.norm64[q], a.cosine.norm64[j]);
    return sqrt(dist2_f64(a.qraw + q * a.d, a.rraw + (int64_t)j * a.d, a.d));
}

__device__ __forceinline__ float key_r(unsigned long long key) { return key_float((uint32_t)(key >> 32)); }
__device__ __forceinline__ uint32_t key_id(unsigned long long key) { return (uint32_t)key; }

// Rows of the reference with the same bits in every coordinate.
__device__ __forceinline__ bool rows_equal(const float* __restrict__ u, const float* __restrict__ v, int d) {
    const uint32_t* x = reinterpret_cast<const uint32_t*>(u);
    const uint32_t* y = reinterpret_cast<const uint32_t*>(v);
    for (int t0 = 0; t0 < d; t0 += 8) {
        bool eq = true;
#pragma unroll
        for (int t = 0; t < 8; ++t)
            if (t0 + t < d) eq &= __ldg(x + t0 + t) == __ldg(y + t0 + t);
        if (!eq) return false;
    }
    return true;
}

// Tie groups are runs of consecutive sorted candidates whose FP32 values the
// difference form cannot order.  A group that reaches the first k positions
// is ordered by FP64 (distance, id), and its members take FP64 distances --
// unless every member's row has the same bits as the first member's row
// (duplicated cells): the FP32 values are then equal, the order by id that
// the sort left is already the FP64 order, and the FP32 value is the
// distance.  Cosine rows always take FP64 values: in a pass of their own where
// the solve has one (`post`; equal rows have equal FP64 distances, too), else
// here.
enum : uint8_t { TIE_NONE = 0, TIE_SAME = 1, TIE_DIFF = 2 };

// Writes the first k of the sorted candidates keys[0..m), resolving tie
// groups as above; dbl and flags hold m entries of scratch.
template <class Team>
__device__ void finalize_row(const Team& team, const RerankArgs& a, int64_t q,
                             const unsigned long long* keys, int m, double* dbl, uint8_t* flags) {
    const int k = a.k;
    const bool cosine = a.metric == SCRUST_METRIC_COSINE;
    for (int p = team.rank; p < m; p += team.size()) {
        int gs = p;
        while (gs > 0 && tied(a, key_r(keys[gs - 1]), key_r(keys[gs]))) gs--;
        if (gs >= k) continue;
        int ge = p;
        while (ge + 1 < m && tied(a, key_r(keys[ge]), key_r(keys[ge + 1]))) ge++;
        uint8_t f = TIE_NONE;
        if (ge > gs && (!cosine || a.post))
            f = (p == gs || rows_equal(a.rraw + (int64_t)key_id(keys[gs]) * a.d,
                                       a.rraw + (int64_t)key_id(keys[p]) * a.d, a.d))
                    ? TIE_SAME
                    : TIE_DIFF;
        flags[p] = f;
    }
    team.sync();
    for (int p = team.rank; p < m; p += team.size()) {
        int gs = p;
        while (gs > 0 && tied(a, key_r(keys[gs - 1]), key_r(keys[gs]))) gs--;
        if (gs >= k) continue;
        int ge = p;
        while (ge + 1 < m && tied(a, key_r(keys[ge]), key_r(keys[ge + 1]))) ge++;
        bool fp64 = cosine && !a.post;
        if (ge > gs && !fp64)
            for (int o = gs; o <= ge; ++o) fp64 |= flags[o] == TIE_DIFF;
        if (fp64) dbl[p] = adjudicate(a, q, key_id(keys[p]));
    }
    team.sync();
    for (int p = team.rank; p < m; p += team.size()) {
        int gs = p;
        while (gs > 0 && tied(a, key_r(keys[gs - 1]), key_r(keys[gs]))) gs--;
        if (gs >= k) continue;
        int ge = p;
        while (ge + 1 < m && tied(a, key_r(keys[ge]), key_r(keys[ge + 1]))) ge++;
        bool fp64 = cosine && !a.post;
        if (ge > gs && !fp64)
            for (int o = gs; o <= ge; ++o) fp64 |= flags[o] == TIE_DIFF;
        const uint32_t id = key_id(keys[p]);
        int pos = p;
        if (fp64 && ge > gs) {
            const double dv = dbl[p];
            int rank = 0;
            for (int o = gs; o <= ge; ++o) {
                const double dq = dbl[o];
                const uint32_t io = key_id(keys[o]);
                rank += (dq < dv) || (dq == dv && io < id);
            }
            pos = gs + rank;
        }
        if (pos < k) {
            const float dist = fp64 ? __double2float_rn(dbl[p]) : sqrtf(key_r(keys[p]));
            a.out_idx[q * k + pos] = a.row_lo ? id - a.row_lo[q] : id;
            a.out_dist[q * k + pos] = dist;
        }
    }
    team.sync();
}

// A row without k columns that can be ranked (NaN coordinates, more ties than
// the fallback holds): the first k columns of its solve other than itself, at
// distance NaN, so that no later kernel meets an id that was never written.
template <class Team>
__device__ void write_open_row(const Team& team, const RerankArgs& a, int64_t q) {
    const int64_t lo = a.row_lo ? (int64_t)a.row_lo[q] : 0, own = a.self ? q + a.self_offset : -1;
    for (int t = team.rank; t < a.k; t += team.size()) {
        const int64_t j = lo + t + (own >= 0 && lo + t >= own ? 1 : 0);
        a.out_idx[q * a.k + t] = (uint32_t)(j - lo);
        a.out_dist[q * a.k + t] = __int_as_float(0x7fc00000);
    }
}

__device__ void push_fallback(const RerankArgs& a, int64_t slot) {
    uint32_t pos = atomicAdd(a.fb_count, 1u);
    a.fb_rows[pos] = (uint32_t)slot;
}

__device__ __forceinline__ int64_t input_row(const RerankArgs& a, int64_t s) {
    return a.perm ? (int64_t)a.perm[s] : s;
}
// The input query row of list row `slot`.
__device__ __forceinline__ int64_t query_row(const RerankArgs& a, int64_t slot) {
    return a.qperm ? (int64_t)a.qperm[slot] : slot;
}

// (Shared memory leaves room for three blocks an SM; told so, the compiler keeps
// more of a row's loads in flight: 700 x 100, k = 40, plain form: 381 us a solve
// at 40 registers, 348 so.)
__global__ void __launch_bounds__(RR_WARPS * 32, 3) rerank_warp_kernel(RerankArgs a) {
    extern __shared__ unsigned long long rr_smem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    unsigned long long* A = rr_smem + (size_t)warp * 2 * RC;
    unsigned long long* B = A + RC;
    uint8_t* flags = reinterpret_cast<uint8_t*>(rr_smem + (size_t)RR_WARPS * 2 * RC) + (size_t)warp * RC;
    const int64_t slot = (int64_t)blockIdx.x * RR_WARPS + warp;  // list row
    if (slot >= a.nq || (a.qperm && a.qperm[slot] == 0xffffffffu)) return;
    WarpTeam team;
    if (a.lists.overflow[slot]) {
        if (lane == 0) push_fallback(a, slot);
        return;
    }
    const int64_t q = query_row(a, slot);
    const int segs = a.lists.segments;
    int m0 = 0;
    for (int s = 0; s < segs; ++s) m0 += (int)min(a.lists.cnt[slot * segs + s], (uint32_t)a.lists.ctot);
    if (m0 > RC || m0 < a.k) {
        if (lane == 0) push_fallback(a, slot);
        return;
    }
    int off = 0;
    for (int s = 0; s < segs; ++s) {
        const int c = (int)min(a.lists.cnt[slot * segs + s], (uint32_t)a.lists.ctot);
        const int64_t base = (slot * segs + s) * (int64_t)a.lists.ctot;
        for (int p = lane; p < c; p += 32) {
            uint32_t id = a.lists.ids[base + p];
            float v = a.lists.vals[base + p];
            if ((int64_t)id >= a.nr) {  // never written by a candidate kernel: refuse to read it
                atomicExch(a.err + DERR_CANDIDATES, 1);
                id = 0;
                v = __int_as_float(0x7f800000);
            }
            if (a.perm) id = a.perm[id];
            A[off + p] = ((unsigned long long)float_key(v) << 32) | id;
        }
        off += c;
    }
    __syncwarp();
    const uint32_t kth = team_select_hi(team, A, m0, a.k);
    const float theta = a.bounds.margin ? PlainBound{a.bounds.margin[slot]}.theta(key_float(kth))
                                        : TensorBound{a.bounds.A[slot], a.bounds.delta[slot], a.bounds.eps2[slot]}.theta(
                                              key_float(kth));
    int m = 0;
    for (int b0 = 0; b0 < m0; b0 += 32) {
        const int p = b0 + lane;
        bool keep = false;
        uint32_t id = 0;
        if (p < m0) {
            const unsigned long long kk = A[p];
            keep = key_r(kk) < theta;
            id = key_id(kk);
        }
        const uint32_t ballot = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const float r = compute_r(a, q, id);
            B[m + __popc(ballot & lanemask_lt())] = ((unsigned long long)float_key(r) << 32) | id;
        }
        m += __popc(ballot);
    }
    if (m < a.k) {  // no threshold: bounds of NaN
        write_open_row(team, a, q);
        return;
    }
    __syncwarp();
    const int P = next_pow2(m);
    for (int p = m + lane; p < P; p += 32) B[p] = ~0ull;
    __syncwarp();
    team_bitonic_sort(team, B, P);
    finalize_row(team, a, q, B, m, reinterpret_cast<double*>(A), flags);
}

// The cosine distance of rows q and j in f32 pairs (the Dot2 scheme of Ogita,
// Rump and Oishi, SIAM J. Sci. Comput. 26 (2005), in eight chains, times the
// norms' reciprocals): h + l, h rounded, within cosine_pair_error of the true
// value and of cosine_f64's.  NaN for rows without reciprocals, whose products
// may leave f32's range.
//
// With u = 2^-24, m terms a chain and S = sum |x y| <= |x| |y|: a chain's low
// part sums 2 m terms that come to at most (m + 1) u of its share of S, so it
// is off by 2 m (m + 1) u^2 of that; combining the chains adds 16 (m + 2)
// u^2 S; the two products with reciprocals, themselves within u^2, and the
// subtraction 32 u^2.  cosine_f64 is off by (d + 4) 2^-53.
__device__ __forceinline__ float cosine_pair_error(int stride, int d) {
    const float m = (float)(stride / 8);
    return (2.f * m * (m + 1.f) + 16.f * (m + 2.f) + 32.f + 0.0625f * (d + 4)) * 4.44089210e-15f;  // 1.25 u^2
}
__device__ __forceinline__ void two_sum(float a, float b, float* sum, float* error) {
    const float z = __fadd_rn(a, b), t = __fsub_rn(z, a);
    *error = __fadd_rn(__fsub_rn(a, __fsub_rn(z, t)), __fsub_rn(b, t));
    *sum = z;
}
__device__ __forceinline__ void cosine_pair(const CosineRows& rows, int stride, int64_t q, int64_t j, float* high,
                                            float* low) {
    const float* x = rows.raw + q * stride;
    const float* y = rows.raw + j * stride;
    float s[8], c[8];
#pragma unroll
    for (int h = 0; h < 8; ++h) s[h] = c[h] = 0.f;
    for (int t = 0; t < stride; t += 8) {
        float xv[8], yv[8];
        ldg_v8(x + t, xv);
        ldg_v8(y + t, yv);
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            const float p = __fmul_rn(xv[h], yv[h]);
            const float pe = __fmaf_rn(xv[h], yv[h], -p);
            float ze;
            two_sum(s[h], p, &s[h], &ze);
            c[h] = __fadd_rn(c[h], __fadd_rn(pe, ze));
        }
    }
#pragma unroll
    for (int w = 4; w > 0; w >>= 1) {
#pragma unroll
        for (int h = 0; h < w; ++h) {
            float ze;
            two_sum(s[h], s[h + w], &s[h], &ze);
            c[h] = __fadd_rn(__fadd_rn(c[h], c[h + w]), ze);
        }
    }
    float th = s[0], tl = c[0];
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        const float2 inv = __ldg(rows.inverse + (side ? j : q));
        const float p = __fmul_rn(th, inv.x);
        float e = __fmaf_rn(th, inv.x, -p);
        e = __fmaf_rn(th, inv.y, e);
        e = __fmaf_rn(tl, inv.x, e);
        th = __fadd_rn(p, e);
        tl = __fsub_rn(e, __fsub_rn(th, p));
    }
    float z, ze;
    two_sum(1.f, -th, &z, &ze);
    const float rest = __fsub_rn(ze, tl);
    *high = __fadd_rn(z, rest);
    *low = __fsub_rn(rest, __fsub_rn(*high, z));
}
// Tensor-form solves: the candidate pass left every list with a threshold no
// smaller than the final one, so the rerank needs no selection.  A warp per
// list row keeps the entries below the smaller of its lists' thresholds,
// measures them on the working rows laid out in list order (for an ordered
// solve neighbouring rows share candidates, which stay in cache), and
// finishes as above with input ids.  A row with more than RS_KEYS survivors
// (many cells inside the bound of the k-th, as for queries off the data's
// manifold in high dimension) is finished by a second pass with room for
// RS_BIG_KEYS; beyond that, by the fallback.
constexpr int RS_WARPS = 8;
constexpr int RS_KEYS = 128;
constexpr int RS_BIG_WARPS = 4;
constexpr int RS_BIG_KEYS = 2048;

// 0: done; 1: more than `cap` survivors; 2: needs the fallback.
template <int CAP>
__device__ int sorted_row(const RerankArgs& a, int64_t slot, unsigned long long* keys, double* dbl, uint8_t* flags) {
    const int lane = threadIdx.x & 31;
    WarpTeam team;
    if (a.lists.overflow[slot]) return 2;
    const int segs = a.lists.segments;
    float theta = __int_as_float(0x7f800000);
    for (int l = 0; l < segs; ++l) theta = fminf(theta, a.theta[slot * segs + l]);
    const float* xq = a.xs + slot * a.xs_stride;
    int m = 0;
    for (int l = 0; l < segs; ++l) {
        const int c = (int)min(a.lists.cnt[slot * segs + l], (uint32_t)a.lists.ctot);
        const int64_t base = (slot * segs + l) * (int64_t)a.lists.ctot;
        for (int b0 = 0; b0 < c; b0 += 32) {
            const int p = b0 + lane;
            bool keep = false;
            uint32_t id = 0;
            if (p < c) {
                id = a.lists.ids[base + p];
                if ((int64_t)id >= a.nr) {  // never written by a candidate kernel: refuse to read it
                    atomicExch(a.err + DERR_CANDIDATES, 1);
                } else {
                    keep = a.ids_only || a.lists.vals[base + p] < theta;
                }
            }
            const uint32_t ballot = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const int pos = m + __popc(ballot & lanemask_lt());
                if (pos < CAP) {
                    const float* xr = a.xr_list + (int64_t)id * a.xs_stride;
                    const float r = a.xs_v8 ? dist2_f32_v8(xq, xr, a.xs_stride / 8) : dist2_f32(xq, xr, a.d);
                    keys[pos] = ((unsigned long long)float_key(r) << 32) | (uint32_t)input_row(a, id);
                }
            }
            m += __popc(ballot);
        }
    }
    if (m < a.k) return 2;
    if (m > CAP) return 1;
    __syncwarp();
    const int P = next_pow2(m);
    for (int p = m + lane; p < P; p += 32) keys[p] = ~0ull;
    __syncwarp();
    team_bitonic_sort(team, keys, P);
    finalize_row(team, a, query_row(a, slot), keys, m, dbl, flags);
    return 0;
}

__device__ __forceinline__ unsigned long long min_u64(unsigned long long x, unsigned long long y) {
    return x < y ? x : y;
}
__device__ __forceinline__ unsigned long long max_u64(unsigned long long x, unsigned long long y) {
    return x < y ? y : x;
}

// Ascending bitonic sort across the warp of P = 32 or 64 keys, position
// lane + 32 r in key[r] (key[1] unused when P = 32); fully unrolled.
template <int P>
__device__ __forceinline__ void warp_sort_keys(unsigned long long (&key)[2]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int size = 2; size <= P; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride == 32) {
                const unsigned long long lo = min_u64(key[0], key[1]), hi = max_u64(key[0], key[1]);
                key[0] = lo;
                key[1] = hi;
            } else {
#pragma unroll
                for (int r = 0; r < P / 32; ++r) {
                    const int i = lane + 32 * r;
                    const unsigned long long o = __shfl_xor_sync(0xffffffffu, key[r], stride);
                    const bool take_min = ((i & stride) == 0) == ((i & size) == 0);
                    key[r] = ((key[r] < o) == take_min) ? key[r] : o;
                }
            }
        }
    }
}

// Rows whose lists hold at most 64 entries in all (nearly every row): the
// entries are read two per lane, the survivors measured, and the (distance,
// id) keys sorted in registers across the warp (bitonic over 64 positions,
// position lane + 32 r in key[r]); tie groups are then found from a ballot of
// the positions that start one.  The result is finalize_row's.  Returns 0
// when done, 2 for the fallback, 3 when the lists hold more than 64 entries.
__device__ int sorted_row_regs(const RerankArgs& a, int64_t slot, unsigned long long* keys_s, double* dbl) {
    const int lane = threadIdx.x & 31;
    const int segs = a.lists.segments;
    if (segs > 32 && !a.ids_only) return 3;  // the threshold below is that of the first 32 lists
    // The row's header, its own coordinates and -- with two lists, the
    // common case -- the first 32 slots of both lists are read at once (the
    // lists hold at least 64 slots each); only then is anything tested.
    // Slots 32..63 of a list are read only when it holds more than 32.
    const uint32_t ovf = a.lists.overflow[slot];
    const int cl = lane < segs ? (int)min(a.lists.cnt[slot * segs + lane], (uint32_t)a.lists.ctot) : 0;
    const float tl = lane < segs ? a.theta[slot * segs + lane] : __int_as_float(0x7f800000);
    const int64_t base0 = slot * segs * (int64_t)a.lists.ctot;
    uint32_t sid[2][2] = {{0u, 0u}, {0u, 0u}};
    float sval[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
    if (segs == 2) {
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            sid[l][0] = a.lists.ids[base0 + l * (int64_t)a.lists.ctot + lane];
            sval[l][0] = a.ids_only ? __int_as_float(0xff800000) : a.lists.vals[base0 + l * (int64_t)a.lists.ctot + lane];
        }
    }
    if (ovf) return 2;
    float theta = tl;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) theta = fminf(theta, __shfl_xor_sync(0xffffffffu, theta, o));
    int m0 = 0;
    uint32_t eid[2] = {0u, 0u};
    float eval[2] = {0.f, 0.f};
    bool have[2] = {false, false};
    if (segs == 2) {
        const int c0 = __shfl_sync(0xffffffffu, cl, 0), c1 = __shfl_sync(0xffffffffu, cl, 1);
        m0 = c0 + c1;
        if (m0 > 64) return 3;
#pragma unroll
        for (int l = 0; l < 2; ++l)
            if ((l == 0 ? c0 : c1) > 32) {
                sid[l][1] = a.lists.ids[base0 + l * (int64_t)a.lists.ctot + lane + 32];
                sval[l][1] = a.ids_only ? __int_as_float(0xff800000)
                                        : a.lists.vals[base0 + l * (int64_t)a.lists.ctot + lane + 32];
            }
        // Position e = lane + 32 r: list 0 slot e below c0, else list 1 slot e - c0.
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int e = lane + 32 * r;
            const int p1 = max(e - c0, 0);
            const uint32_t i10 = __shfl_sync(0xffffffffu, sid[1][0], p1 & 31);
            const uint32_t i11 = __shfl_sync(0xffffffffu, sid[1][1], p1 & 31);
            const float v10 = __shfl_sync(0xffffffffu, sval[1][0], p1 & 31);
            const float v11 = __shfl_sync(0xffffffffu, sval[1][1], p1 & 31);
            have[r] = e < m0;
            eid[r] = e < c0 ? sid[0][r] : (p1 < 32 ? i10 : i11);
            eval[r] = e < c0 ? sval[0][r] : (p1 < 32 ? v10 : v11);
        }
    } else {
        // Entry e of the row's lists (in list order) -> list and position.
        int list[2] = {-1, -1}, pos[2] = {0, 0};
        for (int l0 = 0; l0 < segs; l0 += 32) {
            const int own = l0 == 0 ? cl
                            : l0 + lane < segs
                                ? (int)min(a.lists.cnt[slot * segs + l0 + lane], (uint32_t)a.lists.ctot)
                                : 0;
            // Only lists that hold something are looked at.
            for (uint32_t some = __ballot_sync(0xffffffffu, own != 0); some; some &= some - 1) {
                const int l = __ffs(some) - 1;
                const int c = __shfl_sync(0xffffffffu, own, l);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int e = lane + 32 * r;
                    if (list[r] < 0 && e < m0 + c) {
                        list[r] = l0 + l;
                        pos[r] = e - m0;
                    }
                }
                m0 += c;
            }
        }
        if (m0 > 64) return 3;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (list[r] >= 0) {
                const int64_t at = base0 + list[r] * (int64_t)a.lists.ctot + pos[r];
                have[r] = true;
                eid[r] = a.lists.ids[at];
                eval[r] = a.ids_only ? __int_as_float(0xff800000) : a.lists.vals[at];
            }
        }
    }
    const float* xq = a.xs + slot * a.xs_stride;
    unsigned long long key[2] = {~0ull, ~0ull};
    int m = 0;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        bool keep = false;
        const uint32_t id = eid[r];
        if (have[r]) {
            if ((int64_t)id >= a.nr) {  // never written by a candidate kernel: refuse to read it
                atomicExch(a.err + DERR_CANDIDATES, 1);
            } else {
                keep = eval[r] < theta;
            }
        }
        if (keep) {
            const float* xr = a.xr_list + (int64_t)id * a.xs_stride;
            const float d2 = a.xs_v8 ? dist2_f32_v8(xq, xr, a.xs_stride / 8) : dist2_f32(xq, xr, a.d);
            key[r] = ((unsigned long long)float_key(d2) << 32) | (uint32_t)input_row(a, id);
        }
        m += __popc(__ballot_sync(0xffffffffu, keep));
    }
    if (m < a.k) return 2;
    // Bitonic sort of the 64 positions (32 when the second half is empty).
    if (m0 > 32)
        warp_sort_keys<64>(key);
    else
        warp_sort_keys<32>(key);
    // Positions that start a tie group (runs of consecutive tied values).
    const unsigned long long up0 = __shfl_up_sync(0xffffffffu, key[0], 1);
    const unsigned long long up1 = __shfl_up_sync(0xffffffffu, key[1], 1);
    const unsigned long long last0 = __shfl_sync(0xffffffffu, key[0], 31);
    bool start[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int p = lane + 32 * r;
        const unsigned long long prev = r == 0 ? up0 : (lane == 0 ? last0 : up1);
        start[r] = p == 0 || p >= m || !tied(a, key_r(prev), key_r(key[r]));
    }
    const unsigned long long S =
        (unsigned long long)__ballot_sync(0xffffffffu, start[0]) |
        ((unsigned long long)__ballot_sync(0xffffffffu, start[1]) << 32);
    const int k = a.k;
    const bool cosine = a.metric == SCRUST_METRIC_COSINE;
    const int64_t q = query_row(a, slot);
    // The common case: positions 0..k all start a group, so the first k are
    // singletons and the sort's order and FP32 values are final.
    if ((!cosine || a.post) && k < 63 && (S & ((2ull << k) - 1)) == ((2ull << k) - 1)) {
        if (lane < k) {
            const uint32_t id = key_id(key[0]);
            a.out_idx[q * k + lane] = a.row_lo ? id - a.row_lo[q] : id;
            a.out_dist[q * k + lane] = sqrtf(key_r(key[0]));
        }
        if (lane + 32 < k) {
            const uint32_t id = key_id(key[1]);
            a.out_idx[q * k + lane + 32] = a.row_lo ? id - a.row_lo[q] : id;
            a.out_dist[q * k + lane + 32] = sqrtf(key_r(key[1]));
        }
        return 0;
    }
    int gs[2], ge[2];
    bool grouped[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int p = lane + 32 * r;
        const unsigned long long upto = p == 63 ? ~0ull : (2ull << p) - 1;  // positions 0..p
        gs[r] = 63 - __clzll(S & upto);
        const unsigned long long after = S & ~upto;
        ge[r] = min(after ? __ffsll(after) - 2 : 63, m - 1);
        grouped[r] = p < m && gs[r] < k && ge[r] > gs[r];
    }
    // Members whose row differs from their group's first member's row.
    unsigned long long D = 0;
    if ((!cosine || a.post) && __any_sync(0xffffffffu, grouped[0] || grouped[1])) {
        bool differs[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int p = lane + 32 * r;
            const uint32_t f0 = __shfl_sync(0xffffffffu, key_id(key[0]), gs[r] & 31);
            const uint32_t f1 = __shfl_sync(0xffffffffu, key_id(key[1]), gs[r] & 31);
            const uint32_t first = gs[r] < 32 ? f0 : f1;
            differs[r] = grouped[r] && p != gs[r] &&
                         !rows_equal(a.rraw + (int64_t)first * a.d, a.rraw + (int64_t)key_id(key[r]) * a.d, a.d);
        }
        D = (unsigned long long)__ballot_sync(0xffffffffu, differs[0]) |
            ((unsigned long long)__ballot_sync(0xffffffffu, differs[1]) << 32);
    }
    bool need[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int p = lane + 32 * r;
        const unsigned long long span =
            (ge[r] == 63 ? ~0ull : (2ull << ge[r]) - 1) & ~((1ull << gs[r]) - 1);  // positions gs..ge
        need[r] = p < m && gs[r] < k && ((cosine && !a.post) || (grouped[r] && (D & span) != 0));
    }
    const bool any_group = __any_sync(0xffffffffu, need[0] || need[1]);
    if (any_group) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int p = lane + 32 * r;
            if (p < m) keys_s[p] = key[r];
            if (need[r]) dbl[p] = adjudicate(a, q, key_id(key[r]));
        }
        __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int p = lane + 32 * r;
        if (p >= m || gs[r] >= k) continue;
        const uint32_t id = key_id(key[r]);
        int at = p;
        if (need[r] && ge[r] > gs[r]) {
            const double dv = dbl[p];
            int rank = 0;
            for (int o = gs[r]; o <= ge[r]; ++o) {
                const double dq = dbl[o];
                const uint32_t io = key_id(keys_s[o]);
                rank += (dq < dv) || (dq == dv && io < id);
            }
            at = gs[r] + rank;
        }
        if (at < k) {
            const float dist = need[r] ? __double2float_rn(dbl[p]) : sqrtf(key_r(key[r]));
            a.out_idx[q * k + at] = a.row_lo ? id - a.row_lo[q] : id;
            a.out_dist[q * k + at] = dist;
        }
    }
    __syncwarp();
    return 0;
}

// Ascending bitonic sort across the warp of 32 R keys, position lane + 32 r in
// key[r]; fully unrolled.
template <int R>
__device__ __forceinline__ void warp_sort_wide(unsigned long long (&key)[R]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int size = 2; size <= 32 * R; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= 32) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int o = r ^ (stride / 32);
                    if (o > r) {
                        const unsigned long long lo = min_u64(key[r], key[o]), hi = max_u64(key[r], key[o]);
                        const bool up = ((32 * r) & size) == 0;
                        key[r] = up ? lo : hi;
                        key[o] = up ? hi : lo;
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int i = lane + 32 * r;
                    const unsigned long long o = __shfl_xor_sync(0xffffffffu, key[r], stride);
                    const bool take_min = ((i & stride) == 0) == ((i & size) == 0);
                    key[r] = ((key[r] < o) == take_min) ? key[r] : o;
                }
            }
        }
    }
}

// sorted_row_regs for collected lists (ids below their thresholds) of up to
// 32 R entries in all: R entries a lane, the same result.  Solves of more than
// 32 neighbours keep 1.2 to 1.5 k candidates a row, past the 64 that
// sorted_row_regs holds (its shared-memory form, with the queue of rows above
// 128 entries, took 3.1 ms for 50,021 rows at k = 50 and 4.3 ms at k = 100).
// Returns 0 when done, 2 for the fallback, 3 for more entries than that.
template <int R>
__device__ int sorted_row_wide(const RerankArgs& a, int64_t slot, unsigned long long* keys_s, double* dbl) {
    constexpr uint32_t FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int segs = a.lists.segments;
    if (a.lists.overflow[slot]) return 2;
    // Entry e of the row's lists (in list order) -> list and position.
    int list[R], pos[R];
#pragma unroll
    for (int r = 0; r < R; ++r) list[r] = -1;
    int m = 0;
    for (int l0 = 0; l0 < segs; l0 += 32) {
        const int own =
            l0 + lane < segs ? (int)min(a.lists.cnt[slot * segs + l0 + lane], (uint32_t)a.lists.ctot) : 0;
        for (uint32_t some = __ballot_sync(FULL, own != 0); some; some &= some - 1) {
            const int l = __ffs(some) - 1;
            const int c = __shfl_sync(FULL, own, l);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int e = lane + 32 * r;
                if (list[r] < 0 && e < m + c) {
                    list[r] = l0 + l;
                    pos[r] = e - m;
                }
            }
            m += c;
        }
    }
    if (m > 32 * R) return 3;
    if (m < a.k) return 2;
    const float* xq = a.xs + slot * a.xs_stride;
    uint32_t id[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
        id[r] = list[r] >= 0 ? a.lists.ids[(slot * segs + list[r]) * (int64_t)a.lists.ctot + pos[r]] : 0xffffffffu;
    unsigned long long key[R];
    bool bad = false;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        key[r] = ~0ull;
        if (list[r] < 0) continue;
        if ((int64_t)id[r] >= a.nr) {  // never written by a candidate kernel: refuse to read it
            bad = true;
            continue;
        }
        const float* xr = a.xr_list + (int64_t)id[r] * a.xs_stride;
        const float d2 = a.xs_v8 ? dist2_f32_v8(xq, xr, a.xs_stride / 8) : dist2_f32(xq, xr, a.d);
        key[r] = ((unsigned long long)float_key(d2) << 32) | (uint32_t)input_row(a, id[r]);
    }
    if (__any_sync(FULL, bad)) {
        if (lane == 0) atomicExch(a.err + DERR_CANDIDATES, 1);
        return 2;
    }
    warp_sort_wide<R>(key);
    // Positions that start a tie group (runs of consecutive tied values).
    uint32_t S[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int p = lane + 32 * r;
        const unsigned long long up = __shfl_up_sync(FULL, key[r], 1);
        const unsigned long long last = __shfl_sync(FULL, key[r > 0 ? r - 1 : 0], 31);
        const unsigned long long prev = lane == 0 ? last : up;
        S[r] = __ballot_sync(FULL, p == 0 || p >= m || !tied(a, key_r(prev), key_r(key[r])));
    }
    const int k = a.k;
    const bool cosine = a.metric == SCRUST_METRIC_COSINE;
    const int64_t q = query_row(a, slot);
    // The common case: positions 0..k all start a group.
    bool plain = (!cosine || a.post) && k < 32 * R;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int bits = k + 1 - 32 * r;  // of this word that must be set
        const uint32_t want = bits >= 32 ? FULL : bits > 0 ? (1u << bits) - 1u : 0u;
        plain &= (S[r] & want) == want;
    }
    if (plain) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int p = lane + 32 * r;
            if (p < k) {
                const uint32_t c = key_id(key[r]);
                a.out_idx[q * k + p] = a.row_lo ? c - a.row_lo[q] : c;
                a.out_dist[q * k + p] = sqrtf(key_r(key[r]));
            }
        }
        return 0;
    }
    int gs[R], ge[R];
    bool grouped[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int p = lane + 32 * r;
        // The last start at or before p, and the one before the next start.
        gs[r] = 0;
        ge[r] = 32 * R - 1;
#pragma unroll
        for (int w = 0; w < R; ++w) {
            const uint32_t upto = w < r ? FULL : w == r ? FULL >> (31 - lane) : 0u;
            if (S[w] & upto) gs[r] = 32 * w + 31 - __clz(S[w] & upto);
        }
#pragma unroll
        for (int w = R - 1; w >= 0; --w) {
            const uint32_t after = w > r ? FULL : w == r ? ~(FULL >> (31 - lane)) : 0u;
            if (S[w] & after) ge[r] = 32 * w + __ffs(S[w] & after) - 2;
        }
        ge[r] = min(ge[r], m - 1);
        grouped[r] = p < m && gs[r] < k && ge[r] > gs[r];
        keys_s[p] = key[r];
    }
    __syncwarp();
    // Members whose row differs from their group's first member's row.
    uint32_t D[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int p = lane + 32 * r;
        const bool differs = (!cosine || a.post) && grouped[r] && p != gs[r] &&
                             !rows_equal(a.rraw + (int64_t)key_id(keys_s[gs[r]]) * a.d,
                                         a.rraw + (int64_t)key_id(key[r]) * a.d, a.d);
        D[r] = __ballot_sync(FULL, differs);
    }
    bool need[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int p = lane + 32 * r;
        bool any = false;  // a differing member in positions gs..ge
#pragma unroll
        for (int w = 0; w < R; ++w) {
            const int lo = max(gs[r] - 32 * w, 0), hi = min(ge[r] - 32 * w, 31);
            if (lo <= hi) any |= (D[w] & (FULL >> (31 - hi)) & (FULL << lo)) != 0u;
        }
        need[r] = p < m && gs[r] < k && ((cosine && !a.post) || (grouped[r] && any));
        if (need[r]) dbl[p] = adjudicate(a, q, key_id(key[r]));
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int p = lane + 32 * r;
        if (p >= m || gs[r] >= k) continue;
        const uint32_t c = key_id(key[r]);
        int at = p;
        if (need[r] && ge[r] > gs[r]) {
            const double dv = dbl[p];
            int rank = 0;
            for (int o = gs[r]; o <= ge[r]; ++o) {
                const double dq = dbl[o];
                const uint32_t io = key_id(keys_s[o]);
                rank += (dq < dv) || (dq == dv && io < c);
            }
            at = gs[r] + rank;
        }
        if (at < k) {
            const float dist = need[r] ? __double2float_rn(dbl[p]) : sqrtf(key_r(key[r]));
            a.out_idx[q * k + at] = a.row_lo ? c - a.row_lo[q] : c;
            a.out_dist[q * k + at] = dist;
        }
    }
    __syncwarp();
    return 0;
}

// rerank_sorted_kernel's rows by sorted_row_wide, four entries a lane: 0.27 ms
// for 50,021 rows at k = 50 (eight a lane takes twice as long for the same
// rows: twice the network, half the warps).
__global__ void __launch_bounds__(RS_WARPS * 32, 4) rerank_wide_kernel(RerankArgs a, int64_t span) {
    __shared__ unsigned long long keys[RS_WARPS][128];
    __shared__ double dbl[RS_WARPS][128];
    const int warp = threadIdx.x >> 5;
    const int64_t lo = (int64_t)blockIdx.x * span, hi = min(a.nq, lo + span);
    for (int64_t slot = lo + warp; slot < hi; slot += RS_WARPS) {
        if (a.qperm && a.qperm[slot] == 0xffffffffu) continue;  // padding of a batch layout
        const int r = sorted_row_wide<4>(a, slot, keys[warp], dbl[warp]);
        if (r && (threadIdx.x & 31) == 0) {
            if (r == 3) {
                a.wide_rows[atomicAdd(a.wide_count, 1u)] = (uint32_t)slot;
            } else {
                push_fallback(a, slot);
            }
        }
        __syncwarp();
    }
}

// Collected rows of more entries than the kernel before holds (a query's 64, or
// 128 above 32 neighbours), up to 256, eight a lane: warps take them from a
// queue (at k = 100 half of the rows are among them).
__global__ void __launch_bounds__(RS_WARPS * 32, 2) rerank_wide_queue_kernel(RerankArgs a) {
    __shared__ unsigned long long keys[RS_WARPS][256];
    __shared__ double dbl[RS_WARPS][256];
    const int warp = threadIdx.x >> 5;
    const uint32_t count = *a.wide_count;
    for (;;) {
        uint32_t i = 0;
        if ((threadIdx.x & 31) == 0) i = atomicAdd(a.wide_next, 1u);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= count) break;
        const int64_t slot = a.wide_rows[i];
        const int r = sorted_row_wide<8>(a, slot, keys[warp], dbl[warp]);
        if (r && (threadIdx.x & 31) == 0) {
            if (r == 3) {
                a.big_rows[atomicAdd(a.big_count, 1u)] = (uint32_t)slot;
            } else {
                push_fallback(a, slot);
            }
        }
        __syncwarp();
    }
}

// Each block walks its own contiguous range of list rows, its warps on
// consecutive rows: the rows an SM holds at once come from a few ranges, and
// neighbouring rows' candidate rows (mostly the same cells) stay in its L1.
__global__ void __launch_bounds__(RS_WARPS * 32, 6) rerank_sorted_kernel(RerankArgs a, int64_t span) {
    extern __shared__ unsigned long long rs_smem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    unsigned long long* keys = rs_smem + (size_t)warp * 2 * RS_KEYS;
    double* dbl = reinterpret_cast<double*>(keys + RS_KEYS);
    uint8_t* flags = reinterpret_cast<uint8_t*>(rs_smem + (size_t)RS_WARPS * 2 * RS_KEYS) + (size_t)warp * RS_KEYS;
    const int64_t lo = (int64_t)blockIdx.x * span, hi = min(a.nq, lo + span);
    for (int64_t slot = lo + warp; slot < hi; slot += RS_WARPS) {
        if (a.qperm && a.qperm[slot] == 0xffffffffu) continue;  // padding of a batch layout
        int r = sorted_row_regs(a, slot, keys, dbl);
        // A query's collected rows over 64 entries are often far over; a self
        // solve's are few, and cheapest here (1M x 50, k = 15: 90 us less than
        // through the queue).
        if (r == 3 && !(a.ids_only && !a.self)) r = sorted_row<RS_KEYS>(a, slot, keys, dbl, flags);
        if (r && lane == 0) {
            if (r == 3) {
                a.wide_rows[atomicAdd(a.wide_count, 1u)] = (uint32_t)slot;
            } else if (r == 1) {
                a.big_rows[atomicAdd(a.big_count, 1u)] = (uint32_t)slot;
            } else {
                push_fallback(a, slot);
            }
        }
        __syncwarp();
    }
}

// The rows with more survivors than the first pass holds: warps take them
// from a queue.
__global__ void __launch_bounds__(RS_BIG_WARPS * 32) rerank_sorted_big_kernel(RerankArgs a) {
    extern __shared__ unsigned long long rb_smem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    unsigned long long* keys = rb_smem + (size_t)warp * 2 * RS_BIG_KEYS;
    double* dbl = reinterpret_cast<double*>(keys + RS_BIG_KEYS);
    uint8_t* flags =
        reinterpret_cast<uint8_t*>(rb_smem + (size_t)RS_BIG_WARPS * 2 * RS_BIG_KEYS) + (size_t)warp * RS_BIG_KEYS;
    for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(a.big_next, 1u);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= *a.big_count) break;
        const int64_t slot = a.big_rows[i];
        const int r = sorted_row<RS_BIG_KEYS>(a, slot, keys, dbl, flags);
        if (r && lane == 0) push_fallback(a, slot);
        __syncwarp();
    }
}

// A cluster (or block) per row, over every reference row of its solve: used for rows whose
// candidate lists overflowed (many cells within the margin, e.g. duplicates, or
// data of few dimensions).  Bound by the latency of one SM's row reads: each
// block measures and counts its share of the columns, and the first one
// gathers the candidates in its shared memory, sorts and finishes them
// (300,000 rows of 10 dimensions, k = 20, some 350 rows here: 10.6 ms with a
// block a row, 1.6 ms so; a launch without rows returns at once).
template <int CLUSTER>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(FB_THREADS) rerank_fallback_kernel(RerankArgs a) {
    if (*a.fb_count == 0u) return;
    namespace cg = cooperative_groups;
    extern __shared__ unsigned long long fb_smem[];
    unsigned long long* keys = fb_smem;  // the first block's: the row's candidates
    double* dbl = reinterpret_cast<double*>(fb_smem + FB_CAP);
    uint8_t* flags = reinterpret_cast<uint8_t*>(fb_smem + 2 * FB_CAP);
    __shared__ int scratch;
    __shared__ uint32_t hist[256], all[256];
    __shared__ uint32_t row_s, sel_prefix;
    __shared__ int sel_rank, cnt_s, outside_s;
    __shared__ float limit_s, next_s;
    __shared__ int again_s;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = CLUSTER == 1 ? 0 : (int)cluster.block_rank(), tid = threadIdx.x;
    const bool first = rank == 0;
    auto of_block = [&](auto* p, int b) {
        if constexpr (CLUSTER == 1)
            return p;
        else
            return cluster.map_shared_rank(p, b);
    };
    auto of_first = [&](auto* p) { return of_block(p, 0); };
    auto sync = [&]() {
        if constexpr (CLUSTER == 1)
            __syncthreads();
        else
            cluster.sync();
    };
    BlockTeam team(&scratch);
    float* sc = a.fb_scratch + (int64_t)(blockIdx.x / CLUSTER) * a.nr;
    for (;;) {
        if (first && tid == 0) {
            const uint32_t i = atomicAdd(a.fb_next, 1u);
            row_s = i < *a.fb_count ? a.fb_rows[i] : 0xffffffffu;
            sel_prefix = 0;
            sel_rank = a.k;
        }
        sync();
        const uint32_t row = *of_first(&row_s);
        if (row == 0xffffffffu) break;
        const int64_t q = query_row(a, row);
        // The columns of the row's own solve, [lo, hi) of the input rows, and
        // the block's share of them.
        const int64_t lo = a.row_lo ? (int64_t)a.row_lo[q] : 0, hi = a.row_lo ? (int64_t)a.row_hi[q] : a.nr;
        const int64_t j0 = lo + (hi - lo) * rank / CLUSTER, j1 = lo + (hi - lo) * (rank + 1) / CLUSTER;
        for (int64_t j = j0 + tid; j < j1; j += FB_THREADS)
            sc[j] = a.self && j == q + a.self_offset ? __int_as_float(0x7f800000) : compute_r(a, q, (uint32_t)j);
        // k-th smallest of the row: four 8-bit radix passes.
        uint32_t mask = 0;
        for (int pass = 0; pass < 4; ++pass) {
            const int shift = 24 - 8 * pass;
            hist[tid] = 0;
            const uint32_t prefix = *of_first(&sel_prefix);
            __syncthreads();
            for (int64_t j = j0 + tid; j < j1; j += FB_THREADS) {
                const uint32_t key = float_key(sc[j]);
                if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
            }
            sync();
            if (first) {
                uint32_t sum = 0;
                for (int b = 0; b < CLUSTER; ++b) sum += *of_block(&hist[tid], b);
                all[tid] = sum;
                __syncthreads();
                if (tid == 0) {
                    int left = sel_rank;
                    uint32_t b = 0;
                    for (; b < 256; ++b) {
                        if ((int)all[b] >= left) break;
                        left -= (int)all[b];
                    }
                    sel_rank = left;
                    sel_prefix = prefix | (b << shift);
                }
            }
            mask |= 255u << shift;
            sync();
        }
        if (first && tid == 0) {
            const float vk = key_float(sel_prefix);
            limit_s = vk;
            if (a.mode != SCRUST_MODE_REFERENCE_SNAP)
                limit_s = vk + 4.0f * (a.gamma * 2.0f * vk + kTieAbs) + (a.metric == SCRUST_METRIC_COSINE ? 1e-6f : 0.0f);
        }
        int m = 0;
        for (int attempt = 0; attempt < 8; ++attempt) {
            if (first && tid == 0) cnt_s = outside_s = again_s = 0;
            sync();
            const float T = *of_first(&limit_s);
            int* cnt = of_first(&cnt_s);
            unsigned long long* out = of_first(keys);
            for (int64_t j = j0 + tid; j < j1; j += FB_THREADS) {
                const float r = sc[j];
                if (r <= T) {
                    const int pos = atomicAdd(cnt, 1);
                    if (pos < FB_CAP) out[pos] = ((unsigned long long)float_key(r) << 32) | (uint32_t)j;
                }
            }
            sync();
            m = *cnt;
            if (m > FB_CAP) break;
            if (first) {
                const int P = next_pow2(m);
                for (int p = m + tid; p < P; p += FB_THREADS) keys[p] = ~0ull;
                __syncthreads();
                team_bitonic_sort(team, keys, P);
                // If the tie group holding the last collected candidate reaches
                // position k-1, make sure nothing just outside T could join it.
                if (tid == 0 && a.mode != SCRUST_MODE_REFERENCE_SNAP && m > 0) {
                    const float rl = key_r(keys[m - 1]);
                    int gs = m - 1;
                    while (gs > 0 && tied(a, key_r(keys[gs - 1]), key_r(keys[gs]))) gs--;
                    again_s = gs < a.k;
                    next_s = rl + 2.0f * (a.gamma * 2.0f * rl + kTieAbs) +
                             (a.metric == SCRUST_METRIC_COSINE ? 1e-6f : 0.0f);
                }
            }
            sync();
            if (!*of_first(&again_s)) break;
            const float T2 = *of_first(&next_s);
            int outside = 0;
            for (int64_t j = j0 + tid; j < j1; j += FB_THREADS) outside += (sc[j] > T && sc[j] <= T2);
            outside = team.sum(outside);
            if (tid == 0 && outside) atomicAdd(of_first(&outside_s), outside);
            sync();
            if (*of_first(&outside_s) == 0) break;
            sync();  // all have read it before it is cleared
            if (first && tid == 0) limit_s = T2;
        }
        if (first) {
            if (m > FB_CAP || m < a.k) {
                if (tid == 0) atomicExch(a.err + (m > FB_CAP ? DERR_TIE_OVERFLOW : DERR_CANDIDATES), 1);
                write_open_row(team, a, q);
            } else {
                finalize_row(team, a, q, keys, m, dbl, flags);
            }
        }
        sync();  // the first block's shared memory is free for the next row
    }
    sync();  // it stays until all have read the last row
}

// Distances of cosine rows' neighbours, one a thread: the f32 value that the
// FP64 form (cosine_f64) rounds to, from f32 pairs wherever every value within
// the two forms' error bounds rounds alike; else by cosine_f64 itself.  Bound
// by the row gathers (30,011 rows of 50, k = 30: with f64 products, three
// 64-clock instructions a coordinate, the rerank took 409 us; now it takes
// 80 us and this pass 52).
__global__ void __launch_bounds__(256) cosine_distances_kernel(RerankArgs a, int64_t total, int stride) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const int64_t q = i / a.k;
    const uint32_t j = a.out_idx[i] + (a.row_lo ? a.row_lo[q] : 0u);
    if ((int64_t)j >= a.cosine.n) return;
    float h, l;
    cosine_pair(a.cosine, stride, q, (int64_t)j, &h, &l);
    a.out_dist[i] = rounds_surely(h, l, cosine_pair_error(stride, a.d))
                        ? h
                        : __double2float_rn(cosine_f64(a.qraw + q * a.d, a.rraw + (int64_t)j * a.d, a.d,
                                                       a.cosine.norm64[q], a.cosine.norm64[j]));
}

}  // namespace

cudaError_t launch_rerank(scrust_context* ctx, const KnnPlan& plan, const float* qx,
                          const float* rx, const float* qnorm2, const float* rnorm2,
                          const CosineRows& cosine, const float* qraw,
                          const float* rraw, const RowBounds& bounds, const Lists& lists,
                          const uint32_t* perm, const float* xs, const float* theta, uint32_t* out_idx,
                          float* out_dist, const uint32_t* row_lo, const uint32_t* row_hi, const float* xr_list,
                          int xs_stride, bool ids_only, const uint32_t* qperm) {
    cudaError_t e;
    uint32_t* fb_rows = (uint32_t*)ws_get(ctx, SLOT_FALLBACK_ROWS, sizeof(uint32_t) * (size_t)plan.nq, &e);
    if (!fb_rows) return e;
    const bool fb_blocks = plan.nr <= FB_BLOCK_COLUMNS;
    const int fb_at_once = fb_blocks ? (int)std::min<int64_t>(plan.nq, 3 * ctx->sm_count) : FB_ROWS;
    float* fb_scratch =
        (float*)ws_get(ctx, SLOT_FALLBACK_SCRATCH, sizeof(float) * (size_t)plan.nr * fb_at_once, &e);
    if (!fb_scratch) return e;
    RerankArgs a;
    a.qx = qx;
    a.rx = rx;
    a.qn2 = qnorm2;
    a.rn2 = rnorm2;
    a.cosine = cosine;
    a.raw_stride = padded_row_floats(plan.d);
    a.post = plan.metric == SCRUST_METRIC_COSINE && plan.mode != SCRUST_MODE_REFERENCE_SNAP && cosine.raw ? 1 : 0;
    a.qraw = qraw;
    a.rraw = rraw;
    a.bounds = bounds;
    a.lists = lists;
    a.perm = perm;
    a.qperm = qperm ? qperm : perm;
    a.xs = xs;
    a.xr_list = xr_list ? xr_list : xs;
    a.xs_stride = xs_stride > 0 ? xs_stride : plan.d;
    a.ids_only = ids_only ? 1 : 0;
    // 32-byte loads need rows padded to 8 floats on both sides: the lists'
    // query rows and the reference rows the candidate ids index.
    a.xs_v8 = xs && a.xs_stride % 8 == 0 && ((uintptr_t)xs & 31) == 0 && ((uintptr_t)a.xr_list & 31) == 0 &&
              (!xr_list || a.xs_stride == padded_row_floats(plan.d));
    a.theta = theta;
    a.row_lo = row_lo;
    a.row_hi = row_hi;
    a.nq = plan.nq;
    a.nr = plan.nr;
    a.d = plan.d;
    a.k = plan.k;
    a.mode = plan.mode;
    a.metric = plan.metric;
    a.self = plan.self ? 1 : 0;
    a.self_offset = plan.self_offset;
    a.gamma = dist2_f32_gamma(plan.d);
    a.out_idx = out_idx;
    a.out_dist = out_dist;
    a.fb_rows = fb_rows;
    a.fb_count = ctx->d_counter;
    a.fb_next = ctx->d_counter + 1;
    a.big_count = ctx->d_counter + 2;
    a.big_next = ctx->d_counter + 3;
    a.big_rows = nullptr;
    a.wide_rows = nullptr;
    a.wide_count = ctx->d_counter + 4;
    a.wide_next = ctx->d_counter + 5;
    if (xs && theta) {
        a.big_rows = (uint32_t*)ws_get(ctx, SLOT_RERANK_BIG, sizeof(uint32_t) * 2 * (size_t)plan.nq, &e);
        if (!a.big_rows) return e;
        a.wide_rows = a.big_rows + plan.nq;
    }
    a.fb_scratch = fb_scratch;
    a.err = ctx->d_err;
    e = cudaMemsetAsync(ctx->d_counter, 0, 6 * sizeof(uint32_t), ctx->stream);
    if (e != cudaSuccess) return e;
    if (xs && theta) {
        const size_t smem_s = (size_t)RS_WARPS * (2 * RS_KEYS * sizeof(unsigned long long) + RS_KEYS);
        // As many blocks as stay resident (6 an SM), each over a contiguous
        // range of rows.
        const int64_t groups = (plan.nq + RS_WARPS - 1) / RS_WARPS;
        const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>(groups, 6 * (int64_t)ctx->sm_count));
        const int64_t span = (groups + blocks - 1) / blocks * RS_WARPS;
        // Most rows need no shared memory (the register path): leave the rest
        // of the SM's unified memory to L1, which caches the candidate rows
        // that neighbouring rows share.
        static_assert(RS_WARPS * (2 * RS_KEYS * 8 + RS_KEYS) <= 24 * 1024, "rerank block smem");
        const unsigned grid = (unsigned)((plan.nq + span - 1) / span);
        if (ids_only && plan.k > 32) {  // most rows hold more than 64 entries
            rerank_wide_kernel<<<grid, RS_WARPS * 32, 0, ctx->stream>>>(a, span);
        } else {
            if ((e = set_smem_carveout(ctx, (const void*)rerank_sorted_kernel, 50)) != cudaSuccess) return e;
            rerank_sorted_kernel<<<grid, RS_WARPS * 32, smem_s, ctx->stream>>>(a, span);
        }
        if (ids_only && (plan.k > 32 || !plan.self)) {
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
            const int64_t most = (plan.nq + RS_WARPS - 1) / RS_WARPS;
            rerank_wide_queue_kernel<<<(unsigned)std::min<int64_t>(most, 2 * ctx->sm_count), RS_WARPS * 32, 0,
                                       ctx->stream>>>(a);
            ctx->launches += 1;
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        const size_t smem_b = (size_t)RS_BIG_WARPS * (2 * RS_BIG_KEYS * sizeof(unsigned long long) + RS_BIG_KEYS);
        if ((e = set_smem_limit(ctx, (const void*)rerank_sorted_big_kernel, (int)smem_b)) != cudaSuccess) return e;
        const int64_t most = (plan.nq + RS_BIG_WARPS - 1) / RS_BIG_WARPS;
        rerank_sorted_big_kernel<<<(unsigned)std::min<int64_t>(most, 2 * ctx->sm_count), RS_BIG_WARPS * 32, smem_b,
                                   ctx->stream>>>(a);
        ctx->launches += 2;
    } else {
        const size_t smem_w = (size_t)RR_WARPS * (2 * RC * sizeof(unsigned long long) + RC);
        e = set_smem_limit(ctx, (const void*)rerank_warp_kernel, (int)smem_w);
        if (e != cudaSuccess) return e;
        const unsigned blocks = (unsigned)((plan.nq + RR_WARPS - 1) / RR_WARPS);
        rerank_warp_kernel<<<blocks, RR_WARPS * 32, smem_w, ctx->stream>>>(a);
        ctx->launches += 1;
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const size_t smem_f = (size_t)FB_CAP * (sizeof(unsigned long long) + sizeof(double) + 1);
    const auto fallback = fb_blocks ? rerank_fallback_kernel<1> : rerank_fallback_kernel<FB_CLUSTER>;
    e = set_smem_limit(ctx, (const void*)fallback, (int)smem_f);
    if (e != cudaSuccess) return e;
    fallback<<<fb_at_once * (fb_blocks ? 1 : FB_CLUSTER), FB_THREADS, smem_f, ctx->stream>>>(a);
    ctx->launches += 1;
    if (a.post) {
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        const int64_t total = cosine.n * plan.k;
        cosine_distances_kernel<<<(unsigned)((total + 255) / 256), 256, 0, ctx->stream>>>(a, total, a.raw_stride);
        ctx->launches += 1;
    }
    return cudaGetLastError();
}

}  // namespace scrust
