// cluster.cu -- Leiden and Louvain community detection on the GPU, on the
// connectivities graph this library builds (crates/scrust-core/src/cluster.rs:88,125).
//
// The objective is the reference's RBConfiguration modularity
// Q = (1/2m) sum_ij (A_ij - gamma k_i k_j / 2m) [c_i = c_j] on the graph
// (A + A^T) / 2 (cluster.rs:214-290), and the structure is the reference's:
// local moving, then (Leiden) refinement of every community into
// well-connected subcommunities, aggregation, and repeat until nothing
// moves; Leiden restarts from its own result n_iterations times, stopping
// early when a pass changes nothing; labels are numbered by descending
// community size (cluster.rs:828-850).
//
// The reference moves one node at a time from a queue.  Here every pass is
// parallel and deterministic (the same graph and seed give the same labels):
//   - Local moving runs in rounds.  In each round half of the nodes (chosen
//     by a hash of node, seed and level, alternating) look at the
//     communities of their neighbours as the round began, and move to the
//     one of largest gain, ties to the smaller id, if that beats staying
//     (cluster.rs:425-455).  A node alone in its community joins another
//     lone node's community only when that id is smaller, so two lone
//     nodes never swap.  Rounds continue until two in a row move nothing.
//   - A node's edge weight per neighbouring community is summed in a
//     shared-memory table.  Where every sum of a level's weights is exact in
//     f64 (their lowest set bit against the largest row sum), the weights are
//     taken as integers and added in any order; else a warp per node adds
//     them 32 neighbours at a time, each community's partial in lane order,
//     so every sum is formed in one fixed order.  Both give the same bits.
//   - Community strengths are fixed-point (int64, scale 2^s with
//     2m * 2^s <= 2^61) and change by integer atomics, whose result does not
//     depend on their order.
//   - Refinement: within each community, lone well-connected nodes merge
//     into a neighbouring subcommunity of non-negative gain that is well
//     connected to the rest of the community (cluster.rs:507-641), drawn with
//     probability proportional to exp((gain - max) / 0.01) by a counter-based
//     hash; a node moving in a round never joins a subcommunity whose own
//     lone node may move in that round.  Cuts are recomputed each round.
//   - Aggregation: entries keyed by (community, community) with two stable
//     radix sorts and per-key sums in sorted order.
// Nodes whose neighbours span more than 2048 communities do not move (the
// table's limit); on kNN graphs no node comes near it.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace scrust {

namespace {

constexpr uint32_t kEmpty = 0xffffffffu;
constexpr int kSmallTable = 128;  // nodes with at most 64 neighbour entries, 4 warps a block
constexpr int kSmallWarps = 4;
constexpr int kBigTable = 2048;   // the rest, one warp a block
constexpr int kSmallDegree = 64;
constexpr int kMaxRounds = 200;
constexpr double kTheta = 0.01;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

inline uint64_t mix_host(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ bool active_in(uint32_t v, int round, uint64_t salt) {
    return ((mix64(salt ^ (uint64_t)v) + (uint64_t)round) & 1ull) == 0ull;
}

// ---- the symmetric graph ----------------------------------------------------

__global__ void cl_rows_kernel(const uint32_t* __restrict__ indptr, int64_t n, uint32_t* __restrict__ erow) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    for (uint32_t e = indptr[r], e1 = indptr[r + 1]; e < e1; ++e) erow[e] = (uint32_t)r;
}

__global__ void cl_check_kernel(const float* __restrict__ values, int64_t nnz, int* __restrict__ bad) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += (int64_t)gridDim.x * blockDim.x) {
        const float v = values[e];
        if (!(v >= 0.f) || isinf(v)) atomicExch(bad, 1);
    }
}

// Entry i < nnz is row(i) -> col(i), entry nnz + i the reverse; keyed by
// their first node.
__global__ void cl_sym_keys_kernel(const uint32_t* __restrict__ erow, const uint32_t* __restrict__ indices,
                                   int64_t nnz, uint32_t* __restrict__ keys, unsigned long long* __restrict__ vals) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * nnz) return;
    keys[i] = i < nnz ? erow[i] : indices[i - nnz];
    vals[i] = (unsigned long long)i;
}

// start[c] = number of sorted keys below c, c in [0, n].
__global__ void cl_starts_kernel(const uint32_t* __restrict__ keys, int64_t m, int64_t n, uint32_t* __restrict__ start) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p > m) return;
    const int64_t lo = p == 0 ? 0 : (int64_t)keys[p - 1] + 1;
    const int64_t hi = p == m ? n : (int64_t)keys[p];
    for (int64_t c = lo; c <= hi && c <= n; ++c) start[c] = (uint32_t)p;
}

__global__ void cl_sym_fill_kernel(const unsigned long long* __restrict__ order, int64_t m, int64_t nnz,
                                   const uint32_t* __restrict__ erow, const uint32_t* __restrict__ indices,
                                   const float* __restrict__ values, uint32_t* __restrict__ nb,
                                   double* __restrict__ w) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= m) return;
    const int64_t i = (int64_t)(order[p] & 0xffffffffull);
    const int64_t e = i < nnz ? i : i - nnz;
    nb[p] = i < nnz ? indices[e] : erow[e];
    w[p] = (double)values[e] / 2.0;
}

// Node strengths (row sums in row order).
__global__ void cl_strength_kernel(const uint32_t* __restrict__ ptr, const double* __restrict__ w, int64_t n,
                                   double* __restrict__ k) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    double s = 0.0;
    for (uint32_t p = ptr[v], p1 = ptr[v + 1]; p < p1; ++p) s += w[p];
    k[v] = s;
}

// Sum of `count` doubles: blocks of 256 by a tree each, then the blocks'
// totals in order (one block doing both took 300 us for 60,000).
__global__ void cl_sum_blocks_kernel(const double* __restrict__ x, int64_t count, double* __restrict__ totals) {
    __shared__ double part[256];
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    part[threadIdx.x] = i < count ? x[i] : 0.0;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = part[0];
}
__global__ void cl_sum_totals_kernel(const double* __restrict__ totals, int64_t blocks, double* __restrict__ out) {
    double total = 0.0;
#pragma unroll 8
    for (int64_t b = 0; b < blocks; ++b) total += totals[b];
    out[0] = total;
}

// The lowest set bit of any positive weight as an exponent (min into
// exps[0]) and the exponent above the largest strength (max into exps[1]).
__global__ void cl_exponents_kernel(const double* __restrict__ w, int64_t m, const double* __restrict__ k, int64_t n,
                                    int* __restrict__ exps) {
    int low = 2000, high = -2000;
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = t0; i < m; i += step) {
        const unsigned long long u = (unsigned long long)__double_as_longlong(w[i]) & 0x7fffffffffffffffull;
        if (!u) continue;
        const int e = (int)(u >> 52);
        const unsigned long long mant = (u & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull);
        low = min(low, (e ? e : 1) - 1075 + __ffsll((long long)mant) - 1);
    }
    for (int64_t i = t0; i < n; i += step) {
        const unsigned long long u = (unsigned long long)__double_as_longlong(k[i]) & 0x7fffffffffffffffull;
        if (u) high = max(high, (int)(u >> 52) - 1022);
    }
    low = __reduce_min_sync(0xffffffffu, low);
    high = __reduce_max_sync(0xffffffffu, high);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(exps, low);
        atomicMax(exps + 1, high);
    }
}

// Weights as integers: w[i] 2^shift, exact (and below 2^53); and those in f32.
__global__ void cl_integers_kernel(const double* __restrict__ w, int64_t m, double scale, long long* __restrict__ out,
                                   float* __restrict__ flt) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const double x = w[i] * scale;  // scale: a power of two
    out[i] = (long long)x;
    flt[i] = (float)x;
}

__global__ void cl_fix_kernel(const double* __restrict__ x, int64_t count, double scale, long long* __restrict__ fx) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) fx[i] = llrint(x[i] * scale);
}

// ---- community bookkeeping --------------------------------------------------

__global__ void cl_iota_kernel(int64_t n, uint32_t* __restrict__ out) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) out[v] = (uint32_t)v;
}

__global__ void cl_ones_kernel(int64_t n, int* __restrict__ out) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) out[v] = 1;
}

__global__ void cl_comm_init_kernel(const uint32_t* __restrict__ labels, const long long* __restrict__ kfix, int64_t n,
                                    long long* __restrict__ K, int* __restrict__ size) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    atomicAdd((unsigned long long*)(K + labels[v]), (unsigned long long)kfix[v]);
    atomicAdd(size + labels[v], 1);
}

// Sum over the lanes in `peers`, at its lowest lane, in lane order (wbuf: 32
// values of the warp's own), or for integers in any order, in log2 of the
// largest group's size steps: each lane adds the next lane left in its group,
// then every second lane leaves.  For all lanes of a warp.
__device__ __forceinline__ double peer_sum(uint32_t peers, bool lead, double x, double* wbuf) {
    wbuf[threadIdx.x & 31] = x;
    __syncwarp();
    double s = 0.0;
    if (lead)
        for (uint32_t b = peers; b; b &= b - 1) s += wbuf[__ffs(b) - 1];
    __syncwarp();
    return s;
}
template <class V>
__device__ __forceinline__ V peer_tree(uint32_t peers, V x) {
    const int lane = threadIdx.x & 31;
    uint32_t above = peers & (0xfffffffeu << lane);
    int rank = __popc(peers & ((1u << lane) - 1u));
    while (__any_sync(0xffffffffu, above != 0u)) {
        const int next = __ffs(above);
        const V t = __shfl_sync(0xffffffffu, x, next ? next - 1 : lane);
        if (next) x += t;
        above &= ~__ballot_sync(0xffffffffu, rank & 1);
        rank >>= 1;
    }
    return x;
}
__device__ __forceinline__ long long peer_sum(uint32_t peers, bool, long long x, long long*) {
    return peer_tree(peers, x);
}

// The per-node table of edge weight to each neighbouring community (or
// subcommunity), one warp per node: neighbours in chunks of 32; in a chunk
// each community's partial is summed by its lowest lane in lane order, then
// added to the table, so each entry is summed in one fixed order.  V: double,
// or long long for weights as integers.  With `group_of`, only neighbours in
// the node's own group count.  slots receives the table's occupied places;
// returns their count, or -1 when the table overflowed.  (The callers look at
// the occupied places alone: testing all T, 32 at a time, cost a node up to 64
// rounds of f64 divisions, 64 clocks an instruction.)
template <int T, class V>
__device__ int gather_table(const uint32_t* __restrict__ nb, const V* __restrict__ w, uint32_t p0, uint32_t p1,
                            uint32_t self, const uint32_t* __restrict__ label, const uint32_t* __restrict__ group_of,
                            uint32_t group, uint32_t* keys, V* vals, V* wbuf, uint16_t* slots, int* count,
                            int* overflow) {
    const int lane = threadIdx.x & 31;
    for (int t = lane; t < T; t += 32) keys[t] = kEmpty;
    if (lane == 0) {
        *overflow = 0;
        *count = 0;
    }
    __syncwarp();
    for (uint32_t base = p0; base < p1; base += 32) {
        const uint32_t p = base + lane;
        uint32_t c = kEmpty;
        V wt = 0;
        if (p < p1) {
            const uint32_t u = nb[p];
            if (u != self && (!group_of || group_of[u] == group)) {
                c = label[u];
                wt = w[p];
            }
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, c);
        const bool lead = c != kEmpty && (__ffs(peers) - 1) == lane;
        const V s = peer_sum(c == kEmpty ? 0u : peers, lead, wt, wbuf);
        if (lead) {
            uint32_t slot = (uint32_t)(mix64(c) & (T - 1));
            bool placed = false;
            for (int probe = 0; probe < T; ++probe) {
                const uint32_t prev = atomicCAS(keys + slot, kEmpty, c);
                if (prev == kEmpty || prev == c) {
                    if (prev == kEmpty) {
                        vals[slot] = 0;
                        slots[atomicAdd(count, 1)] = (uint16_t)slot;
                    }
                    vals[slot] += s;
                    placed = true;
                    break;
                }
                slot = (slot + 1) & (T - 1);
            }
            if (!placed) *overflow = 1;
        }
        __syncwarp();
    }
    return *overflow ? -1 : *count;
}

// An f64 as an unsigned integer of the same order (both zeros alike, no NaN).
__device__ __forceinline__ unsigned long long order_key(double x) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x + 0.0);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double key_order(unsigned long long k) {
    return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
}

// What a move decision reads besides the node's own table.
struct MoveArgs {
    const uint32_t* ptr;
    const uint32_t* nb;
    const long long* wint;   // weights as integers, w 2^wshift
    const float* wflt;       // the same in f32
    const double* w;
    const long long* kfix;
    const uint32_t* comm;
    const long long* K;
    const int* size;
    int64_t n_level;
    double unit;             // 2^-wshift
    float gain_unit;         // res inv_scale^2 / total / unit 2^31, or a NaN when that has no safe f32
    double inv_scale, res, total;
    uint32_t* moved;         // the round's moves: node and community
    uint32_t* to;
    unsigned int* moves;
};

// The node's end of a round (cluster.rs:420-455): the neighbouring community
// of largest gain when it beats staying; a node whose best gain, staying
// included, is negative goes alone to its reserved id n + v, when that
// community is empty.
__device__ __forceinline__ uint32_t destination(const MoveArgs& a, uint32_t v, uint32_t own, double best,
                                                uint32_t best_c, double stay) {
    uint32_t to = own;
    if (best_c != kEmpty && best > stay) to = best_c;
    const double top = to == own ? stay : best;
    const uint32_t fresh = (uint32_t)(a.n_level + v);
    if (top < 0.0 && own != fresh && a.size[fresh] == 0) to = fresh;
    return to;
}
__device__ __forceinline__ void record_move(const MoveArgs& a, uint32_t v, uint32_t own, uint32_t to) {
    if (to == own) return;
    const unsigned int i = atomicAdd(a.moves, 1u);
    a.moved[i] = v;
    a.to[i] = to;
}

// Gain of community strength k for a node of strength kv and weight e to it.
__device__ __forceinline__ double move_gain(const MoveArgs& a, double e, long long k, double kv) {
    return e - a.res * ((double)k * a.inv_scale) * kv / a.total;
}

// A non-negative integer in f32 by its halves, within 2 roundings of 2^-24 (the
// conversion instruction for 64 bits is an f64-rate one: 64 clocks a warp).
__device__ __forceinline__ float to_f32(long long x) {
    return fmaf((float)(uint32_t)((unsigned long long)x >> 32), 4294967296.0f, (float)(uint32_t)x);
}
// The same gain in f32, in units of the integer weights, as bounds: e the
// node's weight to the community, f its strength times gain_unit.  At most 9
// roundings of 2^-24 on either product or their difference (the weight summed
// in f32 in up to five steps, too), within 2^-20 of their sum; the constant
// covers what underflows (k f below 2^62 2^-126).  A NaN bounds nothing.
__device__ __forceinline__ void gain_bounds(float e, long long k, float f, float* low, float* high) {
    const float q = to_f32(k) * f;
    const float g = e - q, err = (e + fabsf(q)) * 9.5367431640625e-7f + 1e-18f;
    *low = g - err;
    *high = g + err;
}
__device__ __forceinline__ float gain_factor(const MoveArgs& a, long long kfix) {
    return (to_f32(kfix) * 4.656612873077393e-10f) * a.gain_unit;
}
// f32 as an unsigned integer of the same order (no NaN); 0 stands for none and
// reads back as a NaN, below which nothing is.
__device__ __forceinline__ uint32_t order_key(float x) {
    const uint32_t u = __float_as_uint(x);
    return (u >> 31) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_order(uint32_t k) { return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k); }

// Where a node of community `own` goes by the bounds of its gains, one warp:
// each lane holds up to E neighbouring communities c (kEmpty: none) with the
// node's weight s to them and their strength k; e_own is its weight to its own
// and k_own that one's strength without it.  One community above all others
// and above zero decides; kEmpty when the bounds leave it open.
template <int E>
__device__ __forceinline__ uint32_t bounded_move(uint32_t own, float f, const uint32_t (&c)[E], const float (&s)[E],
                                                 const long long (&k)[E], float e_own, long long k_own) {
    float own_low, own_high, high[E];
    gain_bounds(e_own, k_own, f, &own_low, &own_high);
    uint32_t key = own_low == own_low ? order_key(own_low) : 0u;
#pragma unroll
    for (int i = 0; i < E; ++i) {
        float low;
        gain_bounds(s[i], k[i], f, &low, &high[i]);
        if (c[i] != kEmpty && low == low) key = max(key, order_key(low));
    }
    key = __reduce_max_sync(0xffffffffu, key);
    const float least = key_order(key);
    const bool stays = !(own_high < least);
    int cands = stays ? 1 : 0;
    uint32_t to = own;
#pragma unroll
    for (int i = 0; i < E; ++i) {
        const uint32_t who = __ballot_sync(0xffffffffu, c[i] != kEmpty && !(high[i] < least));
        cands += __popc(who);
        if (who) to = __shfl_sync(0xffffffffu, c[i], __ffs(who) - 1);
    }
    return cands == 1 && least > 0.0f ? to : kEmpty;
}

// The same by the f64 gains (some 25 instructions of 64 clocks each), from the
// warp's table of `found` places: the largest wins, ties to the smaller id.
template <int T>
__device__ uint32_t exact_move(const MoveArgs& a, uint32_t v, uint32_t own, bool alone, long long kf, long long k_own,
                               const uint32_t* keys, const long long* vals, const uint16_t* slots, int found) {
    const int lane = threadIdx.x & 31;
    const double kv = (double)kf * a.inv_scale;
    double best = -INFINITY;
    long long e_own = 0;
    uint32_t best_c = kEmpty;
    for (int i0 = 0; i0 < found; i0 += 32) {
        uint32_t c = kEmpty;
        long long e = 0;
        if (i0 + lane < found) {
            c = keys[slots[i0 + lane]];
            e = vals[slots[i0 + lane]];
        }
        const uint32_t home = __ballot_sync(0xffffffffu, c == own);
        if (home) e_own = __shfl_sync(0xffffffffu, e, __ffs(home) - 1);
        // Lone nodes only join smaller lone ids.
        if (c == kEmpty || c == own || (alone && c > own && a.size[c] == 1)) continue;
        const double g = move_gain(a, (double)e * a.unit, a.K[c], kv);
        if (g > best || (g == best && c < best_c)) {
            best = g;
            best_c = c;
        }
    }
    __syncwarp();
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const uint32_t oc = __shfl_xor_sync(0xffffffffu, best_c, o);
        if (ob > best || (ob == best && oc < best_c)) {
            best = ob;
            best_c = oc;
        }
    }
    return destination(a, v, own, best, best_c, move_gain(a, (double)e_own * a.unit, k_own, kv));
}

// Local moving, one round, exact integer weights, nodes of at most
// kSmallDegree entries, kMoveNodes nodes a warp: a node's weights are summed
// per community in registers where its entries are one chunk of 32, else by
// the warp's table.  Bound by the latency of node -> neighbours -> labels ->
// strengths, so the warp's nodes are in flight together, and before by f64
// units, so sums and gains are bounded in f32 first.  A late round of 60,000
// nodes of 46 entries (23 merged): 112 us (a warp per node, f64 gains at 128
// places), 32 us (f64 gains, one thread per occupied place of a block), 22 us
// (bounds in f32, places of a block), 16 us (two nodes a warp), 11 us with
// nodes of more than one chunk a warp each and first, and the larger ones of
// up to kFusedTable / 2 entries in the same launch (5 us of their own before).
constexpr int kMoveWarps = 4;
constexpr int kMoveNodes = 2;
struct SmallTables {
    uint32_t keys[kMoveWarps][kSmallTable];
    long long vals[kMoveWarps][kSmallTable];
    uint16_t slots[kMoveWarps][kSmallTable];
    int count[kMoveWarps], over[kMoveWarps];
};
__device__ __forceinline__ void move_small_nodes(const MoveArgs& a, const uint32_t* __restrict__ nodes, int64_t count,
                                                 const uint32_t* __restrict__ mids, int64_t mid_count, int64_t block,
                                                 SmallTables& tab) {
    constexpr int T = kSmallTable, P = kMoveNodes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // The first warps take a node of more than one chunk each, being the longest.
    const int64_t g = block * kMoveWarps + warp;
    const bool mid = g < mid_count;
    const uint32_t* list = mid ? mids : nodes;
    const int64_t i0 = mid ? g : (g - mid_count) * P;
    if (!mid && i0 >= count) return;
    const int here = mid ? 1 : (int)min((int64_t)P, count - i0);
    // Lane j holds node j.
    uint32_t my_v = 0, my_own = 0, my_p0 = 0, my_deg = 0;
    long long my_kf = 0, my_kown = 0;
    bool my_alone = false;
    if (lane < here) {
        my_v = list[i0 + lane];
        my_own = a.comm[my_v];
        my_p0 = a.ptr[my_v];
        my_deg = a.ptr[my_v + 1] - my_p0;
        my_kf = a.kfix[my_v];
        my_kown = a.K[my_own] - my_kf;
        my_alone = a.size[my_own] == 1;
    }
    const float my_f = gain_factor(a, my_kf);
    uint32_t my_to = lane < here ? kEmpty : my_own;
    uint32_t c[P];
    float s[P], e_own[P];
    long long k[P];
#pragma unroll
    for (int j = 0; j < P; ++j) {
        const uint32_t v = __shfl_sync(0xffffffffu, my_v, j), p = __shfl_sync(0xffffffffu, my_p0, j) + lane;
        const uint32_t deg = __shfl_sync(0xffffffffu, my_deg, j);
        c[j] = kEmpty;
        s[j] = 0.0f;
        if (deg <= 32u && (uint32_t)lane < deg) {
            const uint32_t u = a.nb[p];
            s[j] = a.wflt[p];
            if (u != v) c[j] = u;
        }
    }
#pragma unroll
    for (int j = 0; j < P; ++j)
        if (c[j] != kEmpty) c[j] = a.comm[c[j]];
#pragma unroll
    for (int j = 0; j < P; ++j) {
        const uint32_t own = __shfl_sync(0xffffffffu, my_own, j);
        const bool alone = __shfl_sync(0xffffffffu, my_alone, j);
        const uint32_t peers = __match_any_sync(0xffffffffu, c[j]);
        s[j] = peer_tree(c[j] == kEmpty ? 0u : peers, s[j]);
        if ((__ffs(peers) - 1) != lane) c[j] = kEmpty;
        const uint32_t home = __ballot_sync(0xffffffffu, c[j] == own);
        e_own[j] = __shfl_sync(0xffffffffu, s[j], home ? __ffs(home) - 1 : 0);
        if (!home) e_own[j] = 0.0f;
        if (c[j] == own) c[j] = kEmpty;
        // Lone nodes only join smaller lone ids.
        if (alone && c[j] != kEmpty && c[j] > own && a.size[c[j]] == 1) c[j] = kEmpty;
        k[j] = c[j] != kEmpty ? a.K[c[j]] : 0ll;
    }
#pragma unroll
    for (int j = 0; j < P; ++j) {
        const uint32_t c1[1] = {c[j]};
        const float s1[1] = {s[j]};
        const long long k1[1] = {k[j]};
        const uint32_t to = bounded_move<1>(__shfl_sync(0xffffffffu, my_own, j), __shfl_sync(0xffffffffu, my_f, j), c1,
                                            s1, k1, e_own[j], __shfl_sync(0xffffffffu, my_kown, j));
        if (lane == j && j < here && my_deg <= 32u) my_to = to;
    }
    // Nodes of more than one chunk, and those that the bounds leave open.  (At
    // most kSmallDegree communities: the table never overflows.)
    for (uint32_t rest = __ballot_sync(0xffffffffu, my_to == kEmpty); rest; rest &= rest - 1) {
        const int j = __ffs(rest) - 1;
        const uint32_t v = __shfl_sync(0xffffffffu, my_v, j), own = __shfl_sync(0xffffffffu, my_own, j);
        const uint32_t p0 = __shfl_sync(0xffffffffu, my_p0, j), deg = __shfl_sync(0xffffffffu, my_deg, j);
        const bool alone = __shfl_sync(0xffffffffu, my_alone, j);
        const int found = gather_table<T>(a.nb, a.wint, p0, p0 + deg, v, a.comm, nullptr, 0u, tab.keys[warp],
                                          tab.vals[warp], (long long*)nullptr, tab.slots[warp], &tab.count[warp],
                                          &tab.over[warp]);
        const long long k_own = __shfl_sync(0xffffffffu, my_kown, j);
        uint32_t to = kEmpty;
        if (deg > 32u) {
            uint32_t c2[2];
            float s2[2], e2 = 0.0f;
            long long k2[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                c2[i] = kEmpty;
                s2[i] = 0.0f;
                k2[i] = 0;
                if (lane + 32 * i < found) {
                    const int t = tab.slots[warp][lane + 32 * i];
                    c2[i] = tab.keys[warp][t];
                    s2[i] = to_f32(tab.vals[warp][t]);
                }
                const uint32_t home = __ballot_sync(0xffffffffu, c2[i] == own);
                if (home) e2 = __shfl_sync(0xffffffffu, s2[i], __ffs(home) - 1);
                if (c2[i] == own || (alone && c2[i] != kEmpty && c2[i] > own && a.size[c2[i]] == 1)) c2[i] = kEmpty;
                if (c2[i] != kEmpty) k2[i] = a.K[c2[i]];
            }
            to = bounded_move<2>(own, __shfl_sync(0xffffffffu, my_f, j), c2, s2, k2, e2, k_own);
        }
        if (to == kEmpty)
            to = exact_move<T>(a, v, own, alone, __shfl_sync(0xffffffffu, my_kf, j), k_own, tab.keys[warp], tab.vals[warp],
                               tab.slots[warp], found);
        if (lane == j) my_to = to;
        __syncwarp();
    }
    const uint32_t movers = __ballot_sync(0xffffffffu, my_to != my_own);
    if (!movers) return;
    unsigned int at = 0;
    if (lane == 0) at = atomicAdd(a.moves, (unsigned int)__popc(movers));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(movers & ((1u << lane) - 1u));
    if (my_to != my_own) {
        a.moved[at] = my_v;
        a.to[at] = my_to;
    }
}

// The same for nodes of more entries, a block per node: the warps add their
// chunks to one table by atomics, of twice the node's entries up to kBigTable
// places (a warp per node, clearing and testing 2,048 places: 59 us a round).
template <int T>
struct BigTable {
    uint32_t keys[T];
    unsigned long long vals[T];
    float high[T];
    uint16_t slots[T], cand[T];
    int found, over, cands;
    uint32_t low, best_c;
    unsigned long long best, own_val;
    double stay;
};
template <int T>
__device__ __forceinline__ void move_big_node(const MoveArgs& a, uint32_t v, BigTable<T>& tab) {
    constexpr int N = 32 * kMoveWarps;
    uint32_t* keys = tab.keys;
    unsigned long long* vals = tab.vals;
    float* high = tab.high;
    uint16_t *slots = tab.slots, *cand = tab.cand;
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t own = a.comm[v];
    const uint32_t p0 = a.ptr[v], p1 = a.ptr[v + 1];
    const long long kf = a.kfix[v];
    const float factor = gain_factor(a, kf);
    uint32_t mask = T - 1;
    while (mask >= 255u && (mask >> 1) >= 2u * (p1 - p0)) mask >>= 1;
    for (uint32_t t = tid; t <= mask; t += N) {
        keys[t] = kEmpty;
        vals[t] = 0ull;
    }
    if (tid == 0) {
        tab.found = 0;
        tab.over = 0;
        tab.cands = 0;
        tab.low = 0u;
        tab.best = 0ull;
        tab.own_val = 0ull;
        tab.best_c = kEmpty;
        tab.stay = -INFINITY;
    }
    __syncthreads();
    for (uint32_t base = p0 + (uint32_t)(tid - lane); base < p1; base += N) {
        const uint32_t p = base + lane;
        uint32_t c = kEmpty;
        long long wt = 0;
        if (p < p1) {
            const uint32_t u = a.nb[p];
            if (u != v) {
                c = a.comm[u];
                wt = a.wint[p];
            }
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, c);
        const long long s = peer_sum(c == kEmpty ? 0u : peers, false, wt, nullptr);
        if (c != kEmpty && (__ffs(peers) - 1) == lane) {
            uint32_t slot = (uint32_t)mix64(c) & mask;
            bool placed = false;
            for (uint32_t probe = 0; probe <= mask; ++probe) {
                const uint32_t prev = atomicCAS(keys + slot, kEmpty, c);
                if (prev == kEmpty || prev == c) {
                    if (prev == kEmpty) slots[atomicAdd(&tab.found, 1)] = (uint16_t)slot;
                    atomicAdd(&vals[slot], (unsigned long long)s);
                    placed = true;
                    break;
                }
                slot = (slot + 1) & mask;
            }
            if (!placed) tab.over = 1;
        }
        __syncwarp();
    }
    __syncthreads();
    if (tab.over) return;
    const int found = tab.found;
    const bool alone = a.size[own] == 1;
    for (int i = tid; i < found; i += N) {
        const int s = slots[i];
        const uint32_t c = keys[s];
        high[s] = -INFINITY;
        if (c == own) {
            tab.own_val = vals[s];
            keys[s] = kEmpty;
        } else if (alone && c > own && a.size[c] == 1) {
            keys[s] = kEmpty;
        } else {
            float lo;
            gain_bounds(to_f32((long long)vals[s]), a.K[c], factor, &lo, &high[s]);
            if (lo == lo) atomicMax(&tab.low, order_key(lo));
        }
    }
    __syncthreads();
    // The node's own community, adjacent or not.
    const long long k_own = a.K[own] - kf;
    float own_low, own_high;
    gain_bounds(to_f32((long long)tab.own_val), k_own, factor, &own_low, &own_high);
    if (tid == 0 && own_low == own_low) atomicMax(&tab.low, order_key(own_low));
    __syncthreads();
    const float least = key_order(tab.low);
    for (int i = tid; i < found; i += N) {
        const int s = slots[i];
        if (keys[s] != kEmpty && !(high[s] < least)) cand[atomicAdd(&tab.cands, 1)] = (uint16_t)s;
    }
    __syncthreads();
    const int cands = tab.cands;
    const bool stays = !(own_high < least);
    if (cands + (stays ? 1 : 0) == 1 && least > 0.0f) {
        if (tid == 0 && !stays) record_move(a, v, own, keys[cand[0]]);
        return;
    }
    const double kv = (double)kf * a.inv_scale;
    for (int t = tid; t <= cands; t += N) {
        if (!t && !stays) continue;
        const int s = t ? cand[t - 1] : 0;
        const double g = t ? move_gain(a, (double)(long long)vals[s] * a.unit, a.K[keys[s]], kv)
                           : move_gain(a, (double)(long long)tab.own_val * a.unit, k_own, kv);
        if (!t) {
            tab.stay = g;
        } else if (g == g) {
            vals[s] = order_key(g);
            atomicMax(&tab.best, vals[s]);
        } else {
            keys[s] = kEmpty;
        }
    }
    __syncthreads();
    for (int t = tid; t < cands; t += N)
        if (keys[cand[t]] != kEmpty && vals[cand[t]] == tab.best) atomicMin(&tab.best_c, keys[cand[t]]);
    __syncthreads();
    if (tid == 0) record_move(a, v, own, destination(a, v, own, key_order(tab.best), tab.best_c, tab.stay));
}

constexpr int kFusedTable = 512;  // nodes of at most half as many entries share a launch with the small ones
__global__ void __launch_bounds__(32 * kMoveWarps) cl_move_kernel_all(MoveArgs a, const uint32_t* __restrict__ bigs,
                                                                      int64_t big_count,
                                                                      const uint32_t* __restrict__ nodes, int64_t count,
                                                                      const uint32_t* __restrict__ mids,
                                                                      int64_t mid_count) {
    __shared__ union {
        SmallTables small;
        BigTable<kFusedTable> big;
    } tab;
    if ((int64_t)blockIdx.x < big_count)
        move_big_node(a, bigs[blockIdx.x], tab.big);
    else
        move_small_nodes(a, nodes, count, mids, mid_count, (int64_t)blockIdx.x - big_count, tab.small);
}
__global__ void __launch_bounds__(32 * kMoveWarps) cl_move_big_kernel(MoveArgs a, const uint32_t* __restrict__ nodes) {
    __shared__ BigTable<kBigTable> tab;
    move_big_node(a, nodes[blockIdx.x], tab);
}

// Local moving, one round, one warp per node, f64 weights whose sums round:
// the fixed order of gather_table.
template <int T, int W>
__global__ void __launch_bounds__(32 * W) cl_move_kernel(MoveArgs a, const uint32_t* __restrict__ nodes, int64_t count) {
    __shared__ uint32_t keys[W][T];
    __shared__ double vals[W][T];
    __shared__ double wbuf[W][32];
    __shared__ uint16_t slots[W][T];
    __shared__ int found_s[W], overflow[W];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t idx = (int64_t)blockIdx.x * W + warp;
    if (idx >= count) return;
    const uint32_t v = nodes[idx];
    const uint32_t own = a.comm[v];
    const int found = gather_table<T>(a.nb, a.w, a.ptr[v], a.ptr[v + 1], v, a.comm, nullptr, 0u, keys[warp], vals[warp],
                                      wbuf[warp], slots[warp], &found_s[warp], &overflow[warp]);
    if (found < 0) return;
    const double kv = (double)a.kfix[v] * a.inv_scale;
    double e_own = 0.0;
    double best = -INFINITY;
    uint32_t best_c = kEmpty;
    const bool alone = a.size[own] == 1;
    for (int i = lane; i < found; i += 32) {
        const int t = slots[warp][i];
        const uint32_t c = keys[warp][t];
        if (c == own) {
            e_own = vals[warp][t];
            continue;
        }
        if (alone && a.size[c] == 1 && c > own) continue;  // lone nodes only join smaller lone ids
        const double g = move_gain(a, vals[warp][t], a.K[c], kv);
        if (g > best || (g == best && c < best_c)) {
            best = g;
            best_c = c;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const uint32_t oc = __shfl_xor_sync(0xffffffffu, best_c, o);
        e_own += __shfl_xor_sync(0xffffffffu, e_own, o);  // one lane holds it, the rest hold 0
        if (ob > best || (ob == best && oc < best_c)) {
            best = ob;
            best_c = oc;
        }
    }
    if (lane == 0)
        record_move(a, v, own, destination(a, v, own, best, best_c, move_gain(a, e_own, a.K[own] - a.kfix[v], kv)));
}

// The round's moves applied (each node at most once).
__global__ void cl_apply_kernel(const unsigned int* __restrict__ count, const uint32_t* __restrict__ moved,
                                const uint32_t* __restrict__ to, const long long* __restrict__ kfix,
                                uint32_t* __restrict__ comm, long long* __restrict__ K, int* __restrict__ size) {
    const unsigned int moves = *count;
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < moves; i += gridDim.x * blockDim.x) {
        const uint32_t v = moved[i], a = comm[v], b = to[i];
        atomicAdd((unsigned long long*)(K + a), (unsigned long long)(-kfix[v]));
        atomicAdd((unsigned long long*)(K + b), (unsigned long long)kfix[v]);
        atomicSub(size + a, 1);
        atomicAdd(size + b, 1);
        comm[v] = b;
    }
}

// ---- refinement -------------------------------------------------------------

// Per node: its weight to the rest of its community (fixed order), and
// whether it is well connected to it (cluster.rs:507-515).
__global__ void cl_to_subset_kernel(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ nb,
                                    const double* __restrict__ w, const double* __restrict__ k, int64_t n,
                                    const uint32_t* __restrict__ part, const long long* __restrict__ K,
                                    double inv_scale, double res, double total, double* __restrict__ to_subset,
                                    unsigned char* __restrict__ well) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const uint32_t c = part[v];
    double s = 0.0;
    for (uint32_t p = ptr[v], p1 = ptr[v + 1]; p < p1; ++p) {
        const uint32_t u = nb[p];
        if (u != (uint32_t)v && part[u] == c) s += w[p];
    }
    to_subset[v] = s;
    const double kc = (double)K[c] * inv_scale;
    well[v] = s >= res * k[v] * (kc - k[v]) / total;
}

// Per subcommunity, its cut to the rest of its community:
// sum over members of (to_subset - weight to the subcommunity), fixed point.
__global__ void cl_cut_kernel(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ nb,
                              const double* __restrict__ w, int64_t n, const uint32_t* __restrict__ sub,
                              const double* __restrict__ to_subset, double scale, long long* __restrict__ cut) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const uint32_t s = sub[v];
    double inside = 0.0;
    for (uint32_t p = ptr[v], p1 = ptr[v + 1]; p < p1; ++p) {
        const uint32_t u = nb[p];
        if (u != (uint32_t)v && sub[u] == s) inside += w[p];
    }
    atomicAdd((unsigned long long*)(cut + s), (unsigned long long)llrint((to_subset[v] - inside) * scale));
}
// The same with weights as integers, eight lanes a node (latency of a row's
// scattered reads: 23 us a round at 60,000 nodes with a thread a node).
__global__ void cl_cut_int_kernel(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ nb,
                                  const long long* __restrict__ w, double unit, int64_t n,
                                  const uint32_t* __restrict__ sub, const double* __restrict__ to_subset, double scale,
                                  long long* __restrict__ cut) {
    const int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int lane = threadIdx.x & 7;
    long long inside = 0;
    uint32_t s = 0;
    if (v < n) {
        s = sub[v];
        const uint32_t p1 = ptr[v + 1];
#pragma unroll 4
        for (uint32_t p = ptr[v] + lane; p < p1; p += 8) {
            const uint32_t u = nb[p];
            if (u != (uint32_t)v && sub[u] == s) inside += w[p];
        }
    }
    for (int o = 4; o > 0; o >>= 1) inside += __shfl_xor_sync(0xffffffffu, inside, o);
    if (v < n && lane == 0)
        atomicAdd((unsigned long long*)(cut + s),
                  (unsigned long long)llrint((to_subset[v] - (double)inside * unit) * scale));
}

// Refinement, one round, one warp per node (cluster.rs:560-641): a lone,
// well-connected node of this round's half merges into a subcommunity of
// its community with non-negative gain whose cut to the rest of the
// community passes the well-connectedness test, drawn with probability
// proportional to exp(gain / 0.01) by the Gumbel-max rule (the largest
// gain / 0.01 + G, G a Gumbel variate from a hash of seed, node,
// subcommunity and round).  A lone node that may itself move in this round
// is not a target.
template <int T, int W, class V>
__global__ void __launch_bounds__(32 * W) cl_refine_kernel(const uint32_t* __restrict__ ptr,
                                                           const uint32_t* __restrict__ nb, const V* __restrict__ w,
                                                           double unit, const long long* __restrict__ kfix,
                                                           const uint32_t* __restrict__ nodes, int64_t count,
                                                           const uint32_t* __restrict__ part,
                                                           const uint32_t* __restrict__ sub,
                                                           const long long* __restrict__ Ksub,
                                                           const int* __restrict__ subsize,
                                                           const long long* __restrict__ K,
                                                           const long long* __restrict__ cut,
                                                           const unsigned char* __restrict__ well, double inv_scale,
                                                           double res, double total, int round, uint64_t salt,
                                                           uint32_t* __restrict__ moved, uint32_t* __restrict__ to,
                                                           unsigned int* __restrict__ moves) {
    __shared__ uint32_t keys[W][T];
    __shared__ V vals[W][T];
    __shared__ V wbuf[W][32];
    __shared__ uint16_t slots[W][T];
    __shared__ int found_s[W], overflow[W];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t idx = (int64_t)blockIdx.x * W + warp;
    if (idx >= count) return;
    const uint32_t v = nodes[idx];
    if (sub[v] != v || subsize[v] != 1 || !well[v]) return;
    const uint32_t c = part[v];
    const int found = gather_table<T>(nb, w, ptr[v], ptr[v + 1], v, sub, part, c, keys[warp], vals[warp], wbuf[warp],
                                      slots[warp], &found_s[warp], &overflow[warp]);
    if (found < 0) return;
    const double kv = (double)kfix[v] * inv_scale;
    const double kc = (double)K[c] * inv_scale;
    double best = -INFINITY;
    uint32_t best_s = kEmpty;
    for (int i = lane; i < found; i += 32) {
        const int t = slots[warp][i];
        const uint32_t s = keys[warp][t];
        const double ks = (double)Ksub[s] * inv_scale;
        const double gain = (double)vals[warp][t] * unit - res * ks * kv / total;
        const bool frozen = !(subsize[s] == 1 && well[s] && active_in(s, round, salt));
        if (!(gain >= 0.0 && frozen && (double)cut[s] * inv_scale >= res * ks * (kc - ks) / total)) continue;
        const uint64_t h = mix64(salt ^ mix64(((uint64_t)v << 32 | s) ^ mix64((uint64_t)round + 0x51ed27ull)));
        const double u = ((double)(h >> 11) + 0.5) * 1.1102230246251565e-16;
        const double key = gain / kTheta - log(-log(u));
        if (key > best || (key == best && s < best_s)) {
            best = key;
            best_s = s;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const uint32_t os = __shfl_xor_sync(0xffffffffu, best_s, o);
        if (ob > best || (ob == best && os < best_s)) {
            best = ob;
            best_s = os;
        }
    }
    if (lane == 0 && best_s != kEmpty) {
        const unsigned int i = atomicAdd(moves, 1u);
        moved[i] = v;
        to[i] = best_s;
    }
}

// ---- aggregation ------------------------------------------------------------

__global__ void cl_flag_kernel(const uint32_t* __restrict__ labels, int64_t n, uint32_t* __restrict__ flag) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) flag[labels[v]] = 1u;
}

__global__ void cl_relabel_kernel(const uint32_t* __restrict__ in, int64_t n, const uint32_t* __restrict__ id,
                                  uint32_t* __restrict__ out) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) out[v] = id[in[v]];
}

__global__ void cl_agg_keys_kernel(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ nb, int64_t n,
                                   const uint32_t* __restrict__ lab, uint32_t* __restrict__ krow,
                                   uint32_t* __restrict__ kcol) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    for (uint32_t p = ptr[v], p1 = ptr[v + 1]; p < p1; ++p) {
        krow[p] = lab[v];
        kcol[p] = lab[nb[p]];
    }
}

__global__ void cl_seq_kernel(int64_t m, unsigned long long* __restrict__ vals) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < m) vals[p] = (unsigned long long)p;
}

// kA[p] = kcol[order[p]] for the second (stable) sort, by row.
__global__ void cl_gather_u32_kernel(const uint32_t* __restrict__ src, const unsigned long long* __restrict__ order,
                                     int64_t m, uint32_t* __restrict__ dst) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < m) dst[p] = src[order[p] & 0xffffffffull];
}

// Segment heads of the sorted (row, col) keys.
__global__ void cl_heads_kernel(const unsigned long long* __restrict__ order, const uint32_t* __restrict__ krow,
                                const uint32_t* __restrict__ kcol, int64_t m, uint32_t* __restrict__ head) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= m) return;
    const int64_t e = (int64_t)(order[p] & 0xffffffffull);
    if (p == 0) {
        head[p] = 1u;
        return;
    }
    const int64_t f = (int64_t)(order[p - 1] & 0xffffffffull);
    head[p] = (krow[e] != krow[f] || kcol[e] != kcol[f]) ? 1u : 0u;
}

// One thread per coarse entry: its weight summed over its run in sorted order.
__global__ void cl_segsum_kernel(const unsigned long long* __restrict__ order, const uint32_t* __restrict__ head,
                                 const uint32_t* __restrict__ pos, const uint32_t* __restrict__ krow,
                                 const uint32_t* __restrict__ kcol, const double* __restrict__ w, int64_t m,
                                 uint32_t* __restrict__ out_row, uint32_t* __restrict__ out_nb,
                                 double* __restrict__ out_w) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= m || !head[p]) return;
    const int64_t e0 = (int64_t)(order[p] & 0xffffffffull);
    double s = 0.0;
    for (int64_t q = p; q < m && (q == p || !head[q]); ++q) s += w[order[q] & 0xffffffffull];
    const uint32_t id = pos[p];
    out_row[id] = krow[e0];
    out_nb[id] = kcol[e0];
    out_w[id] = s;
}

// ---- scoring and output -----------------------------------------------------

__global__ void cl_score_kernel(const uint32_t* __restrict__ ptr, const uint32_t* __restrict__ nb,
                                const double* __restrict__ w, const long long* __restrict__ kfix, int64_t n,
                                const uint32_t* __restrict__ lab, double scale, long long* __restrict__ internal,
                                long long* __restrict__ strength) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const uint32_t c = lab[v];
    double s = 0.0;
    for (uint32_t p = ptr[v], p1 = ptr[v + 1]; p < p1; ++p)
        if (lab[nb[p]] == c) s += w[p];
    atomicAdd((unsigned long long*)(internal + c), (unsigned long long)llrint(s * scale));
    atomicAdd((unsigned long long*)(strength + c), (unsigned long long)kfix[v]);
}

__global__ void cl_q_kernel(const long long* __restrict__ internal, const long long* __restrict__ strength, int64_t nc,
                            double inv_scale, double res, double total, double* __restrict__ out) {
    __shared__ double part[256];
    double q = 0.0;
    for (int64_t base = 0; base < nc; base += 256) {
        const int64_t c = base + threadIdx.x;
        double t = 0.0;
        if (c < nc) {
            const double in = (double)internal[c] * inv_scale, st = (double)strength[c] * inv_scale;
            t = in / total - res * (st / total) * (st / total);
        }
        part[threadIdx.x] = t;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) q += part[0];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = q;
}

__global__ void cl_differ_kernel(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, int64_t n,
                                 unsigned int* __restrict__ differ) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n && a[v] != b[v]) *differ = 1u;
}

__global__ void cl_size_keys_kernel(const int* __restrict__ size, int64_t nc, uint32_t* __restrict__ keys,
                                    unsigned long long* __restrict__ vals) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc) return;
    keys[c] = 0xffffffffu - (uint32_t)size[c];
    vals[c] = (unsigned long long)c;
}

__global__ void cl_rank_kernel(const unsigned long long* __restrict__ order, int64_t nc, uint32_t* __restrict__ rank) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nc) rank[order[i] & 0xffffffffull] = (uint32_t)i;
}

// The nodes by degree and by the half of the rounds they are active in
// (active_in): nodes of at most `chunk` entries of even and odd rounds from
// the two ends of `small`, those of up to kSmallDegree from the ends of `mid`,
// the rest from the ends of `big`.
__global__ void cl_node_lists_kernel(const uint32_t* __restrict__ ptr, int64_t n, uint64_t salt, uint32_t chunk,
                                     uint32_t* __restrict__ small, uint32_t* __restrict__ mid,
                                     uint32_t* __restrict__ big, unsigned int* __restrict__ counts) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const uint32_t degree = v < n ? ptr[v + 1] - ptr[v] : 0u;
    const int kind = v >= n ? 6
                            : (degree <= chunk ? 0 : degree <= (uint32_t)kSmallDegree ? 2 : 4) +
                                  (active_in((uint32_t)v, 0, salt) ? 0 : 1);
    const uint32_t peers = __match_any_sync(0xffffffffu, kind);
    unsigned int at = 0;
    if (kind < 6 && (__ffs(peers) - 1) == lane) at = atomicAdd(counts + kind, (unsigned int)__popc(peers));
    at = __shfl_sync(0xffffffffu, at, __ffs(peers) - 1) + __popc(peers & ((1u << lane) - 1u));
    if (kind >= 6) return;
    if (kind >= 4) atomicMax(counts + 8, degree);
    uint32_t* list = kind < 2 ? small : kind < 4 ? mid : big;
    list[(kind & 1) ? n - 1 - (int64_t)at : (int64_t)at] = (uint32_t)v;
}

__global__ void cl_scatter_kernel(const uint32_t* __restrict__ collapse, const uint32_t* __restrict__ partition,
                                  int64_t n, uint32_t* __restrict__ out) {
    // Every member of a subcommunity lies in the same community, so the
    // writes to one slot agree.
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) out[collapse[v]] = partition[v];
}

struct Level {
    int64_t n = 0, m = 0;
    uint32_t* ptr = nullptr;
    uint32_t* nb = nullptr;
    double* w = nullptr;
    double* k = nullptr;
    long long* kfix = nullptr;
    // The graph that moves read: where every sum over a row is exact, entries
    // of one neighbour merged and weights as integers (w 2^shift); else the
    // graph itself and wint null.
    const uint32_t* mptr = nullptr;
    const uint32_t* mnb = nullptr;
    long long* wint = nullptr;
    float* wflt = nullptr;
    int shift = 0;
};

unsigned grid_for(int64_t n) { return (unsigned)std::max<int64_t>(1, (n + 255) / 256); }

}  // namespace

// The whole algorithm on device buffers, under the context lock.  Buffers
// are cut from blocks of 32 MB or more, of which the context keeps at most
// kKeepBytes from call to call (some hundred cudaMalloc and cudaFree pairs
// took milliseconds).
class Clusterer {
    static constexpr size_t kKeepBytes = (size_t)1 << 30;

public:
    Clusterer(scrust_context* ctx, scrust_status* st) : ctx_(ctx), st_(st), s_(ctx->stream) {}
    ~Clusterer() {
        cudaStreamSynchronize(s_);
        auto& blocks = ctx_->cluster_blocks;
        size_t total = 0;
        for (auto& b : blocks) total += b.second;
        if (blocks.size() < 2 && total <= kKeepBytes) return;
        // One block of the same size serves the next call without gaps.
        for (auto& b : blocks) cudaFree(b.first);
        blocks.clear();
        void* p = nullptr;
        if (total <= kKeepBytes && cudaMalloc(&p, total) == cudaSuccess) blocks.emplace_back(p, total);
        cudaGetLastError();
    }

    template <class T>
    T* alloc(size_t count) {
        const size_t bytes = (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~(size_t)255;
        auto& blocks = ctx_->cluster_blocks;
        while (block_ < blocks.size() && used_ + bytes > blocks[block_].second) {
            ++block_;
            used_ = 0;
        }
        if (block_ == blocks.size()) {
            const size_t want = std::max(bytes, (size_t)32 << 20);
            void* p = nullptr;
            if (cudaMalloc(&p, want) != cudaSuccess) {
                cudaGetLastError();
                ok_ = false;
                return nullptr;
            }
            blocks.emplace_back(p, want);
            used_ = 0;
        }
        void* p = (char*)blocks[block_].first + used_;
        used_ += bytes;
        return (T*)p;
    }

    int32_t build(const uint32_t* indptr, const uint32_t* indices, const float* values, int64_t n, int64_t nnz);
    int32_t run(bool leiden, double res, int n_iterations, uint64_t seed, uint32_t* out_labels, double* out_q,
                uint64_t* out_nc);
    int32_t score_only(const uint32_t* labels, int64_t nc, double res, double* out_q);

private:
    int32_t oom() { return fail(st_, SCRUST_OOM, "clustering: device allocation failed"); }
    template <class V>
    bool download(V* host, const V* dev, size_t count) {
        if (cudaMemcpyAsync(host, dev, sizeof(V) * count, cudaMemcpyDeviceToHost, s_) != cudaSuccess ||
            cudaStreamSynchronize(s_) != cudaSuccess) {
            cudaGetLastError();
            ok_ = false;
        }
        return ok_;
    }
    cudaError_t sort_pairs(uint32_t* kA, unsigned long long* vA, uint32_t* kB, unsigned long long* vB, int64_t m,
                           int bits, uint32_t** kout, unsigned long long** vout);
    int64_t compact(const uint32_t* labels, int64_t n, int64_t width, uint32_t* out);
    int32_t node_lists(const Level& L, uint64_t salt, uint32_t chunk);
    int32_t integer_weights(Level* L, bool merged);
    int32_t local_moving(const Level& L, uint32_t* comm, long long* K, int* size, double res, bool* moved_any);
    int32_t refine(const Level& L, const uint32_t* part, const long long* K, double res, uint64_t salt,
                   uint32_t* sub);
    int32_t aggregate(const Level& L, const uint32_t* lab, int64_t nc, Level* out);
    int32_t optimise(const uint32_t* initial, double res, bool leiden, uint64_t salt, uint32_t* out,
                     int64_t* out_nc);
    double score(const Level& L, const uint32_t* lab, int64_t nc, double res);

    scrust_context* ctx_;
    scrust_status* st_;
    cudaStream_t s_;
    bool ok_ = true;
    size_t block_ = 0, used_ = 0;  // the next free byte of the context's blocks
    Level g0_;
    double total_ = 0.0, scale_ = 1.0, inv_scale_ = 1.0;
    unsigned int* counter_ = nullptr;  // 6 list counts, 2 exponents, the largest degree of a big node, the moves of each round, labels changed
    // Node lists of the current level (cl_node_lists_kernel) and their counts.
    uint32_t* small_ = nullptr;
    uint32_t* mid_ = nullptr;
    uint32_t* big_ = nullptr;
    unsigned int counts_[9] = {};
    // The list of small (0), mid (1) or big (2) nodes active in `round`, and its length.
    const uint32_t* active(const Level& L, int kind, int round, int64_t* count) const {
        const int odd = round & 1;
        *count = counts_[2 * kind + odd];
        const uint32_t* list = kind == 2 ? big_ : kind ? mid_ : small_;
        return odd ? list + (L.n - *count) : list;
    }
};

// Rounds enqueued between two looks at their move counts.  Two rounds without
// a move leave every later one without any (nothing they read has changed), so
// the rounds past the last do nothing; a look after every round left the GPU
// idle for as long as a round took.
constexpr int kRoundBatch = 8;
constexpr int kCounterMoves = 9;
static_assert(kMaxRounds % kRoundBatch == 0, "whole batches");

cudaError_t Clusterer::sort_pairs(uint32_t* kA, unsigned long long* vA, uint32_t* kB, unsigned long long* vB,
                                  int64_t m, int bits, uint32_t** kout, unsigned long long** vout) {
    const int nb = radix_blocks(std::max<int64_t>(m, 1));
    const size_t scan_elems = scan_scratch_elems((int64_t)256 * nb);
    uint32_t* hist = alloc<uint32_t>((size_t)256 * nb + 16);
    uint32_t* scan = alloc<uint32_t>(scan_elems);
    if (!ok_) return cudaErrorMemoryAllocation;
    return radix_sort_pairs(ctx_, kA, vA, kB, vB, m, bits, hist, scan, scan_elems, kout, vout);
}

// Ids in use (below `width`) renumbered 0.. in ascending order (cluster.rs:807-826).
int64_t Clusterer::compact(const uint32_t* labels, int64_t n, int64_t width, uint32_t* out) {
    uint32_t* flag = alloc<uint32_t>((size_t)width + 1);
    uint32_t* scan = alloc<uint32_t>(scan_scratch_elems(width + 1));
    if (!ok_) return -1;
    cudaMemsetAsync(flag, 0, sizeof(uint32_t) * ((size_t)width + 1), s_);
    cl_flag_kernel<<<grid_for(n), 256, 0, s_>>>(labels, n, flag);
    if (device_exclusive_scan(ctx_, flag, flag, width + 1, scan, scan_scratch_elems(width + 1)) != cudaSuccess) {
        ok_ = false;
        return -1;
    }
    cl_relabel_kernel<<<grid_for(n), 256, 0, s_>>>(labels, n, flag, out);
    ctx_->launches += 2;
    uint32_t nc = 0;
    if (!download(&nc, flag + width, 1)) return -1;
    return (int64_t)nc;
}

int32_t Clusterer::build(const uint32_t* indptr, const uint32_t* indices, const float* values, int64_t n,
                         int64_t nnz) {
    if (nnz == 0)
        return fail(st_, SCRUST_INVALID_PARAMETER, "the graph needs at least one edge of positive weight");
    int* bad = alloc<int>(1);
    uint32_t* erow = alloc<uint32_t>(nnz);
    const int64_t m = 2 * nnz;
    uint32_t* kA = alloc<uint32_t>(m);
    uint32_t* kB = alloc<uint32_t>(m);
    unsigned long long* vA = alloc<unsigned long long>(m);
    unsigned long long* vB = alloc<unsigned long long>(m);
    g0_.n = n;
    g0_.m = m;
    g0_.ptr = alloc<uint32_t>(n + 1);
    g0_.nb = alloc<uint32_t>(m);
    g0_.w = alloc<double>(m);
    g0_.k = alloc<double>(n);
    g0_.kfix = alloc<long long>(n);
    double* tot = alloc<double>(1);
    double* tots = alloc<double>((size_t)(n / 256 + 1));
    counter_ = alloc<unsigned int>(kCounterMoves + kMaxRounds + 1);
    if (!ok_) return oom();
    cudaMemsetAsync(bad, 0, sizeof(int), s_);
    cl_check_kernel<<<(unsigned)std::min<int64_t>(1024, nnz / 256 + 1), 256, 0, s_>>>(values, nnz, bad);
    int hbad = 0;
    if (!download(&hbad, bad, 1)) return fail(st_, SCRUST_KERNEL, "clustering: graph check");
    if (hbad) return fail(st_, SCRUST_INVALID_PARAMETER, "graph weights must be finite and non-negative");
    cl_rows_kernel<<<grid_for(n), 256, 0, s_>>>(indptr, n, erow);
    cl_sym_keys_kernel<<<grid_for(m), 256, 0, s_>>>(erow, indices, nnz, kA, vA);
    int bits = 1;
    while (((int64_t)1 << bits) <= n) bits++;
    uint32_t* keys = nullptr;
    unsigned long long* order = nullptr;
    cudaError_t e;
    if ((e = sort_pairs(kA, vA, kB, vB, m, bits, &keys, &order)) != cudaSuccess)
        return cuda_fail(st_, e, "clustering: graph");
    cl_starts_kernel<<<grid_for(m + 1), 256, 0, s_>>>(keys, m, n, g0_.ptr);
    cl_sym_fill_kernel<<<grid_for(m), 256, 0, s_>>>(order, m, nnz, erow, indices, values, g0_.nb, g0_.w);
    cl_strength_kernel<<<grid_for(n), 256, 0, s_>>>(g0_.ptr, g0_.w, n, g0_.k);
    cl_sum_blocks_kernel<<<grid_for(n), 256, 0, s_>>>(g0_.k, n, tots);
    cl_sum_totals_kernel<<<1, 1, 0, s_>>>(tots, (int64_t)grid_for(n), tot);
    ctx_->launches += 8;
    if (!download(&total_, tot, 1)) return fail(st_, SCRUST_KERNEL, "clustering: graph");
    if (!(total_ > 0.0))
        return fail(st_, SCRUST_INVALID_PARAMETER, "the graph needs at least one edge of positive weight");
    // Fixed point for strengths: the total at 2^61 leaves room for the
    // rounding of up to 2^31 terms below 2^63.
    const int sexp = (int)std::floor(61.0 - std::log2(total_));
    scale_ = std::ldexp(1.0, sexp);
    inv_scale_ = std::ldexp(1.0, -sexp);
    cl_fix_kernel<<<grid_for(n), 256, 0, s_>>>(g0_.k, n, scale_, g0_.kfix);
    ctx_->launches += 1;
    return ok(st_);
}

int32_t Clusterer::node_lists(const Level& L, uint64_t salt, uint32_t chunk) {
    small_ = alloc<uint32_t>(L.n);
    mid_ = alloc<uint32_t>(L.n);
    big_ = alloc<uint32_t>(L.n);
    if (!ok_) return oom();
    cudaMemsetAsync(counter_, 0, 9 * sizeof(unsigned int), s_);
    cl_node_lists_kernel<<<grid_for(L.n), 256, 0, s_>>>(L.mptr, L.n, salt, chunk, small_, mid_, big_, counter_);
    ctx_->launches += 1;
    if (!download(counts_, counter_, 9)) return fail(st_, SCRUST_KERNEL, "clustering: node lists");
    return ok(st_);
}

// The level's weights as integers, where every sum over a row is exact: a
// multiple of their lowest set bit, below 2^53 of it.  Entries of one neighbour
// are merged then (the symmetric graph holds most edges twice; half the
// entries make most rows one chunk of 32), unless they already are.
int32_t Clusterer::integer_weights(Level* L, bool merged) {
    L->mptr = L->ptr;
    L->mnb = L->nb;
    L->wint = nullptr;
    int exps[2] = {2000, -2000};
    cudaMemcpyAsync(counter_ + 6, exps, sizeof(exps), cudaMemcpyHostToDevice, s_);
    cl_exponents_kernel<<<(unsigned)std::min<int64_t>(4 * ctx_->sm_count, grid_for(L->m)), 256, 0, s_>>>(
        L->w, L->m, L->k, L->n, (int*)(counter_ + 6));
    ctx_->launches += 1;
    if (!download(exps, (const int*)(counter_ + 6), 2)) return fail(st_, SCRUST_KERNEL, "clustering: weights");
    // (|shift| <= 1000 keeps 2^-shift an f64; a strength rounds up to at most
    // the next power of two.)
    if (exps[0] >= 2000 || exps[1] + 1 - exps[0] > 53 || exps[0] < -1000 || exps[0] > 900) return ok(st_);
    Level g = *L;
    if (!merged) {
        uint32_t* each = alloc<uint32_t>(L->n);
        if (!ok_) return oom();
        cl_iota_kernel<<<grid_for(L->n), 256, 0, s_>>>(L->n, each);
        ctx_->launches += 1;
        const int32_t rc = aggregate(*L, each, L->n, &g);
        if (rc) return rc;
    }
    L->shift = -exps[0];
    L->wint = alloc<long long>(g.m);
    L->wflt = alloc<float>(g.m);
    if (!ok_) return oom();
    L->mptr = g.ptr;
    L->mnb = g.nb;
    cl_integers_kernel<<<grid_for(g.m), 256, 0, s_>>>(g.w, g.m, std::ldexp(1.0, L->shift), L->wint, L->wflt);
    ctx_->launches += 1;
    return ok(st_);
}

int32_t Clusterer::local_moving(const Level& L, uint32_t* comm, long long* K, int* size, double res, bool* moved_any) {
    MoveArgs a;
    a.ptr = L.mptr;
    a.nb = L.mnb;
    a.wint = L.wint;
    a.wflt = L.wflt;
    a.w = L.w;
    a.kfix = L.kfix;
    a.comm = comm;
    a.K = K;
    a.size = size;
    a.n_level = L.n;
    a.unit = std::ldexp(1.0, -L.shift);
    a.inv_scale = inv_scale_;
    a.res = res;
    a.total = total_;
    const double gu = res * inv_scale_ * inv_scale_ / total_ / a.unit * 2147483648.0;
    a.gain_unit = gu > 1e-28 && gu < 1e28 ? (float)gu : NAN;
    a.moved = alloc<uint32_t>(L.n);
    a.to = alloc<uint32_t>(L.n);
    if (!ok_) return oom();
    uint32_t* seen = alloc<uint32_t>(L.n);
    if (!ok_) return oom();
    *moved_any = false;
    const unsigned apply_blocks = std::min<unsigned>(grid_for(L.n), 2u * (unsigned)ctx_->sm_count);
    cudaMemsetAsync(counter_ + kCounterMoves, 0, sizeof(unsigned int) * (kMaxRounds + 1), s_);
    int quiet = 0, end = kMaxRounds, seen_batch = -1;
    for (int r0 = 0; r0 < end && quiet < 2; r0 += kRoundBatch) {
        for (int round = r0; round < r0 + kRoundBatch; ++round) {
            a.moves = counter_ + kCounterMoves + round;
            int64_t ns = 0, nm = 0, nb = 0;
            const uint32_t* small = active(L, 0, round, &ns);
            const uint32_t* mid = active(L, 1, round, &nm);
            const uint32_t* big = active(L, 2, round, &nb);
            if (L.wint && ns + nm + nb) {
                const bool fused = counts_[8] <= kFusedTable / 2;
                const int64_t warps = nm + (ns + kMoveNodes - 1) / kMoveNodes, with = fused ? nb : 0;
                const int64_t blocks = with + (warps + kMoveWarps - 1) / kMoveWarps;
                if (blocks)
                    cl_move_kernel_all<<<(unsigned)blocks, 32 * kMoveWarps, 0, s_>>>(a, big, with, small, ns, mid, nm);
                nb -= with;
            }
            if (ns && !L.wint)
                cl_move_kernel<kSmallTable, kSmallWarps>
                    <<<(unsigned)((ns + kSmallWarps - 1) / kSmallWarps), 32 * kSmallWarps, 0, s_>>>(a, small, ns);
            if (nb && L.wint)
                cl_move_big_kernel<<<(unsigned)nb, 32 * kMoveWarps, 0, s_>>>(a, big);
            else if (nb)
                cl_move_kernel<kBigTable, 1><<<(unsigned)nb, 32, 0, s_>>>(a, big, nb);
            cl_apply_kernel<<<apply_blocks, 256, 0, s_>>>(a.moves, a.moved, a.to, L.kfix, comm, K, size);
            ctx_->launches += 3;
        }
        // Rounds read the labels and the round's parity alone (strengths and
        // sizes follow from the labels, in integers), so labels equal to those
        // some whole batches ago repeat from there: only what is left over of
        // the remaining batches after whole repeats has to run.  (On a graph of
        // 60,000 cells ten nodes that swap for ever kept the first level going
        // to kMaxRounds, the last 60 rounds of it such a repeat.)
        // `seen` is taken at batches 1, 2, 4, 8 .. (Brent's rule).
        const int batch = r0 / kRoundBatch;
        unsigned int got[kRoundBatch], differ = 1;
        unsigned int* d_differ = counter_ + kCounterMoves + kMaxRounds;
        const bool look = end == kMaxRounds && seen_batch >= 0;
        if (look) {
            cudaMemsetAsync(d_differ, 0, sizeof(unsigned int), s_);
            cl_differ_kernel<<<grid_for(L.n), 256, 0, s_>>>(seen, comm, L.n, d_differ);
            cudaMemcpyAsync(&differ, d_differ, sizeof(differ), cudaMemcpyDeviceToHost, s_);
            ctx_->launches += 1;
        }
        if (!download(got, counter_ + kCounterMoves + r0, kRoundBatch))
            return fail(st_, SCRUST_KERNEL, "clustering: local moving");
        for (int i = 0; i < kRoundBatch && quiet < 2; ++i) {
            if (got[i]) *moved_any = true;
            quiet = got[i] ? 0 : quiet + 1;
        }
        if (look && !differ) {
            const int left = (kMaxRounds - r0) / kRoundBatch - 1;
            end = r0 + kRoundBatch * (1 + left % (batch - seen_batch));
        } else if (batch && !(batch & (batch - 1))) {
            cudaMemcpyAsync(seen, comm, sizeof(uint32_t) * L.n, cudaMemcpyDeviceToDevice, s_);
            seen_batch = batch;
        }
    }
    return ok(st_);
}

int32_t Clusterer::refine(const Level& L, const uint32_t* part, const long long* K, double res, uint64_t salt,
                          uint32_t* sub) {
    const int64_t n = L.n;
    double* to_subset = alloc<double>(n);
    unsigned char* well = alloc<unsigned char>(n);
    long long* Ksub = alloc<long long>(n);
    int* subsize = alloc<int>(n);
    long long* cut = alloc<long long>(n);
    uint32_t* moved = alloc<uint32_t>(n);
    uint32_t* to = alloc<uint32_t>(n);
    if (!ok_) return oom();
    int32_t rc = node_lists(L, salt, kSmallDegree);
    if (rc) return rc;
    const unsigned nb = grid_for(n);
    cl_to_subset_kernel<<<nb, 256, 0, s_>>>(L.ptr, L.nb, L.w, L.k, n, part, K, inv_scale_, res, total_, to_subset,
                                           well);
    cl_iota_kernel<<<nb, 256, 0, s_>>>(n, sub);
    cl_ones_kernel<<<nb, 256, 0, s_>>>(n, subsize);
    cudaMemcpyAsync(Ksub, L.kfix, sizeof(long long) * n, cudaMemcpyDeviceToDevice, s_);
    ctx_->launches += 3;
    const unsigned apply_blocks = std::min<unsigned>(nb, 2u * (unsigned)ctx_->sm_count);
    const double unit = std::ldexp(1.0, -L.shift);
    cudaMemsetAsync(counter_ + kCounterMoves, 0, sizeof(unsigned int) * kMaxRounds, s_);
    int quiet = 0;
    for (int r0 = 0; r0 < kMaxRounds && quiet < 2; r0 += kRoundBatch) {
        for (int round = r0; round < r0 + kRoundBatch; ++round) {
            unsigned int* moves = counter_ + kCounterMoves + round;
            cudaMemsetAsync(cut, 0, sizeof(long long) * n, s_);
            if (L.wint)
                cl_cut_int_kernel<<<grid_for(8 * n), 256, 0, s_>>>(L.mptr, L.mnb, L.wint, unit, n, sub, to_subset,
                                                                  scale_, cut);
            else
                cl_cut_kernel<<<nb, 256, 0, s_>>>(L.ptr, L.nb, L.w, n, sub, to_subset, scale_, cut);
            for (int kind = 0; kind < 2; ++kind) {
                int64_t count = 0;
                const uint32_t* nodes = active(L, 2 * kind, round, &count);
                if (!count) continue;
                const unsigned grid = kind ? (unsigned)count : (unsigned)((count + kSmallWarps - 1) / kSmallWarps);
                auto go = [&](auto kernel, auto* w, double u) {
                    kernel<<<grid, kind ? 32 : 32 * kSmallWarps, 0, s_>>>(
                        L.mptr, L.mnb, w, u, L.kfix, nodes, count, part, sub, Ksub, subsize, K, cut, well, inv_scale_, res,
                        total_, round, salt, moved, to, moves);
                };
                if (L.wint) {
                    if (kind)
                        go(cl_refine_kernel<kBigTable, 1, long long>, (const long long*)L.wint, unit);
                    else
                        go(cl_refine_kernel<kSmallTable, kSmallWarps, long long>, (const long long*)L.wint, unit);
                } else if (kind) {
                    go(cl_refine_kernel<kBigTable, 1, double>, (const double*)L.w, 1.0);
                } else {
                    go(cl_refine_kernel<kSmallTable, kSmallWarps, double>, (const double*)L.w, 1.0);
                }
            }
            cl_apply_kernel<<<apply_blocks, 256, 0, s_>>>(moves, moved, to, L.kfix, sub, Ksub, subsize);
            ctx_->launches += 4;
        }
        unsigned int moves[kRoundBatch];
        if (!download(moves, counter_ + kCounterMoves + r0, kRoundBatch))
            return fail(st_, SCRUST_KERNEL, "clustering: refinement");
        for (int i = 0; i < kRoundBatch && quiet < 2; ++i) quiet = moves[i] ? 0 : quiet + 1;
    }
    return ok(st_);
}

// The graph of communities (cluster.rs:681-730): entries keyed by
// (community of row, community of neighbour) in ascending order, weights
// summed per key in the order of the finer graph's entries.
int32_t Clusterer::aggregate(const Level& L, const uint32_t* lab, int64_t nc, Level* out) {
    const int64_t m = L.m;
    uint32_t* krow = alloc<uint32_t>(m);
    uint32_t* kcol = alloc<uint32_t>(m);
    uint32_t* kA = alloc<uint32_t>(m);
    uint32_t* kB = alloc<uint32_t>(m);
    unsigned long long* vA = alloc<unsigned long long>(m);
    unsigned long long* vB = alloc<unsigned long long>(m);
    uint32_t* head = alloc<uint32_t>(m + 1);
    uint32_t* pos = alloc<uint32_t>(m + 1);
    uint32_t* scan = alloc<uint32_t>(scan_scratch_elems(m + 1));
    uint32_t* orow = alloc<uint32_t>(m);
    if (!ok_) return oom();
    const unsigned eb = grid_for(m);
    cl_agg_keys_kernel<<<grid_for(L.n), 256, 0, s_>>>(L.ptr, L.nb, L.n, lab, krow, kcol);
    cl_seq_kernel<<<eb, 256, 0, s_>>>(m, vA);
    cudaMemcpyAsync(kA, kcol, sizeof(uint32_t) * m, cudaMemcpyDeviceToDevice, s_);
    ctx_->launches += 2;
    int bits = 1;
    while (((int64_t)1 << bits) <= nc) bits++;
    uint32_t* keys = nullptr;
    unsigned long long* order = nullptr;
    cudaError_t e;
    if ((e = sort_pairs(kA, vA, kB, vB, m, bits, &keys, &order)) != cudaSuccess)
        return cuda_fail(st_, e, "clustering: aggregate");
    // Then a stable pass by row.
    unsigned long long* o2 = order == vA ? vB : vA;
    uint32_t* k2 = keys == kA ? kB : kA;
    cl_gather_u32_kernel<<<eb, 256, 0, s_>>>(krow, order, m, k2);
    ctx_->launches += 1;
    if ((e = sort_pairs(k2, order, keys, o2, m, bits, &keys, &order)) != cudaSuccess)
        return cuda_fail(st_, e, "clustering: aggregate");
    cl_heads_kernel<<<eb, 256, 0, s_>>>(order, krow, kcol, m, head);
    cudaMemsetAsync(head + m, 0, sizeof(uint32_t), s_);
    if ((e = device_exclusive_scan(ctx_, head, pos, m + 1, scan, scan_scratch_elems(m + 1))) != cudaSuccess)
        return cuda_fail(st_, e, "clustering: aggregate");
    ctx_->launches += 1;
    uint32_t mo = 0;
    if (!download(&mo, pos + m, 1)) return fail(st_, SCRUST_KERNEL, "clustering: aggregate");
    out->n = nc;
    out->m = mo;
    out->ptr = alloc<uint32_t>(nc + 1);
    out->nb = alloc<uint32_t>(mo);
    out->w = alloc<double>(mo);
    out->k = alloc<double>(nc);
    out->kfix = alloc<long long>(nc);
    if (!ok_) return oom();
    cl_segsum_kernel<<<eb, 256, 0, s_>>>(order, head, pos, krow, kcol, L.w, m, orow, out->nb, out->w);
    cl_starts_kernel<<<grid_for(mo + 1), 256, 0, s_>>>(orow, mo, nc, out->ptr);
    cl_strength_kernel<<<grid_for(nc), 256, 0, s_>>>(out->ptr, out->w, nc, out->k);
    cl_fix_kernel<<<grid_for(nc), 256, 0, s_>>>(out->k, nc, scale_, out->kfix);
    ctx_->launches += 4;
    return ok(st_);
}

double Clusterer::score(const Level& L, const uint32_t* lab, int64_t nc, double res) {
    long long* internal = alloc<long long>(nc);
    long long* strength = alloc<long long>(nc);
    double* q = alloc<double>(1);
    if (!ok_) return NAN;
    cudaMemsetAsync(internal, 0, sizeof(long long) * nc, s_);
    cudaMemsetAsync(strength, 0, sizeof(long long) * nc, s_);
    cl_score_kernel<<<grid_for(L.n), 256, 0, s_>>>(L.ptr, L.nb, L.w, L.kfix, L.n, lab, scale_, internal, strength);
    cl_q_kernel<<<1, 256, 0, s_>>>(internal, strength, nc, inv_scale_, res, total_, q);
    ctx_->launches += 2;
    double h = NAN;
    download(&h, q, 1);
    return h;
}

// One pass (cluster.rs:732-784) from `initial` labels of the nodes; writes
// the nodes' labels, compacted, and their count.
int32_t Clusterer::optimise(const uint32_t* initial, double res, bool leiden, uint64_t salt, uint32_t* out,
                            int64_t* out_nc) {
    Level level = g0_;
    const int64_t n0 = g0_.n;
    uint32_t* fold = alloc<uint32_t>(n0);
    uint32_t* labels = alloc<uint32_t>(n0);
    if (!ok_) return oom();
    cl_iota_kernel<<<grid_for(n0), 256, 0, s_>>>(n0, fold);
    cudaMemcpyAsync(labels, initial, sizeof(uint32_t) * n0, cudaMemcpyDeviceToDevice, s_);
    ctx_->launches += 1;
    for (int depth = 0; depth < 64; ++depth) {
        const int64_t n = level.n;
        // Community ids below 2n: the labels in use, and n + v reserved for v.
        long long* K = alloc<long long>(2 * n);
        int* size = alloc<int>(2 * n);
        uint32_t* partition = alloc<uint32_t>(n);
        if (!ok_) return oom();
        cudaMemsetAsync(K, 0, sizeof(long long) * 2 * n, s_);
        cudaMemsetAsync(size, 0, sizeof(int) * 2 * n, s_);
        cl_comm_init_kernel<<<grid_for(n), 256, 0, s_>>>(labels, level.kfix, n, K, size);
        ctx_->launches += 1;
        const uint64_t level_salt = mix_host(salt ^ ((uint64_t)depth * 0xD1B54A32D192ED03ull));
        int32_t rc = SCRUST_OK;
        if (depth && (rc = integer_weights(&level, true))) return rc;
        if ((rc = node_lists(level, level_salt, level.wint ? 32 : kSmallDegree))) return rc;
        bool moved = false;
        if ((rc = local_moving(level, labels, K, size, res, &moved))) return rc;
        const int64_t nc = compact(labels, n, 2 * n, partition);
        if (nc < 0) return fail(st_, SCRUST_KERNEL, "clustering: compact");
        if (!moved || nc == n) {
            cl_relabel_kernel<<<grid_for(n0), 256, 0, s_>>>(fold, n0, partition, out);
            ctx_->launches += 1;
            *out_nc = nc;
            return ok(st_);
        }
        uint32_t* collapse = alloc<uint32_t>(n);
        if (!ok_) return oom();
        int64_t ncol = nc;
        if (leiden) {
            long long* Kp = alloc<long long>(nc);
            int* sp = alloc<int>(nc);
            uint32_t* sub = alloc<uint32_t>(n);
            if (!ok_) return oom();
            cudaMemsetAsync(Kp, 0, sizeof(long long) * nc, s_);
            cudaMemsetAsync(sp, 0, sizeof(int) * nc, s_);
            cl_comm_init_kernel<<<grid_for(n), 256, 0, s_>>>(partition, level.kfix, n, Kp, sp);
            ctx_->launches += 1;
            if ((rc = refine(level, partition, Kp, res, mix_host(level_salt ^ 0x5bd1e995ull), sub))) return rc;
            ncol = compact(sub, n, n, collapse);
            if (ncol < 0) return fail(st_, SCRUST_KERNEL, "clustering: compact");
        } else {
            cudaMemcpyAsync(collapse, partition, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s_);
        }
        Level next;
        if ((rc = aggregate(level, collapse, ncol, &next))) return rc;
        // The coarser level starts with each node in its members' community.
        uint32_t* next_labels = alloc<uint32_t>(ncol);
        uint32_t* fold2 = alloc<uint32_t>(n0);
        if (!ok_) return oom();
        cl_scatter_kernel<<<grid_for(n), 256, 0, s_>>>(collapse, partition, n, next_labels);
        cl_relabel_kernel<<<grid_for(n0), 256, 0, s_>>>(fold, n0, collapse, fold2);
        ctx_->launches += 2;
        fold = fold2;
        level = next;
        labels = next_labels;
    }
    return fail(st_, SCRUST_KERNEL, "clustering: no convergence after 64 levels");
}

int32_t Clusterer::run(bool leiden, double res, int n_iterations, uint64_t seed, uint32_t* out_labels,
                       double* out_q, uint64_t* out_nc) {
    const int64_t n = g0_.n;
    uint32_t* cur = alloc<uint32_t>(n);
    uint32_t* found = alloc<uint32_t>(n);
    unsigned int* differ = alloc<unsigned int>(1);
    if (!ok_) return oom();
    cl_iota_kernel<<<grid_for(n), 256, 0, s_>>>(n, cur);
    ctx_->launches += 1;
    int32_t rc = integer_weights(&g0_, false);
    if (rc) return rc;
    int64_t nc = n;
    const int passes = leiden ? n_iterations : 1;
    for (int pass = 0; pass < passes; ++pass) {
        int64_t fnc = 0;
        rc = optimise(cur, res, leiden, mix_host(seed ^ ((uint64_t)pass << 40)), found, &fnc);
        if (rc) return rc;
        if (leiden) {
            // A pass that returns its own input has converged (cluster.rs:104-118).
            cudaMemsetAsync(differ, 0, sizeof(unsigned int), s_);
            cl_differ_kernel<<<grid_for(n), 256, 0, s_>>>(found, cur, n, differ);
            ctx_->launches += 1;
            unsigned int hd = 0;
            if (!download(&hd, differ, 1)) return fail(st_, SCRUST_KERNEL, "clustering: compare");
            if (!hd) break;
        }
        cudaMemcpyAsync(cur, found, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s_);
        nc = fnc;
    }
    // Labels by descending community size, ties to the smaller id (cluster.rs:828-850).
    int* size = alloc<int>(nc);
    long long* strength = alloc<long long>(nc);
    uint32_t* kA = alloc<uint32_t>(nc);
    uint32_t* kB = alloc<uint32_t>(nc);
    unsigned long long* vA = alloc<unsigned long long>(nc);
    unsigned long long* vB = alloc<unsigned long long>(nc);
    uint32_t* rank = alloc<uint32_t>(nc);
    if (!ok_) return oom();
    cudaMemsetAsync(size, 0, sizeof(int) * nc, s_);
    cudaMemsetAsync(strength, 0, sizeof(long long) * nc, s_);
    cl_comm_init_kernel<<<grid_for(n), 256, 0, s_>>>(cur, g0_.kfix, n, strength, size);
    cl_size_keys_kernel<<<grid_for(nc), 256, 0, s_>>>(size, nc, kA, vA);
    ctx_->launches += 2;
    uint32_t* keys = nullptr;
    unsigned long long* order = nullptr;
    cudaError_t e;
    if ((e = sort_pairs(kA, vA, kB, vB, nc, 32, &keys, &order)) != cudaSuccess)
        return cuda_fail(st_, e, "clustering: label order");
    cl_rank_kernel<<<grid_for(nc), 256, 0, s_>>>(order, nc, rank);
    cl_relabel_kernel<<<grid_for(n), 256, 0, s_>>>(cur, n, rank, out_labels);
    ctx_->launches += 2;
    *out_q = score(g0_, out_labels, nc, res);
    *out_nc = (uint64_t)nc;
    if (!ok_) return fail(st_, SCRUST_KERNEL, "clustering: score");
    return ok(st_);
}

int32_t Clusterer::score_only(const uint32_t* labels, int64_t nc, double res, double* out_q) {
    *out_q = score(g0_, labels, nc, res);
    if (!ok_) return fail(st_, SCRUST_KERNEL, "clustering: score");
    return ok(st_);
}

}  // namespace scrust

using namespace scrust;

namespace {

int32_t check_graph(const uint32_t* indptr, const uint32_t* indices, uint64_t n, uint64_t n_cols, scrust_status* st) {
    if (n == 0 || n_cols != n)
        return fail(st, SCRUST_SHAPE, "expected a square graph with at least one node, got %llu x %llu",
                    (unsigned long long)n, (unsigned long long)n_cols);
    if (!indptr) return fail(st, SCRUST_SHAPE, "expected non-null pointers");
    const uint64_t nnz = indptr[n];
    if (nnz && !indices) return fail(st, SCRUST_SHAPE, "expected non-null pointers");
    if (indptr[0] != 0) return fail(st, SCRUST_SHAPE, "expected indptr to start at 0");
    for (uint64_t r = 0; r < n; ++r)
        if (indptr[r + 1] < indptr[r]) return fail(st, SCRUST_SHAPE, "expected a non-decreasing indptr");
    for (uint64_t i = 0; i < nnz; ++i)
        if (indices[i] >= n_cols) return fail(st, SCRUST_SHAPE, "expected column indices below %llu", (unsigned long long)n_cols);
    if (n >= 0x7fffff00ull || 2 * nnz >= 0xffffff00ull) return fail(st, SCRUST_SHAPE, "expected fewer than 2^31 entries");
    return SCRUST_OK;
}

int32_t check_resolution(double res, scrust_status* st) {
    if (!std::isfinite(res) || res <= 0.0)
        return fail(st, SCRUST_INVALID_PARAMETER, "resolution must be finite and greater than zero, got %g", res);
    return SCRUST_OK;
}

// Host CSR in; runs `body` with the device copy.
template <class Fn>
int32_t with_device_graph(scrust_context* ctx, const uint32_t* indptr, const uint32_t* indices, const float* values,
                          uint64_t n, scrust_status* st, Fn body) {
    const uint64_t nnz = indptr[n];
    cudaError_t e;
    const size_t o_ix = ((sizeof(uint32_t) * (n + 1)) + 255) & ~(size_t)255;
    const size_t o_vl = o_ix + (((sizeof(uint32_t) * std::max<uint64_t>(nnz, 1)) + 255) & ~(size_t)255);
    const size_t bytes = o_vl + sizeof(float) * std::max<uint64_t>(nnz, 1);
    char* buf = (char*)ws_get(ctx, SLOT_HOST_IN, bytes, &e);
    if (!buf) return cuda_fail(st, e, "workspace");
    if ((e = cudaMemcpyAsync(buf, indptr, sizeof(uint32_t) * (n + 1), cudaMemcpyHostToDevice, ctx->stream)) !=
            cudaSuccess ||
        (nnz && (e = cudaMemcpyAsync(buf + o_ix, indices, sizeof(uint32_t) * nnz, cudaMemcpyHostToDevice, ctx->stream)) !=
                    cudaSuccess) ||
        (nnz && (e = cudaMemcpyAsync(buf + o_vl, values, sizeof(float) * nnz, cudaMemcpyHostToDevice, ctx->stream)) !=
                    cudaSuccess))
        return cuda_fail(st, e, "upload");
    return body((const uint32_t*)buf, (const uint32_t*)(buf + o_ix), (const float*)(buf + o_vl), (int64_t)nnz);
}

int32_t cluster_host(scrust_context* ctx, const uint32_t* indptr, const uint32_t* indices, const float* values,
                     uint64_t n, uint64_t n_cols, bool leiden, double res, uint32_t n_iterations, uint64_t seed,
                     uint32_t* out_labels, double* out_q, uint64_t* out_nc, scrust_status* st) {
    int32_t rc = check_resolution(res, st);
    if (rc) return rc;
    if (leiden && n_iterations == 0) return fail(st, SCRUST_INVALID_PARAMETER, "n_iterations must be at least 1, got 0");
    if ((rc = check_graph(indptr, indices, n, n_cols, st))) return rc;
    if (!out_labels || !out_q || !out_nc || (indptr[n] && !values)) return fail(st, SCRUST_SHAPE, "expected non-null pointers");
    if (!ctx) return fail(st, SCRUST_NO_GPU, "no CUDA context (no usable GPU)");
    std::lock_guard<std::mutex> lock(ctx->mu);
    DeviceGuard device_guard(ctx->device);
    return with_device_graph(ctx, indptr, indices, values, n, st,
                             [&](const uint32_t* dip, const uint32_t* dix, const float* dvl, int64_t nnz) -> int32_t {
                                 Clusterer c(ctx, st);
                                 int32_t r = c.build(dip, dix, dvl, (int64_t)n, nnz);
                                 if (r) return r;
                                 uint32_t* dl = c.alloc<uint32_t>(n);
                                 if (!dl) return fail(st, SCRUST_OOM, "clustering: device allocation failed");
                                 if ((r = c.run(leiden, res, (int)n_iterations, seed, dl, out_q, out_nc))) return r;
                                 cudaError_t e = cudaMemcpyAsync(out_labels, dl, sizeof(uint32_t) * n,
                                                                 cudaMemcpyDeviceToHost, ctx->stream);
                                 if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
                                 if (e != cudaSuccess) return cuda_fail(st, e, "download");
                                 return collect_device_errors(ctx, st);
                             });
}

}  // namespace

extern "C" {

int32_t scrust_cuda_leiden(scrust_context* ctx, const uint32_t* indptr, const uint32_t* indices, const float* values,
                           uint64_t n_rows, uint64_t n_cols, double resolution, uint32_t n_iterations, uint64_t seed,
                           uint32_t* out_labels, double* out_modularity, uint64_t* out_n_communities,
                           scrust_status* st) {
    return cluster_host(ctx, indptr, indices, values, n_rows, n_cols, true, resolution, n_iterations, seed, out_labels,
                        out_modularity, out_n_communities, st);
}

int32_t scrust_cuda_louvain(scrust_context* ctx, const uint32_t* indptr, const uint32_t* indices, const float* values,
                            uint64_t n_rows, uint64_t n_cols, double resolution, uint64_t seed, uint32_t* out_labels,
                            double* out_modularity, uint64_t* out_n_communities, scrust_status* st) {
    return cluster_host(ctx, indptr, indices, values, n_rows, n_cols, false, resolution, 1, seed, out_labels,
                        out_modularity, out_n_communities, st);
}

int32_t scrust_cuda_modularity(scrust_context* ctx, const uint32_t* indptr, const uint32_t* indices,
                               const float* values, uint64_t n_rows, uint64_t n_cols, const uint32_t* labels,
                               uint64_t n_labels, double resolution, double* out, scrust_status* st) {
    int32_t rc = check_resolution(resolution, st);
    if (rc) return rc;
    if ((rc = check_graph(indptr, indices, n_rows, n_cols, st))) return rc;
    if (!labels || !out || (indptr[n_rows] && !values)) return fail(st, SCRUST_SHAPE, "expected non-null pointers");
    if (n_labels != n_rows)
        return fail(st, SCRUST_SHAPE, "expected %llu labels, one per node, got %llu", (unsigned long long)n_rows,
                    (unsigned long long)n_labels);
    uint32_t mx = 0;
    for (uint64_t i = 0; i < n_labels; ++i) mx = std::max(mx, labels[i]);
    if ((uint64_t)mx + 1 > n_rows)
        return fail(st, SCRUST_INVALID_PARAMETER, "labels must be community ids below the node count, got %u", mx);
    if (!ctx) return fail(st, SCRUST_NO_GPU, "no CUDA context (no usable GPU)");
    std::lock_guard<std::mutex> lock(ctx->mu);
    DeviceGuard device_guard(ctx->device);
    return with_device_graph(ctx, indptr, indices, values, n_rows, st,
                             [&](const uint32_t* dip, const uint32_t* dix, const float* dvl, int64_t nnz) -> int32_t {
                                 Clusterer c(ctx, st);
                                 int32_t r = c.build(dip, dix, dvl, (int64_t)n_rows, nnz);
                                 if (r) return r;
                                 uint32_t* dl = c.alloc<uint32_t>(n_rows);
                                 if (!dl) return fail(st, SCRUST_OOM, "clustering: device allocation failed");
                                 cudaMemcpyAsync(dl, labels, sizeof(uint32_t) * n_rows, cudaMemcpyHostToDevice,
                                                 ctx->stream);
                                 return c.score_only(dl, (int64_t)mx + 1, resolution, out);
                             });
}

}  // extern "C"
