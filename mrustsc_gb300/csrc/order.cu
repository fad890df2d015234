// order.cu -- a spatial ordering of the rows for the tensor sweep.
//
// Exactness never depends on the order in which a row meets its columns, but
// speed does: a row's threshold only tightens once it has seen columns near
// it, and until then every column it meets is appended to its list.  So
// before the sweep the rows are grouped into cells around anchors (every
// n/m-th row), the cells are laid out consecutively, and every 256-row work
// item gets a short list of priority tiles: the tiles holding its own cells
// and the cells of the anchors nearest to them.  The sweep visits those
// first (knn_tensor.cu).  Nearest anchors come from the tensor candidate lists
// of a points x anchors pass with k = 1 (an approximate assignment is enough
// for an ordering); anchor neighbourhoods from an FP32 anchors x anchors kNN.
//
// The sweep then runs in two passes.  The first visits only the priority
// tiles and leaves every row with a threshold.  Between the passes the rows of
// each cell within a 256-row block (a segment) get a bounding ball of their
// quantised values (centre c, radius R) and the largest distance U that can
// still matter to one of them: the MMA value of a pair is at least
// |a_i - b_j|^2 - A_i - delta_i, so a column j can join row i's list only while
// |a_i - b_j| < sqrt(theta_i + A_i + delta_i).  A tile all of whose segments t
// have |c_s - c_t| - R_s - R_t >= U_s for every segment s of a row block cannot
// add to any row of it and is left out of the collect pass, which visits the
// rest.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace scrust {

namespace {

size_t align_up(size_t v) { return (v + 255) & ~(size_t)255; }

// Anchor c is input row floor(c * n / m); its coordinates are copied out
// for the anchor neighbourhoods.
__global__ void anchors_kernel(const float* __restrict__ x, int d, int64_t n, int64_t m, uint32_t* __restrict__ src,
                               float* __restrict__ out) {
    const int64_t c = blockIdx.x;
    if (c >= m) return;
    const int64_t r = (c * n) / m;
    if (threadIdx.x == 0) src[c] = (uint32_t)r;
    for (int t = threadIdx.x; t < d; t += blockDim.x) out[c * d + t] = x[r * d + t];
}

// Squared FP32 distances between all anchors (a sequential fma chain over
// the dimensions per pair), 64 x 64 per block and 4 x 4 per thread; the
// diagonal is +inf.
__global__ void __launch_bounds__(256) anchor_dist_kernel(const float* __restrict__ anc, int m, int d,
                                                          float* __restrict__ dist) {
    __shared__ __align__(16) float As[64][64 + 4];  // padded as in segment_pairs_kernel
    __shared__ __align__(16) float Bs[64][64 + 4];
    const int i0 = blockIdx.y * 64, j0 = blockIdx.x * 64;
    const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
    float acc[4][4] = {};
    for (int t0 = 0; t0 < d; t0 += 64) {  // 64 dimensions at a time
        const int dc = min(64, d - t0);
        __syncthreads();
        for (int p = threadIdx.x; p < 64 * 64; p += blockDim.x) {
            const int r = p / 64, t = p % 64;
            As[t][r] = (i0 + r < m && t < dc) ? anc[(int64_t)(i0 + r) * d + t0 + t] : 0.f;
            Bs[t][r] = (j0 + r < m && t < dc) ? anc[(int64_t)(j0 + r) * d + t0 + t] : 0.f;
        }
        __syncthreads();
        for (int t = 0; t < dc; ++t) {
            const float4 a4 = *reinterpret_cast<const float4*>(&As[t][ty * 4]);
            const float4 b4 = *reinterpret_cast<const float4*>(&Bs[t][tx * 4]);
            const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float df = av[p] - bv[q];
                    acc[p][q] = fmaf(df, df, acc[p][q]);
                }
        }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int i = i0 + ty * 4 + p;
        if (i >= m) continue;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int j = j0 + tx * 4 + q;
            if (j < m) dist[(int64_t)i * m + j] = i == j ? __int_as_float(0x7f800000) : acc[p][q];
        }
    }
}

// One warp per anchor: its kAnchorNeighbours nearest other anchors, nearest
// first, ties to the smaller id; 0xffffffff past the last.  The largest of the
// lanes' smallest distances has kAnchorNeighbours <= 32 at or below it, one of
// each lane: the candidates, some hundred and thirty of 3,906, are collected
// and sorted (a sorted top-32 in every lane, which some lane entered at almost
// every step, took 150 us for 3,906 anchors; 87 us so).  More of them than
// kTopCap (many anchors at one distance) go through such lists.
constexpr int kTopCap = 256;
static_assert(kAnchorNeighbours <= 32, "a bound from one distance a lane");
__global__ void __launch_bounds__(128) anchor_top_kernel(const float* __restrict__ dist, int m,
                                                         uint32_t* __restrict__ nb) {
    __shared__ unsigned long long found_s[4][kTopCap];
    const int lane = threadIdx.x & 31;
    const int64_t c = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (c >= m) return;
    constexpr int K = kAnchorNeighbours;
    const uint32_t none = float_key(__int_as_float(0x7f800000));
    const float* row = dist + c * m;
    uint32_t least = 0xffffffffu;
#pragma unroll 8
    for (int j = lane; j < m; j += 32) least = min(least, float_key(row[j]));
    const uint32_t bound = __reduce_max_sync(0xffffffffu, least);
    unsigned long long* found = found_s[threadIdx.x >> 5];
    int count = 0;
#pragma unroll 4
    for (int j0 = 0; j0 < m; j0 += 32) {
        const uint32_t key = j0 + lane < m ? float_key(row[j0 + lane]) : 0xffffffffu;
        const bool in = j0 + lane < m && key <= bound;
        const uint32_t who = __ballot_sync(0xffffffffu, in);
        const int at = count + __popc(who & lanemask_lt());
        if (in && at < kTopCap) found[at] = ((unsigned long long)key << 32) | (uint32_t)(j0 + lane);
        count += __popc(who);
    }
    __syncwarp();
    if (count <= kTopCap) {
        constexpr int R = kTopCap / 32;
        unsigned long long key[R];
#pragma unroll
        for (int r = 0; r < R; ++r) key[r] = lane + 32 * r < count ? found[lane + 32 * r] : ~0ull;
        // (Ascending bitonic sort, position lane + 32 r in key[r]; the halves
        // past `count` hold nothing and are left out.)
#pragma unroll
        for (int size = 2; size <= kTopCap; size <<= 1) {
            if (size > 32 && size / 2 >= count) break;
#pragma unroll
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                if (stride >= 32) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const int o = r ^ (stride / 32);
                        if (o > r) {
                            const bool up = ((32 * r) & size) == 0;
                            const unsigned long long a = key[r], b = key[o];
                            key[r] = (a < b) == up ? a : b;
                            key[o] = (a < b) == up ? b : a;
                        }
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const int i = lane + 32 * r;
                        const unsigned long long o = __shfl_xor_sync(0xffffffffu, key[r], stride);
                        const bool take_min = ((i & stride) == 0) == ((i & size) == 0);
                        key[r] = (key[r] < o) == take_min ? key[r] : o;
                    }
                }
            }
        }
        if (lane < K) nb[c * K + lane] = (uint32_t)(key[0] >> 32) < none ? (uint32_t)key[0] : 0xffffffffu;
        return;
    }
    unsigned long long top[K];
#pragma unroll
    for (int r = 0; r < K; ++r) top[r] = ~0ull;
    for (int j = lane; j < m; j += 32) {
        unsigned long long key = ((unsigned long long)float_key(row[j]) << 32) | (uint32_t)j;
        if (key < top[K - 1]) {
#pragma unroll
            for (int r = 0; r < K; ++r) {
                const unsigned long long lo = key < top[r] ? key : top[r];
                key = key < top[r] ? top[r] : key;
                top[r] = lo;
            }
        }
    }
    for (int r = 0; r < K; ++r) {
        unsigned long long best = top[0];
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
            best = other < best ? other : best;
        }
        if (top[0] == best) {  // the owning lane pops its head (keys are distinct)
#pragma unroll
            for (int q = 0; q < K - 1; ++q) top[q] = top[q + 1];
            top[K - 1] = ~0ull;
        }
        if (lane == 0) nb[c * K + r] = (uint32_t)(best >> 32) < none ? (uint32_t)best : 0xffffffffu;
    }
}

// Cells are laid out in the order of a walk over the anchors: from each
// anchor to its nearest unvisited neighbouring anchor, or, when all of them
// have been visited, to the lowest unvisited anchor.  Consecutive cells are
// then mostly neighbours, so a 256-row block rarely mixes far-apart cells.
// The block stages the first kChainNb neighbours of every anchor (16-bit
// ids) in shared memory, many loads in flight; then one warp walks, since
// every step depends on the one before.  rank[a] is anchor a's place.
constexpr int kChainNb = 12;
constexpr int kChainThreads = 1024;
__global__ void __launch_bounds__(kChainThreads) anchor_chain_kernel(const uint32_t* __restrict__ nb, int m,
                                                                     uint32_t* __restrict__ rank) {
    extern __shared__ uint32_t ch_smem[];
    const int words = (m + 3) / 4 + 1;                      // visited bytes, then one full word past them
    uint8_t* vis = reinterpret_cast<uint8_t*>(ch_smem);     // m bytes (+ padding), 1 = visited
    uint16_t* nbs = reinterpret_cast<uint16_t*>(ch_smem + (words + 1) / 2 * 2);  // m * kChainNb, 8-byte aligned
    for (int i = threadIdx.x; i < words; i += blockDim.x) ch_smem[i] = 0u;
    __syncthreads();
    // Bytes past m read as visited, so neither the tests nor the scan for
    // the lowest unvisited anchor ever pick one.
    for (int i = m + threadIdx.x; i < 4 * words; i += blockDim.x) vis[i] = 1;
    for (int a = threadIdx.x; a < m; a += blockDim.x) {
        const uint4* src = reinterpret_cast<const uint4*>(nb + (int64_t)a * kAnchorNeighbours);
        uint32_t c[kChainNb];
#pragma unroll
        for (int q = 0; q < kChainNb / 4; ++q) {
            const uint4 w = src[q];
            c[4 * q] = w.x;
            c[4 * q + 1] = w.y;
            c[4 * q + 2] = w.z;
            c[4 * q + 3] = w.w;
        }
        // Missing neighbours point past m (a visited byte).
#pragma unroll
        for (int j = 0; j < kChainNb; ++j)
            nbs[(int64_t)a * kChainNb + j] = c[j] < (uint32_t)m ? (uint16_t)c[j] : (uint16_t)m;
    }
    __syncthreads();
    // Lane j looks at the j-th neighbour of the current anchor: a step is two
    // dependent shared loads, a ballot and a shuffle.  (One thread looking at
    // all twelve: 655 us for 3,906 anchors, 62 us for 390; 502 and 52 us so.)
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    if (lane == 0) {
        vis[0] = 1;
        rank[0] = 0;
    }
    __syncwarp();
    const uint32_t* vis4 = ch_smem;
    int cur = 0, scan = 0, pos = 1;
    for (; pos < m; ++pos) {
        const int c = lane < kChainNb ? (int)nbs[(size_t)cur * kChainNb + lane] : m;
        const uint32_t free = __ballot_sync(0xffffffffu, lane < kChainNb && !vis[c]);
        int next;
        if (free) {
            next = __shfl_sync(0xffffffffu, c, __ffs(free) - 1);
        } else {
            // The lowest unvisited anchor (words below `scan` are all visited).
            uint32_t open = 0u;
            for (; scan < words; scan += 32) {
                open = __ballot_sync(0xffffffffu, scan + lane < words && vis4[scan + lane] != 0x01010101u);
                if (open) break;
            }
            if (!open) break;          // cannot happen: an unvisited anchor exists while pos < m
            scan += __ffs(open) - 1;
            const uint32_t v = vis4[scan];
            int b = 0;
            while (b < 3 && ((v >> (8 * b)) & 0xffu)) ++b;
            next = 4 * scan + b;
            if (next >= m) break;      // cannot happen: bytes past m are marked visited
        }
        if (lane == 0) {
            vis[next] = 1;
            rank[next] = (uint32_t)pos;
        }
        __syncwarp();
        cur = next;
    }
    if (lane != 0) return;
    // Every anchor gets a rank whatever happened above.
    for (int a = 0; a < m && pos < m; ++a)
        if (!vis[a]) {
            vis[a] = 1;
            rank[a] = (uint32_t)pos++;
        }
}

// Anchor neighbourhoods renamed into walk order: row rank[a] of out holds
// the ranks of a's neighbours.
__global__ void relabel_neighbours_kernel(const uint32_t* __restrict__ nb, const uint32_t* __restrict__ rank, int m,
                                          uint32_t* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)m * kAnchorNeighbours) return;
    const int64_t a = i / kAnchorNeighbours, j = i % kAnchorNeighbours;
    const uint32_t c = nb[i];
    out[(int64_t)rank[a] * kAnchorNeighbours + j] = c < (uint32_t)m ? rank[c] : 0xffffffffu;
}

// Each row's nearest anchor from the nearest-group pass: the best of its
// `parts` groups (one of each column part and segment), then the group's eight anchors measured on the same
// 16-bit operands (a row's [a, 1, 1, 1] times an anchor's [-2b, three norm
// parts], summed in f32 over the `words` 16-byte words that hold them) and
// the smallest taken (ties to the lower anchor): an approximately nearest
// anchor, which is all an ordering needs.  Eight lanes per row, lane l
// holding word l (and word l + 8, of two operand blocks) of the row and of
// each of the eight anchors, so that every load of an anchor row is one contiguous line for the eight lanes; the
// partial sums meet by shuffles.  keys[i] receives the anchor
// (anchor_rank_kernel turns it into the sort key once the walk is done),
// vals[i] the row.
template <class T>
__device__ __forceinline__ float dot_word(uint4 x, uint4 y) {
    const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
    float acc = 0.f;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        float2 p, q;
        if constexpr (std::is_same<T, __nv_bfloat16>::value) {
            p = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xs[h]));
            q = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ys[h]));
        } else {
            p = __half22float2(*reinterpret_cast<const __half2*>(&xs[h]));
            q = __half22float2(*reinterpret_cast<const __half2*>(&ys[h]));
        }
        acc = fmaf(p.x, q.x, acc);
        acc = fmaf(p.y, q.y, acc);
    }
    return acc;
}

template <class T, int BLOCKS>
__global__ void nearest_anchor_kernel(const unsigned long long* __restrict__ best, int parts, int64_t n, int64_t m,
                                      const T* __restrict__ A, const T* __restrict__ B, int words,
                                      uint32_t* __restrict__ keys, unsigned long long* __restrict__ vals) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t i = t >> 3;
    const int l = (int)(t & 7);
    const bool row_ok = i < n;
    unsigned long long near = ~0ull;
    if (parts == 2) {
        if (row_ok) near = min(best[2 * i], best[2 * i + 1]);
    } else {
        for (int p = l; p < parts && row_ok; p += 8) near = min(near, best[i * parts + p]);
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) near = min(near, __shfl_xor_sync(0xffffffffu, near, o));
    }
    const uint32_t g = row_ok ? (uint32_t)near : 0u;
    const int64_t c0 = (int64_t)g * 8;
    float part[8];
#pragma unroll
    for (int a = 0; a < 8; ++a) part[a] = 0.f;
#pragma unroll
    for (int b = 0; b < BLOCKS; ++b) {
        const int lw = l + 8 * b;
        const bool lane_ok = row_ok && lw < words;
        const uint4 x =
            lane_ok ? __ldg(reinterpret_cast<const uint4*>(A + i * 64 * BLOCKS) + lw) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int a = 0; a < 8; ++a)
            if (lane_ok && c0 + a < m)
                part[a] += dot_word<T>(x, __ldg(reinterpret_cast<const uint4*>(B + (c0 + a) * 64 * BLOCKS) + lw));
    }
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) part[a] += __shfl_xor_sync(0xffffffffu, part[a], o);
    if (row_ok && l == 0) {
        int arg = 0;
        float bv = c0 < m ? part[0] : __int_as_float(0x7f800000);
#pragma unroll
        for (int a = 1; a < 8; ++a)
            if (c0 + a < m && part[a] < bv) {
                bv = part[a];
                arg = a;
            }
        const int64_t col = c0 + arg;
        keys[i] = (uint32_t)(col < m ? col : m - 1);
        vals[i] = (unsigned long long)i;
    }
}

// keys[i] = rank[keys[i]]: each row's anchor becomes the anchor's walk rank.
__global__ void anchor_rank_kernel(uint32_t* __restrict__ keys, int64_t n, const uint32_t* __restrict__ rank) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) keys[i] = rank[keys[i]];
}

// The sorted pairs taken apart, and (unless null) the m + 1 first places of the
// cells, each written by the first row past the cells before it.  (Counting
// rows by atomics took 22 us for 100,000 rows in 390 cells, 50 us for a
// million, and a scan after it; 2 and 5 us so.)
__global__ void unpack_perm_kernel(const uint32_t* __restrict__ skeys, const unsigned long long* __restrict__ svals,
                                   int64_t n, uint32_t m, uint32_t* __restrict__ perm,
                                   uint32_t* __restrict__ cell_of_pos, uint32_t* __restrict__ cell_start) {
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t key = skeys[s];
    perm[s] = (uint32_t)svals[s];
    cell_of_pos[s] = key;
    if (!cell_start) return;
    for (uint32_t c = s ? skeys[s - 1] + 1u : 0u; c <= key && c <= m; ++c) cell_start[c] = (uint32_t)s;
    if (s == n - 1)
        for (uint32_t c = key + 1u; c <= m; ++c) cell_start[c] = (uint32_t)n;
}

// anchor_rank_kernel, the stable sort by rank and unpack_perm_kernel by one
// block, for up to kRowsOneBlock rows: rank and row in one word, 7-bit radix
// passes in shared memory, a warp on R groups of 32 consecutive rows.  (Five
// launches for ranks below 256, eight above, of 1.3 to 6 us and as many gaps
// of 2: 27 us at 2,638 rows, 35 at one query; the chain of dependent steps,
// not the data, is the time here.)
constexpr int kRowsOneBlock = 8192;
constexpr int kRowBits = 13;
static_assert(kRowsOneBlock <= 1 << kRowBits && kMaxAnchors <= 1 << kRowBits, "rank and row in one word");
template <int R>
__global__ void __launch_bounds__(1024) order_rows_kernel(const uint32_t* __restrict__ anchor, int n,
                                                          const uint32_t* __restrict__ rank, int bits, uint32_t m,
                                                          uint32_t* __restrict__ perm,
                                                          uint32_t* __restrict__ cell_of_pos,
                                                          uint32_t* __restrict__ cell_start) {
    __shared__ uint32_t words[R * 1024];
    __shared__ uint16_t cnt[32][130];  // per warp and digit; the odd number of words spreads a digit's warps over the banks
    __shared__ uint32_t wsum[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, base = warp * R * 32 + lane;
    uint32_t key[R], at[R];
    // Places past the rows hold the largest word and come last in every pass.
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = base + r * 32;
        key[r] = i < n ? rank[anchor[i]] << kRowBits | (uint32_t)i : 0xffffffffu;
    }
    for (int shift = kRowBits; shift < kRowBits + bits; shift += 7) {
        for (int d = lane; d < 128; d += 32) cnt[warp][d] = 0;
        __syncwarp();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t d = key[r] >> shift & 127u;
            const uint32_t peers = __match_any_sync(0xffffffffu, d), before = cnt[warp][d];
            at[r] = before + __popc(peers & lanemask_lt());
            __syncwarp();
            if (__ffs(peers) - 1 == lane) cnt[warp][d] = (uint16_t)(before + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        // First places by digit, then warp: four warps' counts of a digit a thread.
        const int d = threadIdx.x >> 3, w0 = (threadIdx.x & 7) * 4;
        uint32_t c[4], sum = 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            c[j] = cnt[w0 + j][d];
            sum += c[j];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        uint32_t first = incl - sum + __reduce_add_sync(0xffffffffu, lane < warp ? wsum[lane] : 0u);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            cnt[w0 + j][d] = (uint16_t)first;
            first += c[j];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) words[cnt[warp][key[r] >> shift & 127u] + at[r]] = key[r];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; ++r) key[r] = words[base + r * 32];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int s = base + r * 32;
        if (s >= n) continue;
        const uint32_t cell = key[r] >> kRowBits;
        perm[s] = key[r] & ((1u << kRowBits) - 1u);
        cell_of_pos[s] = cell;
        if (!cell_start) continue;
        for (uint32_t c = s ? (words[s - 1] >> kRowBits) + 1u : 0u; c <= cell && c <= m; ++c) cell_start[c] = (uint32_t)s;
        if (s == n - 1)
            for (uint32_t c = cell + 1u; c <= m; ++c) cell_start[c] = (uint32_t)n;
    }
}

// One warp per 256-row work item: the column tiles holding the item's own
// cells, then those holding the cells of their nearest anchors, nearest
// anchors first; distinct, at most kPrioMax.  In a self solve the item's own
// tile always comes first, so no list is empty.
// (With the first 8 home cells only, a block of many small cells gave the rows
// past them thresholds from other clusters: 40 rows of one million overflowed
// their lists, and the exact fallback took 32 ms for them.)
constexpr int kHomeMax = 32;
__global__ void prio_tiles_kernel(const uint32_t* __restrict__ cell_of_pos, int64_t n,
                                  const uint32_t* __restrict__ cell_start, int m,
                                  const uint32_t* __restrict__ anchor_nb, int ka, int items, int col_tiles,
                                  uint32_t* __restrict__ prio, uint32_t* __restrict__ prio_cnt) {
    __shared__ uint32_t outs[4][kPrioMax];
    __shared__ uint32_t homes[4][kHomeMax];
    __shared__ int nhome[4];
    __shared__ uint32_t seen[4][(kMaxAnchors + 31) / 32];
    const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * 4 + wi;
    if (item >= items) return;
    for (int w = lane; w < (m + 31) / 32; w += 32) seen[wi][w] = 0u;
    uint32_t* out = outs[wi];
    const int64_t s0 = (int64_t)item * 256, s1 = min(n, s0 + 256);
    if (lane == 0) nhome[wi] = 0;
    __syncwarp();
    bool heads[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int64_t sp = s0 + 32 * r + lane;
        heads[r] = sp < s1 && (sp == s0 || cell_of_pos[sp] != cell_of_pos[sp - 1]);
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int64_t sp = s0 + 32 * r + lane;
        const bool head = heads[r];
        const uint32_t bal = __ballot_sync(0xffffffffu, head);
        if (head) {
            const int pos = nhome[wi] + __popc(bal & lanemask_lt());
            if (pos < kHomeMax) homes[wi][pos] = cell_of_pos[sp];
        }
        __syncwarp();
        if (lane == 0) nhome[wi] = min(kHomeMax, nhome[wi] + __popc(bal));
        __syncwarp();
    }
    const int nh = nhome[wi];
    int cnt = 0;
    // Appends tile t unless present (every lane tracks cnt).
    auto add = [&](uint32_t t) {
        if (cnt >= kPrioMax || t >= (uint32_t)col_tiles) return;
        const bool dup = (lane < cnt && out[lane] == t) || (lane + 32 < cnt && out[lane + 32] == t);
        if (__any_sync(0xffffffffu, dup)) return;
        if (lane == 0) out[cnt] = t;
        cnt++;
        __syncwarp();
    };
    add((uint32_t)item);
    // The cells in turn (each home, then each home's nearest neighbour, its
    // second nearest ..), 32 at a time so that their loads are in flight
    // together, and each cell once: homes share neighbours (adding the tiles
    // of every repeat, 41 us for 100,000 rows, 21 us so; 54 and 25 us for a million).
    const int cells = (min(ka, kAnchorNeighbours) + 1) * nh;
    auto cell_at = [&](int i) {
        if (i >= cells) return 0xffffffffu;
        const int j = i / nh - 1;
        const uint32_t h = homes[wi][i % nh];
        return j < 0 ? h : anchor_nb[(int64_t)h * ka + j];
    };
    uint32_t ahead = cell_at(lane);
    for (int i0 = 0; i0 < cells && cnt < kPrioMax; i0 += 32) {
        const uint32_t c = ahead;
        ahead = cell_at(i0 + 32 + lane);
        const uint32_t peers = __match_any_sync(0xffffffffu, c);
        bool first = c < (uint32_t)m && (__ffs(peers) - 1) == lane && !((seen[wi][c >> 5] >> (c & 31)) & 1u);
        if (!__any_sync(0xffffffffu, first)) continue;
        uint32_t a = 0u, b = 0u;
        if (first) {
            atomicOr(&seen[wi][c >> 5], 1u << (c & 31));
            a = cell_start[c];
            b = cell_start[c + 1];
            first = b > a;
        }
        for (uint32_t live = __ballot_sync(0xffffffffu, first); live && cnt < kPrioMax; live &= live - 1) {
            const int l = __ffs(live) - 1;
            const uint32_t t0 = __shfl_sync(0xffffffffu, a, l) / 256, t1 = (__shfl_sync(0xffffffffu, b, l) - 1) / 256;
            for (uint32_t t = t0; t <= t1 && cnt < kPrioMax; ++t) add(t);
        }
        __syncwarp();
    }
    __syncwarp();
    for (int t = lane; t < cnt; t += 32) prio[(int64_t)item * kPrioMax + t] = out[t];
    if (lane == 0) prio_cnt[item] = (uint32_t)cnt;
}


__device__ __forceinline__ float op_float(__half v) { return __half2float(v); }
__device__ __forceinline__ float op_float(__nv_bfloat16 v) { return __bfloat162float(v); }
// A 16-bit operand value from the low half of a word.
template <class T>
__device__ __forceinline__ float op_bits(uint32_t w);
template <>
__device__ __forceinline__ float op_bits<__half>(uint32_t w) {
    return __half2float(__ushort_as_half((unsigned short)(w & 0xffffu)));
}
template <>
__device__ __forceinline__ float op_bits<__nv_bfloat16>(uint32_t w) {
    return __bfloat162float(__ushort_as_bfloat16((unsigned short)(w & 0xffffu)));
}

// Balls of a tile's cell segments (runs of rows of one cell; a cell lies in one
// region of the data, while a tile may straddle two far-apart cells).  Centres
// are stored dimension-major for coalesced pair tests.
// Segments past kSegMax share the last ball, which then reaches everywhere: with
// 8, one block of a million cells kept all 3,900 tiles and its CTA took 6.4 ms
// of a collect pass of 1.3 ms.
constexpr int kSegMax = 32;
struct TileBalls {
    float* seg_centre;  // [kSegMax][d][tiles]
    float* seg_radius;  // [kSegMax][tiles]
    float* seg_reach;   // [kSegMax][tiles]
    uint32_t* nseg;     // [tiles + 1], the last 0
};

// One block of 256 threads per column tile (= row block, the solve being a
// self-kNN): centres (means) and radii of the quantised rows of its segments,
// and the reach U = max over the rows of sqrt(theta + A + delta), theta being
// the smaller of the row's two list thresholds.
template <class T, int BLOCKS>
__global__ void __launch_bounds__(256) tile_balls_kernel(const T* __restrict__ ops, int64_t n, int d, int tiles,
                                                         const uint32_t* __restrict__ cell_of_pos,
                                                         const float* __restrict__ theta, const float* __restrict__ bA,
                                                         const float* __restrict__ bdelta, TileBalls b) {
    constexpr int W = 64 * BLOCKS;  // halves per operand row
    __shared__ float scentre[kSegMax][W];
    __shared__ int sstart[kSegMax + 1];
    __shared__ int wheads[8];
    __shared__ uint32_t rmax_seg[kSegMax], umax_seg[kSegMax];
    const int tile = blockIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t j = (int64_t)tile * 256 + threadIdx.x;
    const bool valid = j < n;
    const int rows = (int)min((int64_t)256, n - (int64_t)tile * 256);
    const T* row = ops + j * W;
    // The row's 16-bit values, read once as 16-byte words.
    uint32_t rw[W / 2];
#pragma unroll
    for (int q = 0; q < W / 8; ++q) {
        const uint4 u = valid ? reinterpret_cast<const uint4*>(row)[q] : make_uint4(0u, 0u, 0u, 0u);
        rw[4 * q] = u.x;
        rw[4 * q + 1] = u.y;
        rw[4 * q + 2] = u.z;
        rw[4 * q + 3] = u.w;
    }
    // Segment of each row: the number of run heads at or before it, less one.
    const bool head = valid && (threadIdx.x == 0 || cell_of_pos[j] != cell_of_pos[j - 1]);
    const uint32_t hb = __ballot_sync(0xffffffffu, head);
    if (lane == 0) wheads[w] = __popc(hb);
    if (threadIdx.x < kSegMax) {
        rmax_seg[threadIdx.x] = 0u;
        umax_seg[threadIdx.x] = 0u;
    }
    __syncthreads();
    int before = 0, nheads = 0;
    for (int q = 0; q < 8; ++q) {
        before += q < w ? wheads[q] : 0;
        nheads += wheads[q];
    }
    const int nseg = min(nheads, kSegMax);
    const int seg = min(before + __popc(hb & lanemask_lt()) + (head ? 1 : 0) - 1, kSegMax - 1);
    if (head && seg == before + __popc(hb & lanemask_lt())) sstart[seg] = threadIdx.x;
    if (threadIdx.x == 0) sstart[nseg] = rows;
    __syncthreads();
    for (int p = threadIdx.x; p < nseg * d; p += blockDim.x) {
        const int sg = p / d, t = p % d;
        float sum = 0.f;
        for (int r = sstart[sg]; r < sstart[sg + 1]; ++r) sum += op_float(ops[((int64_t)tile * 256 + r) * W + t]);
        const float c = sum / (float)(sstart[sg + 1] - sstart[sg]);
        scentre[sg][t] = c;
        b.seg_centre[((int64_t)sg * d + t) * tiles + tile] = c;
    }
    __syncthreads();
    if (valid) {
        // The squared distance to the centre in f32: a sum of d non-negative
        // rounded squares of rounded differences is at most (d + 2) units of
        // the last place below the exact value, so scaling by
        // 1 + (d + 4) 2^-23 (rounded up) bounds it from above.
        float s2 = 0.f;
#pragma unroll
        for (int t = 0; t < W; ++t) {
            if (t < d) {
                const float ds = op_bits<T>(rw[t >> 1] >> (16 * (t & 1))) - scentre[seg][t];
                s2 = fmaf(ds, ds, s2);
            }
        }
        const float grow = 1.0f + (float)(d + 4) * 1.1920929e-07f;
        s2 = __fmul_ru(s2, grow);
        const float th = fminf(theta[2 * j], theta[2 * j + 1]);
        // The reach sqrt(theta + A + delta), every step rounded up.
        const float v = __fadd_ru(__fadd_ru(th, bA[j]), bdelta[j]);
        const float u = isinf(th) && th > 0.f ? th : (v > 0.f ? __fsqrt_ru(v) : 0.f);
        // Non-negative floats order like their bit patterns.
        atomicMax(&rmax_seg[seg], __float_as_uint(s2));
        atomicMax(&umax_seg[seg], __float_as_uint(u));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        b.nseg[tile] = (uint32_t)nseg;
        if (tile == 0) b.nseg[tiles] = 0u;  // for the scan
    }
    if (threadIdx.x < nseg) {
        const int sg = threadIdx.x;
        b.seg_radius[(int64_t)sg * tiles + tile] = __fmul_ru(__fsqrt_ru(__uint_as_float(rmax_seg[sg])), 1.0f + 1e-6f);
        b.seg_reach[(int64_t)sg * tiles + tile] = __uint_as_float(umax_seg[sg]);
    }
}

// Whether a ball of reach u around centre I may hold a point within u of a
// point of ball T (conservatively true).  The f32 centre distance is within
// 1e-5 relative plus 3e-5 absolute (centre coordinates are at most 64 in
// magnitude); the slack covers both.  The test is made on squares in f32,
// each side moved past its own rounding (a few units of 2^-24 relative), so
// it never drops a tile the exact test keeps; a NaN keeps the tile.
__device__ __forceinline__ bool tile_needed(float dc2, float rI, float rT, float uI) {
    const float reach = (rI + rT + uI * (1.0f + 1e-5f) + 1e-4f) * (1.0f + 1e-6f);
    const float lhs = dc2 * ((1.0f - 1e-5f) * (1.0f - 1e-5f) * (1.0f - 1e-6f));
    return !(lhs >= reach * reach * (1.0f + 1e-6f));
}

// No more than the squared distance of two centres, from their squared norms and
// product, all f32 sums of d terms: each is off by at most (d + 1) u of itself
// (u = 2^-24; twice the product is at most the norms' sum), and adding them up
// by 6 u of the sum.  Half the instructions of summing squared differences,
// and its error lies well below that of the thresholds (a few 1e-2 against
// 0.4, in the operands' scale).  0 for anything not finite, which keeps the tile.
__device__ __forceinline__ float centres_apart(float a2, float b2, float product, int d) {
    const float sum = a2 + b2;
    return fmaxf(0.f, fmaf(-2.f, product, sum) - (2.f * d + 16.f) * 5.9604645e-8f * sum);
}

// The cell-segment balls of all tiles, one row each (centres padded to `width`
// = 64 or 128 dimensions with zeros), in tile order.
__global__ void flatten_segments_kernel(TileBalls b, int d, int width, int tiles, const uint32_t* __restrict__ seg_off,
                                        float* __restrict__ fc, float* __restrict__ fr, float* __restrict__ fu,
                                        uint32_t* __restrict__ fo) {
    const int T = blockIdx.x;
    const int ns = (int)min(b.nseg[T], (uint32_t)kSegMax);
    const uint32_t o = seg_off[T];
    for (int p = threadIdx.x; p < ns * width; p += blockDim.x) {
        const int sg = p / width, t = p % width;
        fc[(int64_t)(o + sg) * width + t] = t < d ? b.seg_centre[((int64_t)sg * d + t) * tiles + T] : 0.f;
    }
    if (threadIdx.x < ns) {
        fr[o + threadIdx.x] = b.seg_radius[(int64_t)threadIdx.x * tiles + T];
        fu[o + threadIdx.x] = b.seg_reach[(int64_t)threadIdx.x * tiles + T];
        fo[o + threadIdx.x] = (uint32_t)T;
    }
}

// All pairs of segment balls, 64 x 64 per block step, 4 x 4 per thread (7,800
// segments of 50 dimensions: 211 us with squared differences and 4-way bank
// conflicts in the staging, 194 us so; 1,300 of 100: 18 and 11 us):
// when segment i (of row block owner[i]) may reach segment j (of tile
// owner[j]), bit (owner[i], owner[j]) of the reach bitmap is set.  The
// segment count S is read on the device; blocks stride over the block pairs
// of the upper triangle, and each centre distance serves both directions.
constexpr int SP = 64;
template <int BLOCKS>
__global__ void __launch_bounds__(256) segment_pairs_kernel(const float* __restrict__ fc, const float* __restrict__ fr,
                                                            const float* __restrict__ fu,
                                                            const uint32_t* __restrict__ fo,
                                                            const uint32_t* __restrict__ S_ptr, int d, int words,
                                                            uint32_t* __restrict__ bitmap) {
    __shared__ __align__(16) float As[64][SP + 4];
    __shared__ __align__(16) float Bs[64][SP + 4];
    __shared__ float norms[2][4][SP];
    const int S = (int)*S_ptr;
    const int nb = (S + SP - 1) / SP;
    const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
    for (int64_t bp = blockIdx.x; bp < (int64_t)nb * nb; bp += gridDim.x) {
        const int bi = (int)(bp / nb), bj = (int)(bp % nb);
        if (bi > bj) continue;
        const int i0 = bi * SP, j0 = bj * SP;
        float acc[4][4] = {};
        // Thread t stages four dimensions of segment t % 64 at a time (conflict
        // free) and sums their squares.
        const int r = threadIdx.x % SP, part = threadIdx.x / SP;
        float a2 = 0.f, b2 = 0.f;
#pragma unroll
        for (int blk = 0; blk < BLOCKS; ++blk) {  // 64 dimensions at a time
            __syncthreads();
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int t = 4 * (part + 4 * c);
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 x = i0 + r < S ? __ldg(reinterpret_cast<const float4*>(fc + ((int64_t)(i0 + r) * BLOCKS + blk) * 64 + t)) : zero;
                const float4 y = j0 + r < S ? __ldg(reinterpret_cast<const float4*>(fc + ((int64_t)(j0 + r) * BLOCKS + blk) * 64 + t)) : zero;
                As[t][r] = x.x, As[t + 1][r] = x.y, As[t + 2][r] = x.z, As[t + 3][r] = x.w;
                Bs[t][r] = y.x, Bs[t + 1][r] = y.y, Bs[t + 2][r] = y.z, Bs[t + 3][r] = y.w;
                a2 += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
                b2 += y.x * y.x + y.y * y.y + y.z * y.z + y.w * y.w;
            }
            if (blk == BLOCKS - 1) {
                norms[0][part][r] = a2;
                norms[1][part][r] = b2;
            }
            __syncthreads();
            const int dims = min(64, d - 64 * blk);
            for (int t = 0; t < dims; ++t) {
                const float4 a4 = *reinterpret_cast<const float4*>(&As[t][ty * 4]);
                const float4 b4 = *reinterpret_cast<const float4*>(&Bs[t][tx * 4]);
                const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int q = 0; q < 4; ++q) acc[p][q] = fmaf(av[p], bv[q], acc[p][q]);
            }
        }
        auto norm = [&](int side, int row) {
            return norms[side][0][row] + norms[side][1][row] + norms[side][2][row] + norms[side][3][row];
        };
        float nb2[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) nb2[q] = norm(1, tx * 4 + q);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int i = i0 + ty * 4 + p;
            if (i >= S) continue;
            const float na2 = norm(0, ty * 4 + p);
            const float ri = fr[i], ui = fu[i];
            const uint32_t oi = fo[i];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = j0 + tx * 4 + q;
                if (j >= S) continue;
                const float rj = fr[j];
                const uint32_t oj = fo[j];
                const float apart = centres_apart(na2, nb2[q], acc[p][q], d);
                if (tile_needed(apart, ri, rj, ui))
                    atomicOr(bitmap + (int64_t)oi * words + (oj >> 5), 1u << (oj & 31));
                // Off the diagonal block, the same distance for j reaching i.
                if (bi != bj && tile_needed(apart, rj, ri, fu[j]))
                    atomicOr(bitmap + (int64_t)oj * words + (oi >> 5), 1u << (oi & 31));
            }
        }
    }
}

// One block per row block I: the tiles of its reach bitmap row (all tiles where
// there is no bitmap) that are not in its priority list, ascending, at
// entries[I * tiles ...].
__global__ void __launch_bounds__(256) tile_lists_kernel(const uint32_t* __restrict__ bitmap, int words, int tiles,
                                                         const uint32_t* __restrict__ prio,
                                                         const uint32_t* __restrict__ prio_cnt,
                                                         uint32_t* __restrict__ counts, uint32_t* __restrict__ entries,
                                                         int prio_stride = kPrioMax) {
    extern __shared__ uint32_t in_prio[];  // words
    __shared__ int wsum[8];
    const int I = blockIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int pc = (int)min(prio_cnt[I], (uint32_t)prio_stride);
    for (int i = threadIdx.x; i < words; i += blockDim.x) in_prio[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < pc; i += blockDim.x) {
        const uint32_t t = prio[(int64_t)I * prio_stride + i];
        if (t < (uint32_t)tiles) atomicOr(&in_prio[t >> 5], 1u << (t & 31));
    }
    __syncthreads();
    const uint32_t* row = bitmap ? bitmap + (int64_t)I * words : nullptr;
    uint32_t* out = entries + (int64_t)I * tiles;
    int base = 0;
    for (int w0 = 0; w0 < words; w0 += 256) {
        const int wd = w0 + threadIdx.x;
        const uint32_t all = tiles - wd * 32 >= 32 ? 0xffffffffu : (1u << (tiles & 31)) - 1u;
        uint32_t bits = wd < words ? (row ? row[wd] : all) & ~in_prio[wd] : 0u;
        int c = __popc(bits);
        int incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[w] = incl;
        __syncthreads();
        int before = 0, total = 0;
        for (int q = 0; q < 8; ++q) {
            before += q < w ? wsum[q] : 0;
            total += wsum[q];
        }
        int pos = base + before + incl - c;
        while (bits) {
            const int bt = __ffs(bits) - 1;
            bits &= bits - 1;
            out[pos++] = (uint32_t)(wd * 32 + bt);
        }
        base += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) counts[I] = (uint32_t)base;
}

// Operand rows (128 BLOCKS bytes each) and their per-row terms moved into list
// order; padding rows are zero like the operand kernel writes them.
// Eight lanes per block of a row: lane q copies the row's q-th 16-byte word of
// A and B (a warp writes whole 128-byte lines).
template <int BLOCKS>
__global__ void gather_operands_kernel(const uint4* __restrict__ A0, const uint4* __restrict__ B0,
                                       const float* __restrict__ bA0, const float* __restrict__ eps0,
                                       const uint32_t* __restrict__ perm, int64_t n, int64_t n_pad,
                                       uint4* __restrict__ A16, uint4* __restrict__ B16, float* __restrict__ bA,
                                       float* __restrict__ eps, const uint32_t* __restrict__ max_eps_bits,
                                       const uint32_t* __restrict__ max_bhat_bits, float* __restrict__ bdelta,
                                       float* __restrict__ beps2) {
    constexpr int WORDS = 8 * BLOCKS;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t s = t / WORDS;
    const int q = (int)(t % WORDS);
    if (s >= n_pad) return;
    if (s < n) {
        const int64_t r = perm[s];
        A16[s * WORDS + q] = A0[r * WORDS + q];
        B16[s * WORDS + q] = B0[r * WORDS + q];
        if (q == 0) {
            const float A = bA0[r], ep = eps0[r];
            bA[s] = A;
            eps[s] = ep;
            tensor_row_bounds(A, ep, __uint_as_float(*max_eps_bits), __uint_as_float(*max_bhat_bits), 64 * BLOCKS,
                              bdelta + s, beps2 + s);
        }
    } else {
        const uint4 z = make_uint4(0u, 0u, 0u, 0u);
        A16[s * WORDS + q] = z;
        B16[s * WORDS + q] = z;
        if (q == 0) {
            bA[s] = 0.f;
            eps[s] = 0.f;
        }
    }
}

// Keys that sort row blocks by decreasing count (stable, so ties keep
// block order).
__global__ void work_keys_kernel(const uint32_t* __restrict__ counts, int items, uint32_t* __restrict__ keys,
                                 unsigned long long* __restrict__ vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= items) return;
    keys[i] = 0xffffu - min(counts[i], 0xffffu);
    vals[i] = (unsigned long long)i;
}

// The same order by one block, for up to kOrderOneBlock row blocks: bitonic
// over (key, block) words, all distinct.  (Keys, two radix passes of three
// launches and the ids taken out again: eight launches, 33 us of a solve of
// any size below that, twice; this is one, of 5 us at 400 and 18 us at 4,000.)
constexpr int kOrderOneBlock = 8192;
// R words a thread: word r of thread t is element t + r blockDim.x.  Distances
// below a warp go by shuffles, at or above a block between a thread's words.
template <int R>
__global__ void __launch_bounds__(1024) order_one_block_kernel(const uint32_t* __restrict__ counts, int items,
                                                               uint32_t* __restrict__ order) {
    __shared__ uint32_t swap[R * 1024];
    const int tid = threadIdx.x, n = blockDim.x;
    uint32_t key[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = tid + r * n;
        key[r] = i < items ? (0xffffu - min(counts[i], 0xffffu)) << 16 | (uint32_t)i : 0xffffffffu;
    }
    for (int size = 2; size <= R * n; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= n) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
#pragma unroll
                    for (int o = 1; o < R; o <<= 1) {
                        if (stride != o * n || (r & o)) continue;
                        const uint32_t lo = min(key[r], key[r ^ o]), hi = max(key[r], key[r ^ o]);
                        const bool up = ((tid + r * n) & size) == 0;
                        key[r] = up ? lo : hi;
                        key[r ^ o] = up ? hi : lo;
                    }
                }
                continue;
            }
            if (stride >= 32) {
                __syncthreads();
#pragma unroll
                for (int r = 0; r < R; ++r) swap[tid + r * n] = key[r];
                __syncthreads();
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int i = tid + r * n;
                const uint32_t o = stride >= 32 ? swap[i ^ stride] : __shfl_xor_sync(0xffffffffu, key[r], stride);
                key[r] = ((i & stride) == 0) == ((i & size) == 0) ? min(key[r], o) : max(key[r], o);
            }
        }
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (tid + r * n < items) order[tid + r * n] = key[r] & 0xffffu;
}

__global__ void narrow_kernel(const unsigned long long* __restrict__ vals, int items, uint32_t* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < items) out[i] = (uint32_t)vals[i];
}

// Segment centres transposed to [64][segs], so that threads reading one
// dimension of consecutive segments read consecutive words.
__global__ void transpose_centres_kernel(const float* __restrict__ fc, int64_t segs, float* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= segs * 64) return;
    out[(i % 64) * segs + i / 64] = fc[i];
}

// Query rows against atlas tiles: the atlas tile of a segment ball may hold a
// candidate of a query while tile_needed holds for the query as a ball of
// radius 0 and of its own reach sqrt(theta + A + delta); the row block takes
// the tiles of all its queries.  64 queries x 64 atlas segments a block, 4 x 4
// a thread, distances in f32 on the quantised rows.  Testing every query costs
// 2 d operations a segment (5,000 x 8,000 segments: 200 us with squared
// differences and bank conflicts in the staging, 141 us so), and a block of
// queries sorted by cell falls in a hundred cells or more: balls around runs
// of its queries (eight at most, tested one by one in 276 us) covered so much
// that nearly every tile was kept, three passes of 600 us and more.
template <class T>
__global__ void __launch_bounds__(256) query_tiles_kernel(const T* __restrict__ ops, int64_t q,
                                                          const uint32_t* __restrict__ row_theta,
                                                          const float* __restrict__ bA,
                                                          const float* __restrict__ bdelta,
                                                          const float* __restrict__ act, const float* __restrict__ ar,
                                                          const uint32_t* __restrict__ ao, int64_t asegs, int d,
                                                          int words, uint32_t* __restrict__ bitmap) {
    __shared__ __align__(16) float As[64][64 + 4];
    __shared__ __align__(16) float Bs[64][64 + 4];
    __shared__ float reach[64], query2[64], centre2[4][64];
    __shared__ uint32_t hit[64];
    const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
    const int64_t i0 = (int64_t)blockIdx.y * 64, j0 = (int64_t)blockIdx.x * 64;
    const int r = threadIdx.x % 64, part = threadIdx.x / 64;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int t = 8 * (part + 4 * c);
        uint4 w = make_uint4(0u, 0u, 0u, 0u);
        if (i0 + r < q) w = __ldg(reinterpret_cast<const uint4*>(ops + (i0 + r) * 64 + t));
        const T* v = reinterpret_cast<const T*>(&w);
#pragma unroll
        for (int e = 0; e < 8; ++e) As[t + e][r] = t + e < d ? op_float(v[e]) : 0.f;
    }
    float c2 = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) {  // (the centres come dimension by dimension)
        const int t = part + 4 * c;
        const float v = j0 + r < asegs && t < d ? __ldg(act + (int64_t)t * asegs + j0 + r) : 0.f;
        Bs[t][r] = v;
        c2 += v * v;
    }
    centre2[part][r] = c2;
    if (threadIdx.x < 64) {
        hit[threadIdx.x] = 0u;
        const int64_t i = i0 + threadIdx.x;
        float u = 0.f;
        query2[threadIdx.x] = i < q ? bA[i] : 0.f;
        if (i < q) {
            // Every step rounded up; a row without a threshold reaches all.
            const uint32_t key = row_theta[i];
            const float th = key == 0xffffffffu ? __int_as_float(0x7f800000) : key_float(key);
            const float v = __fadd_ru(__fadd_ru(th, bA[i]), bdelta[i]);
            u = isinf(th) && th > 0.f ? th : (v > 0.f ? __fsqrt_ru(v) : 0.f);
        }
        reach[threadIdx.x] = u;
    }
    __syncthreads();
    float acc[4][4] = {};
    for (int t = 0; t < d; ++t) {
        const float4 a4 = *reinterpret_cast<const float4*>(&As[t][ty * 4]);
        const float4 b4 = *reinterpret_cast<const float4*>(&Bs[t][tx * 4]);
        const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[p][c] = fmaf(av[p], bv[c], acc[p][c]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int64_t j = j0 + tx * 4 + c;
        if (j >= asegs) continue;
        const float rj = ar[j];
        const int cj = tx * 4 + c;
        const float b2 = centre2[0][cj] + centre2[1][cj] + centre2[2][cj] + centre2[3][cj];
        bool any = false;
#pragma unroll
        for (int p = 0; p < 4; ++p)
            any |= i0 + ty * 4 + p < q &&
                   tile_needed(centres_apart(query2[ty * 4 + p], b2, acc[p][c], d), 0.f, rj, reach[ty * 4 + p]);
        if (any) hit[tx * 4 + c] = 1u;
    }
    __syncthreads();
    if (threadIdx.x < 64 && hit[threadIdx.x]) {
        const uint32_t tile = ao[j0 + threadIdx.x];
        atomicOr(bitmap + i0 / 256 * words + (tile >> 5), 1u << (tile & 31));
    }
}

// Exclusive prefix of `v` over the block's 256 threads, and the total.
__device__ __forceinline__ int block_prefix(int v, int* wsum, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    __syncthreads();
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    int before = 0, all = 0;
    for (int i = 0; i < 8; ++i) {
        before += i < w ? wsum[i] : 0;
        all += wsum[i];
    }
    *total = all;
    return before + incl - v;
}

// Priority tiles of a block of routed queries.  A block of 256 queries sorted
// by cell may span many cells (queries are few per cell), so every cell of
// its rows counts: the tiles holding those cells, then, for small cells, the
// nearest neighbouring cells until they hold `want` rows between them (16 k: the
// threshold pass looks at groups of 8 columns, and k of them must come from
// the query's own surroundings), up to kQueryPrio tiles; and while fewer than kQueryPrioNear have been taken,
// the tiles of the cells' eight nearest neighbours, lowest first.  The tiles come
// in ascending order, so that the chunks they are cut into hold whole
// clusters.  (A query whose cell was small, or whose tiles were left out, kept
// a threshold from another cluster, and its block then every tile of the
// atlas: 11,691 second tiles of 20 blocks for 5,000 queries of a million
// cells, 3,651 of one block for 100.)
// One block of 256 threads per query block; three tile bitmaps in shared memory,
// or two and no tiles of nearest neighbours for an atlas whose third does not
// fit (from some 155 million cells on).
constexpr int kQueryPrio = 512;
constexpr int kQueryPrioNear = 256;
constexpr int kQueryPrioNb = 8;

// Column segments that give two work items an SM where `tiles` tiles and `most`
// allow it, and that cutting the tiles into equal runs reproduces.
int column_segments(int most, int tiles, int items, int sms) {
    int c = std::max(1, std::min({most, tiles, (2 * sms + items - 1) / items}));
    while (c > 1 && (tiles + (tiles + c - 1) / c - 1) / ((tiles + c - 1) / c) != c) c--;
    return c;
}
__global__ void __launch_bounds__(256) query_prio_kernel(const uint32_t* __restrict__ cell_of_pos, int64_t n,
                                                         const uint32_t* __restrict__ cell_start, int m,
                                                         const uint32_t* __restrict__ cell_nb, int col_tiles,
                                                         uint32_t want, int maps, uint32_t* __restrict__ prio,
                                                         uint32_t* __restrict__ prio_cnt) {
    extern __shared__ uint32_t qp_bm[];
    __shared__ int wsum[8];
    const int words = (col_tiles + 31) / 32;
    uint32_t* home = qp_bm;
    uint32_t* more = qp_bm + words;
    uint32_t* near = maps == 3 ? qp_bm + 2 * words : nullptr;
    const int I = blockIdx.x;
    for (int i = threadIdx.x; i < maps * words; i += blockDim.x) qp_bm[i] = 0u;
    __syncthreads();
    const int64_t p = (int64_t)I * 256 + threadIdx.x;
    // Marks the tiles of cell c; its rows.
    auto mark = [&](uint32_t* bm, uint32_t c) {
        if (c >= (uint32_t)m) return 0u;
        const uint32_t a = cell_start[c], b = cell_start[c + 1];
        if (b <= a) return 0u;
        for (uint32_t t = a / 256; t <= (b - 1) / 256 && t < (uint32_t)col_tiles; ++t)
            atomicOr(&bm[t >> 5], 1u << (t & 31));
        return b - a;
    };
    if (p < n) {
        const uint32_t c = cell_of_pos[p];
        // Rows of one cell come together: the first of each run marks for all.
        if (p == (int64_t)I * 256 || cell_of_pos[p - 1] != c) {
            uint32_t rows = mark(home, c);
            if (c < (uint32_t)m) {
                const uint32_t* nb = cell_nb + (int64_t)c * kAnchorNeighbours;
                int j = 0;
                for (; j < kAnchorNeighbours && rows < want; ++j) rows += mark(more, nb[j]);
                if (near)
                    for (const int j1 = min(j + kQueryPrioNb, kAnchorNeighbours); j < j1; ++j) mark(near, nb[j]);
            }
        }
    }
    __syncthreads();
    // Each thread has a run of words; a bit stays while its place among the
    // bits of its kind is within the budget.
    const int per = (words + 255) / 256, w0 = min(words, (int)threadIdx.x * per), w1 = min(words, w0 + per);
    auto keep = [&](uint32_t* bm, int budget) {
        int c = 0, total = 0;
        for (int w = w0; w < w1; ++w) c += __popc(bm[w]);
        int at = block_prefix(c, wsum, &total);
        for (int w = w0; w < w1; ++w) {
            uint32_t bits = bm[w];
            const int here = __popc(bits);
            for (int over = min(here, at + here - budget); over > 0; --over) bits &= ~(0x80000000u >> __clz(bits));
            bm[w] = bits;
            at += here;
        }
        return min(total, budget);
    };
    int taken = keep(home, kQueryPrio);
    for (int w = w0; w < w1; ++w) more[w] &= ~home[w];
    taken += keep(more, kQueryPrio - taken);
    if (near) {
        for (int w = w0; w < w1; ++w) near[w] &= ~(home[w] | more[w]);
        keep(near, max(0, kQueryPrioNear - taken));
    }
    int c = 0, total = 0;
    for (int w = w0; w < w1; ++w) {
        home[w] |= more[w] | (near ? near[w] : 0u);
        c += __popc(home[w]);
    }
    int at = block_prefix(c, wsum, &total);
    uint32_t* out = prio + (int64_t)I * kQueryPrio;
    for (int w = w0; w < w1; ++w)
        for (uint32_t bits = home[w]; bits; bits &= bits - 1) out[at++] = (uint32_t)(w * 32 + __ffs(bits) - 1);
    if (threadIdx.x == 0) prio_cnt[I] = (uint32_t)total;
}

// Up to five runs of words set, each to its value: one launch where every run
// had its own: a request of one query 320 -> 312 us, 300 queries 667 -> 655.
struct WordRuns {
    uint32_t* p[5];
    int64_t n[5];
    uint32_t value[5];
};
__global__ void __launch_bounds__(256) set_words_kernel(WordRuns r) {
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
#pragma unroll
    for (int j = 0; j < 5; ++j)
        for (int64_t i = first; i < r.n[j]; i += step) r.p[j][i] = r.value[j];
}

// A row block's tile list cut into `segs` contiguous chunks of equal size,
// one per column segment, so that each segment of a row block is its own
// work item: dst row (block * segs + segment), `dst_stride` entries apart.
// Contiguous, not dealt round robin: the list starts with the tiles nearest
// the block, and one segment that sees them all finds a threshold near the
// rows' k-th distance, which the others then share; tiles dealt out one by
// one would leave every segment's own k-th smallest far out.  One block per
// row block.
__global__ void split_lists_kernel(const uint32_t* __restrict__ src, int src_stride, const uint32_t* __restrict__ cnt,
                                   int segs, uint32_t* __restrict__ dst, int dst_stride,
                                   uint32_t* __restrict__ dst_cnt) {
    const int I = blockIdx.x;
    const int c = (int)min(cnt[I], (uint32_t)src_stride);
    const int chunk = (c + segs - 1) / segs;  // <= dst_stride = ceil(src_stride / segs)
    for (int t = threadIdx.x; t < c; t += blockDim.x)
        dst[((int64_t)I * segs + t / chunk) * dst_stride + t % chunk] = src[(int64_t)I * src_stride + t];
    if (threadIdx.x < segs)
        dst_cnt[(int64_t)I * segs + threadIdx.x] = (uint32_t)max(0, min(chunk, c - (int)threadIdx.x * chunk));
}

__global__ void gather_rows_kernel(const float* __restrict__ x, const uint32_t* __restrict__ perm, int64_t n, int d,
                                   int stride, float* __restrict__ xs) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if ((stride & 3) == 0) {
        const int groups = stride >> 2;
        if (i >= n * groups) return;
        const int64_t s = i / groups;
        const int t0 = (int)(i - s * groups) * 4;
        const uint32_t r = perm[s];
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = (r == 0xffffffffu || t0 + e >= d) ? 0.f : x[(int64_t)r * d + t0 + e];
        reinterpret_cast<float4*>(xs + s * stride)[t0 >> 2] = make_float4(v[0], v[1], v[2], v[3]);
        return;
    }
    if (i >= n * stride) return;
    const int64_t s = i / stride, t = i % stride;
    const uint32_t r = perm[s];
    xs[i] = (r == 0xffffffffu || t >= d) ? 0.f : x[(int64_t)r * d + t];
}

// One thread per (list, segment, tile of the segment).
__global__ void deal_tiles_kernel(const uint32_t* __restrict__ src, const uint32_t* __restrict__ cnt,
                                  const uint32_t* __restrict__ order, int items, int stride, int parts,
                                  uint32_t* __restrict__ dst, uint32_t* __restrict__ dst_cnt,
                                  uint32_t* __restrict__ dst_order) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int share = (stride + parts - 1) / parts;
    const int64_t list = t / share;
    const int p = (int)(t % share);
    if (list >= (int64_t)parts * items) return;
    const int64_t i = list / parts;
    const int s = (int)(list % parts);
    const int c = (int)min(cnt[i], (uint32_t)stride);
    if (parts * p + s < c) dst[list * stride + p] = src[i * stride + parts * p + s];
    if (p == 0) {
        dst_cnt[list] = (uint32_t)((c + parts - 1 - s) / parts);
        dst_order[list] = (uint32_t)parts * order[i] + (uint32_t)s;
    }
}

// The operand type and width pick the instantiation.
void launch_tile_balls(bool bf16, const void* ops, int64_t n, int d, int tiles, const uint32_t* cell_of_pos,
                       const float* theta, const float* bA, const float* bdelta, const TileBalls& b, cudaStream_t s) {
    const bool one = operand_blocks(d) == 1;
    if (bf16) {
        const auto kern = one ? tile_balls_kernel<__nv_bfloat16, 1> : tile_balls_kernel<__nv_bfloat16, 2>;
        kern<<<tiles, 256, 0, s>>>((const __nv_bfloat16*)ops, n, d, tiles, cell_of_pos, theta, bA, bdelta, b);
    } else {
        const auto kern = one ? tile_balls_kernel<__half, 1> : tile_balls_kernel<__half, 2>;
        kern<<<tiles, 256, 0, s>>>((const __half*)ops, n, d, tiles, cell_of_pos, theta, bA, bdelta, b);
    }
}

void launch_nearest_anchor(bool bf16, const unsigned long long* best, int parts, int64_t n, int64_t m, const void* A, const void* B,
                           int blocks, int words, uint32_t* keys, unsigned long long* vals, cudaStream_t s) {
    const unsigned grid = (unsigned)((n * 8 + 255) / 256);
    if (bf16) {
        const auto kern = blocks == 1 ? nearest_anchor_kernel<__nv_bfloat16, 1> : nearest_anchor_kernel<__nv_bfloat16, 2>;
        kern<<<grid, 256, 0, s>>>(best, parts, n, m, (const __nv_bfloat16*)A, (const __nv_bfloat16*)B, words, keys, vals);
    } else {
        const auto kern = blocks == 1 ? nearest_anchor_kernel<__half, 1> : nearest_anchor_kernel<__half, 2>;
        kern<<<grid, 256, 0, s>>>(best, parts, n, m, (const __half*)A, (const __half*)B, words, keys, vals);
    }
}

// The rows in the order of their anchors' walk ranks (stable): kA holds the
// anchors and vA the rows, both overwritten; hist and scan as the radix sort
// wants them.  cell_start (m + 1 places) may be null.
cudaError_t order_rows(scrust_context* ctx, uint32_t* kA, unsigned long long* vA, uint32_t* kB, unsigned long long* vB,
                       int64_t n, const uint32_t* rank, int64_t m, uint32_t* hist, uint32_t* scan, size_t scan_elems,
                       uint32_t* perm, uint32_t* cell_of_pos, uint32_t* cell_start) {
    cudaStream_t s = ctx->stream;
    int bits = 1;
    while (((int64_t)1 << bits) < m) bits++;
    if (n <= kRowsOneBlock) {
        const auto kern = n <= 1024   ? order_rows_kernel<1>
                          : n <= 2048 ? order_rows_kernel<2>
                          : n <= 4096 ? order_rows_kernel<4>
                                      : order_rows_kernel<8>;
        kern<<<1, 1024, 0, s>>>(kA, (int)n, rank, bits, (uint32_t)m, perm, cell_of_pos, cell_start);
        ctx->launches += 1;
        return cudaGetLastError();
    }
    anchor_rank_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(kA, n, rank);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    uint32_t* skeys = nullptr;
    unsigned long long* svals = nullptr;
    if ((e = radix_sort_pairs(ctx, kA, vA, kB, vB, n, bits, hist, scan, scan_elems, &skeys, &svals)) != cudaSuccess)
        return e;
    unpack_perm_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(skeys, svals, n, (uint32_t)m, perm, cell_of_pos,
                                                                   cell_start);
    ctx->launches += 2;
    return cudaGetLastError();
}

}  // namespace

// Row blocks sorted by decreasing count into `order`; scratch holds
// work_order_scratch(items) bytes.
size_t work_order_scratch(int items) {
    const int nb = radix_blocks(items);
    return align_up(4 * (size_t)items) * 2 + align_up(8 * (size_t)items) * 2 + align_up(4 * ((size_t)256 * nb + 16)) +
           align_up(4 * scan_scratch_elems((int64_t)256 * nb));
}

cudaError_t sort_by_work(scrust_context* ctx, const uint32_t* counts, int items, char* scratch, uint32_t* order) {
    if (items <= kOrderOneBlock) {
        int width = 32;
        while (width < items) width *= 2;
        const int threads = std::min(1024, width);
        const auto kern = width <= 1024   ? order_one_block_kernel<1>
                          : width == 2048 ? order_one_block_kernel<2>
                          : width == 4096 ? order_one_block_kernel<4>
                                          : order_one_block_kernel<8>;
        kern<<<1, threads, 0, ctx->stream>>>(counts, items, order);
        ctx->launches += 1;
        return cudaGetLastError();
    }
    const int nb = radix_blocks(items);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = scratch + off;
        off += align_up(bytes);
        return p;
    };
    uint32_t* kA = (uint32_t*)take(4 * (size_t)items);
    uint32_t* kB = (uint32_t*)take(4 * (size_t)items);
    unsigned long long* vA = (unsigned long long*)take(8 * (size_t)items);
    unsigned long long* vB = (unsigned long long*)take(8 * (size_t)items);
    uint32_t* hist = (uint32_t*)take(4 * ((size_t)256 * nb + 16));
    const size_t scan_elems = scan_scratch_elems((int64_t)256 * nb);
    uint32_t* scan = (uint32_t*)take(4 * scan_elems);
    work_keys_kernel<<<(items + 255) / 256, 256, 0, ctx->stream>>>(counts, items, kA, vA);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    uint32_t* ks = nullptr;
    unsigned long long* vs = nullptr;
    if ((e = radix_sort_pairs(ctx, kA, vA, kB, vB, items, 16, hist, scan, scan_elems, &ks, &vs)) != cudaSuccess)
        return e;
    narrow_kernel<<<(items + 255) / 256, 256, 0, ctx->stream>>>(vs, items, order);
    ctx->launches += 2;
    return cudaGetLastError();
}

cudaError_t launch_deal_tiles(const uint32_t* src, const uint32_t* cnt, const uint32_t* order, int items, int stride,
                              int parts, uint32_t* dst, uint32_t* dst_cnt, uint32_t* dst_order, cudaStream_t s) {
    const int64_t threads = (int64_t)parts * items * ((stride + parts - 1) / parts);
    deal_tiles_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(src, cnt, order, items, stride, parts, dst,
                                                                        dst_cnt, dst_order);
    return cudaGetLastError();
}

cudaError_t launch_gather_rows(const float* x, const uint32_t* perm, int64_t n, int d, int stride, float* xs,
                               cudaStream_t s) {
    const int64_t threads = (stride & 3) == 0 ? n * (stride >> 2) : n * stride;
    gather_rows_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(x, perm, n, d, stride, xs);
    return cudaGetLastError();
}


int32_t build_row_order(scrust_context* ctx, const float* x, int64_t n, int d, const double* means,
                        uint32_t* max_bits, bool cosine, bool bf16, void* A16, void* B16, float* bA, float* beps,
                        float* bdelta, float* beps2, RowOrder* out, scrust_status* st) {
    cudaStream_t s = ctx->stream;
    cudaError_t e = cudaSuccess;
    const int64_t n_pad = (n + 255) / 256 * 256;
    const int items = (int)(n_pad / 256);
    const int64_t m = std::min<int64_t>(std::max<int64_t>(n / 256, 2), kMaxAnchors);
    const int64_t m_pad = (m + 255) / 256 * 256;
    const int nblocks = radix_blocks(n);
    const int blocks = operand_blocks(d);
    const size_t row_bytes = operand_row_bytes(d);
    const size_t scan_elems = scan_scratch_elems(std::max<int64_t>((int64_t)256 * nblocks, m + 1));

    // Carve the ordering slot.
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = align_up(off + bytes);
        return o;
    };
    const size_t o_src = take(4 * (size_t)m), o_anc = take(4 * (size_t)m * d), o_aA = take(row_bytes * (size_t)m_pad),
                 o_aB = take(row_bytes * (size_t)m_pad), o_arb = take(8 * (size_t)m_pad), o_kA = take(4 * (size_t)n),
                 o_kB = take(4 * (size_t)n), o_vA = take(8 * (size_t)n), o_vB = take(8 * (size_t)n),
                 o_perm = take(4 * (size_t)n), o_cell = take(4 * (size_t)n), o_cst = take(4 * (size_t)(m + 1)), o_nb = take(4 * (size_t)m * kAnchorNeighbours),
                 o_nb2 = take(4 * (size_t)m * kAnchorNeighbours), o_rank = take(4 * (size_t)m),
                 o_adist = take(4 * (size_t)m * (size_t)m),
                 o_prio = take(4 * (size_t)items * kPrioMax), o_pc = take(4 * (size_t)items),
                 o_theta = take(8 * (size_t)n_pad), o_po = take(4 * (size_t)items),
                 o_best = take(16 * (size_t)n_pad), o_A0 = take(row_bytes * (size_t)n_pad),
                 o_B0 = take(row_bytes * (size_t)n_pad), o_bA0 = take(4 * (size_t)n_pad), o_eps0 = take(4 * (size_t)n_pad),
                 o_ws = take(work_order_scratch(items)),
                 o_hist = take(4 * ((size_t)256 * nblocks + 16)), o_scan = take(4 * scan_elems);
    char* base = (char*)ws_get(ctx, SLOT_ORDER, off, &e);
    if (!base) return cuda_fail(st, e, "ordering: workspace");
    uint32_t* src = (uint32_t*)(base + o_src);
    float* anc = (float*)(base + o_anc);
    uint32_t *keysA = (uint32_t*)(base + o_kA), *keysB = (uint32_t*)(base + o_kB);
    unsigned long long *valsA = (unsigned long long*)(base + o_vA), *valsB = (unsigned long long*)(base + o_vB);
    uint32_t* perm = (uint32_t*)(base + o_perm);
    uint32_t* cell_of_pos = (uint32_t*)(base + o_cell);
    uint32_t* cell_start = (uint32_t*)(base + o_cst);
    uint32_t* anchor_nb = (uint32_t*)(base + o_nb);
    uint32_t* cell_nb = (uint32_t*)(base + o_nb2);
    uint32_t* rank = (uint32_t*)(base + o_rank);
    uint32_t* prio = (uint32_t*)(base + o_prio);
    uint32_t* prio_cnt = (uint32_t*)(base + o_pc);
    float* arb = (float*)(base + o_arb);

    // Anchors, and both operand sets in the input order.
    anchors_kernel<<<(unsigned)m, 64, 0, s>>>(x, d, n, m, src, anc);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "ordering: anchors");
    // The anchor neighbourhoods and the walk that orders the cells run on the
    // copy stream beside the operands and the rows x anchors pass below; the
    // main stream waits for them before the cells are formed.
    const size_t chain_smem = 4 * (size_t)((((m + 3) / 4 + 1) + 1) / 2 * 2) + 2 * (size_t)m * kChainNb;
    if ((e = set_smem_limit(ctx, (const void*)anchor_chain_kernel, (int)chain_smem)) != cudaSuccess ||
        (e = cudaEventRecord(ctx->copy_ev, s)) != cudaSuccess ||
        (e = cudaStreamWaitEvent(ctx->copy_stream, ctx->copy_ev, 0)) != cudaSuccess)
        return cuda_fail(st, e, "ordering: anchor walk");
    {
        float* adist = (float*)(base + o_adist);
        const dim3 grid((unsigned)((m + 63) / 64), (unsigned)((m + 63) / 64));
        anchor_dist_kernel<<<grid, 256, 0, ctx->copy_stream>>>(anc, (int)m, d, adist);
        anchor_top_kernel<<<(unsigned)((m + 3) / 4), 128, 0, ctx->copy_stream>>>(adist, (int)m, anchor_nb);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "ordering: anchor neighbours");
        ctx->launches += 2;
    }
    anchor_chain_kernel<<<1, kChainThreads, chain_smem, ctx->copy_stream>>>(anchor_nb, (int)m, rank);
    // The relabelling indexes by rank: never launched without the walk.
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "ordering: anchor walk");
    relabel_neighbours_kernel<<<(unsigned)((m * kAnchorNeighbours + 255) / 256), 256, 0, ctx->copy_stream>>>(
        anchor_nb, rank, (int)m, cell_nb);
    if ((e = cudaGetLastError()) != cudaSuccess || (e = cudaEventRecord(ctx->copy_ev, ctx->copy_stream)) != cudaSuccess)
        return cuda_fail(st, e, "ordering: anchor walk");
    ctx->launches += 2;

    void* A0 = base + o_A0;
    void* B0 = base + o_B0;
    float* bA0 = (float*)(base + o_bA0);
    float* eps0 = (float*)(base + o_eps0);
    if ((e = launch_tensor_operands(x, n, n_pad, d, means, max_bits, cosine, bf16, nullptr, A0, B0, bA0, eps0,
                                    max_bits + 1, max_bits + 2, ctx->sm_count, s)) != cudaSuccess ||
        (e = launch_tensor_operands(x, m, m_pad, d, means, max_bits, cosine, bf16, src, base + o_aA, base + o_aB, arb,
                                    arb + m_pad, max_bits + 1, max_bits + 2, ctx->sm_count, s)) != cudaSuccess)
        return cuda_fail(st, e, "ordering: operands");
    ctx->launches += 3;

    // Rows x anchors with k = 1 on the tensor cores, keeping only each row's
    // nearest anchor.
    KnnPlan px;
    px.nq = n;
    px.nr = m;
    px.d = d;
    px.k = 1;
    px.self = false;
    px.form = SCRUST_FORM_TENSOR;
    Lists lx;  // no storage: the pass keeps no lists
    lx.cap = 64;
    lx.ctot = 64 + 128;
    lx.segments = 2;
    px.cap = lx.cap;
    px.ctot = lx.ctot;
    px.segments = lx.segments;
    px.max_ctas = ctx->sm_count - 1;
    unsigned long long* best = (unsigned long long*)(base + o_best);
    if ((e = launch_tensor_candidates(ctx, px, A0, n_pad, base + o_aB, m_pad, bA0, bdelta, beps2, lx, bf16, nullptr,
                                      false, nullptr, nullptr, nullptr, best)) != cudaSuccess)
        return cuda_fail(st, e, "ordering: anchor candidates");
    const int op_words = (d + 3 + 7) / 8;  // 16-byte words of an operand row holding values
    launch_nearest_anchor(bf16, best, 2, n, m, A0, base + o_aB, blocks, op_words, keysA, valsA, s);
    // The walk ranks (copy stream) are needed from here on.
    if ((e = cudaGetLastError()) != cudaSuccess || (e = cudaStreamWaitEvent(s, ctx->copy_ev, 0)) != cudaSuccess)
        return cuda_fail(st, e, "ordering: nearest anchor");
    ctx->launches += 2;

    // Stable sort of the rows by anchor: the permutation and the cells.
    if ((e = order_rows(ctx, keysA, valsA, keysB, valsB, n, rank, m, (uint32_t*)(base + o_hist),
                        (uint32_t*)(base + o_scan), scan_elems, perm, cell_of_pos, cell_start)) != cudaSuccess)
        return cuda_fail(st, e, "ordering: sort");

    // The priority tiles of every work item.
    prio_tiles_kernel<<<(unsigned)((items + 3) / 4), 128, 0, s>>>(cell_of_pos, n, cell_start, (int)m, cell_nb,
                                                                  kAnchorNeighbours, items, items, prio, prio_cnt);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "ordering: priority tiles");
    ctx->launches += 1;
    if ((e = sort_by_work(ctx, prio_cnt, items, base + o_ws, (uint32_t*)(base + o_po))) != cudaSuccess)
        return cuda_fail(st, e, "ordering: work order");
    // The operands and bounds in list order.
    const auto gather = blocks == 1 ? gather_operands_kernel<1> : gather_operands_kernel<2>;
    gather<<<(unsigned)((n_pad * 8 * blocks + 255) / 256), 256, 0, s>>>(
        (const uint4*)A0, (const uint4*)B0, bA0, eps0, perm, n, n_pad, (uint4*)A16, (uint4*)B16, bA, beps, max_bits + 1,
        max_bits + 2, bdelta, beps2);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "ordering: operands");
    ctx->launches += 1;
    out->perm = perm;
    out->prio = prio;
    out->prio_cnt = prio_cnt;
    out->prio_order = (const uint32_t*)(base + o_po);
    out->theta = (float*)(base + o_theta);
    out->cell_of_pos = cell_of_pos;
    out->anchors = m;
    out->anchors_pad = m_pad;
    out->anchor_B16 = base + o_aB;
    out->anchor_rank = rank;
    out->cell_start = cell_start;
    out->cell_nb = cell_nb;
    return SCRUST_OK;
}

int32_t build_second_pass(scrust_context* ctx, const void* A16, bool bf16, int64_t n, int d, const RowOrder& order,
                          const float* bA, const float* bdelta, TileLists* out, scrust_status* st) {
    cudaStream_t s = ctx->stream;
    cudaError_t e = cudaSuccess;
    const int tiles = (int)((n + 255) / 256);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = align_up(off + bytes);
        return o;
    };
    const int words = (tiles + 31) / 32;
    const int blocks = operand_blocks(d);
    const int64_t smax = (int64_t)tiles * kSegMax;
    const size_t scan_elems = scan_scratch_elems((int64_t)tiles + 1);
    const size_t o_sc = take(4 * (size_t)kSegMax * d * tiles), o_sr = take(4 * (size_t)kSegMax * tiles),
                 o_su = take(4 * (size_t)kSegMax * tiles), o_ns = take(4 * ((size_t)tiles + 1)),
                 o_so = take(4 * ((size_t)tiles + 1)), o_fc = take(4 * 64 * blocks * (size_t)smax), o_fr = take(4 * (size_t)smax),
                 o_fu = take(4 * (size_t)smax), o_fo = take(4 * (size_t)smax), o_scan = take(4 * scan_elems),
                 o_bm = take(4 * (size_t)tiles * words), o_cnt = take(4 * ((size_t)tiles + 1)),
                 o_ent = take(4 * (size_t)tiles * (size_t)tiles);
    char* base = (char*)ws_get(ctx, SLOT_PRUNE, off, &e);
    if (!base) return cuda_fail(st, e, "pruning: workspace");
    TileBalls balls;
    balls.seg_centre = (float*)(base + o_sc);
    balls.seg_radius = (float*)(base + o_sr);
    balls.seg_reach = (float*)(base + o_su);
    balls.nseg = (uint32_t*)(base + o_ns);
    uint32_t* seg_off = (uint32_t*)(base + o_so);
    float* fc = (float*)(base + o_fc);
    float* fr = (float*)(base + o_fr);
    float* fu = (float*)(base + o_fu);
    uint32_t* fo = (uint32_t*)(base + o_fo);
    uint32_t* bitmap = (uint32_t*)(base + o_bm);
    uint32_t* counts = (uint32_t*)(base + o_cnt);
    uint32_t* entries = (uint32_t*)(base + o_ent);
    // Up to 17 anchors are all among each other's 16 nearest, so the priority
    // lists hold every tile and there is nothing to test: the lists are what is
    // left of all tiles, by one launch instead of six (2,638 rows, with the
    // unused work order of these lists gone: 501 -> 482 us; from 18 anchors, 4,608
    // rows, the balls rule tiles out).
    const bool few = order.anchors <= kAnchorNeighbours + 1;
    if (!few) {
        if ((e = cudaMemsetAsync(bitmap, 0, 4 * (size_t)tiles * words, s)) != cudaSuccess)
            return cuda_fail(st, e, "pruning: memset");
        launch_tile_balls(bf16, A16, n, d, tiles, order.cell_of_pos, order.theta, bA, bdelta, balls, s);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "pruning: tile balls");
        if ((e = device_exclusive_scan(ctx, balls.nseg, seg_off, (int64_t)tiles + 1, (uint32_t*)(base + o_scan),
                                       scan_elems)) != cudaSuccess)
            return cuda_fail(st, e, "pruning: segment scan");
        flatten_segments_kernel<<<tiles, 64, 0, s>>>(balls, d, 64 * blocks, tiles, seg_off, fc, fr, fu, fo);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "pruning: segments");
        const auto pairs = blocks == 1 ? segment_pairs_kernel<1> : segment_pairs_kernel<2>;
        pairs<<<8 * ctx->sm_count, 256, 0, s>>>(fc, fr, fu, fo, seg_off + tiles, d, words, bitmap);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "pruning: segment pairs");
        ctx->launches += 3;
    }
    const size_t lists_smem = 4 * (size_t)words;
    if ((e = set_smem_limit(ctx, (const void*)tile_lists_kernel, (int)lists_smem)) != cudaSuccess)
        return cuda_fail(st, e, "pruning: tile lists");
    tile_lists_kernel<<<tiles, 256, lists_smem, s>>>(few ? nullptr : bitmap, words, tiles, order.prio, order.prio_cnt,
                                                     counts, entries);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "pruning: tile lists");
    ctx->launches += 1;
    out->tiles = entries;
    out->offset = nullptr;
    out->count = counts;
    out->stride = tiles;
    out->order = nullptr;  // the collect pass keeps the priority lists' order
    return SCRUST_OK;
}

// ---- query solves against an ordered atlas -------------------------------------

namespace {

// The per-tile ball arrays of `tiles` tiles, laid out from byte `at` of
// `base`; returns the end of the layout.
size_t carve_balls(char* base, size_t at, int tiles, int d, TileBalls* b) {
    auto take = [&](size_t bytes) {
        const size_t a = at;
        at = align_up(at + bytes);
        return base + a;
    };
    b->seg_centre = (float*)take(4 * (size_t)kSegMax * d * tiles);
    b->seg_radius = (float*)take(4 * (size_t)kSegMax * tiles);
    b->seg_reach = (float*)take(4 * (size_t)kSegMax * tiles);
    b->nseg = (uint32_t*)take(4 * ((size_t)tiles + 1));
    return at;
}

}  // namespace

void atlas_order_free(AtlasOrder* o) {
    if (!o) return;
    void* ptrs[] = {o->B16, o->perm, o->rows, o->anchor_B16, o->anchor_rank, o->cell_start,
                    o->cell_nb, o->seg_centre_t, o->seg_radius, o->seg_tile};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    *o = AtlasOrder{};
}

int32_t atlas_order_build(scrust_context* ctx, const float* atlas, int64_t m, int d, const double* means,
                          uint32_t* words, bool bf16, AtlasOrder* out, scrust_status* st) {
    cudaStream_t s = ctx->stream;
    cudaError_t e = cudaSuccess;
    AtlasOrder o;
    o.m = m;
    o.m_pad = (m + 255) / 256 * 256;
    o.d = d;
    o.bf16 = bf16;
    const int tiles = (int)(o.m_pad / 256);
    const int P = padded_row_floats(d);
    // Scratch of the build: operands and row terms in list order, the tile
    // balls and their flattened segments.
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t at = off;
        off = align_up(off + bytes);
        return at;
    };
    const int64_t smax = (int64_t)tiles * kSegMax;
    const size_t scan_elems = scan_scratch_elems((int64_t)tiles + 1);
    const size_t o_A = take(128 * (size_t)o.m_pad), o_t = take(4 * 4 * (size_t)o.m_pad),
                 o_th = take(4 * 2 * (size_t)o.m_pad), o_so = take(4 * ((size_t)tiles + 1)),
                 o_fc = take(4 * 64 * (size_t)smax), o_fr = take(4 * (size_t)smax), o_fu = take(4 * (size_t)smax),
                 o_fo = take(4 * (size_t)smax), o_scan = take(4 * scan_elems);
    TileBalls balls;
    const size_t total = carve_balls(nullptr, off, tiles, d, &balls);
    char* base = nullptr;
    if ((e = cudaMalloc(&base, total)) != cudaSuccess || (e = cudaMalloc(&o.B16, 128 * (size_t)o.m_pad)) != cudaSuccess) {
        cudaFree(base);
        atlas_order_free(&o);
        cudaGetLastError();
        return cuda_fail(st, e, "atlas ordering: allocation");
    }
    carve_balls(base, off, tiles, d, &balls);
    float* terms = (float*)(base + o_t);
    float *bA = terms, *beps = terms + o.m_pad, *bdelta = terms + 2 * o.m_pad, *beps2 = terms + 3 * o.m_pad;
    RowOrder ord;
    int32_t rc = build_row_order(ctx, atlas, m, d, means, words, false, bf16, base + o_A, o.B16, bA, beps, bdelta,
                                 beps2, &ord, st);
    auto bail = [&](int32_t code) {
        cudaStreamSynchronize(s);
        cudaFree(base);
        atlas_order_free(&o);
        cudaGetLastError();
        return code;
    };
    if (rc) return bail(rc);
    o.anchors = ord.anchors;
    o.anchors_pad = ord.anchors_pad;
    const size_t na = (size_t)o.anchors;
    if ((e = cudaMalloc(&o.perm, 4 * (size_t)m)) != cudaSuccess ||
        (e = cudaMalloc(&o.rows, 4 * (size_t)m * P)) != cudaSuccess ||
        (e = cudaMalloc(&o.anchor_B16, 128 * (size_t)o.anchors_pad)) != cudaSuccess ||
        (e = cudaMalloc(&o.anchor_rank, 4 * na)) != cudaSuccess ||
        (e = cudaMalloc(&o.cell_start, 4 * (na + 1))) != cudaSuccess ||
        (e = cudaMalloc(&o.cell_nb, 4 * na * kAnchorNeighbours)) != cudaSuccess ||
        (e = cudaMemcpyAsync(o.perm, ord.perm, 4 * (size_t)m, cudaMemcpyDeviceToDevice, s)) != cudaSuccess ||
        (e = cudaMemcpyAsync(o.anchor_B16, ord.anchor_B16, 128 * (size_t)o.anchors_pad, cudaMemcpyDeviceToDevice,
                             s)) != cudaSuccess ||
        (e = cudaMemcpyAsync(o.anchor_rank, ord.anchor_rank, 4 * na, cudaMemcpyDeviceToDevice, s)) != cudaSuccess ||
        (e = cudaMemcpyAsync(o.cell_start, ord.cell_start, 4 * (na + 1), cudaMemcpyDeviceToDevice, s)) !=
            cudaSuccess ||
        (e = cudaMemcpyAsync(o.cell_nb, ord.cell_nb, 4 * na * kAnchorNeighbours, cudaMemcpyDeviceToDevice, s)) !=
            cudaSuccess ||
        (e = launch_gather_rows(atlas, ord.perm, m, d, P, o.rows, s)) != cudaSuccess ||
        (e = cudaMemsetAsync(base + o_th, 0, 4 * 2 * (size_t)o.m_pad, s)) != cudaSuccess)
        return bail(cuda_fail(st, e, "atlas ordering"));
    // The cell-segment balls of the atlas tiles (their reach is not used).
    uint32_t* seg_off = (uint32_t*)(base + o_so);
    float* fc = (float*)(base + o_fc);
    launch_tile_balls(bf16, base + o_A, m, d, tiles, ord.cell_of_pos, (const float*)(base + o_th), bA, bdelta,
                              balls, s);
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = device_exclusive_scan(ctx, balls.nseg, seg_off, (int64_t)tiles + 1, (uint32_t*)(base + o_scan),
                                   scan_elems)) != cudaSuccess)
        return bail(cuda_fail(st, e, "atlas ordering: tile balls"));
    flatten_segments_kernel<<<tiles, 64, 0, s>>>(balls, d, 64, tiles, seg_off, fc, (float*)(base + o_fr),
                                                 (float*)(base + o_fu), (uint32_t*)(base + o_fo));
    uint32_t segs = 0;
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = cudaMemcpyAsync(&segs, seg_off + tiles, sizeof(uint32_t), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return bail(cuda_fail(st, e, "atlas ordering: segments"));
    o.segs = segs;
    if ((e = cudaMalloc(&o.seg_centre_t, 4 * 64 * (size_t)std::max<uint32_t>(segs, 1))) != cudaSuccess ||
        (e = cudaMalloc(&o.seg_radius, 4 * (size_t)std::max<uint32_t>(segs, 1))) != cudaSuccess ||
        (e = cudaMalloc(&o.seg_tile, 4 * (size_t)std::max<uint32_t>(segs, 1))) != cudaSuccess ||
        (e = cudaMemcpyAsync(o.seg_radius, base + o_fr, 4 * (size_t)segs, cudaMemcpyDeviceToDevice, s)) !=
            cudaSuccess ||
        (e = cudaMemcpyAsync(o.seg_tile, base + o_fo, 4 * (size_t)segs, cudaMemcpyDeviceToDevice, s)) != cudaSuccess)
        return bail(cuda_fail(st, e, "atlas ordering: segments"));
    if (segs) transpose_centres_kernel<<<(unsigned)((64 * (int64_t)segs + 255) / 256), 256, 0, s>>>(fc, segs,
                                                                                                 o.seg_centre_t);
    if ((e = cudaGetLastError()) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return bail(cuda_fail(st, e, "atlas ordering: segments"));
    ctx->launches += 4;
    cudaFree(base);
    *out = o;
    return ok(st);
}

namespace {
constexpr int kRoutedCap = 256, kRoutedTotal = 256 + 128;  // a routed batch's lists: capacity and storage
}

size_t routed_list_bytes(const AtlasOrder& at, int64_t q, int k, int sm_count, int most_segments) {
    const int64_t q_pad = (q + 255) / 256 * 256;
    const int col_tiles = (int)(at.m_pad / 256);
    const size_t lists = 2 * (size_t)column_segments(std::min(most_segments, kQuerySegments), col_tiles,
                                                     (int)(q_pad / 256), sm_count);
    const size_t top = k < 2 ? 0 : k <= 16 ? 16 : 32;
    const size_t row = lists * (kRoutedTotal * 8 + 4 + 4 + 4 * top) + 8;  // ids and values, count, threshold, top-K
    return (size_t)q_pad * row * 9 / 8;                                   // the workspace grows by an eighth more
}

int32_t cross_ordered_enqueue(scrust_context* ctx, const AtlasOrder& at, const float* atlas_rows, const double* means,
                              const uint32_t* words, const float* dq, int64_t q, int k, uint32_t* d_idx,
                              float* d_dist, scrust_status* st, int most_segments) {
    cudaStream_t s = ctx->stream;
    cudaError_t e = cudaSuccess;
    const int d = at.d;
    const bool bf16 = at.bf16;
    const int64_t q_pad = (q + 255) / 256 * 256;
    const int items = (int)(q_pad / 256), col_tiles = (int)(at.m_pad / 256), words_t = (col_tiles + 31) / 32;
    // Column segments per row block, so that a small batch still fills the
    // GPU: each segment of a block is its own work item, and the segments of
    // a row share its threshold through HBM.
    const int csegs = column_segments(std::min(most_segments, kQuerySegments), col_tiles, items, ctx->sm_count);
    // The anchors likewise: one query had one CTA pass over all 16 tiles of
    // 3,906 anchors (23 us of its 320; 8 in 16 segments).
    const int anchor_tiles = (int)(at.anchors_pad / 256);
    const int anchor_segs = column_segments(anchor_tiles, anchor_tiles, items, ctx->sm_count);
    const int work = items * csegs;
    const int ps = (kQueryPrio + csegs - 1) / csegs, es = (col_tiles + csegs - 1) / csegs;
    const int P = padded_row_floats(d);
    const int nblocks = radix_blocks(q);
    const size_t scan_elems =
        scan_scratch_elems(std::max<int64_t>((int64_t)256 * nblocks, std::max<int64_t>(items, at.anchors) + 1));
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t a = off;
        off = align_up(off + bytes);
        return a;
    };
    const size_t o_A0 = take(128 * (size_t)q_pad), o_B0 = take(128 * (size_t)q_pad), o_t0 = take(4 * 2 * (size_t)q_pad),
                 o_As = take(128 * (size_t)q_pad), o_Bs = take(128 * (size_t)q_pad), o_ts = take(4 * 4 * (size_t)q_pad),
                 o_w = take(64), o_best = take(16 * (size_t)anchor_segs * q_pad), o_kA = take(4 * (size_t)q), o_kB = take(4 * (size_t)q),
                 o_vA = take(8 * (size_t)q), o_vB = take(8 * (size_t)q), o_qp = take(4 * (size_t)q),
                 o_cell = take(4 * (size_t)q),
                 o_xs = take(4 * (size_t)q * P), o_prio = take(4 * (size_t)items * kQueryPrio),
                 o_pc = take(4 * (size_t)items), o_ps = take(4 * (size_t)work * ps), o_psc = take(4 * (size_t)work),
                 o_po = take(4 * (size_t)work), o_po2 = take(4 * (size_t)work), o_ws = take(work_order_scratch(work)),
                 o_rt = take(4 * (size_t)q_pad), o_th = take(4 * 2 * (size_t)csegs * q_pad),
                 o_bm = take(4 * (size_t)items * words_t), o_cnt = take(4 * ((size_t)items + 1)), o_ent = take(4 * (size_t)items * col_tiles),
                 o_es = take(4 * (size_t)work * es), o_esc = take(4 * (size_t)work),
                 o_hist = take(4 * ((size_t)256 * nblocks + 16)), o_scan = take(4 * scan_elems);
    char* base = (char*)ws_get(ctx, SLOT_XORDER, off, &e);
    if (!base) return cuda_fail(st, e, "query routing: workspace");
    float* t0 = (float*)(base + o_t0);
    float *bA0 = t0, *eps0 = t0 + q_pad;
    float* ts = (float*)(base + o_ts);
    float *bA = ts, *beps = ts + q_pad, *bdelta = ts + 2 * q_pad, *beps2 = ts + 3 * q_pad;
    uint32_t* qwords = (uint32_t*)(base + o_w);
    uint32_t* qperm = (uint32_t*)(base + o_qp);
    uint32_t* cell_of_pos = (uint32_t*)(base + o_cell);
    uint32_t* prio = (uint32_t*)(base + o_prio);
    uint32_t* prio_cnt = (uint32_t*)(base + o_pc);
    uint32_t* row_theta = (uint32_t*)(base + o_rt);
    float* theta = (float*)(base + o_th);
    float* xs = (float*)(base + o_xs);
    uint32_t* bitmap = (uint32_t*)(base + o_bm);
    uint32_t* counts = (uint32_t*)(base + o_cnt);
    uint32_t* entries = (uint32_t*)(base + o_ent);
    unsigned long long* best = (unsigned long long*)(base + o_best);

    Lists lists;
    lists.cap = kRoutedCap;
    lists.ctot = kRoutedTotal;
    lists.segments = 2 * csegs;
    int32_t rc = alloc_lists(ctx, q_pad, &lists, st, false);
    if (rc) return rc;
    // The queries' operands, in input order; every query's nearest anchor.
    // Everything that starts from a set value.  A list the threshold pass leaves
    // without a threshold (a segment with no tile) keeps a huge one; a row
    // without any keeps reach everywhere.
    const size_t slots = (size_t)q_pad * lists.segments;
    const WordRuns runs = {{qwords, lists.cnt, (uint32_t*)theta, row_theta, bitmap},
                           {16, (int64_t)slots + q_pad, 2 * (int64_t)csegs * q_pad, q_pad, (int64_t)items * words_t},
                           {0u, 0u, 0x7f7f7f7fu, 0xffffffffu, 0u}};
    const int64_t longest = std::max((int64_t)slots + q_pad, (int64_t)items * words_t);
    set_words_kernel<<<(unsigned)std::min<int64_t>((longest + 255) / 256, 4 * ctx->sm_count), 256, 0, s>>>(runs);
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = launch_tensor_operands(dq, q, q_pad, d, means, words, false, bf16, nullptr, base + o_A0, base + o_B0, bA0,
                                    eps0, qwords, qwords + 1, ctx->sm_count, s)) != cudaSuccess)
        return cuda_fail(st, e, "query routing: operands");
    KnnPlan px;
    px.nq = q;
    px.nr = at.anchors;
    px.d = d;
    px.k = 1;
    px.self = false;
    px.form = SCRUST_FORM_TENSOR;
    Lists lx;  // no storage: the pass keeps no lists
    lx.cap = 64;
    lx.ctot = 64 + 128;
    lx.segments = 2 * anchor_segs;
    px.cap = lx.cap;
    px.ctot = lx.ctot;
    px.segments = lx.segments;
    if ((e = launch_tensor_candidates(ctx, px, base + o_A0, q_pad, at.anchor_B16, at.anchors_pad, bA0, eps0, eps0, lx,
                                      bf16, nullptr, false, nullptr, nullptr, nullptr, best)) != cudaSuccess)
        return cuda_fail(st, e, "query routing: nearest anchor");
    const int op_words = (d + 3 + 7) / 8;  // 16-byte words of an operand row holding values
    launch_nearest_anchor(bf16, best, lx.segments, q, at.anchors, base + o_A0, at.anchor_B16, 1, op_words, (uint32_t*)(base + o_kA),
                          (unsigned long long*)(base + o_vA), s);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "query routing: nearest anchor");
    ctx->launches += 4;
    // The queries sorted by the walk place of their cell; their operands,
    // bounds and rows in that order.
    if ((e = order_rows(ctx, (uint32_t*)(base + o_kA), (unsigned long long*)(base + o_vA), (uint32_t*)(base + o_kB),
                        (unsigned long long*)(base + o_vB), q, at.anchor_rank, at.anchors, (uint32_t*)(base + o_hist),
                        (uint32_t*)(base + o_scan), scan_elems, qperm, cell_of_pos, nullptr)) != cudaSuccess)
        return cuda_fail(st, e, "query routing: sort");
    gather_operands_kernel<1><<<(unsigned)((q_pad * 8 + 255) / 256), 256, 0, s>>>(
        (const uint4*)(base + o_A0), (const uint4*)(base + o_B0), bA0, eps0, qperm, q, q_pad, (uint4*)(base + o_As),
        (uint4*)(base + o_Bs), bA, beps, words + 1, words + 2, bdelta, beps2);
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = launch_gather_rows(dq, qperm, q, d, P, xs, s)) != cudaSuccess)
        return cuda_fail(st, e, "query routing: gather");
    // Priority tiles per row block, dealt over its column segments.
    const int maps = 12 * (size_t)words_t + 1024 <= ctx->smem_optin ? 3 : 2;
    const size_t prio_smem = 4 * maps * (size_t)words_t;
    if ((e = set_smem_limit(ctx, (const void*)query_prio_kernel, (int)prio_smem)) != cudaSuccess)
        return cuda_fail(st, e, "query routing: priority tiles");
    query_prio_kernel<<<items, 256, prio_smem, s>>>(cell_of_pos, q, at.cell_start, (int)at.anchors, at.cell_nb,
                                                    col_tiles, 16u * (uint32_t)k, maps, prio, prio_cnt);
    split_lists_kernel<<<items, 256, 0, s>>>(prio, kQueryPrio, prio_cnt, csegs, (uint32_t*)(base + o_ps), ps,
                                             (uint32_t*)(base + o_psc));
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "query routing: priority tiles");
    if ((e = sort_by_work(ctx, (uint32_t*)(base + o_psc), work, base + o_ws, (uint32_t*)(base + o_po))) != cudaSuccess)
        return cuda_fail(st, e, "query routing: work order");
    ctx->launches += 5;

    // The threshold pass over the priority tiles.
    KnnPlan plan;
    plan.nq = q;
    plan.nr = at.m;
    plan.d = d;
    plan.k = k;
    plan.self = false;
    plan.form = SCRUST_FORM_TENSOR;
    plan.precision = bf16 ? SCRUST_PRECISION_BF16 : SCRUST_PRECISION_FP16;
    plan.cap = lists.cap;
    plan.ctot = lists.ctot;
    plan.segments = lists.segments;
    TileLists first;
    first.tiles = (const uint32_t*)(base + o_ps);
    first.count = (const uint32_t*)(base + o_psc);
    first.stride = ps;
    first.order = (const uint32_t*)(base + o_po);
    first.row_theta = row_theta;
    // Each row's threshold is then taken from its lists together: a list sees
    // one column part of one segment's few tiles, so the best list's own k-th
    // lies far beyond the row's (one query alone, 13 tiles over 16 segments,
    // kept some 400 candidates).
    const int width = k <= 16 ? 16 : 32;
    float* topk = nullptr;
    if (k >= 2) {
        topk = (float*)ws_get(ctx, SLOT_TOPK, sizeof(float) * (size_t)lists.segments * width * q_pad, &e);
        if (!topk) return cuda_fail(st, e, "query knn: workspace");
    }
    if ((e = launch_tensor_candidates(ctx, plan, base + o_As, q_pad, at.B16, at.m_pad, bA, bdelta, beps2, lists, bf16,
                                      &first, false, theta, nullptr, nullptr, nullptr, kPassThresholds, topk)) !=
            cudaSuccess ||
        (topk && (e = launch_merge_segment_thresholds(topk, width, q, q_pad, k, lists.segments, first.count, bA, bdelta,
                                                      beps2, row_theta, s)) != cudaSuccess))
        return cuda_fail(st, e, "query knn: threshold pass");
    ctx->launches += topk ? 1 : 0;
    // The atlas tiles each row block cannot rule out: its queries, with the
    // reach of their shared thresholds, against the atlas segment balls.
    // (A grid's second dimension ends at 65,535: more groups of 64 queries take
    // more launches, whole row blocks each.)
    constexpr int64_t kMostGroups = 65532;
    static_assert(kMostGroups % 4 == 0 && kMostGroups <= 65535, "whole row blocks of 256 queries");
    for (int64_t i0 = 0; at.segs && i0 < q; i0 += 64 * kMostGroups) {
        const int64_t here = std::min<int64_t>(q - i0, 64 * kMostGroups);
        const dim3 grid((unsigned)((at.segs + 63) / 64), (unsigned)((here + 63) / 64));
        const char* ops = base + o_As + 128 * (size_t)i0;
        uint32_t* bits = bitmap + i0 / 256 * words_t;
        if (bf16)
            query_tiles_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>((const __nv_bfloat16*)ops, here, row_theta + i0, bA + i0,
                                                                   bdelta + i0, at.seg_centre_t, at.seg_radius,
                                                                   at.seg_tile, at.segs, d, words_t, bits);
        else
            query_tiles_kernel<__half><<<grid, 256, 0, s>>>((const __half*)ops, here, row_theta + i0, bA + i0, bdelta + i0,
                                                            at.seg_centre_t, at.seg_radius, at.seg_tile, at.segs, d,
                                                            words_t, bits);
    }
    const size_t lists_smem = 4 * (size_t)words_t;
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = set_smem_limit(ctx, (const void*)tile_lists_kernel, (int)lists_smem)) != cudaSuccess)
        return cuda_fail(st, e, "query knn: tile lists");
    tile_lists_kernel<<<items, 256, lists_smem, s>>>(bitmap, words_t, col_tiles, prio, prio_cnt, counts, entries,
                                                     kQueryPrio);
    split_lists_kernel<<<items, 256, 0, s>>>(entries, col_tiles, counts, csegs, (uint32_t*)(base + o_es), es,
                                             (uint32_t*)(base + o_esc));
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "query knn: tile lists");
    ctx->launches += 7;
    // The thresholds tightened over the kept tiles too: a query's neighbours
    // spread over its cluster, so a block whose queries fall in many cells
    // leaves the first pass with loose thresholds, and collecting at those
    // would overflow the lists.
    TileLists second;
    second.tiles = (const uint32_t*)(base + o_es);
    second.count = (const uint32_t*)(base + o_esc);
    second.stride = es;
    second.row_theta = row_theta;
    if ((e = sort_by_work(ctx, (uint32_t*)(base + o_esc), work, base + o_ws, (uint32_t*)(base + o_po2))) != cudaSuccess)
        return cuda_fail(st, e, "query knn: work order");
    second.order = (const uint32_t*)(base + o_po2);
    if ((e = launch_tensor_candidates(ctx, plan, base + o_As, q_pad, at.B16, at.m_pad, bA, bdelta, beps2, lists, bf16,
                                      &second, true, theta, nullptr, nullptr, nullptr, kPassThresholds)) != cudaSuccess)
        return cuda_fail(st, e, "query knn: second threshold pass");
    // One collect pass over both lists, then the exact finish.
    TileLists both = first;
    both.tiles2 = second.tiles;
    both.count2 = second.count;
    both.stride2 = es;
    if ((e = launch_tensor_candidates(ctx, plan, base + o_As, q_pad, at.B16, at.m_pad, bA, bdelta, beps2, lists, bf16,
                                      &both, false, theta, nullptr, nullptr, nullptr, kPassCollect)) != cudaSuccess)
        return cuda_fail(st, e, "query knn: collect pass");
    RowBounds bounds;
    bounds.A = bA;
    bounds.delta = bdelta;
    bounds.eps2 = beps2;
    if ((e = launch_rerank(ctx, plan, dq, atlas_rows, nullptr, nullptr, CosineRows(), dq, atlas_rows, bounds,
                           lists, at.perm, xs, theta, d_idx, d_dist, nullptr, nullptr, at.rows, P, true, qperm)) !=
        cudaSuccess)
        return cuda_fail(st, e, "query knn: rerank");
    ctx->launches += 3;
    return ok(st);
}

}  // namespace scrust
