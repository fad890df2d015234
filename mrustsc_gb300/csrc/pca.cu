// pca.cu -- truncated PCA of a cells x genes CSR matrix on the GPU, the step
// before the neighbours path (crates/scrust-core/src/pca.rs:74): its
// embedding can stay in HBM and go straight into the kNN graph build.
//
// The algorithm is the reference's randomised SVD (pca.rs:74-216): per-gene
// means and total variance (ddof 1 centred, 0 uncentred), a Gaussian sketch
// of n_components + 24 columns, power iterations (7 when fewer than a tenth
// of the spectrum is asked for, else 4) with an orthonormalisation after
// every product, then the eigendecomposition of (X^T Q)^T (X^T Q), singular
// values from its eigenvalues, the largest-loading sign fix (pca.rs:497-519)
// and scanpy's explained variance (S^2 / (n - 1) centred, the score columns'
// population variance uncentred).  Centring is a rank-one correction of
// every product, so the centred matrix is never formed.
//
// Device layout and order:
//   - X @ V: one warp per cell row and 32 columns, the row's entries in CSR
//     order; X^T @ U: the same per gene over a stable CSC copy (made once by
//     the library's radix sort), entries in row order.  No atomics: the same
//     inputs give the same bits.
//   - Grams: each block sums its rows' products in f32 groups of 32 rows into
//     f64, the blocks' partial Grams then add up in block order.
//   - Orthonormalisation: shifted CholeskyQR, twice (the shift, 1e-7 of the
//     largest diagonal entry, keeps a numerically rank-deficient sketch
//     factorable, as the reference's eigenvalue floor does).  Any orthonormal
//     basis of the sketch gives the same components; the reference whitens
//     by the Gram's eigenvectors instead.
//   - The final small eigenproblem: one-sided Jacobi in f64 over a cluster of
//     blocks.
// The Gaussian sketch comes from a counter-based generator (splitmix64 of
// the seed and the entry's index, Box-Muller in f64) instead of the
// reference's StdRng stream, so results agree with the reference's
// subspace, not its bits.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace scrust {

namespace {

constexpr int kOversampling = 24;
constexpr int kPcaMaxWidth = 128;  // sketch columns (n_components + 24) at most
constexpr double kShift = 1e-7;
constexpr int kJacobiSweeps = 60;
constexpr int kGramRows = 32;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Omega (g x w, rows ld apart): standard normals by Box-Muller from two
// uniforms in (0, 1] drawn from the seed and the pair's index; entries count
// row by row.
__global__ void pca_gaussian_kernel(int64_t count, int w, int ld, uint64_t seed, float* __restrict__ omega) {
    const int64_t pair = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (2 * pair >= count) return;
    const uint64_t h1 = mix64(seed ^ mix64((uint64_t)pair * 2 + 1));
    const uint64_t h2 = mix64(seed ^ mix64((uint64_t)pair * 2 + 2));
    const double u1 = ((double)(h1 >> 11) + 1.0) * 1.1102230246251565e-16;  // (0, 1]
    const double u2 = (double)(h2 >> 11) * 1.1102230246251565e-16;          // [0, 1)
    const double r = sqrt(-2.0 * log(u1));
    const double t = 6.283185307179586 * u2;
    omega[2 * pair / w * ld + 2 * pair % w] = (float)(r * cos(t));
    if (2 * pair + 1 < count) omega[(2 * pair + 1) / w * ld + (2 * pair + 1) % w] = (float)(r * sin(t));
}

// One warp per cell row (one thread per row read its entries alone: 88 us for
// 30,000 rows of 200, 13 us so).
__global__ void pca_csc_keys_kernel(const uint32_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
                                    const float* __restrict__ values, int64_t n, uint32_t* __restrict__ keys,
                                    unsigned long long* __restrict__ vals) {
    const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (r >= n) return;
    for (uint32_t e = indptr[r] + (threadIdx.x & 31), e1 = indptr[r + 1]; e < e1; e += 32) {
        keys[e] = indices[e];
        vals[e] = ((unsigned long long)(uint32_t)r << 32) | __float_as_uint(values[e]);
    }
}

// start[c] = number of sorted keys below c, c in [0, g].
__global__ void pca_starts_kernel(const uint32_t* __restrict__ keys, int64_t nnz, int64_t g,
                                  uint32_t* __restrict__ start) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p > nnz) return;
    const int64_t lo = p == 0 ? 0 : (int64_t)keys[p - 1] + 1;
    const int64_t hi = p == nnz ? g : (int64_t)keys[p];
    for (int64_t c = lo; c <= hi && c <= g; ++c) start[c] = (uint32_t)p;
}

// Sum over the block's 128 threads in a fixed tree; every thread gets it.
constexpr int kSumThreads = 128;
__device__ __forceinline__ double block_sum(double v, double* part) {
    part[threadIdx.x] = v;
    __syncthreads();
#pragma unroll
    for (int o = kSumThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
        __syncthreads();
    }
    const double total = part[0];
    __syncthreads();
    return total;
}

// Per gene: f64 sum and sum of squares over its entries, the f32 mean, and
// the gene's variance term (pca.rs:227-255).  One block per gene, strided
// threads and a fixed tree; a thread per gene waited on every entry in turn
// (2.2 ms for 2,000 genes of 3,000 entries).
__global__ void __launch_bounds__(kSumThreads)
    pca_column_stats_kernel(const uint32_t* __restrict__ cstart, const unsigned long long* __restrict__ cv, int64_t n,
                            double ddof, float* __restrict__ mean, double* __restrict__ var_term) {
    __shared__ double part[kSumThreads];
    const int64_t c = blockIdx.x;
    double s = 0.0, q = 0.0;
    for (uint32_t p = cstart[c] + threadIdx.x, p1 = cstart[c + 1]; p < p1; p += kSumThreads) {
        const double v = (double)__uint_as_float((uint32_t)cv[p]);
        s += v;
        q += v * v;
    }
    s = block_sum(s, part);
    q = block_sum(q, part);
    if (threadIdx.x) return;
    const double dn = (double)n;
    mean[c] = (float)(s / dn);
    var_term[c] = fmax(q - s * s / dn, 0.0) / (dn - ddof);
}

// Sum of `count` doubles in index order by one block (fixed tree per block of
// 256, blocks in order), into out[0].
__global__ void pca_sum_kernel(const double* __restrict__ x, int64_t count, double* __restrict__ out) {
    __shared__ double part[256];
    double total = 0.0;
    for (int64_t base = 0; base < count; base += 256) {
        const int64_t i = base + threadIdx.x;
        part[threadIdx.x] = i < count ? x[i] : 0.0;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) total += part[0];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = total;
}

// m[j] = sum_g mean[g] * B[g, j] in f64, one block per column (one thread per
// column read the genes one after another: 264 us for 2,000).
__global__ void __launch_bounds__(kSumThreads)
    pca_mean_row_kernel(const float* __restrict__ mean, const float* __restrict__ B, int64_t g, int ld,
                        float* __restrict__ m) {
    __shared__ double part[kSumThreads];
    const int j = blockIdx.x;
    double s = 0.0;
    for (int64_t c = threadIdx.x; c < g; c += kSumThreads) s += (double)mean[c] * (double)B[c * ld + j];
    s = block_sum(s, part);
    if (threadIdx.x == 0) m[j] = (float)s;
}

// Column sums of U (n x w) in f64 in two fixed-order levels: per block of
// rows, then over the blocks.  128 rows a block keeps every SM busy (with
// 4096, 30,000 rows were eight blocks: 400 us; 12 us so).
constexpr int kColRows = 128;
__global__ void pca_colsum_part_kernel(const float* __restrict__ U, int64_t n, int w, int ld, double* __restrict__ part) {
    const int64_t r0 = (int64_t)blockIdx.x * kColRows;
    const int64_t r1 = min(n, r0 + kColRows);
    for (int j = threadIdx.x; j < w; j += blockDim.x) {
        double s = 0.0;
#pragma unroll 8
        for (int64_t r = r0; r < r1; ++r) s += (double)U[r * ld + j];
        part[(int64_t)blockIdx.x * w + j] = s;
    }
}
__global__ void __launch_bounds__(kSumThreads)
    pca_colsum_final_kernel(const double* __restrict__ part, int blocks, int w, float* __restrict__ out) {
    __shared__ double sums[kSumThreads];
    const int j = blockIdx.x;
    double s = 0.0;
    for (int b = threadIdx.x; b < blocks; b += kSumThreads) s += part[(int64_t)b * w + j];
    s = block_sum(s, sums);
    if (threadIdx.x == 0) out[j] = (float)s;
}

// Both products keep every output one chain of fused adds over the sparse
// row's entries in order; rows of B and Y are ld floats apart, a multiple of 4
// with zeros past w, and a lane takes four columns of its warp's sparse row.
// Both are bound by the reads of B rows out of L2 (4 w bytes an entry).
__device__ __forceinline__ void fma4(float x, const float4& y, float4& acc) {
    acc.x = fmaf(x, y.x, acc.x);
    acc.y = fmaf(x, y.y, acc.y);
    acc.z = fmaf(x, y.z, acc.z);
    acc.w = fmaf(x, y.w, acc.w);
}

// Y (n x w) = X (n CSR rows) @ B (g x w) - ones * m (when m is given: the
// centring of X, X_c B = X B - 1 (mean^T B)); one warp per row.  30,000 x 2,000
// with 200 entries a row, w = 74: 175 us, 10 TB/s out of L2 (a lane per column
// 177 us).
__global__ void __launch_bounds__(128) pca_spmm_kernel(const uint32_t* __restrict__ start,
                                                       const uint32_t* __restrict__ idx,
                                                       const float* __restrict__ val, int64_t n,
                                                       const float* __restrict__ B, int w, int ld,
                                                       const float* __restrict__ m, float* __restrict__ Y) {
    constexpr uint32_t FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (r >= n) return;
    const int ld4 = ld / 4;
    const bool mine = lane < ld4;
    const float4* bq = reinterpret_cast<const float4*>(B) + (mine ? lane : 0);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t e1 = start[r + 1];
    for (uint32_t e = start[r]; e < e1; e += 32) {
        const int count = (int)min(32u, e1 - e);
        const uint32_t c = lane < count ? idx[e + lane] : 0u;
        const float v = lane < count ? val[e + lane] : 0.f;
        if (count == 32) {
#pragma unroll
            for (int u = 0; u < 32; ++u)
                fma4(__shfl_sync(FULL, v, u), bq[(int64_t)__shfl_sync(FULL, c, u) * ld4], acc);
        } else {
#pragma unroll 4
            for (int u = 0; u < count; ++u)
                fma4(__shfl_sync(FULL, v, u), bq[(int64_t)__shfl_sync(FULL, c, u) * ld4], acc);
        }
    }
    if (!mine) return;
    float y[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
    for (int t = 0; t < 4; ++t)
        if (m && 4 * lane + t < w) y[t] -= m[4 * lane + t];
    reinterpret_cast<float4*>(Y)[r * ld4 + lane] = make_float4(y[0], y[1], y[2], y[3]);
}

// Z (g x w) = X^T @ U (n x w) - mean sums^T (when mean is given: the centring,
// X_c^T U = X^T U - mean (1^T U)); one warp per gene over the CSC copy (entries
// as row << 32 | value, rows ascending).  Genes are few and long (2,000 of
// 3,000 entries, some four times that), so the latency of a chain of rows
// decides: each warp keeps two stages of kStageRows rows of U on their way
// into shared memory while it adds a third.  The same size: 496 us; one entry
// fetched after another 2.5 ms, a lane per column and three warps a gene
// 674 us, four columns a lane out of registers 1.25 ms (the compiler kept few
// loads in flight).
constexpr int kStageRows = 16;
constexpr int kStages = 3;
constexpr int kSpmmTWarps = 4;
size_t spmm_t_smem_bytes(int ld) { return sizeof(float) * (size_t)kSpmmTWarps * kStages * kStageRows * ld; }

__global__ void __launch_bounds__(kSpmmTWarps * 32)
    pca_spmm_t_kernel(const uint32_t* __restrict__ start, const unsigned long long* __restrict__ packed, int64_t g,
                      const float* __restrict__ U, int w, int ld, const float* __restrict__ mean,
                      const float* __restrict__ sums, float* __restrict__ Z) {
    extern __shared__ float4 ring4[];
    constexpr uint32_t FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t r = (int64_t)blockIdx.x * kSpmmTWarps + warp;
    if (r >= g) return;
    const int ld4 = ld / 4;
    const bool mine = lane < ld4;
    const float4* uq = reinterpret_cast<const float4*>(U) + lane;
    // This lane's column of each slot; it reads only what it copied itself.
    float4* ring = ring4 + (size_t)warp * kStages * kStageRows * ld4 + lane;
    const uint32_t ring_addr = (uint32_t)__cvta_generic_to_shared(ring);
    const uint32_t e0 = start[r], len = start[r + 1] - e0;
    const uint32_t stages = (len + kStageRows - 1) / kStageRows;
    // 32 entries a lane each: the chunk being added, the one whose rows are on
    // their way, and the one after.
    auto fetch = [&](uint32_t chunk) {
        const uint32_t at = chunk * 32 + lane;
        return at < len ? packed[e0 + at] : 0ull;
    };
    auto issue = [&](uint32_t stage, unsigned long long entries) {
        if (stage < stages) {
            const int count = (int)min((uint32_t)kStageRows, len - stage * kStageRows);
            const uint32_t slot = ring_addr + (stage % kStages) * (uint32_t)(kStageRows * ld4 * 16);
            const uint32_t rows = (uint32_t)(entries >> 32);
            const int first = (int)(stage & 1) * kStageRows;
#pragma unroll
            for (int u = 0; u < kStageRows; ++u) {
                const uint32_t row = __shfl_sync(FULL, rows, first + u);
                if (mine && u < count)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(slot + (uint32_t)(u * ld4 * 16)),
                                 "l"(uq + (int64_t)row * ld4)
                                 : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    static_assert(kStages == 3 && kStageRows == 16, "a chunk of 32 entries is two stages, issued one chunk ahead");
    unsigned long long cur = fetch(0), next = fetch(1);
    issue(0, cur);
    issue(1, cur);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t chunk = 0; chunk * 2 < stages; ++chunk) {
        const unsigned long long after = fetch(chunk + 2);
        const float v = __uint_as_float((uint32_t)cur);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const uint32_t stage = chunk * 2 + half;
            issue(stage + 2, next);
            asm volatile("cp.async.wait_group 2;" ::: "memory");
            if (stage < stages) {
                const int count = (int)min((uint32_t)kStageRows, len - stage * kStageRows);
                const float4* slot = ring + (size_t)(stage % kStages) * kStageRows * ld4;
                if (count == kStageRows) {
#pragma unroll
                    for (int u = 0; u < kStageRows; ++u)
                        fma4(__shfl_sync(FULL, v, half * kStageRows + u), mine ? slot[u * ld4] : acc, acc);
                } else {
                    for (int u = 0; u < count; ++u)
                        fma4(__shfl_sync(FULL, v, half * kStageRows + u), mine ? slot[u * ld4] : acc, acc);
                }
            }
        }
        cur = next;
        next = after;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!mine) return;
    float y[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
    for (int t = 0; t < 4; ++t)
        if (mean && 4 * lane + t < w) y[t] -= mean[r] * sums[4 * lane + t];
    reinterpret_cast<float4*>(Z)[r * ld4 + lane] = make_float4(y[0], y[1], y[2], y[3]);
}

// Partial Grams: block b sums, over its rows, groups of kGramRows rows' f32
// products added into f64 accumulators; entries (i, j), i <= j, row by row
// of the upper triangle.  A thread per 4 x 4 tile of entries, its sums in
// registers: two shared-memory reads per 16 products instead of two per
// product (30,000 x 74: 23 -> 21 us; what is left is the blocks' partials, a
// part per 50 rows, going out to memory).
__host__ __device__ constexpr int gram_tiles(int w) { return ((w + 3) / 4) * ((w + 3) / 4 + 1) / 2; }
constexpr int kGramThreads = (gram_tiles(kPcaMaxWidth) + 31) / 32 * 32;

__global__ void __launch_bounds__(kGramThreads)
    pca_gram_part_kernel(const float* __restrict__ Y, int64_t n, int w, int ld, int64_t rows_per_block,
                         double* __restrict__ part) {
    __shared__ float4 tile[kGramRows][kPcaMaxWidth / 4];
    const int entries = w * (w + 1) / 2, ld4 = ld / 4;
    // This thread's tile of entries: row block ib, column block jb >= ib.
    int ib = 0, rem = threadIdx.x;
    while (ib < ld4 && rem >= ld4 - ib) {
        rem -= ld4 - ib;
        ++ib;
    }
    const int jb = ib + rem;
    const bool mine = ib < ld4;
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    const int64_t r0 = (int64_t)blockIdx.x * rows_per_block;
    const int64_t r1 = min(n, r0 + rows_per_block);
    for (int64_t base = r0; base < r1; base += kGramRows) {
        const int rows = (int)min((int64_t)kGramRows, r1 - base);
        for (int t = threadIdx.x; t < rows * ld4; t += blockDim.x)
            tile[t / ld4][t % ld4] = reinterpret_cast<const float4*>(Y)[base * ld4 + t];
        __syncthreads();
        if (mine) {
            float s[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
            for (int r = 0; r < rows; ++r) {
                const float4 x4 = tile[r][ib], y4 = tile[r][jb];
                const float x[4] = {x4.x, x4.y, x4.z, x4.w}, y[4] = {y4.x, y4.y, y4.z, y4.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[i][j] = fmaf(x[i], y[j], s[i][j]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] += (double)s[i][j];
        }
        __syncthreads();
    }
    if (!mine) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gi = 4 * ib + i;
        const int64_t row = (int64_t)gi * w - (int64_t)gi * (gi - 1) / 2 - gi;  // entry (gi, j) at row + j
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gj = 4 * jb + j;
            if (gi < w && gj < w && gj >= gi) part[(int64_t)blockIdx.x * entries + row + gj] = acc[i][j];
        }
    }
}

// The blocks' partial Grams added up: 32 entries a block, each by eight
// threads over every eighth partial and then in a fixed order (a thread per
// entry over up to 608 partials waited 32 us).
constexpr int kGramFinalLanes = 8;
__global__ void __launch_bounds__(32 * kGramFinalLanes)
    pca_gram_final_kernel(const double* __restrict__ part, int blocks, int w, double* __restrict__ G) {
    __shared__ double sums[kGramFinalLanes][32];
    const int entries = w * (w + 1) / 2;
    const int t = blockIdx.x * 32 + threadIdx.x;
    double s = 0.0;
    if (t < entries) {
#pragma unroll 4
        for (int b = threadIdx.y; b < blocks; b += kGramFinalLanes) s += part[(int64_t)b * entries + t];
    }
    sums[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y || t >= entries) return;
#pragma unroll
    for (int y = 1; y < kGramFinalLanes; ++y) s += sums[y][threadIdx.x];
    int i = 0, rem = t;
    while (i < w && rem >= w - i) {
        rem -= w - i;
        ++i;
    }
    const int j = i + rem;
    G[i * w + j] = s;
    G[j * w + i] = s;
}

// T = L^-T of the shifted Cholesky factor of G (w x w, f64), as f32.  Every
// block factors G in its shared memory (right-looking: each entry still loses
// its products in the order of the columns), then a warp solves each of the
// block's columns of L^-1, its entries across the lanes.  Bound by f64 issue
// (a warp's f64 instruction holds its scheduler for 64 clocks): the trailing
// updates of one SM, the reciprocal root of every column in a row, and the
// solves, which are spread over kCholeskyBlocks SMs.  G is scaled by a power
// of two so that its largest diagonal entry lies in [1, 4), which no ratio
// sees; the reciprocal diagonal stands in for sqrt and divisions, and warp 0
// forms the next one while the others update the triangle.  At w = 74: 470 us
// when one thread summed every diagonal entry out of L2 and one thread solved
// each column; 148 us with a square root and divisions after every update;
// 75 us so.
constexpr int kCholeskyBlocks = 16;
constexpr int kCholeskyThreads = 512;
size_t cholesky_smem_bytes(int w) { return sizeof(double) * ((size_t)w * (w | 1) + 2 * (size_t)w); }

__global__ void __launch_bounds__(kCholeskyThreads)
    pca_cholesky_kernel(const double* __restrict__ G, int w, float* __restrict__ T, int* __restrict__ err) {
    extern __shared__ double csm[];
    __shared__ double shift, root_scale;
    const int ld = w | 1;
    double* A = csm;             // w x ld, the lower triangle
    double* col = csm + w * ld;  // the current column of L
    double* inv = col + w;       // reciprocal diagonal of L
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) {
        double mx = 0.0;
        for (int i = lane; i < w; i += 32) mx = fmax(mx, G[i * w + i]);
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) {
            // An even power of two, so that its root is one too.
            int ex = 1;
            if (mx > 0.0 && mx < 1e300) frexp(mx, &ex);
            ex = (ex - 1) / 2 - (ex - 1 < 0 && (ex - 1) % 2 != 0 ? 1 : 0);
            root_scale = ldexp(1.0, -ex);
            shift = mx > 0.0 ? kShift * mx * root_scale * root_scale : 1.0;
        }
    }
    __syncthreads();
    const double scale = root_scale * root_scale;
    for (int t = tid; t < w * w; t += kCholeskyThreads) {
        const int i = t / w, j = t % w;
        if (j <= i) A[i * ld + j] = G[t] * scale + (i == j ? shift : 0.0);
    }
    __syncthreads();
    auto pivot = [&](int k, double d) {  // warp 0
        if (!(d > 0.0)) {
            d = shift;
            if (lane == 0) atomicExch(err, 1);
        }
        const double y = rsqrt(d);
        if (lane == 0) inv[k] = y;
    };
    if (warp == 0) pivot(0, A[0]);
    __syncthreads();
    for (int k = 0; k < w; ++k) {
        const double inv_diag = inv[k];
        for (int i = k + 1 + tid; i < w; i += kCholeskyThreads) {
            const double v = A[i * ld + k] * inv_diag;
            A[i * ld + k] = v;
            col[i] = v;
        }
        __syncthreads();
        if (warp == 0) {
            if (k + 1 < w) pivot(k + 1, A[(k + 1) * ld + k + 1] - col[k + 1] * col[k + 1]);
        } else {
            // The rest of the trailing triangle, eight lanes a row.
            for (int i = k + 2 + (tid - 32) / 8; i < w; i += (kCholeskyThreads - 32) / 8) {
                const double li = col[i];
                for (int j = k + 1 + (tid & 7); j <= i; j += 8) A[i * ld + j] -= li * col[j];
            }
        }
        __syncthreads();
    }
    // x = column c of L^-1 by forward substitution, entry i in lane i % 32:
    // row c of L^-T (zero before c).
    for (int c = blockIdx.x + kCholeskyBlocks * warp; c < w; c += kCholeskyBlocks * (kCholeskyThreads / 32)) {
        double v[kPcaMaxWidth / 32], x[kPcaMaxWidth / 32];
#pragma unroll
        for (int t = 0; t < kPcaMaxWidth / 32; ++t) {
            v[t] = t * 32 + lane == c ? root_scale : 0.0;
            x[t] = 0.0;
        }
#pragma unroll
        for (int tr = 0; tr < kPcaMaxWidth / 32; ++tr) {
            for (int l = 0; l < 32; ++l) {
                const int r = tr * 32 + l;
                if (r < c) continue;
                if (r >= w) break;
                const double xr = __shfl_sync(0xffffffffu, v[tr], l) * inv[r];
                if (lane == l) x[tr] = xr;
#pragma unroll
                for (int t = tr; t < kPcaMaxWidth / 32; ++t) {
                    const int i = t * 32 + lane;
                    if (t * 32 < w && i > r && i < w) v[t] -= A[i * ld + r] * xr;
                }
            }
        }
#pragma unroll
        for (int t = 0; t < kPcaMaxWidth / 32; ++t)
            if (t * 32 + lane < w) T[c * w + t * 32 + lane] = (float)x[t];
    }
}

// Out (rows x m, ldo apart) = A (rows x w, lda apart) @ M (w x m); Out may be
// A itself when m = w.
// kMulRows rows of A and all of M in shared memory, a thread per 4 rows x 4
// columns, each output one chain of fused adds over w in order.  Bound by the
// shared-memory reads (5 for 16 fused adds): 32 products of 2,000 or 30,000
// rows by 74 x 74 take 0.7 ms, 1.4 ms with a warp per row and M through L1.
constexpr int kMulRows = 32;
constexpr int kMulThreads = 256;
size_t mul_smem_bytes(int w, int m) { return sizeof(float) * ((size_t)kMulRows * (w | 1) + (size_t)w * ((m + 3) / 4 * 4)); }

__global__ void __launch_bounds__(kMulThreads)
    pca_rows_mul_kernel(const float* A, int lda, int64_t rows, int w, const float* __restrict__ M, int m, float* out,
                        int ldo) {
    extern __shared__ float4 msm4[];
    const int mp = (m + 3) / 4 * 4, lds = w | 1;
    float* sM = reinterpret_cast<float*>(msm4);  // w x mp, zeros past m
    float* sA = sM + (size_t)w * mp;             // kMulRows x lds
    const int64_t r0 = (int64_t)blockIdx.x * kMulRows;
    const int here = (int)min((int64_t)kMulRows, rows - r0);
    for (int t = threadIdx.x; t < w * mp; t += kMulThreads) sM[t] = t % mp < m ? M[(t / mp) * m + t % mp] : 0.f;
    for (int t = threadIdx.x; t < kMulRows * w; t += kMulThreads)
        sA[(t / w) * lds + t % w] = t / w < here ? A[(r0 + t / w) * lda + t % w] : 0.f;
    __syncthreads();
    const int groups = mp / 4;
    for (int t = threadIdx.x; t < groups * (kMulRows / 4); t += kMulThreads) {
        const int jc = (t % groups) * 4, ir = (t / groups) * 4;
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 4
        for (int k = 0; k < w; ++k) {
            const float4 b = *reinterpret_cast<const float4*>(sM + k * mp + jc);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float x = sA[(ir + i) * lds + k];
                acc[i][0] = fmaf(x, b.x, acc[i][0]);
                acc[i][1] = fmaf(x, b.y, acc[i][1]);
                acc[i][2] = fmaf(x, b.z, acc[i][2]);
                acc[i][3] = fmaf(x, b.w, acc[i][3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (ir + i < here && jc + j < m) out[(r0 + ir + i) * ldo + jc + j] = acc[i][j];
    }
}

// Eigenpairs of the symmetric H (w x w, f64) by one-sided Jacobi rotations of
// its columns, the same rotations applied to the columns of V, the identity at
// first: at the end column j of V is the j-th eigenvector and its product with
// column j of the rotated H, H V, the eigenvalue (pca.rs:388-447 rotates H from
// both sides; the eigenpairs are the same).  A round rotates w / 2
// disjoint pairs, a warp each, over a cluster of kJacobiBlocks blocks; the
// columns pass through L2 between rounds.  A sweep of rounds meets every pair
// once.  A pair is done when its columns are orthogonal to f64 rounding, or
// when one of them is zero.
// (V stays orthonormal whatever H's columns are, and the sign of an eigenvalue
// is kept, which a column's norm loses.  With eigenvectors from the columns
// alone, and columns below 1e-13 of the trace left as they were, those past the
// rank lay along the leading ones: their loadings had norms of 1e6 and more.)
// Bound by the latency of a round, most of it f64 issue (64 clocks a warp
// instruction): so the squared norms are kept beside the columns and followed
// through the rotations (measured anew each sweep), the angle is taken in f32
// (a pair comes out orthogonal to 1e-7 instead of 1e-16, and the next sweep
// meets it again), and only the rotation's length is exact to f64.  One block
// rotating one pair after another took 55 ms at w = 74; this form with norms,
// angle and roots in f64 4.3 ms; with the angle in f32 2.2 ms; V adds 0.3 ms.
constexpr int kJacobiBlocks = 8;
constexpr int kJacobiThreads = 256;  // kJacobiBlocks * 8 warps: kPcaMaxWidth / 2 pairs
static_assert(kJacobiBlocks * kJacobiThreads / 32 * 2 >= kPcaMaxWidth, "a warp for every pair");

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// H: w x w, symmetric, so its rows serve as its columns; overwritten with the
// rotated columns (column j at H + j w), scaled by a power of two.  V: w x w,
// column j at V + j w.  lambda: w eigenvalues (between sweeps: squared norms).
// rotated: kJacobiSweeps flags, zero on entry.  root: w values of scratch.
// An eigenvalue below zero, or one that f32 cannot resolve, is 0 on return: the
// loadings B^T v / sqrt(lambda) are f32 sums of terms of up to
// |b_a| |v_a| / sqrt(lambda), b_a the rows of B, |b_a|^2 the diagonal of H, and
// where those come to 2^24 and more nothing of the unit vector they stand for
// is left (constant columns of 300 x 40: loadings of norm 2e5, and infinite ones).
__global__ void __cluster_dims__(kJacobiBlocks, 1, 1) __launch_bounds__(kJacobiThreads)
    pca_jacobi_kernel(double* H, double* V, int w, double* lambda, double* root, int* rotated, int* __restrict__ err) {
    constexpr int SLOTS = kPcaMaxWidth / 32;
    constexpr int WARPS = kJacobiBlocks * kJacobiThreads / 32;
    constexpr double EPS = 2.220446049250313e-16;
    const int lane = threadIdx.x & 31;
    const int slot = (int)(blockIdx.x * kJacobiThreads + threadIdx.x) >> 5;
    const int players = w + (w & 1);  // odd: one column sits out each round
    // The trace, no smaller than the largest eigenvalue, brought into
    // [1/2, 1), so that squares of norms stay inside the f32 range.
    double trace = 0.0;
    for (int i = lane; i < w; i += 32) trace += fabs(__ldcg(H + (int64_t)i * w + i));
    trace = warp_sum(trace);
    int ex = 0;
    if (trace > 0.0 && trace < 1e300) frexp(trace, &ex);
    const double scale = ldexp(1.0, -ex);
    cluster_barrier();  // everyone has read the diagonal
    for (int c = slot; c < w; c += WARPS)
        for (int i = lane; i < w; i += 32) {
            const double h = __ldcg(H + (int64_t)c * w + i);
            if (i == c) __stcg(root + c, sqrt(fmax(h, 0.0)));
            __stcg(H + (int64_t)c * w + i, h * scale);
            __stcg(V + (int64_t)c * w + i, i == c ? 1.0 : 0.0);
        }
    // Orthogonal: to 16 roundings, whatever the columns' sizes (the Gram of a
    // graded basis holds its small eigenvalues to as many digits as the large
    // ones).  Zero: a column whose squared norm leaves f64's range.
    constexpr double ORTHO2 = (16 * EPS) * (16 * EPS), TINY2 = 1e-280;
    int sweep = 0;
    bool done = w < 2;
    auto norms = [&]() {  // each column's squared norm, by the warp that owns it
        for (int c = slot; c < w; c += WARPS) {
            double s = 0.0;
            for (int i = lane; i < w; i += 32) {
                const double v = __ldcg(H + (int64_t)c * w + i);
                s += v * v;
            }
            s = warp_sum(s);
            if (lane == 0) __stcg(lambda + c, s);
        }
    };
    for (; sweep < kJacobiSweeps && !done; ++sweep) {
        norms();
        cluster_barrier();
        for (int round = 0; round < players - 1; ++round) {
            if (slot < players / 2) {
                const int a = slot == 0 ? players - 1 : (round + slot) % (players - 1);
                const int b = (round - slot + players - 1) % (players - 1);
                const int p = min(a, b), q = max(a, b);
                if (q < w) {
                    double x[SLOTS], y[SLOTS], vx[SLOTS], vy[SLOTS];
                    const double pp = __ldcg(lambda + p), qq = __ldcg(lambda + q);
#pragma unroll
                    for (int t = 0; t < SLOTS; ++t) {
                        const int i = t * 32 + lane;
                        x[t] = i < w ? __ldcg(H + (int64_t)p * w + i) : 0.0;
                        y[t] = i < w ? __ldcg(H + (int64_t)q * w + i) : 0.0;
                        vx[t] = i < w ? __ldcg(V + (int64_t)p * w + i) : 0.0;
                        vy[t] = i < w ? __ldcg(V + (int64_t)q * w + i) : 0.0;
                    }
                    double pq = 0.0;
#pragma unroll
                    for (int t = 0; t < SLOTS; ++t)
                        if (t * 32 < w) pq += x[t] * y[t];
                    pq = warp_sum(pq);
                    // (A NaN fails every comparison and keeps rotating, so it
                    // ends as not converged.)
                    if (!(pq * pq <= ORTHO2 * pp * qq) && !(fmin(pp, qq) <= TINY2)) {
                        // By the power of two that brings the larger norm near
                        // one (its exponent negated), so that the f32 quotient
                        // of two small columns is in range.
                        const int top = __double2hiint(fmax(pp, qq)) & 0x7ff00000;
                        const double near_one = __hiloint2double(0x7fe00000 - top, 0);
                        const float theta = (float)((qq - pp) * near_one) / (float)(2.0 * pq * near_one);
                        // (Past 1e6 the root is theta itself to f32, and theta^2
                        // may be out of range; past 1e30 the product of the
                        // columns may be, and the tangent is 1 / (2 theta).)
                        const float root = fabsf(theta) > 1e6f ? fabsf(theta) : sqrtf(fmaf(theta, theta, 1.f));
                        const double tangent = fabsf(theta) > 1e30f
                                                   ? pq / (qq - pp)
                                                   : (double)((theta < 0.f ? -1.f : 1.f) / (fabsf(theta) + root));
                        const double cs = rsqrt(fma(tangent, tangent, 1.0)), sn = tangent * cs;
#pragma unroll
                        for (int t = 0; t < SLOTS; ++t) {
                            const int i = t * 32 + lane;
                            if (i < w) {
                                __stcg(H + (int64_t)p * w + i, cs * x[t] - sn * y[t]);
                                __stcg(H + (int64_t)q * w + i, sn * x[t] + cs * y[t]);
                                __stcg(V + (int64_t)p * w + i, cs * vx[t] - sn * vy[t]);
                                __stcg(V + (int64_t)q * w + i, sn * vx[t] + cs * vy[t]);
                            }
                        }
                        if (lane == 0) {
                            __stcg(lambda + p, pp - tangent * pq);
                            __stcg(lambda + q, qq + tangent * pq);
                            atomicExch(rotated + sweep, 1);
                        }
                    }
                }
            }
            cluster_barrier();
        }
        done = __ldcg(rotated + sweep) == 0;
    }
    if (!done && blockIdx.x == 0 && threadIdx.x == 0) atomicExch(err, 2);
    const double back = ldexp(1.0, ex);
    for (int c = slot; c < w; c += WARPS) {
        double l = 0.0, terms = 0.0;
        for (int i = lane; i < w; i += 32) {
            const double v = __ldcg(V + (int64_t)c * w + i);
            l += v * __ldcg(H + (int64_t)c * w + i);
            terms += fabs(v) * __ldcg(root + i);
        }
        l = warp_sum(l) * back;
        terms = warp_sum(terms) * 5.9604644775390625e-8;  // 2^-24
        if (lane == 0) __stcg(lambda + c, l >= terms * terms && l >= 1.1754943508222875e-38 ? l : 0.0);  // f32's smallest
    }
}

// From the eigenpairs of H = B B^T (w x w; column j of V, w apart, is
// eigenvector j): the n_components largest, their singular values, and
// the two small matrices the outputs are built from: basis[:, j] = v_j * s_j
// (embedding = Q @ basis), scaled[:, j] = v_j / s_j (components^T = B^T @
// scaled).  A warp per eigenpair, placed by how many come before it.
__global__ void pca_select_kernel(const double* __restrict__ lambda, const double* __restrict__ V, int w, int nc,
                                  float* __restrict__ basis, float* __restrict__ scaled, double* __restrict__ sing) {
    const int lane = threadIdx.x & 31;
    const int idx = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (idx >= w) return;
    const double l = lambda[idx];
    int before = 0;  // eigenvalues that come first: larger, or equal and earlier
    for (int i = lane; i < w; i += 32) before += lambda[i] > l || (lambda[i] == l && i < idx);
    const int c = __reduce_add_sync(0xffffffffu, before);
    if (c >= nc) return;
    const double s = sqrt(l);
    if (lane == 0) sing[c] = s;
    const double inv = s > 0.0 ? 1.0 / s : 0.0;
    for (int r = lane; r < w; r += 32) {
        const double e = V[(int64_t)idx * w + r];
        basis[r * nc + c] = (float)(e * s);
        scaled[r * nc + c] = (float)(e * inv);
    }
}

// components (nc x g) from components^T (g x nc); the sign fix of
// pca.rs:497-519: the first largest-magnitude loading of each component is
// made positive (and its embedding column flipped with it).  One block per
// component.
__global__ void __launch_bounds__(kSumThreads)
    pca_signs_kernel(const float* __restrict__ ct, int64_t g, int nc, int* __restrict__ flip) {
    __shared__ float val[kSumThreads];
    __shared__ int64_t at[kSumThreads];
    const int c = blockIdx.x, tid = threadIdx.x;
    float extreme = 0.f;
    int64_t first = g;
    for (int64_t k = tid; k < g; k += kSumThreads) {
        const float v = ct[k * nc + c];
        if (fabsf(v) > fabsf(extreme)) {
            extreme = v;
            first = k;
        }
    }
    val[tid] = extreme;
    at[tid] = first;
    __syncthreads();
    for (int o = kSumThreads / 2; o > 0; o >>= 1) {
        if (tid < o) {
            const float x = fabsf(val[tid]), y = fabsf(val[tid + o]);
            if (y > x || (y == x && at[tid + o] < at[tid])) {
                val[tid] = val[tid + o];
                at[tid] = at[tid + o];
            }
        }
        __syncthreads();
    }
    if (tid == 0) flip[c] = val[0] < 0.f ? 1 : 0;
}

__global__ void pca_finish_kernel(const float* __restrict__ ct, int64_t g, int nc, const int* __restrict__ flip,
                                  float* __restrict__ components, float* __restrict__ emb, int64_t n) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < g * nc) {
        const int64_t k = t / nc;
        const int c = (int)(t % nc);
        const float v = ct[t];
        components[(int64_t)c * g + k] = flip[c] ? -v : v;
    }
    if (t < n * nc) {
        const int c = (int)(t % nc);
        if (flip[c]) emb[t] = -emb[t];
    }
}

// Explained variance: S^2 / (n - 1) centred, else each score column's
// population variance (f64); ratios over the total variance.  One block per
// component.
__global__ void __launch_bounds__(kSumThreads)
    pca_variance_kernel(const double* __restrict__ sing, const float* __restrict__ emb, int64_t n, int nc, int centred,
                        const double* __restrict__ total, float* __restrict__ var, float* __restrict__ ratio) {
    __shared__ double part[kSumThreads];
    const int c = blockIdx.x;
    float v;
    if (centred) {
        v = (float)(sing[c] * sing[c] / (double)(n - 1));
    } else {
        double m = 0.0;
        for (int64_t r = threadIdx.x; r < n; r += kSumThreads) m += (double)emb[r * nc + c];
        m = block_sum(m, part) / (double)n;
        double s = 0.0;
        for (int64_t r = threadIdx.x; r < n; r += kSumThreads) {
            const double d = (double)emb[r * nc + c] - m;
            s += d * d;
        }
        v = (float)(block_sum(s, part) / (double)n);
    }
    if (threadIdx.x) return;
    var[c] = v;
    ratio[c] = total[0] > 0.0 ? (float)((double)v / total[0]) : 0.f;
}

size_t al(size_t v) { return (v + 255) & ~(size_t)255; }

struct PcaWork {
    float *omega, *Y, *Z, *mvec, *colsum, *mean, *T, *basis, *scaled, *ct;
    double *var_term, *total, *gram_part, *G, *V, *lambda, *root, *sing, *colpart;
    uint32_t *kA, *kB, *cstart;
    unsigned long long *vA, *vB;
    uint32_t *hist, *scan;
    size_t scan_elems;
    int* flip;
    const uint32_t* ckeys;
    const unsigned long long* cvals;
};

}  // namespace

int32_t pca_device_impl(scrust_context* ctx, const uint32_t* indptr, const uint32_t* indices, const float* values,
                        int64_t n, int64_t g, int64_t nnz, int nc, bool zero_center, uint64_t seed, float* emb,
                        float* components, float* variance, float* ratio, scrust_status* st) {
    cudaStream_t s = ctx->stream;
    cudaError_t e = cudaSuccess;
    const int64_t maxc = std::min(n, g);
    const int w = (int)std::min<int64_t>(nc + kOversampling, maxc);
    const int ld = (w + 3) / 4 * 4;  // floats between rows of the sketch and the bases, zeros past w
    const int entries = w * (w + 1) / 2;
    // A Gram over `rows` rows runs ceil(rows / max(32, ceil(rows / 4S))) <= 4S
    // blocks (S = SMs).
    const int gram_blocks = 4 * ctx->sm_count;
    const int col_blocks = (int)((n + kColRows - 1) / kColRows);
    const int nb = radix_blocks(std::max<int64_t>(nnz, 1));
    PcaWork wk;
    wk.scan_elems = scan_scratch_elems((int64_t)256 * nb);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t r = off;
        off = al(off + bytes);
        return r;
    };
    const size_t o_om = take(4 * (size_t)g * ld), o_y = take(4 * (size_t)n * ld), o_z = take(4 * (size_t)g * ld),
                 o_mv = take(4 * (size_t)w), o_cs = take(4 * (size_t)w), o_mean = take(4 * (size_t)g),
                 o_t = take(4 * (size_t)w * w), o_basis = take(4 * (size_t)w * nc), o_sc = take(4 * (size_t)w * nc),
                 o_ct = take(4 * (size_t)g * nc), o_vt = take(8 * (size_t)g), o_tot = take(8),
                 o_gp = take(8 * (size_t)gram_blocks * entries), o_g = take(8 * (size_t)w * w),
                 o_v = take(8 * (size_t)w * w), o_lam = take(8 * (size_t)w), o_root = take(8 * (size_t)w), o_sing = take(8 * (size_t)nc),
                 o_cp = take(8 * (size_t)col_blocks * w), o_ka = take(4 * (size_t)nnz), o_kb = take(4 * (size_t)nnz),
                 o_cst = take(4 * (size_t)(g + 1)), o_va = take(8 * (size_t)nnz), o_vb = take(8 * (size_t)nnz),
                 o_hist = take(4 * ((size_t)256 * nb + 16)), o_scan = take(4 * wk.scan_elems),
                 o_flip = take(4 * ((size_t)nc + 1 + kJacobiSweeps));
    char* base = (char*)ws_get(ctx, SLOT_PCA, off, &e);
    if (!base) return cuda_fail(st, e, "pca: workspace");
    wk.omega = (float*)(base + o_om);
    wk.Y = (float*)(base + o_y);
    wk.Z = (float*)(base + o_z);
    wk.mvec = (float*)(base + o_mv);
    wk.colsum = (float*)(base + o_cs);
    wk.mean = (float*)(base + o_mean);
    wk.T = (float*)(base + o_t);
    wk.basis = (float*)(base + o_basis);
    wk.scaled = (float*)(base + o_sc);
    wk.ct = (float*)(base + o_ct);
    wk.var_term = (double*)(base + o_vt);
    wk.total = (double*)(base + o_tot);
    wk.gram_part = (double*)(base + o_gp);
    wk.G = (double*)(base + o_g);
    wk.V = (double*)(base + o_v);
    wk.lambda = (double*)(base + o_lam);
    wk.root = (double*)(base + o_root);
    wk.sing = (double*)(base + o_sing);
    wk.colpart = (double*)(base + o_cp);
    wk.kA = (uint32_t*)(base + o_ka);
    wk.kB = (uint32_t*)(base + o_kb);
    wk.cstart = (uint32_t*)(base + o_cst);
    wk.vA = (unsigned long long*)(base + o_va);
    wk.vB = (unsigned long long*)(base + o_vb);
    wk.hist = (uint32_t*)(base + o_hist);
    wk.scan = (uint32_t*)(base + o_scan);
    wk.flip = (int*)(base + o_flip);
    int* err = wk.flip + nc;  // after the nc sign flags
    int* rotated = err + 1;   // per Jacobi sweep
    if ((e = cudaMemsetAsync(err, 0, sizeof(int) * (1 + kJacobiSweeps), s)) != cudaSuccess ||
        (e = cudaMemsetAsync(wk.omega, 0, sizeof(float) * (size_t)g * ld, s)) != cudaSuccess)
        return cuda_fail(st, e, "pca: memset");
    uint64_t launches = 0;
    // The CSC copy: entries sorted by gene, rows ascending within a gene.
    pca_csc_keys_kernel<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(indptr, indices, values, n, wk.kA, wk.vA);
    int bits = 1;
    while (((int64_t)1 << bits) <= g) bits++;
    uint32_t* ckeys = nullptr;
    unsigned long long* cvals = nullptr;
    if ((e = radix_sort_pairs(ctx, wk.kA, wk.vA, wk.kB, wk.vB, nnz, bits, wk.hist, wk.scan, wk.scan_elems, &ckeys,
                              &cvals)) != cudaSuccess)
        return cuda_fail(st, e, "pca: transpose");
    pca_starts_kernel<<<(unsigned)((nnz + 1 + 255) / 256), 256, 0, s>>>(ckeys, nnz, g, wk.cstart);
    pca_column_stats_kernel<<<(unsigned)g, kSumThreads, 0, s>>>(wk.cstart, cvals, n, zero_center ? 1.0 : 0.0, wk.mean,
                                                                wk.var_term);
    pca_sum_kernel<<<1, 256, 0, s>>>(wk.var_term, g, wk.total);
    launches += 5;
    const unsigned cell_warps = (unsigned)((n * 32 + 127) / 128), gene_blocks = (unsigned)((g + kSpmmTWarps - 1) / kSpmmTWarps);
    const size_t chol_smem = cholesky_smem_bytes(w), spmm_t_smem = spmm_t_smem_bytes(ld), mul_smem = mul_smem_bytes(w, std::max(w, nc));
    if ((e = set_smem_limit(ctx, (const void*)pca_cholesky_kernel, (int)chol_smem)) != cudaSuccess ||
        (e = set_smem_limit(ctx, (const void*)pca_spmm_t_kernel, (int)spmm_t_smem)) != cudaSuccess ||
        (e = set_smem_limit(ctx, (const void*)pca_rows_mul_kernel, (int)mul_smem)) != cudaSuccess)
        return cuda_fail(st, e, "pca: shared memory");
    // out (rows ldo apart) = A @ M (A rows x w, M w x m)
    auto rows_mul = [&](const float* A, int64_t rows, const float* M, int m, float* out, int ldo) {
        pca_rows_mul_kernel<<<(unsigned)((rows + kMulRows - 1) / kMulRows), kMulThreads, mul_smem_bytes(w, m), s>>>(
            A, ld, rows, w, M, m, out, ldo);
    };
    const float* mean = zero_center ? wk.mean : nullptr;
    // X_c @ B into Y
    auto times = [&](const float* B, float* Y) -> cudaError_t {
        if (mean) {
            pca_mean_row_kernel<<<w, kSumThreads, 0, s>>>(wk.mean, B, g, ld, wk.mvec);
            launches += 1;
        }
        pca_spmm_kernel<<<cell_warps, 128, 0, s>>>(indptr, indices, values, n, B, w, ld, mean ? wk.mvec : nullptr, Y);
        launches += 1;
        return cudaGetLastError();
    };
    // X_c^T @ U into Z
    auto transpose_times = [&](const float* U, float* Z) -> cudaError_t {
        if (mean) {
            pca_colsum_part_kernel<<<col_blocks, 128, 0, s>>>(U, n, w, ld, wk.colpart);
            pca_colsum_final_kernel<<<w, kSumThreads, 0, s>>>(wk.colpart, col_blocks, w, wk.colsum);
            launches += 2;
        }
        pca_spmm_t_kernel<<<gene_blocks, kSpmmTWarps * 32, spmm_t_smem, s>>>(wk.cstart, cvals, g, U, w, ld,
                                                                             mean ? wk.mean : nullptr, wk.colsum, Z);
        launches += 1;
        return cudaGetLastError();
    };
    auto gram = [&](const float* Y, int64_t rows) -> cudaError_t {
        const int64_t rpb = std::max<int64_t>(kGramRows, (rows + 4 * ctx->sm_count - 1) / (4 * ctx->sm_count));
        const int blocks = (int)((rows + rpb - 1) / rpb);
        pca_gram_part_kernel<<<blocks, (gram_tiles(w) + 31) / 32 * 32, 0, s>>>(Y, rows, w, ld, rpb, wk.gram_part);
        pca_gram_final_kernel<<<(entries + 31) / 32, dim3(32, kGramFinalLanes), 0, s>>>(wk.gram_part, blocks, w, wk.G);
        launches += 2;
        return cudaGetLastError();
    };
    auto orthonormalize = [&](float* Y, int64_t rows) -> cudaError_t {
        for (int pass = 0; pass < 2; ++pass) {
            cudaError_t e2 = gram(Y, rows);
            if (e2 != cudaSuccess) return e2;
            pca_cholesky_kernel<<<kCholeskyBlocks, kCholeskyThreads, chol_smem, s>>>(wk.G, w, wk.T, err);
            rows_mul(Y, rows, wk.T, w, Y, ld);
            launches += 2;
            if ((e2 = cudaGetLastError()) != cudaSuccess) return e2;
        }
        return cudaSuccess;
    };
    pca_gaussian_kernel<<<(unsigned)(((g * w + 1) / 2 + 255) / 256), 256, 0, s>>>(g * w, w, ld, seed, wk.omega);
    launches += 1;
    if ((e = times(wk.omega, wk.Y)) != cudaSuccess || (e = orthonormalize(wk.Y, n)) != cudaSuccess)
        return cuda_fail(st, e, "pca: sketch");
    const int power = (double)nc < 0.1 * (double)maxc ? 7 : 4;
    for (int it = 0; it < power; ++it) {
        if ((e = transpose_times(wk.Y, wk.Z)) != cudaSuccess || (e = orthonormalize(wk.Z, g)) != cudaSuccess ||
            (e = times(wk.Z, wk.Y)) != cudaSuccess || (e = orthonormalize(wk.Y, n)) != cudaSuccess)
            return cuda_fail(st, e, "pca: power iteration");
    }
    // B^T = X_c^T Q (g x w), its Gram, the eigenpairs, the outputs.
    if ((e = transpose_times(wk.Y, wk.Z)) != cudaSuccess || (e = gram(wk.Z, g)) != cudaSuccess)
        return cuda_fail(st, e, "pca: projection");
    pca_jacobi_kernel<<<kJacobiBlocks, kJacobiThreads, 0, s>>>(wk.G, wk.V, w, wk.lambda, wk.root, rotated, err);
    pca_select_kernel<<<(w + 7) / 8, 256, 0, s>>>(wk.lambda, wk.V, w, nc, wk.basis, wk.scaled, wk.sing);
    rows_mul(wk.Y, n, wk.basis, nc, emb, nc);
    rows_mul(wk.Z, g, wk.scaled, nc, wk.ct, nc);
    pca_signs_kernel<<<nc, kSumThreads, 0, s>>>(wk.ct, g, nc, wk.flip);
    const int64_t span = std::max(g, n) * nc;
    pca_finish_kernel<<<(unsigned)((span + 255) / 256), 256, 0, s>>>(wk.ct, g, nc, wk.flip, components, emb, n);
    pca_variance_kernel<<<nc, kSumThreads, 0, s>>>(wk.sing, emb, n, nc, zero_center ? 1 : 0, wk.total, variance,
                                                     ratio);
    launches += 7;
    ctx->launches += launches;
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(st, e, "pca");
    int herr = 0;
    if ((e = cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return cuda_fail(st, e, "pca: synchronise");
    if (herr == 2)
        return fail(st, SCRUST_NOT_CONVERGED, "Jacobi eigenvalue iteration did not converge in %d sweeps", kJacobiSweeps);
    return ok(st);
}

}  // namespace scrust

using namespace scrust;

namespace {

int32_t check_pca(uint64_t n, uint64_t g, uint32_t nc, scrust_status* st) {
    const uint64_t maxc = std::min(n, g);
    if (nc == 0) return fail(st, SCRUST_INVALID_PARAMETER, "n_components must be at least 1, got 0");
    if (nc > maxc)
        return fail(st, SCRUST_INVALID_PARAMETER, "n_components must be at most min(n_cells, n_genes), got %u", nc);
    if (n < 2) return fail(st, SCRUST_INVALID_PARAMETER, "n_cells must be at least 2, got %llu", (unsigned long long)n);
    if (nc + kOversampling > (uint32_t)kPcaMaxWidth && nc > (uint32_t)(kPcaMaxWidth - kOversampling))
        return fail(st, SCRUST_INVALID_PARAMETER, "n_components must be at most %d, got %u", kPcaMaxWidth - kOversampling,
                    nc);
    if (n >= 0xffffff00ull || g >= 0xffffff00ull) return fail(st, SCRUST_SHAPE, "expected fewer than 2^32 cells and genes");
    return SCRUST_OK;
}

}  // namespace

extern "C" {

int32_t scrust_cuda_pca_device(scrust_context* ctx, const uint32_t* indptr, const uint32_t* indices,
                               const float* values, uint64_t n_cells, uint64_t n_genes, uint64_t nnz,
                               uint32_t n_components, int32_t zero_center, uint64_t seed, float* out_embedding,
                               float* out_components, float* out_variance, float* out_variance_ratio,
                               scrust_status* st) {
    int32_t rc = check_pca(n_cells, n_genes, n_components, st);
    if (rc) return rc;
    if (nnz >= 0xffffff00ull) return fail(st, SCRUST_SHAPE, "expected fewer than 2^32 stored entries");
    if (!ctx) return fail(st, SCRUST_NO_GPU, "no CUDA context (no usable GPU)");
    if (!indptr || (nnz && (!indices || !values)) || !out_embedding || !out_components || !out_variance ||
        !out_variance_ratio)
        return fail(st, SCRUST_SHAPE, "expected non-null pointers");
    std::lock_guard<std::mutex> lock(ctx->mu);
    DeviceGuard device_guard(ctx->device);
    return pca_device_impl(ctx, indptr, indices, values, (int64_t)n_cells, (int64_t)n_genes, (int64_t)nnz,
                           (int)n_components, zero_center != 0, seed, out_embedding, out_components, out_variance,
                           out_variance_ratio, st);
}

int32_t scrust_cuda_pca(scrust_context* ctx, const uint32_t* indptr, const uint32_t* indices, const float* values,
                        uint64_t n_cells, uint64_t n_genes, uint32_t n_components, int32_t zero_center, uint64_t seed,
                        float* out_embedding, float* out_components, float* out_variance, float* out_variance_ratio,
                        scrust_status* st) {
    int32_t rc = check_pca(n_cells, n_genes, n_components, st);
    if (rc) return rc;
    if (!indptr || !out_embedding || !out_components || !out_variance || !out_variance_ratio)
        return fail(st, SCRUST_SHAPE, "expected non-null pointers");
    const uint64_t nnz = indptr[n_cells];
    if (nnz && (!indices || !values)) return fail(st, SCRUST_SHAPE, "expected non-null pointers");
    // CsrMatrix::new's structural checks (crates/scrust-core/src/sparse.rs:18-90).
    if (indptr[0] != 0) return fail(st, SCRUST_SHAPE, "expected indptr to start at 0");
    for (uint64_t r = 0; r < n_cells; ++r)
        if (indptr[r + 1] < indptr[r]) return fail(st, SCRUST_SHAPE, "expected a non-decreasing indptr");
    for (uint64_t i = 0; i < nnz; ++i)
        if (indices[i] >= n_genes)
            return fail(st, SCRUST_SHAPE, "expected column indices below %llu", (unsigned long long)n_genes);
    if (nnz >= 0xffffff00ull) return fail(st, SCRUST_SHAPE, "expected fewer than 2^32 stored entries");
    if (!ctx) return fail(st, SCRUST_NO_GPU, "no CUDA context (no usable GPU)");
    std::lock_guard<std::mutex> lock(ctx->mu);
    DeviceGuard device_guard(ctx->device);
    cudaError_t e;
    const uint32_t nc = n_components;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t r = off;
        off = (off + bytes + 255) & ~(size_t)255;
        return r;
    };
    const size_t o_ip = take(4 * (n_cells + 1)), o_ix = take(4 * std::max<uint64_t>(nnz, 1)),
                 o_vl = take(4 * std::max<uint64_t>(nnz, 1)), o_emb = take(4 * n_cells * nc),
                 o_cmp = take(4 * n_genes * nc), o_var = take(4 * nc), o_rat = take(4 * nc);
    char* buf = (char*)ws_get(ctx, SLOT_HOST_IN, off, &e);
    if (!buf) return cuda_fail(st, e, "workspace");
    if ((e = cudaMemcpyAsync(buf + o_ip, indptr, 4 * (n_cells + 1), cudaMemcpyHostToDevice, ctx->stream)) !=
            cudaSuccess ||
        (nnz && (e = cudaMemcpyAsync(buf + o_ix, indices, 4 * nnz, cudaMemcpyHostToDevice, ctx->stream)) != cudaSuccess) ||
        (nnz && (e = cudaMemcpyAsync(buf + o_vl, values, 4 * nnz, cudaMemcpyHostToDevice, ctx->stream)) != cudaSuccess))
        return cuda_fail(st, e, "upload");
    if ((rc = pca_device_impl(ctx, (const uint32_t*)(buf + o_ip), (const uint32_t*)(buf + o_ix),
                              (const float*)(buf + o_vl), (int64_t)n_cells, (int64_t)n_genes, (int64_t)nnz, (int)nc,
                              zero_center != 0, seed, (float*)(buf + o_emb), (float*)(buf + o_cmp),
                              (float*)(buf + o_var), (float*)(buf + o_rat), st)))
        return rc;
    if ((e = cudaMemcpyAsync(out_embedding, buf + o_emb, 4 * n_cells * nc, cudaMemcpyDeviceToHost, ctx->stream)) !=
            cudaSuccess ||
        (e = cudaMemcpyAsync(out_components, buf + o_cmp, 4 * n_genes * nc, cudaMemcpyDeviceToHost, ctx->stream)) !=
            cudaSuccess ||
        (e = cudaMemcpyAsync(out_variance, buf + o_var, 4 * nc, cudaMemcpyDeviceToHost, ctx->stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(out_variance_ratio, buf + o_rat, 4 * nc, cudaMemcpyDeviceToHost, ctx->stream)) !=
            cudaSuccess)
        return cuda_fail(st, e, "download");
    return collect_device_errors(ctx, st);
}

}  // extern "C"
