// prep.cu -- per-row preparation before candidate generation.
//
//   column means     f64, as crates/scrust-core/src/neighbors.rs:144-154 forms
//                    them (the sequential variant reproduces that order bit for
//                    bit; the parallel one is a deterministic two-level sum)
//   normalise rows   cosine metric: rows divided by their FP64 norm
//   centre/transpose centred f32 coordinates, (D_pad x n_pad) for the plain
//                    form's TMA tiles, squared norms by an fma chain
//                    (crates/scrust-gpu/src/kernels/knn.rs:148-155) and the
//                    largest centred norm
//   margins          per-row candidate margin from the derived error bound
//
// All kernels here are HBM-bound single passes over n x D floats.
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace scrust {

namespace {

constexpr int kMeanRowsPerBlock = 2048;

__global__ void means_sequential_kernel(const float* __restrict__ x, int64_t n, int d,
                                        double* __restrict__ means) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= d) return;
    double s = 0.0;
    for (int64_t r = 0; r < n; r++) s = __dadd_rn(s, (double)__ldg(x + r * d + c));
    means[c] = __ddiv_rn(s, (double)n);
}

__global__ void means_partial_kernel(const float* __restrict__ x, int64_t n, int d,
                                     double* __restrict__ partial) {
    int64_t r0 = (int64_t)blockIdx.x * kMeanRowsPerBlock;
    int64_t r1 = min(n, r0 + kMeanRowsPerBlock);
    for (int c = threadIdx.x; c < d; c += blockDim.x) {
        double s = 0.0;
        for (int64_t r = r0; r < r1; r++) s = __dadd_rn(s, (double)__ldg(x + r * d + c));
        partial[(int64_t)blockIdx.x * d + c] = s;
    }
}

__global__ void means_final_kernel(const double* __restrict__ partial, int blocks, int64_t n, int d,
                                   double* __restrict__ means) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= d) return;
    double s = 0.0;
    for (int b = 0; b < blocks; b++) s = __dadd_rn(s, partial[(int64_t)b * d + c]);
    means[c] = __ddiv_rn(s, (double)n);
}

__global__ void normalise_wide_rows_kernel(const float* __restrict__ x, int64_t n, int d,
                                      float* __restrict__ xn, double* __restrict__ norm64,
                                      int* __restrict__ err) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* row = x + i * d;
    double s = 0.0;
    for (int t = 0; t < d; t++) {
        double v = (double)__ldg(row + t);
        s = __dadd_rn(s, __dmul_rn(v, v));
    }
    double nrm = sqrt(s);
    norm64[i] = nrm;
    if (!(nrm > 0.0)) {
        atomicExch(err + DERR_ZERO_ROW, 1);
        nrm = 1.0;
    }
    for (int t = 0; t < d; t++) xn[i * d + t] = __double2float_rn(__ddiv_rn((double)__ldg(row + t), nrm));
}

// f32 to f64, the conversion by its bits: CUDA's instruction is an f64-rate
// one.  (Zeros, subnormals and non-finite values take it.)
__device__ __forceinline__ double widen(float v) {
    const uint32_t u = __float_as_uint(v), e = u & 0x7f800000u;
    if (e == 0u || e == 0x7f800000u) return (double)v;
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
}

// Rows of up to kCosineMaxDims dimensions, NR_ROWS a block, staged in shared
// memory: FP64 norms by one thread a row in the row's order (a product of two
// floats is exact in f64, so the multiply-add rounds as product and sum do);
// then element by element the quotient x / norm, in f32 from the reciprocal as
// a sum of two floats where that rounds surely, else in f64; and the row's
// padded copy.  Both values are the bits of the f64 forms.  30,011 rows of 50:
// 49 us with a thread a row, f64 throughout and rows read at a stride (16
// f64-rate instructions an element, 64 clocks a warp each), 19 us here.
constexpr int NR_ROWS = 64;
__global__ void __launch_bounds__(256) normalise_rows_kernel(const float* __restrict__ x, int64_t n, int d,
                                                             float* __restrict__ xn, double* __restrict__ norm64,
                                                             float2* __restrict__ inverse, float* __restrict__ raw,
                                                             int raw_stride, int* __restrict__ err) {
    extern __shared__ float nr_rows[];
    __shared__ float2 inv_s[NR_ROWS];
    __shared__ double norm_s[NR_ROWS];
    const int tid = threadIdx.x, stride = d | 1;
    const int64_t first = (int64_t)blockIdx.x * NR_ROWS;
    const int rows = (int)min((int64_t)NR_ROWS, n - first);
#pragma unroll 4
    for (int e = tid; e < rows * d; e += 256) nr_rows[(e / d) * stride + e % d] = __ldg(x + first * d + e);
    __syncthreads();
    if (tid < rows) {
        const float* row = nr_rows + tid * stride;
        double s = 0.0;
#pragma unroll 4
        for (int t = 0; t < d; t++) {
            const double v = widen(row[t]);
            s = __fma_rn(v, v, s);
        }
        double nrm = sqrt(s);
        norm64[first + tid] = nrm;
        if (!(nrm > 0.0)) {
            atomicExch(err + DERR_ZERO_ROW, 1);
            nrm = 1.0;
        }
        norm_s[tid] = nrm;
        float2 inv = make_float2(__int_as_float(0x7fc00000), 0.f);
        if (nrm >= 9.094947017729282e-13 && nrm <= 1.152921504606847e18) {  // [2^-40, 2^60]
            const double r = 1.0 / nrm;
            inv.x = __double2float_rn(r);
            inv.y = __double2float_rn(r - (double)inv.x);
        }
        inv_s[tid] = inv;
        inverse[first + tid] = inv;
    }
    __syncthreads();
    for (int e = tid; e < rows * d; e += 256) {
        const int i = e / d;
        const float v = nr_rows[i * stride + e % d];
        const float2 inv = inv_s[i];
        // v / norm = h + l within 2^-45 of it: one exact product, two roundings
        // of its error term and the reciprocal's own.
        const float p = __fmul_rn(v, inv.x);
        const float r = __fmaf_rn(v, inv.y, __fmaf_rn(v, inv.x, -p));
        const float h = __fadd_rn(p, r), l = __fsub_rn(r, __fsub_rn(h, p));
        const float size = fabsf(h);
        float q = h;
        if (v != 0.f && !(size >= 7.8886091e-31f && rounds_surely(h, l, size * 5.6843419e-14f)))  // 2^-100, 2^-44
            q = __double2float_rn(__ddiv_rn((double)v, norm_s[i]));
        else if (v == 0.f)
            q = v;
        xn[first * d + e] = q;
    }
    for (int e = tid; e < rows * raw_stride; e += 256) {
        const int i = e / raw_stride, t = e % raw_stride;
        raw[first * raw_stride + e] = t < d ? nr_rows[i * stride + t] : 0.f;
    }
}

// One thread per (padded) row: centred coordinates written transposed so the
// plain form's TMA boxes are [64 dims][128 rows]; the squared norm is the
// reference's fma chain; padding rows get +inf so their candidates are never
// admitted.
__global__ void centre_transpose_kernel(const float* __restrict__ x, int64_t n, int64_t n_pad, int d,
                                        int dp, const double* __restrict__ means,
                                        float* __restrict__ coords_t, float* __restrict__ norm2,
                                        float* __restrict__ cnorm, float* __restrict__ xcentred,
                                        uint32_t* __restrict__ max_norm_bits) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    const bool valid = i < n;
    float acc = 0.f;
    for (int t = 0; t < dp; t++) {
        float c = 0.f;
        if (valid && t < d) c = __double2float_rn(__dsub_rn((double)__ldg(x + i * d + t), means[t]));
        if (coords_t) coords_t[(int64_t)t * n_pad + i] = c;
        if (valid && t < d) {
            if (xcentred) xcentred[i * d + t] = c;
            acc = __fmaf_rn(c, c, acc);
        }
    }
    if (norm2) norm2[i] = valid ? acc : __int_as_float(0x7f800000);
    if (valid) {
        // sqrt rounded up by a relative 2^-20 so it bounds the true norm.
        float nrm = __fmul_ru(__fsqrt_ru(acc), 1.0f + 9.5367431640625e-07f);
        cnorm[i] = nrm;
        atomicMax(max_norm_bits, __float_as_uint(nrm));
    } else {
        cnorm[i] = 0.f;
    }
}

// Per-row candidate margin in s-space (s = |b|^2 - 2 a.b; the row's own |a|^2
// is a constant shift and cancels in every comparison made within the row).
//
// For every column j the computed s_ij differs from d_ij^2 - |a_i|^2 (d the
// distance between the caller's rows) by at most beta_i, so a column whose
// lower bound s - beta exceeds the k-th smallest upper bound s + beta cannot
// be among the k nearest: the margin is 2 * beta_i.  beta_i collects
//   plain form (FP32 fused dot, D terms):
//     (gamma_D + u) (M^2 + 2 |a| M)             expansion rounding, gamma_D = (D + 2) u
//     2.01 u (|a| + M)^2                        centring rounding of both rows
//   tensor form (16-bit operands, FP32 accumulate, scale 2^s applied):
//     2 (|e_a| M + |a| E + |e_a| E)             operand quantisation (exact error norms)
//     64 * 2^-24 (2 |a| M + M^2) + (gamma_D + u) M^2 + 2^-30 M^2   accumulation, norm split
//     2.01 u (|a| + M)^2                        centring
//   cosine adds 4.01 u + 1e-12 (f32 rounding of the normalised rows, FP64 noise);
//   reference-snap adds the snap floor ((D+2) 2u)(|a|^2 + M^2) and the
//   sequential chain's (D + 2) u (|a| + M)^2.
// M and E are the largest centred norm and quantisation error norm over all
// reference rows; u = 2^-24.  A 1.5x safety factor is applied.
__global__ void margins_kernel(const float* __restrict__ cnorm, const float* __restrict__ norm2,
                               int64_t n, int d, int mode, int metric, int form,
                               const uint32_t* __restrict__ max_norm_bits,
                               const float* __restrict__ qerr, const uint32_t* __restrict__ max_qerr_bits,
                               float scale2, float* __restrict__ margin) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double u = kUnit32;
    const double M = (double)__uint_as_float(*max_norm_bits);
    const double a = (double)cnorm[i];
    const double gammaD = (double)(d + 2) * u;
    double beta;
    if (form == SCRUST_FORM_PLAIN) {
        beta = (gammaD + u) * (M * M + 2.0 * a * M);
    } else {
        const double E = (double)__uint_as_float(*max_qerr_bits);
        const double ea = (double)qerr[i];
        beta = 2.0 * (ea * M + a * E + ea * E) + 64.0 * u * (2.0 * a * M + M * M) +
               (gammaD + u) * M * M + 9.313225746154785e-10 * M * M;
    }
    beta += 2.01 * u * (a + M) * (a + M);
    if (metric == SCRUST_METRIC_COSINE) beta += (4.01 * u + 1e-12) * (double)scale2;
    if (mode == SCRUST_MODE_REFERENCE_SNAP) {
        const double na = (double)norm2[i];
        beta += (double)(d + 2) * 2.0 * u * (na + M * M) + gammaD * (a + M) * (a + M);
    }
    margin[i] = __double2float_ru(2.0 * 1.5 * beta + 1e-30);
}

}  // namespace

cudaError_t launch_column_means(const float* x, int64_t n, int d, bool sequential, double* means,
                                double* partial, cudaStream_t s) {
    if (sequential) {
        means_sequential_kernel<<<(d + 63) / 64, 64, 0, s>>>(x, n, d, means);
        return cudaGetLastError();
    }
    int blocks = (int)((n + kMeanRowsPerBlock - 1) / kMeanRowsPerBlock);
    int threads = d >= 256 ? 256 : ((d + 31) / 32) * 32;
    means_partial_kernel<<<blocks, threads, 0, s>>>(x, n, d, partial);
    means_final_kernel<<<(d + 127) / 128, 128, 0, s>>>(partial, blocks, n, d, means);
    return cudaGetLastError();
}

namespace {

// Column means for the tensor form, where they only fix a centre (any
// centre serves, as long as every row and query is centred on the same
// one): f32 partial sums over 1024-row blocks, one warp per row at a time,
// then an f64 sum of the partials.  BLOCKS: 64-wide column blocks.  Eight rows
// a warp are fetched ahead of their sums (one after another, 100,000 x 50
// waited 34 us).
constexpr int kMeanRowsF32 = 1024;
template <int BLOCKS>
__global__ void __launch_bounds__(256) means_partial_f32_kernel(const float* __restrict__ x, int64_t n, int d,
                                                                float* __restrict__ partial) {
    __shared__ float acc_s[8][64 * BLOCKS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t r0 = (int64_t)blockIdx.x * kMeanRowsF32;
    const int64_t r1 = min(n, r0 + kMeanRowsF32);
    float acc[2 * BLOCKS];
#pragma unroll
    for (int t = 0; t < 2 * BLOCKS; ++t) acc[t] = 0.f;
    int64_t r = r0 + w;
    for (; r + 56 < r1; r += 64) {
        float v[8][2 * BLOCKS];
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int t = 0; t < 2 * BLOCKS; ++t)
                v[u][t] = lane + 32 * t < d ? __ldg(x + (r + 8 * u) * d + lane + 32 * t) : 0.f;
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int t = 0; t < 2 * BLOCKS; ++t) acc[t] += v[u][t];
    }
    for (; r < r1; r += 8)
#pragma unroll
        for (int t = 0; t < 2 * BLOCKS; ++t)
            if (lane + 32 * t < d) acc[t] += __ldg(x + r * d + lane + 32 * t);
#pragma unroll
    for (int t = 0; t < 2 * BLOCKS; ++t) acc_s[w][lane + 32 * t] = acc[t];
    __syncthreads();
    if (threadIdx.x < d) {
        float t = 0.f;
        for (int q = 0; q < 8; ++q) t += acc_s[q][threadIdx.x];
        partial[(int64_t)blockIdx.x * d + threadIdx.x] = t;
    }
}

// One block of 256 threads per column: strided f32 sums of the partials,
// then a tree.
__global__ void __launch_bounds__(256) means_final_f32_kernel(const float* __restrict__ partial, int blocks,
                                                              int64_t n, int d, double* __restrict__ means) {
    __shared__ float ws[8];
    const int c = blockIdx.x;
    float t = 0.f;
    for (int b = threadIdx.x; b < blocks; b += blockDim.x) t += partial[(int64_t)b * d + c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int w = 0; w < 8; ++w) s += ws[w];
        means[c] = (double)s / (double)n;
    }
}

}  // namespace

// `partial` is the d * (ceil(n / 2048) + 1) doubles that launch_column_means
// takes; the f32 partials of 1024-row blocks fit in it.
cudaError_t launch_column_means_centre(const float* x, int64_t n, int d, double* means, double* partial,
                                       cudaStream_t s) {
    const int blocks = (int)((n + kMeanRowsF32 - 1) / kMeanRowsF32);
    const auto part = operand_blocks(d) == 1 ? means_partial_f32_kernel<1> : means_partial_f32_kernel<2>;
    part<<<blocks, 256, 0, s>>>(x, n, d, reinterpret_cast<float*>(partial));
    means_final_f32_kernel<<<d, 256, 0, s>>>(reinterpret_cast<const float*>(partial), blocks, n, d, means);
    return cudaGetLastError();
}

namespace {
size_t cosine_inverse_at(int64_t n) { return (sizeof(double) * (size_t)n + 255) & ~(size_t)255; }
size_t cosine_raw_at(int64_t n) { return cosine_inverse_at(n) + ((sizeof(float2) * (size_t)n + 255) & ~(size_t)255); }
}  // namespace

size_t cosine_rows_bytes(int64_t n, int d) {
    return d <= kCosineMaxDims ? cosine_raw_at(n) + sizeof(float) * (size_t)n * padded_row_floats(d)
                               : sizeof(double) * (size_t)n;
}

cudaError_t launch_normalise_rows(const float* x, int64_t n, int d, float* xn, void* buf, CosineRows* out, int* d_err,
                                  cudaStream_t s) {
    *out = CosineRows();
    double* norm64 = (double*)buf;
    out->n = n;
    out->norm64 = norm64;
    if (d <= kCosineMaxDims) {
        float2* inverse = (float2*)((char*)buf + cosine_inverse_at(n));
        float* raw = (float*)((char*)buf + cosine_raw_at(n));
        out->inverse = inverse;
        out->raw = raw;
        normalise_rows_kernel<<<(unsigned)((n + NR_ROWS - 1) / NR_ROWS), 256, sizeof(float) * NR_ROWS * (d | 1), s>>>(
            x, n, d, xn, norm64, inverse, raw, padded_row_floats(d), d_err);
    } else {
        normalise_wide_rows_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(x, n, d, xn, norm64, d_err);
    }
    return cudaGetLastError();
}

// The largest norm of a row centred on the f32-rounded column means (as
// the tensor operands centre them), bounded from above; one warp per row,
// lanes over the coordinates (BLOCKS blocks of 64).
template <int BLOCKS>
__global__ void __launch_bounds__(256) max_centred_norm_kernel(const float* __restrict__ x, int64_t n, int d,
                                                               const double* __restrict__ means,
                                                               uint32_t* __restrict__ max_norm_bits) {
    __shared__ float m32[64 * BLOCKS];
    if (threadIdx.x < 64 * BLOCKS) m32[threadIdx.x] = threadIdx.x < d ? __double2float_rn(means[threadIdx.x]) : 0.f;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    float best = 0.f;
#pragma unroll 4
    for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n; r += warps) {
        float acc = 0.f;
#pragma unroll
        for (int t = 0; t < 2 * BLOCKS; ++t) {
            if (lane + 32 * t < d) {
                const float c = __fsub_rn(__ldg(x + r * d + lane + 32 * t), m32[lane + 32 * t]);
                acc = __fmaf_rn(c, c, acc);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        best = fmaxf(best, acc);
    }
    // One atomic a block (with one a warp, half of the 16 us of 100,000 rows was
    // their queue at the one word; 8 us so).
    __shared__ float most[8];
    if (lane == 0) most[threadIdx.x >> 5] = best;
    __syncthreads();
    for (int w = 0; w < 8; ++w) best = fmaxf(best, most[w]);
    if (threadIdx.x == 0 && best > 0.f) {
        // A sum of d rounded non-negative terms, scaled past its rounding.
        const float grow = 1.0f + (float)(d + 4) * 1.1920929e-07f;
        atomicMax(max_norm_bits, __float_as_uint(__fmul_ru(__fsqrt_ru(__fmul_ru(best, grow)), 1.0f + 9.5367431640625e-07f)));
    }
}

cudaError_t launch_max_centred_norm(const float* x, int64_t n, int d, const double* means, uint32_t* max_norm_bits,
                                    int sm_count, cudaStream_t s) {
    const int64_t want = (n + 7) / 8;
    const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sm_count * 8));
    const auto kern = operand_blocks(d) == 1 ? max_centred_norm_kernel<1> : max_centred_norm_kernel<2>;
    kern<<<blocks, 256, 0, s>>>(x, n, d, means, max_norm_bits);
    return cudaGetLastError();
}

cudaError_t launch_centre_transpose(const float* x, int64_t n, int64_t n_pad, int d, int dp,
                                    const double* means, float* coords_t, float* norm2,
                                    float* cnorm, float* xcentred, uint32_t* max_norm_bits,
                                    cudaStream_t s) {
    centre_transpose_kernel<<<(unsigned)((n_pad + 255) / 256), 256, 0, s>>>(
        x, n, n_pad, d, dp, means, coords_t, norm2, cnorm, xcentred, max_norm_bits);
    return cudaGetLastError();
}

cudaError_t launch_margins(const float* cnorm, const float* norm2, int64_t n, int d, int mode,
                           int metric, int form, const uint32_t* max_norm_bits,
                           const float* qerr, const uint32_t* max_qerr_bits, float scale2,
                           float* margin, cudaStream_t s) {
    margins_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
        cnorm, norm2, n, d, mode, metric, form, max_norm_bits, qerr, max_qerr_bits, scale2, margin);
    return cudaGetLastError();
}

}  // namespace scrust
