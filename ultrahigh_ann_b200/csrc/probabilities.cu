// Importance probabilities on the device.
//
// Reference semantics (src/hnsvw25/l2/importance_sampling.cpp:19-45,
// src/hnsvw25/l1/importance_sampling.cpp:19-47): for every pair of rows a < b
// with nonzero distance, L2 contributes min(1, (a_j - b_j)^2 / ||a - b||^2) and
// L1 contributes |a_j - b_j| / ||a - b||_1 to column j; p_j is the maximum
// contribution. Pair distances and the per-column maxima use binary64 (the
// normalisation of the probabilities). The direct backend performs the CPU's
// own operations in the CPU's order (sequential squared differences for L2,
// libstdc++'s transform_reduce grouping for L1, one IEEE division per pair,
// the same two roundings per contribution) and the maximum is exact, so its
// probabilities equal the reference CPU's bit for bit. The Gram backend
// agrees to a few ulps.
//
// Stage 1 (pair kernel): a TILE x TILE block of pairs per CTA, R x R pairs per
// thread. The inverse distance w of every pair a < b (0 for zero distance) goes
// to w[a][b] of an r x r matrix; its mirror slot [b][a] holds the binary32
// weight of the column filter, sqrt(w) (L2) or w (L1).
// Stage 2 (column kernel, run twice): a CTA owns 256 columns and one 32-row
// block A and walks every row block B >= A. With t = |a_j - b_j| * weight in
// binary32, a column's contribution is t^2 (L2) or t (L1) to about 2^-22
// relative. The first run takes the largest t of every column; the second
// evaluates in binary64, with the CPU's roundings, only the pairs whose t lies
// within 2^-20 of it, and combines those across CTAs with a 64-bit atomicMax on
// the bit pattern (nonnegative binary64 values order like their bit patterns).
#include "common.h"
#include "kernels.h"

#include <algorithm>

namespace uha {
namespace {

constexpr int kPairBlock = 32;
constexpr int kPairSlab = 64;
constexpr int kColumns = 256;
// the column kernel: rows a per CTA, columns per thread, threads
constexpr int kMaxRows = 32;
constexpr int kMaxColumns = 2;
constexpr int kMaxThreads = 128;

// The column filter's binary32 weight of a pair with inverse distance w, and
// whether w lies where the filter's relative error holds: the weight and its
// product with a difference then neither overflow nor lose bits to underflow
// unless the product itself is below 2^-126.
__device__ __forceinline__ float filter_weight(int metric, double w, int* odd)
{
    if (w == 0.0) {
        return 0.f;
    }
    const double f = metric == 0 ? sqrt(w) : w;
    if (!(f >= 0x1p-95 && f <= 0x1p95)) {
        atomicOr(odd, 1);
        return 0.f;
    }
    return __double2float_rn(f);
}

__device__ __forceinline__ void store_pair(int metric, double* __restrict__ inverse,
                                           uint64_t row_count, uint64_t a, uint64_t b, double w,
                                           int* odd)
{
    inverse[a * row_count + b] = w;
    reinterpret_cast<float*>(inverse + b * row_count + a)[0] = filter_weight(metric, w, odd);
}

// Binary64 pair distances in the CPU's order: a pair's columns are one chain of
// additions, so what is left to choose is how the pairs spread over the chip.
// Bound: shared-memory reads (two 16-byte reads per 2 x 2 pairs and column) a
// little above the FP64 pipe (3 operations per pair and column) when the chip
// is full, the chain's latency below that. The slab of columns is converted to
// binary64 once, as it is staged, transposed, into one of two buffers, the next
// slab's loads in flight behind the sums.
// Measured, ms at 60,660 columns, L2, by rows (TILE/R):
//            8/1     16/2    32/2    a 32 x 32 tile with 1 x 4 pairs before
//      100   1.04    1.48    2.47
//      200   1.45    1.63    2.47
//      384   3.91    2.53    3.25    6.16
//     1024  16.2     9.05    9.97
//     2048  61.6    32.6    29.7
template <int METRIC, int TILE, int R>
__global__ void __launch_bounds__((TILE / R) * (TILE / R))
    pair_distance_kernel(const float* __restrict__ rows, uint32_t row_count, uint64_t dim,
                         double* __restrict__ inverse, int* odd)
{
    constexpr int kThreads = (TILE / R) * (TILE / R);
    constexpr int kSlab = 32;                 // columns per stage
    constexpr int kPitch = TILE + 2;          // keeps double2 alignment
    constexpr int kGroup = 4;
    constexpr int kLoads = TILE * kSlab / kThreads;
    const uint32_t ta = blockIdx.y;
    const uint32_t tb = blockIdx.x;
    if (tb < ta) {
        return;
    }
    __shared__ __align__(16) double sa[2][kSlab][kPitch];
    __shared__ __align__(16) double sb[2][kSlab][kPitch];
    const int ty = threadIdx.x / (TILE / R);
    const int tx = threadIdx.x % (TILE / R);
    const uint32_t a0 = ta * TILE;
    const uint32_t b0 = tb * TILE;
    double acc[R][R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            acc[i][j] = 0.0;
        }
    }
    float ra[kLoads];
    float rb[kLoads];
    auto fetch = [&](uint64_t c0) {
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            const int e = threadIdx.x + i * kThreads;
            const uint32_t r = e / kSlab;
            const uint64_t col = c0 + e % kSlab;
            ra[i] = col < dim && a0 + r < row_count ? rows[(a0 + r) * dim + col] : 0.f;
            rb[i] = col < dim && b0 + r < row_count ? rows[(b0 + r) * dim + col] : 0.f;
        }
    };
    auto stage = [&](int buffer) {
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            const int e = threadIdx.x + i * kThreads;
            sa[buffer][e % kSlab][e / kSlab] = static_cast<double>(ra[i]);
            sb[buffer][e % kSlab][e / kSlab] = static_cast<double>(rb[i]);
        }
    };
    const uint64_t grouped_end = dim & ~uint64_t(3);
    fetch(0);
    int buffer = 0;
    for (uint64_t c0 = 0; c0 < dim; c0 += kSlab, buffer ^= 1) {
        stage(buffer);
        // one barrier per slab: a thread stages this buffer again only after
        // the next slab's barrier, which every thread reaches past its sums
        __syncthreads();
        if (c0 + kSlab < dim) {
            fetch(c0 + kSlab);
        }
        // groups of kGroup columns: the next group's values are read while
        // this one's terms are formed, and only the additions are a chain
        double va[2][kGroup][R];
        double vb[2][kGroup][R];
        auto read = [&](int slot, int c) {
#pragma unroll
            for (int e = 0; e < kGroup; ++e) {
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    va[slot][e][i] = sa[buffer][c + e][ty * R + i];
                    vb[slot][e][i] = sb[buffer][c + e][tx * R + i];
                }
            }
        };
        read(0, 0);
#pragma unroll
        for (int c = 0; c < kSlab; c += kGroup) {
            const int slot = c / kGroup % 2;
            if (c + kGroup < kSlab) {
                read(slot ^ 1, c + kGroup);
            }
            const bool whole = METRIC == 0 || c0 + c + kGroup <= grouped_end;
#pragma unroll
            for (int i = 0; i < R; ++i) {
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    double t[kGroup];
#pragma unroll
                    for (int e = 0; e < kGroup; ++e) {
                        const double d = __dsub_rn(va[slot][e][i], vb[slot][e][j]);
                        t[e] = METRIC == 0 ? __dmul_rn(d, d) : fabs(d);
                    }
                    if (METRIC == 1 && whole) {
                        // l1_dist: std::transform_reduce as libstdc++ 13
                        // evaluates it (src/core/l1_distance.cpp:17-26): init +
                        // ((t0 + t1) + (t2 + t3)) per group of four from column
                        // 0, then the last dim % 4 columns one by one
                        acc[i][j] = __dadd_rn(acc[i][j], __dadd_rn(__dadd_rn(t[0], t[1]),
                                                                   __dadd_rn(t[2], t[3])));
                    } else {
                        // squared_l2_dist: separately rounded squares in column
                        // order (src/core/l2_distance.cpp:17-23); the zeros
                        // staged past the last column add nothing
#pragma unroll
                        for (int e = 0; e < kGroup; ++e) {
                            acc[i][j] = __dadd_rn(acc[i][j], t[e]);
                        }
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const uint32_t a = a0 + ty * R + i;
            const uint32_t b = b0 + tx * R + j;
            if (a < b && b < row_count) {
                store_pair(METRIC, inverse, row_count, a, b,
                           acc[i][j] != 0.0 ? 1.0 / acc[i][j] : 0.0, odd);
            }
        }
    }
}

// Gram backend, stage 1: G[a][b] = sum_j a_j b_j in binary64 for a <= b,
// same tiling as the pair kernel.
__global__ void __launch_bounds__(256)
    gram_kernel(const float* __restrict__ rows, uint32_t row_count, uint64_t dim,
                double* __restrict__ gram)
{
    const uint32_t ta = blockIdx.y;
    const uint32_t tb = blockIdx.x;
    if (tb < ta) {
        return;
    }
    __shared__ float sa[kPairBlock][kPairSlab + 1];
    __shared__ float sb[kPairBlock][kPairSlab + 1];
    const int ty = threadIdx.x / 8;
    const int tx = threadIdx.x % 8;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const uint32_t a0 = ta * kPairBlock;
    const uint32_t b0 = tb * kPairBlock;
    for (uint64_t c0 = 0; c0 < dim; c0 += kPairSlab) {
        for (int i = threadIdx.x; i < kPairBlock * kPairSlab; i += blockDim.x) {
            const int r = i / kPairSlab;
            const int c = i % kPairSlab;
            const uint64_t col = c0 + c;
            float va = 0.f;
            float vb = 0.f;
            if (col < dim) {
                if (a0 + r < row_count) {
                    va = rows[static_cast<uint64_t>(a0 + r) * dim + col];
                }
                if (b0 + r < row_count) {
                    vb = rows[static_cast<uint64_t>(b0 + r) * dim + col];
                }
            }
            sa[r][c] = va;
            sb[r][c] = vb;
        }
        __syncthreads();
#pragma unroll 4
        for (int c = 0; c < kPairSlab; ++c) {
            const double va = sa[ty][c];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[j] = fma(va, static_cast<double>(sb[tx + 8 * j][c]), acc[j]);
            }
        }
        __syncthreads();
    }
    const uint32_t a = a0 + ty;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t b = b0 + tx + 8 * j;
        if (a < row_count && b < row_count && a <= b) {
            gram[static_cast<uint64_t>(a) * row_count + b] = acc[j];
        }
    }
}

// Gram backend, stage 2: ||a - b||^2 = G_aa + G_bb - 2 G_ab. The identity's
// absolute error is at most about (dim + 2) * 2^-53 * (G_aa + G_bb); pairs
// where that could exceed 2^-24 of the result (binary32-level accuracy) are
// recomputed directly as a binary64 sum of squared differences.
__global__ void gram_to_inverse_kernel(const double* __restrict__ gram,
                                       const float* __restrict__ rows,
                                       uint32_t row_count, uint64_t dim,
                                       double* __restrict__ inverse, int* odd)
{
    const uint64_t pairs = static_cast<uint64_t>(row_count) * row_count;
    for (uint64_t idx = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
         idx < pairs; idx += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint32_t a = static_cast<uint32_t>(idx / row_count);
        const uint32_t b = static_cast<uint32_t>(idx - uint64_t(a) * row_count);
        if (a >= b) {
            continue;
        }
        const double na = gram[uint64_t(a) * row_count + a];
        const double nb = gram[uint64_t(b) * row_count + b];
        double sd = na + nb - 2.0 * gram[idx];
        const double cancellation =
            static_cast<double>(dim + 2) * 1.1102230246251565e-16 * 16777216.0;
        if (!(sd > cancellation * (na + nb))) {
            const float* ra = rows + uint64_t(a) * dim;
            const float* rb = rows + uint64_t(b) * dim;
            sd = 0.0;
            for (uint64_t j = 0; j < dim; ++j) {
                const double d = static_cast<double>(ra[j]) - static_cast<double>(rb[j]);
                sd = fma(d, d, sd);
            }
        }
        store_pair(0, inverse, row_count, a, b, sd != 0.0 ? 1.0 / sd : 0.0, odd);
    }
}

// Two binary32 operations in one instruction (sm_100's packed forms, each half
// rounded as the scalar operation).
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    float2 r;
    asm("add.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long&>(r))
        : "l"(reinterpret_cast<unsigned long long&>(a)),
          "l"(reinterpret_cast<unsigned long long&>(b)));
    return r;
}

__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
    float2 r;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long&>(r))
        : "l"(reinterpret_cast<unsigned long long&>(a)),
          "l"(reinterpret_cast<unsigned long long&>(b)));
    return r;
}

// The largest of three; NaN only where all are.
__device__ __forceinline__ float max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Per-column maxima, one of two runs (see the file comment). top_bits[col]
// holds the bits of the largest t after the first run, 0 only where the column
// has one value in every row (a changing column whose largest t is 0 holds the
// bits 1).
//
// Bound: instruction issue (60 % of the slots busy at 700 rows), 1.5
// instructions per pair and column: packed subtract and multiply, and one
// three-input maximum per two pairs. Row block A stays in registers for two
// columns per thread, so a weight broadcast from shared memory serves two
// pair-columns (with one column per thread the broadcasts themselves were the
// bound: 128 bytes of shared-memory data per pair and warp), and the rows b
// stream through, one ahead. 384 x 60,660, L2, both runs: 1.1 ms against
// 60.8 ms before (every pair folded in binary64, whole row blocks walked again
// for each chunk of 574 pairs); 2,048 rows 27 ms.
//
// Why 2^-20: t is within 3.1 * 2^-24 relative of |a_j - b_j| sqrt(w) (two
// roundings and the weight's), and a contribution's binary64 roundings are
// within 2^-51 of the exact product, so the pair with the largest contribution
// has a t of at least (1 - 6.5 * 2^-24) times the largest. Columns whose
// largest t is not finite or below 2^-60, and every column when some weight was
// out of range, take every pair in binary64.
template <bool EXACT>
__global__ void __launch_bounds__(kMaxThreads)
    coordinate_max_kernel(int metric, const float* __restrict__ rows, uint32_t row_count,
                          uint64_t dim, const double* __restrict__ inverse,
                          unsigned int* __restrict__ top_bits, const int* __restrict__ odd,
                          unsigned long long* __restrict__ maxima_bits, uint32_t first_block)
{
    constexpr int A = kMaxRows;
    constexpr int C = kMaxColumns;
    constexpr uint32_t kChunk = 64;  // rows b whose weights are staged together
    __shared__ __align__(16) float sw[kChunk][A];
    const uint64_t col0 = blockIdx.x * static_cast<uint64_t>(kMaxThreads * C) + threadIdx.x;
    const uint32_t a0 = (first_block + blockIdx.y) * A;
    const uint64_t r64 = row_count;
    float va[C][A];
    float top[C];    // !EXACT: the largest t
    float least[C];  // EXACT: t from here on is evaluated
    double m[C];
#pragma unroll
    for (int k = 0; k < C; ++k) {
        const uint64_t col = col0 + k * kMaxThreads;
#pragma unroll
        for (int r = 0; r < A; ++r) {
            va[k][r] = a0 + r < row_count && col < dim ? rows[(a0 + r) * dim + col] : 0.f;
        }
        top[k] = 0.f;
        m[k] = 0.0;
        if (EXACT) {
            least[k] = __int_as_float(0x7f800000);
            const unsigned int bits = col < dim ? top_bits[col] : 0u;
            if (bits != 0u) {
                const float t = __uint_as_float(bits);
                least[k] = t >= 0x1p-60f && t <= 0x1.fffffep127f && *odd == 0
                               ? __fmul_rd(t, 1.f - 0x1p-20f)
                               : 0.f;
            }
        }
    }
    float next[C];
    auto fetch = [&](uint32_t b) {
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const uint64_t col = col0 + k * kMaxThreads;
            next[k] = b < row_count && col < dim ? rows[b * dim + col] : 0.f;
        }
    };
    fetch(a0 + 1);
    for (uint32_t b0 = a0 + 1; b0 < row_count; b0 += kChunk) {
        __syncthreads();  // the previous chunk's weights are no longer read
        for (uint32_t i = threadIdx.x; i < kChunk * A; i += kMaxThreads) {
            // the weights' slots are [b][a]: consecutive threads, consecutive a
            const uint64_t a = a0 + i % A;
            const uint64_t b = b0 + i / A;
            sw[i / A][i % A] =
                a < b && b < r64 ? reinterpret_cast<const float*>(inverse + b * r64 + a)[0]
                                 : 0.f;
        }
        __syncthreads();
        const uint32_t count = min(kChunk, row_count - b0);
#pragma unroll 1
        for (uint32_t i = 0; i < count; ++i) {
            float vb[C];
#pragma unroll
            for (int k = 0; k < C; ++k) {
                vb[k] = -next[k];
            }
            fetch(b0 + i + 1);
            float t[C][2];
#pragma unroll
            for (int k = 0; k < C; ++k) {
                t[k][0] = EXACT ? 0.f : top[k];
                t[k][1] = 0.f;
            }
#pragma unroll
            for (int r = 0; r < A; r += 4) {
                const float4 w = *reinterpret_cast<const float4*>(&sw[i][r]);
#pragma unroll
                for (int k = 0; k < C; ++k) {
                    const float2 b2 = make_float2(vb[k], vb[k]);
                    const float2 x = mul2(add2(make_float2(va[k][r], va[k][r + 1]), b2),
                                          make_float2(w.x, w.y));
                    const float2 y = mul2(add2(make_float2(va[k][r + 2], va[k][r + 3]), b2),
                                          make_float2(w.z, w.w));
                    t[k][0] = max3(t[k][0], fabsf(x.x), fabsf(x.y));
                    t[k][1] = max3(t[k][1], fabsf(y.x), fabsf(y.y));
                }
            }
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const float both = fmaxf(t[k][0], t[k][1]);
                if (!EXACT) {
                    top[k] = both;
                } else if (both >= least[k]) {
                    // row b's pairs with the block in binary64, with the CPU's
                    // roundings ((d * d) * inverse or |d| * inverse:
                    // importance_sampling.cpp:36-41 of l2, :26-30 of l1); the
                    // values again from memory, since runtime indices would
                    // move va out of registers
                    const uint64_t col = col0 + k * kMaxThreads;
                    const uint64_t b = b0 + i;
                    const double xb = static_cast<double>(rows[b * dim + col]);
#pragma unroll 4
                    for (uint64_t a = a0; a < min(b, static_cast<uint64_t>(a0 + A)); ++a) {
                        const double d =
                            __dsub_rn(static_cast<double>(rows[a * dim + col]), xb);
                        const double w = inverse[a * r64 + b];
                        m[k] = fmax(m[k], metric == 0 ? __dmul_rn(__dmul_rn(d, d), w)
                                                      : __dmul_rn(fabs(d), w));
                    }
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < C; ++k) {
        const uint64_t col = col0 + k * kMaxThreads;
        if (col >= dim) {
            continue;
        }
        if (EXACT) {
            if (m[k] > 0.0) {
                atomicMax(maxima_bits + col,
                          static_cast<unsigned long long>(__double_as_longlong(m[k])));
            }
            continue;
        }
        const float first = rows[col];
        bool changes = false;
#pragma unroll
        for (int r = 0; r < A; ++r) {
            changes = changes || (a0 + r < row_count && va[k][r] != first);
        }
        const unsigned int bits = max(__float_as_uint(top[k]), changes ? 1u : 0u);
        if (bits != 0u) {
            atomicMax(top_bits + col, bits);
        }
    }
}

// The binary32 form of the maxima (the same pairs, the CPU's contributions
// rounded in binary32: within 3e-7 relative): each thread's 32 values of its column of row blocks A and
// B stay in registers (every thread reads only its own column), a pair
// block's inverse distances are rounded to binary32 once in shared memory, and
// the 32 x 32 pairs are unrolled: about four binary32 instructions per
// pair-column. A pair block holding a distance below 2^-100 is folded in
// binary64, with the CPU's roundings.
__global__ void __launch_bounds__(kColumns)
    coordinate_max32_kernel(int metric, const float* __restrict__ rows,
                            uint32_t row_count, uint64_t dim,
                            const double* __restrict__ inverse,
                            unsigned long long* __restrict__ maxima_bits,
                            uint32_t first_block)
{
    __shared__ __align__(16) float sw[kPairBlock * kPairBlock];
    __shared__ double sw64[kPairBlock * kPairBlock];
    const uint64_t col = blockIdx.x * static_cast<uint64_t>(kColumns) + threadIdx.x;
    const uint32_t ta = first_block + blockIdx.y;
    const uint32_t a0 = ta * kPairBlock;
    const uint32_t blocks = (row_count + kPairBlock - 1) / kPairBlock;
    const uint64_t r64 = row_count;
    float va[kPairBlock];
#pragma unroll
    for (int r = 0; r < kPairBlock; ++r) {
        va[r] = a0 + r < row_count && col < dim
                    ? rows[static_cast<uint64_t>(a0 + r) * dim + col]
                    : 0.f;
    }
    float m32[4] = {0.f, 0.f, 0.f, 0.f};  // four chains of the maximum
    double m = 0.0;
    for (uint32_t tb = ta; tb < blocks; ++tb) {
        const uint32_t b0 = tb * kPairBlock;
        float vb[kPairBlock];
#pragma unroll
        for (int r = 0; r < kPairBlock; ++r) {
            vb[r] = b0 + r < row_count && col < dim
                        ? rows[static_cast<uint64_t>(b0 + r) * dim + col]
                        : 0.f;
        }
        __syncthreads();  // the previous block's weights are no longer read
        bool large = false;
        for (int i = threadIdx.x; i < kPairBlock * kPairBlock; i += blockDim.x) {
            const int ra = i / kPairBlock;
            const int rb = i % kPairBlock;
            double v = 0.0;
            const uint64_t a = a0 + ra;
            const uint64_t b = b0 + rb;
            if (a < b && b < row_count) {
                v = inverse[a * r64 + b];
            }
            sw64[i] = v;
            sw[i] = v > 0x1p100 ? 0.f : __double2float_rn(v);
            large = large || v > 0x1p100;
        }
        if (__syncthreads_or(large ? 1 : 0) == 0) {
#pragma unroll
            for (int ra = 0; ra < kPairBlock; ++ra) {
#pragma unroll
                for (int rb = 0; rb < kPairBlock; ++rb) {
                    const float d = __fsub_rn(va[ra], vb[rb]);
                    const float w = sw[ra * kPairBlock + rb];
                    const float c = metric == 0 ? __fmul_rn(__fmul_rn(d, d), w)
                                                : __fmul_rn(fabsf(d), w);
                    m32[ra % 4] = fmaxf(m32[ra % 4], c);
                }
            }
        } else {
#pragma unroll 1
            for (int ra = 0; ra < kPairBlock; ++ra) {
#pragma unroll 1
                for (int rb = 0; rb < kPairBlock; ++rb) {
                    // the values again from memory: runtime indices would
                    // move va and vb out of registers
                    const double xa = a0 + ra < row_count && col < dim
                                          ? rows[static_cast<uint64_t>(a0 + ra) * dim + col]
                                          : 0.f;
                    const double xb = b0 + rb < row_count && col < dim
                                          ? rows[static_cast<uint64_t>(b0 + rb) * dim + col]
                                          : 0.f;
                    const double d = __dsub_rn(xa, xb);
                    const double w = sw64[ra * kPairBlock + rb];
                    const double c = metric == 0 ? __dmul_rn(__dmul_rn(d, d), w)
                                                 : __dmul_rn(fabs(d), w);
                    m = fmax(m, c);
                }
            }
        }
    }
    m = fmax(m, static_cast<double>(fmaxf(fmaxf(m32[0], m32[1]), fmaxf(m32[2], m32[3]))));
    if (col < dim && m > 0.0) {
        atomicMax(maxima_bits + col,
                  static_cast<unsigned long long>(__double_as_longlong(m)));
    }
}

}  // namespace

namespace {

template <int TILE, int R>
void launch_pair_tiles(int metric, const float* rows, uint64_t row_count, uint64_t dim,
                       double* inverse, int* odd, cudaStream_t stream)
{
    const uint64_t blocks = (row_count + TILE - 1) / TILE;
    if (blocks > 65535u) {
        fail(UHA_LENGTH_ERROR, "probability pair grid exceeds device limit");
    }
    const dim3 grid(static_cast<uint32_t>(blocks), static_cast<uint32_t>(blocks));
    constexpr int threads = (TILE / R) * (TILE / R);
    if (metric == 0) {
        pair_distance_kernel<0, TILE, R><<<grid, threads, 0, stream>>>(
            rows, static_cast<uint32_t>(row_count), dim, inverse, odd);
    } else {
        pair_distance_kernel<1, TILE, R><<<grid, threads, 0, stream>>>(
            rows, static_cast<uint32_t>(row_count), dim, inverse, odd);
    }
    check_cuda(cudaGetLastError(), "cannot launch pair distance kernel");
}

}  // namespace

void launch_pair_distances(int metric, const float* rows, uint64_t row_count,
                           uint64_t dim, double* inverse_distances, int* odd,
                           cudaStream_t stream)
{
    // the table at pair_distance_kernel: one pair per thread while the pairs
    // are fewer than the chip's lanes, then 2 x 2, in small tiles until the
    // large ones fill the SMs evenly
    if (row_count < 256) {
        launch_pair_tiles<8, 1>(metric, rows, row_count, dim, inverse_distances, odd, stream);
    } else if (row_count < 1536) {
        launch_pair_tiles<16, 2>(metric, rows, row_count, dim, inverse_distances, odd, stream);
    } else {
        launch_pair_tiles<32, 2>(metric, rows, row_count, dim, inverse_distances, odd, stream);
    }
}

void launch_gram_inverse_distances(const float* rows, uint64_t row_count,
                                   uint64_t dim, double* gram,
                                   double* inverse_distances, int* odd,
                                   cudaStream_t stream)
{
    const uint32_t blocks =
        static_cast<uint32_t>((row_count + kPairBlock - 1) / kPairBlock);
    if (blocks > 65535u) {
        fail(UHA_LENGTH_ERROR, "probability pair grid exceeds device limit");
    }
    gram_kernel<<<dim3(blocks, blocks), 256, 0, stream>>>(
        rows, static_cast<uint32_t>(row_count), dim, gram);
    check_cuda(cudaGetLastError(), "cannot launch Gram kernel");
    gram_to_inverse_kernel<<<148 * 16, 256, 0, stream>>>(
        gram, rows, static_cast<uint32_t>(row_count), dim, inverse_distances, odd);
    check_cuda(cudaGetLastError(), "cannot launch Gram refinement kernel");
}

namespace {

__global__ void finite_check_kernel(const float* __restrict__ values, uint64_t count,
                                    int* flag)
{
    bool bad = false;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
         i < count; i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        bad = bad || !isfinite(values[i]);
    }
    if (__any_sync(0xffffffffu, bad) && threadIdx.x % 32 == 0) {
        atomicOr(flag, 1);
    }
}

}  // namespace

void launch_finite_check(const float* values, uint64_t count, int* flag,
                         cudaStream_t stream)
{
    if (count == 0) {
        return;
    }
    const uint64_t blocks = std::min<uint64_t>((count + 255) / 256, 148ull * 32);
    finite_check_kernel<<<static_cast<uint32_t>(blocks), 256, 0, stream>>>(values, count,
                                                                           flag);
    check_cuda(cudaGetLastError(), "cannot launch the finiteness check");
}

void launch_coordinate_maxima(int metric, const float* rows, uint64_t row_count,
                              uint64_t dim, const double* inverse_distances,
                              unsigned int* top_bits, const int* odd,
                              unsigned long long* maxima_bits, uint64_t pair_chunks,
                              cudaStream_t stream, bool single)
{
    const uint64_t block_rows = single ? kPairBlock : kMaxRows;
    const uint64_t block_columns = single ? kColumns : kMaxThreads * kMaxColumns;
    const uint64_t blocks = (row_count + block_rows - 1) / block_rows;
    const uint64_t column_blocks = (dim + block_columns - 1) / block_columns;
    if (column_blocks > 0x7fffffffull || (row_count + kPairBlock - 1) / kPairBlock > 65535u) {
        fail(UHA_LENGTH_ERROR, "probability column grid exceeds device limit");
    }
    // Up to pair_chunks launches per run, cut at row blocks (a cut inside one
    // would walk its pairs twice) into about equal counts of pairs; fewer where
    // a launch would hold under 2^38 pair-columns (about 20 ms), which keeps
    // the launches of a minutes-long build bounded and small builds whole.
    const double work = 0.5 * static_cast<double>(row_count) * static_cast<double>(row_count) *
                        static_cast<double>(dim);
    const uint64_t launches =
        std::min<uint64_t>(pair_chunks, 1 + static_cast<uint64_t>(work / 0x1p38));
    const uint64_t pair_blocks = blocks * (blocks + 1) / 2;
    auto for_ranges = [&](auto&& launch) {
        uint64_t begin = 0;
        uint64_t done = 0;
        for (uint64_t c = 1; c <= launches && begin < blocks; ++c) {
            uint64_t end = begin;
            const uint64_t until = pair_blocks / launches * c;
            while (end < blocks && end - begin < 65535 && (done < until || c == launches)) {
                done += blocks - end;
                ++end;
            }
            if (end > begin) {
                launch(dim3(static_cast<uint32_t>(column_blocks),
                            static_cast<uint32_t>(end - begin)),
                       static_cast<uint32_t>(begin));
                check_cuda(cudaGetLastError(), "cannot launch probability column kernel");
                begin = end;
            }
            if (c == launches && begin < blocks) {
                --c;  // more row blocks than one grid holds
            }
        }
    };
    const uint32_t rc = static_cast<uint32_t>(row_count);
    if (single) {
        for_ranges([&](dim3 grid, uint32_t first) {
            coordinate_max32_kernel<<<grid, kColumns, 0, stream>>>(
                metric, rows, rc, dim, inverse_distances, maxima_bits, first);
        });
        return;
    }
    for_ranges([&](dim3 grid, uint32_t first) {
        coordinate_max_kernel<false><<<grid, kMaxThreads, 0, stream>>>(
            metric, rows, rc, dim, inverse_distances, top_bits, odd, maxima_bits, first);
    });
    for_ranges([&](dim3 grid, uint32_t first) {
        coordinate_max_kernel<true><<<grid, kMaxThreads, 0, stream>>>(
            metric, rows, rc, dim, inverse_distances, top_bits, odd, maxima_bits, first);
    });
}

}  // namespace uha
