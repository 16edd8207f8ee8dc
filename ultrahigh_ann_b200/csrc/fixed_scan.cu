// Certified L1 scan of larger batches in 16-bit fixed point.
//
// L1 has no contraction form, so its scan is bound by CUDA-core issue: the
// binary32 tile scan spends two instructions per (query, row, column). As in
// the split scan of L2 (split_scan.cu), an estimate with a bounded error is
// enough to list the rows that can be a query's minimum. Per column, with its
// smallest value o over the index's rows, its weight w (1 unless weighted) and
// one step s for all columns, a value x becomes the integer
// v = round(w (x - o) / s) in 0 .. 65,535, and
//   s * (2 sum max(v_q, v_r) - sum v_q - sum v_r) = s * sum |v_q - v_r|
// is exact in integers: two 16-bit maxima per instruction and one two-way dot
// product with ones that adds both to a 32-bit sum, one instruction per two
// columns each, half the binary32 scan's instructions per column. The estimate
// is off by at most R + Q, the sums of |w (x - o) - s v| over the row's and the
// query's columns: about 1e-4 of a distance on expression-like data. A query value
// past the rows' range is clamped: what is past it is the same in the distance to
// every row, a constant of the query that no comparison needs.
//
// Rows whose estimate less their error exceeds some row's estimate plus its own
// cannot be the minimum; the others (usually one or two) are settled from the
// original values in binary64 (certify.cu).
//
// Measured, device queries, one call: 7,028 rows x 60,660 columns, 333 queries:
// 14.1 -> 6.1 ms (the tile kernel 13.0 -> 5.9 ms); 65,536 rows x 128 columns (a
// flat index), 256 queries: 430 -> 154-188 us (tiles 107 us). It was the faster
// one at every size tried (33 to 40,000 rows, 64 to 60,660 columns, 9 to 400
// queries: 1.1 to 9 times), so every direct L1 batch past the streaming scan's 8
// queries takes it.
#include "common.h"
#include "kernels.h"
#include "tile_body.cuh"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>
#include <type_traits>

namespace uha {
namespace {

using tilebody::cp_async16;
using tilebody::cp_async_commit;
using tilebody::cp_async_wait;

constexpr int kThreads = 256;
constexpr int kPrepThreads = 512;         // at most, by the columns of a slice
constexpr uint32_t kRows = 128;          // rows per tile
constexpr uint32_t kStageColumns = 64;   // 128 bytes of a vector
constexpr uint32_t kStageStride = 144;   // bytes, conflict-free 16-byte reads
constexpr int kTileThreads = 128;
constexpr int kStages = 2;
constexpr int kSelectRows = 8;
constexpr uint32_t kRangeRows = 256;     // rows per slice of the range kernel
constexpr uint32_t kRangeSlices = 32768; // and slices of its grid at most (the limit is 65,535)
// steps of error per column that the binary32 arithmetic of the conversion adds
constexpr double kColumnSlack = 0x1p-6;
// The most a row's error can be in steps: half a step per column, the roundings'
// slack and the two of rounding up, unless w (x - o) left binary32. An index with
// a row past this is not usable, which the 32-bit epilogue relies on.
__host__ __device__ constexpr double largest_error(uint64_t dim)
{
    return 2.0 * static_cast<double>(dim) + 64.0;
}
// up to here T and a row's error stay below 2^31
constexpr uint64_t kNarrowColumns = 32000;
static_assert(65535.0 * kNarrowColumns + largest_error(kNarrowColumns) < 2147483647.0,
              "the narrow epilogue's differences fit 32 bits");
constexpr float kLevels = 65535.f;

__device__ __forceinline__ unsigned int ordered(float f)
{
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float from_ordered(unsigned int u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ double block_total(double v, double* scratch)
{
    for (int o = 16; o > 0; o /= 2) {
        v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    __syncthreads();
    if (threadIdx.x % 32 == 0) {
        scratch[threadIdx.x / 32] = v;
    }
    __syncthreads();
    double t = 0.0;
    for (uint32_t w = 0; w < blockDim.x / 32; ++w) {
        t += scratch[w];
    }
    return t;
}

// ---------------------------------------------------------------- index side

// Ordered bits (the smallest's inverted, so both grow from 0) of each column's
// smallest and largest value. grid (columns, slices
// of kRangeRows rows); a grid of kRangeSlices takes every so many-th slice.
__global__ void __launch_bounds__(kThreads)
    column_range_kernel(const float* __restrict__ rows, uint32_t row_count, uint64_t padded,
                        uint64_t dim, unsigned int* __restrict__ low,
                        unsigned int* __restrict__ high)
{
    const uint64_t j = blockIdx.x * static_cast<uint64_t>(kThreads) + threadIdx.x;
    if (j >= dim) {
        return;
    }
    float a = __int_as_float(0x7f800000);
    float b = -a;
    for (uint64_t first = uint64_t(blockIdx.y) * kRangeRows; first < row_count;
         first += uint64_t(gridDim.y) * kRangeRows) {
        const uint32_t end =
            static_cast<uint32_t>(min(uint64_t(row_count), first + kRangeRows));
#pragma unroll 8
        for (uint32_t r = static_cast<uint32_t>(first); r < end; ++r) {
            const float x = rows[r * padded + j];
            a = fminf(a, x);
            b = fmaxf(b, x);
        }
    }
    atomicMax(low + j, ~ordered(a));
    atomicMax(high + j, ordered(b));
}

// offsets[j] = the column's smallest value (0 past dim); step[0] = the largest
// weighted range over 65,535 (its bits, nonnegative; the slot is 0 before).
__global__ void __launch_bounds__(kThreads)
    column_offset_kernel(const unsigned int* __restrict__ low,
                         const unsigned int* __restrict__ high, uint64_t dim, uint64_t pitch,
                         const double* __restrict__ weights, float* __restrict__ offsets,
                         unsigned int* __restrict__ step)
{
    const uint64_t j = blockIdx.x * static_cast<uint64_t>(kThreads) + threadIdx.x;
    float s = 0.f;
    if (j < pitch) {
        const float o = j < dim ? from_ordered(~low[j]) : 0.f;
        offsets[j] = o;
        if (j < dim) {
            const double range =
                static_cast<double>(from_ordered(high[j])) - static_cast<double>(o);
            const double w = weights != nullptr ? weights[j] : 1.0;  // nonnegative
            s = __double2float_ru(w * range / static_cast<double>(kLevels));
        }
    }
    const unsigned int most = __reduce_max_sync(0xffffffffu, __float_as_uint(s));
    if (threadIdx.x % 32 == 0) {
        atomicMax(step, most);
    }
}

// L1 distances of kFixedPairs spread pairs of rows, for the host's estimate of
// whether the step is fine enough for this index.
__global__ void __launch_bounds__(kThreads)
    pair_sample_kernel(const float* __restrict__ rows, uint32_t row_count, uint64_t padded,
                       uint64_t dim, const double* __restrict__ weights,
                       double* __restrict__ out)
{
    __shared__ double scratch[kThreads / 32];
    const uint64_t a = 7919ull * blockIdx.x % row_count;
    const uint64_t b = (104729ull * blockIdx.x + 1) % row_count;
    double acc = 0.0;
    for (uint64_t j = threadIdx.x; j < dim; j += kThreads) {
        const double d = fabs(static_cast<double>(rows[a * padded + j]) -
                              static_cast<double>(rows[b * padded + j]));
        acc += weights != nullptr ? weights[j] * d : d;
    }
    const double total = block_total(acc, scratch);
    if (threadIdx.x == 0) {
        out[blockIdx.x] = total;
    }
}

// grid (slices, vectors): the slice's columns of a vector in fixed point (zeros
// past dim), the sum of their integers and of their errors |w (x - o) - s v|
// (past the range: of what the clamp cuts off, kept apart).
// ROWS: index rows (one slice), terms[i] = the sum and the error in steps, rounded
// up (error_flag is set where it is past largest_error()). Else queries (gathered through `columns` when given, validated, the prepared
// binary32 vector written on the way): parts per slice, and the first slice
// clears the query's words.
//
// Binary32 throughout: whatever integer is chosen, its error is what
// w (x - o) - s v comes to, up to three roundings of at most 65,536 steps times
// 2^-24 (kColumnSlack) and the sum's.
template <bool ROWS>
__global__ void __launch_bounds__(kPrepThreads) fixed_vectors_kernel(const FixedVectors v)
{
    __shared__ double scratch[kPrepThreads / 32];
    const uint64_t i = blockIdx.y;
    const float* in = v.source + i * v.source_pitch;
    uint16_t* out = v.out + i * v.pitch;
    const uint64_t begin = blockIdx.x * v.slice;
    const uint64_t end = min(v.pitch, begin + v.slice);
    const float s = *v.step;
    const float inverse = s > 0.f ? 1.f / s : 0.f;
    float resid = 0.f;
    float past = 0.f;
    unsigned long long sum = 0;
    int bad = 0;
    for (uint64_t j = begin + 4ull * threadIdx.x; j < end; j += 4ull * blockDim.x) {
        float x[4];
        if (v.vector_loads && j < v.source_pitch) {
            const float4 f = *reinterpret_cast<const float4*>(in + j);
            x[0] = f.x;
            x[1] = f.y;
            x[2] = f.z;
            x[3] = f.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x[e] = j + e < v.dim ? in[v.columns != nullptr ? v.columns[j + e] : j + e] : 0.f;
            }
        }
        uint32_t q[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            q[e] = 0;
            if (j + e < v.dim) {
                bad |= isfinite(x[e]) ? 0 : 1;
                float t = x[e] - v.offsets[j + e];
                if (v.weights != nullptr) {
                    t *= static_cast<float>(v.weights[j + e]);
                }
                const float nearest = rintf(t * inverse);
                const float level = fminf(fmaxf(nearest, 0.f), kLevels);
                q[e] = static_cast<uint32_t>(level);
                const float off = fabsf(fmaf(-level, s, t));
                if (ROWS || level == nearest) {
                    resid += off;
                } else {
                    past += off;
                }
                sum += q[e];
            }
        }
        *reinterpret_cast<uint2*>(out + j) = make_uint2(q[0] | q[1] << 16, q[2] | q[3] << 16);
        if (!ROWS && j < v.prepared_pitch) {  // a multiple of 4
            *reinterpret_cast<float4*>(v.prepared + i * v.prepared_pitch + j) =
                make_float4(x[0], x[1], x[2], x[3]);
        }
    }
    if (!ROWS && bad != 0) {
        atomicOr(v.error_flag, 1);
    }
    // in steps; a thread's binary32 sum has at most slice / blockDim + 4 terms
    const double steps = s > 0.f ? 1.0 / static_cast<double>(s) : 0.0;
    const double columns = static_cast<double>(end > begin ? end - begin : 0);
    const double rounding = 1.0 + (columns / blockDim.x + 8.0) * 0x1p-23;
    const double r =
        block_total(static_cast<double>(resid), scratch) * rounding * steps +
        columns * kColumnSlack;
    const double n = block_total(static_cast<double>(sum), scratch);  // below 2^53: exact
    const double c = ROWS ? 0.0 : block_total(static_cast<double>(past), scratch) * steps;
    if (threadIdx.x != 0) {
        return;
    }
    if (ROWS) {
        if (!(r <= largest_error(v.dim) - 2.0)) {
            atomicOr(v.error_flag, 1);
        }
        v.terms[i] = FixedTerms{static_cast<long long>(n),
                                static_cast<long long>(fmin(ceil(r) + 1.0, 0x1p60))};
    } else {
        v.query_parts[i * gridDim.x + blockIdx.x] = FixedParts{n, r, c};
        if (blockIdx.x == 0) {
            v.counts[i] = 0;
            v.upper[i] = ~0ull;
            v.done[i] = 0;
        }
    }
}

// --------------------------------------------------------------------- scan

__device__ __forceinline__ uint32_t max16x2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

struct QueryTerms {
    long long sum;    // of its integers
    long long error;  // in steps, with the roundings below
};

// A query's terms from its slices. Every estimate T = 2 M - (sums) is an exact
// integer, the binary64 reference's roundings ((dim + 64) 2^-51 of the distance,
// the part past the range included) count as the query's error.
__device__ __forceinline__ QueryTerms query_terms(const FixedQuery& f, uint32_t q)
{
    double n = 0.0;
    double r = 0.0;
    double c = 0.0;
    for (uint32_t s = 0; s < f.slices; ++s) {
        const FixedParts p = f.parts[static_cast<uint64_t>(q) * f.slices + s];
        n += p.sum;
        r += p.error;
        c += p.past;
    }
    const double k = static_cast<double>(f.dim);
    r += 2.0 + (k + 64.0) * 0x1p-51 * (65537.0 * k + r + c);
    return QueryTerms{static_cast<long long>(n),
                      static_cast<long long>(fmin(ceil(r), 0x1p60))};  // a NaN too
}

// grid (row tiles, query tiles, splits): sums[split][q][row] = sum of the larger
// of the two integers over the split's columns (at most 65,536 of them: below
// 2^32). 128 rows x 8 J queries per CTA, an 8 x J micro-tile per thread, 64-column
// stages double-buffered with cp.async. Bound: the two instructions per pair of
// columns, 79 % of the issue slots busy (333 queries x 7,028 x 60,660; 73 % at
// 65,536 rows x 128 columns), the dot product's pipe, which runs at half rate,
// being nearly full. (14-bit values, four maxima added before one dot product,
// are 7 instructions for 8 but took 7.0 ms for 5.9: the additions share the
// maxima's pipe.) The 16-byte shared-memory reads serve 8 x J outputs. The column
// loop stays rolled past 8 columns: unrolled it does not fit the instruction
// cache.
// With one split, `least` [q][row tile] is the smallest T - error over the tile's
// rows (0 if negative) and f.upper[q] the smallest T + error, so the selection
// visits only the tiles that hold candidates. Up to kNarrowColumns that epilogue
// is in 32-bit differences (NARROW): at 128 columns it was a fifth of the kernel in
// 64 bits (65,536 rows, 256 queries: 117 us, 107 so).
template <int J, bool NARROW>
__global__ void __launch_bounds__(kTileThreads, J == 8 ? 3 : 4)
    fixed_tile_kernel(const uint16_t* __restrict__ rows, uint32_t row_count,
                      const uint16_t* __restrict__ queries, uint32_t batch, uint64_t pitch,
                      uint32_t columns_per_split, uint32_t* __restrict__ sums,
                      unsigned long long* __restrict__ least, const FixedQuery f)
{
    constexpr uint32_t kQueries = 8 * J;
    constexpr uint32_t kStageBytes = (kRows + kQueries) * kStageStride;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ long long query_sums[kQueries];
    const uint32_t tid = threadIdx.x;
    const uint32_t tr = tid % 16;
    const uint32_t tq = tid / 16;
    const uint32_t row0 = blockIdx.x * kRows;
    const uint32_t q0 = blockIdx.y * kQueries;
    const uint64_t begin = static_cast<uint64_t>(blockIdx.z) * columns_per_split;
    const uint64_t end = min(pitch, begin + columns_per_split);
    const uint32_t stages = static_cast<uint32_t>((end - begin) / kStageColumns);
    auto load = [&](uint32_t stage) {
        unsigned char* to = smem + stage % kStages * kStageBytes;
        const uint64_t column = begin + static_cast<uint64_t>(stage) * kStageColumns;
        // 8 copies of 16 bytes per vector; rows, then queries
#pragma unroll
        for (uint32_t c = tid; c < (kRows + kQueries) * 8; c += kTileThreads) {
            const uint32_t vector = c / 8;
            const bool row = vector < kRows;
            const uint32_t at = row ? row0 + vector : q0 + vector - kRows;
            const bool ok = at < (row ? row_count : batch);
            const uint16_t* from = (row ? rows : queries) + (ok ? at * pitch : 0) + column +
                                   c % 8 * 8;
            cp_async16(to + vector * kStageStride + c % 8 * 16, from, ok);
        }
        cp_async_commit();
    };
    uint32_t acc[8][J];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int j = 0; j < J; ++j) {
            acc[i][j] = 0;
        }
    }
    if (stages > 0) {
        load(0);
    }
    for (uint32_t s = 0; s < stages; ++s) {
        if (s + 1 < stages) {
            load(s + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const unsigned char* r = smem + s % kStages * kStageBytes;
        const unsigned char* q = r + kRows * kStageStride;
#pragma unroll 1
        for (uint32_t k = 0; k < kStageColumns * 2; k += 16) {
            uint4 qv[J];
#pragma unroll
            for (int j = 0; j < J; ++j) {
                qv[j] = *reinterpret_cast<const uint4*>(q + (tq + 8 * j) * kStageStride + k);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint4 rv =
                    *reinterpret_cast<const uint4*>(r + (tr + 16 * i) * kStageStride + k);
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    // both halves of each word, times 1
                    acc[i][j] = __dp2a_lo(max16x2(rv.x, qv[j].x), 0x0101u, acc[i][j]);
                    acc[i][j] = __dp2a_lo(max16x2(rv.y, qv[j].y), 0x0101u, acc[i][j]);
                    acc[i][j] = __dp2a_lo(max16x2(rv.z, qv[j].z), 0x0101u, acc[i][j]);
                    acc[i][j] = __dp2a_lo(max16x2(rv.w, qv[j].w), 0x0101u, acc[i][j]);
                }
            }
        }
        __syncthreads();
    }
    const bool single = gridDim.z == 1;
    using Difference = std::conditional_t<NARROW, int, long long>;
    using Wrapping = std::make_unsigned_t<Difference>;
    constexpr Difference kMost =
        static_cast<Difference>(NARROW ? 0x7fffffffll : 0x7fffffffffffffffll);
    // T - error = 2 M - (query's sum) - under, T + error = 2 M - (query's sum) - over
    Wrapping under[8];
    Wrapping over[8];
    if (single) {
        if (tid < kQueries && q0 + tid < batch) {
            query_sums[tid] = query_terms(f, q0 + tid).sum;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t row = row0 + tr + 16 * i;
            const FixedTerms t = f.terms[min(row, row_count - 1)];
            under[i] = static_cast<Wrapping>(t.sum + t.error);
            over[i] = static_cast<Wrapping>(t.sum - t.error);
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const uint32_t qq = q0 + tq + 8 * j;
        if (single) {
            // the 16 threads of a half-warp share the query; lanes past the batch
            // take part in the shuffles with values that are not stored
            Difference low = kMost;
            Difference high = kMost;
            const Wrapping query = static_cast<Wrapping>(query_sums[tq + 8 * j]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t row = row0 + tr + 16 * i;
                const Wrapping t = 2 * static_cast<Wrapping>(acc[i][j]) - query;
                if (row < row_count) {
                    low = min(low, static_cast<Difference>(t - under[i]));
                    high = min(high, static_cast<Difference>(t - over[i]));
                }
            }
            for (int o = 8; o > 0; o /= 2) {
                low = min(low, __shfl_xor_sync(0xffffffffu, low, o));
                high = min(high, __shfl_xor_sync(0xffffffffu, high, o));
            }
            if (tr == 0 && qq < batch) {
                least[static_cast<uint64_t>(qq) * gridDim.x + blockIdx.x] =
                    static_cast<unsigned long long>(max(low, Difference(0)));
                atomicMin(f.upper + qq,
                          static_cast<unsigned long long>(max(high, Difference(0))));
            }
        }
        if (qq >= batch) {
            continue;
        }
        uint32_t* out = sums + (static_cast<uint64_t>(blockIdx.z) * batch + qq) * row_count;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t row = row0 + tr + 16 * i;
            if (row < row_count) {
                out[row] = acc[i][j];
            }
        }
    }
}

// ---------------------------------------------------------------- selection

// T of a row from its column splits.
__device__ __forceinline__ long long total_of(const uint32_t* base, uint64_t stride,
                                              uint32_t splits, uint32_t row, long long query_sum,
                                              const FixedTerms& terms)
{
    long long m = 0;
    for (uint32_t sp = 0; sp < splits; ++sp) {
        m += base[sp * stride + row];
    }
    return 2 * m - query_sum - terms.sum;
}

// grid (row blocks, queries), more than one split: the smallest T + error over the
// block's rows into upper[q].
__global__ void __launch_bounds__(kThreads)
    fixed_upper_kernel(const uint32_t* __restrict__ sums, uint32_t splits, uint32_t batch,
                       uint32_t row_count, const FixedQuery f)
{
    __shared__ QueryTerms query;
    const uint32_t q = blockIdx.y;
    if (threadIdx.x == 0) {
        query = query_terms(f, q);
    }
    __syncthreads();
    const uint64_t stride = static_cast<uint64_t>(batch) * row_count;
    const uint32_t* base = sums + static_cast<uint64_t>(q) * row_count;
    const uint32_t first = blockIdx.x * kThreads * kSelectRows + threadIdx.x;
    long long best = 0x7fffffffffffffffll;
#pragma unroll
    for (int u = 0; u < kSelectRows; ++u) {
        const uint32_t row = first + u * kThreads;
        if (row < row_count) {
            const FixedTerms t = f.terms[row];
            best = min(best, total_of(base, stride, splits, row, query.sum, t) + t.error);
        }
    }
    for (int o = 16; o > 0; o /= 2) {
        best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
    }
    if (threadIdx.x % 32 == 0) {
        atomicMin(f.upper + q, static_cast<unsigned long long>(max(best, 0ll)));
    }
}

// grid (row blocks, queries): the rows whose T - error is at most the smallest
// T + error, each with the query's error on its side, in any order, into the
// query's list; more than cap of them sets error bit kCandidateOverflow. With
// one split a warp skips the row tiles whose least value is past that.
__global__ void __launch_bounds__(kThreads)
    fixed_collect_kernel(const uint32_t* __restrict__ sums, uint32_t splits, uint32_t batch,
                         uint32_t row_count, const unsigned long long* __restrict__ least,
                         uint32_t tiles, const FixedQuery f, uint32_t cap,
                         uint32_t* __restrict__ candidates, int* error_flag)
{
    __shared__ QueryTerms query;
    const uint32_t q = blockIdx.y;
    if (threadIdx.x == 0) {
        query = query_terms(f, q);
    }
    __syncthreads();
    // both below 2^62
    const long long most =
        static_cast<long long>(min(f.upper[q], 1ull << 61)) + 2 * query.error;
    const uint64_t stride = static_cast<uint64_t>(batch) * row_count;
    const uint32_t* base = sums + static_cast<uint64_t>(q) * row_count;
    auto test = [&](uint32_t row) {
        const FixedTerms t = f.terms[row];
        if (total_of(base, stride, splits, row, query.sum, t) - t.error <= most) {
            const uint32_t slot = atomicAdd(f.counts + q, 1u);
            if (slot < cap) {
                candidates[static_cast<uint64_t>(q) * cap + slot] = row;
            } else {
                atomicOr(error_flag, kCandidateOverflow);
            }
        }
    };
    if (splits > 1) {
        const uint32_t first = blockIdx.x * kThreads * kSelectRows + threadIdx.x;
#pragma unroll
        for (int u = 0; u < kSelectRows; ++u) {
            const uint32_t row = first + u * kThreads;
            if (row < row_count) {
                test(row);
            }
        }
        return;
    }
    const uint32_t lane = threadIdx.x % 32;
    const uint32_t first = (blockIdx.x * kThreads + threadIdx.x) / 32 * 32;
    const uint32_t tile = first + lane;
    const bool in = tile < tiles &&
                    least[static_cast<uint64_t>(q) * tiles + tile] <=
                        static_cast<unsigned long long>(most);
    for (uint32_t set = __ballot_sync(0xffffffffu, in); set != 0; set &= set - 1) {
        const uint32_t row0 = (first + __ffs(set) - 1) * kRows;
        for (uint32_t r = row0 + lane; r < min(row_count, row0 + kRows); r += 32) {
            test(r);
        }
    }
}

template <int J, bool NARROW>
void launch_fixed_tiles(const FixedPlan& plan, const uint16_t* rows, uint32_t row_count,
                        const uint16_t* queries, uint32_t batch, uint64_t pitch, uint32_t* sums,
                        unsigned long long* least, const FixedQuery& f, cudaStream_t stream)
{
    const size_t smem = kStages * (kRows + 8 * J) * kStageStride;
    static std::once_flag once[kMaxDevices];
    std::call_once(once[current_device()], [&] {
        check_cuda(cudaFuncSetAttribute(fixed_tile_kernel<J, NARROW>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(smem)),
                   "cannot configure the fixed-point scan kernel");
    });
    const dim3 grid((row_count + kRows - 1) / kRows, (batch + 8 * J - 1) / (8 * J), plan.splits);
    fixed_tile_kernel<J, NARROW><<<grid, kTileThreads, smem, stream>>>(
        rows, row_count, queries, batch, pitch, plan.columns_per_split, sums, least, f);
    check_cuda(cudaGetLastError(), "cannot launch the fixed-point scan kernel");
}

}  // namespace

static uint32_t prep_threads(uint64_t slice)
{
    return static_cast<uint32_t>(
        std::min<uint64_t>(kPrepThreads, round_up((slice + 3) / 4, 32)));
}

uint64_t fixed_pitch(uint64_t dim)
{
    return round_up(dim == 0 ? 1 : dim, kStageColumns);
}

void launch_fixed_rows(const float* rows, uint64_t row_count, uint64_t padded, uint64_t dim,
                       const double* weights, uint16_t* out, uint64_t pitch, float* offsets,
                       FixedSummary* summary, FixedTerms* terms, unsigned int* ranges,
                       cudaStream_t stream)
{
    const uint32_t rc = static_cast<uint32_t>(row_count);
    unsigned int* low = ranges;
    unsigned int* high = ranges + dim;
    float* step = &summary->step;
    const uint32_t column_blocks = static_cast<uint32_t>((dim + kThreads - 1) / kThreads);
    const uint32_t slices = std::min((rc + kRangeRows - 1) / kRangeRows, kRangeSlices);
    column_range_kernel<<<dim3(column_blocks, slices), kThreads, 0, stream>>>(rows, rc, padded,
                                                                              dim, low, high);
    check_cuda(cudaGetLastError(), "cannot launch the column range kernel");
    column_offset_kernel<<<static_cast<uint32_t>((pitch + kThreads - 1) / kThreads), kThreads, 0,
                           stream>>>(low, high, dim, pitch, weights, offsets,
                                     reinterpret_cast<unsigned int*>(step));
    pair_sample_kernel<<<kFixedPairs, kThreads, 0, stream>>>(rows, rc, padded, dim, weights,
                                                             summary->pairs);
    FixedVectors v{};
    v.source_pitch = padded;
    v.dim = dim;
    v.weights = weights;
    v.offsets = offsets;
    v.step = step;
    v.pitch = pitch;
    v.slice = pitch;
    v.vector_loads = true;  // rows are padded to 16-byte boundaries
    v.error_flag = &summary->coarse;
    for (uint64_t at = 0; at < row_count; at += 65535) {
        const uint64_t count = std::min<uint64_t>(65535, row_count - at);
        v.source = rows + at * padded;
        v.out = out + at * pitch;
        v.terms = terms + at;
        fixed_vectors_kernel<true><<<dim3(1, static_cast<uint32_t>(count)),
                                     prep_threads(v.slice), 0, stream>>>(v);
    }
    check_cuda(cudaGetLastError(), "cannot launch the fixed-point row kernels");
}

bool fixed_usable(const FixedSummary* summary, uint64_t row_count, cudaStream_t stream)
{
    // the summary and the first rows' terms behind it, in one copy
    struct {
        FixedSummary sum;
        FixedTerms terms[kFixedPairs];
    } host;
    static_assert(sizeof(FixedSummary) % alignof(FixedTerms) == 0, "terms follow the summary");
    const uint64_t count = std::min<uint64_t>(row_count, kFixedPairs);
    check_cuda(cudaMemcpyAsync(&host, summary, sizeof(FixedSummary) + count * sizeof(FixedTerms),
                               cudaMemcpyDeviceToHost, stream),
               "cannot copy the rows' errors from the CUDA device");
    check_cuda(cudaStreamSynchronize(stream), "cannot build fixed-point rows");
    double distance = 0.0;
    for (double d : host.sum.pairs) {
        distance += d / kFixedPairs;
    }
    double error = 0.0;
    for (uint64_t i = 0; i < count; ++i) {
        error += static_cast<double>(host.terms[i].error) / static_cast<double>(count);
    }
    const float step = host.sum.step;
    // two vectors' errors within 1/512 of a typical distance: rows closer together
    // than that are rare enough for the candidate lists
    return host.sum.coarse == 0 && std::isfinite(step) && std::isfinite(distance) &&
           step >= 0x1p-100f && 1024.0 * error * static_cast<double>(step) <= distance;
}

uint32_t fixed_slices(uint64_t pitch, uint64_t batch)
{
    const uint64_t want = (2 * 148 + batch - 1) / batch;
    return static_cast<uint32_t>(std::min<uint64_t>(
        {want, (pitch + 2047) / 2048, static_cast<uint64_t>(kSplitSlices)}));
}

void launch_fixed_queries(FixedVectors v, uint64_t batch, cudaStream_t stream)
{
    const uint32_t slices = fixed_slices(v.pitch, batch);
    v.slice = round_up((v.pitch + slices - 1) / slices, kStageColumns);
    v.vector_loads = v.columns == nullptr && v.source_pitch % 4 == 0 &&
                     reinterpret_cast<uintptr_t>(v.source) % 16 == 0;
    fixed_vectors_kernel<false><<<dim3(slices, static_cast<uint32_t>(batch)),
                                  prep_threads(v.slice), 0, stream>>>(v);
    check_cuda(cudaGetLastError(), "cannot launch the fixed-point query kernel");
}

FixedPlan plan_fixed(uint64_t rows, uint64_t pitch, uint64_t batch, int sm_count)
{
    FixedPlan plan{};
    const uint64_t sms = static_cast<uint64_t>(sm_count > 0 ? sm_count : 148);
    const uint64_t row_tiles = (rows + kRows - 1) / kRows;
    const uint64_t most = std::max<uint64_t>(1, pitch / 512);
    // 32-query tiles where they pad less, or where 64-query tiles leave the chip
    // idle however the columns are split
    plan.queries = (round_up(batch, 32) < round_up(batch, 64) && batch < 512) ||
                           row_tiles * ((batch + 63) / 64) * most < 3 * sms
                       ? 32
                       : 64;
    const uint64_t tiles = row_tiles * ((batch + plan.queries - 1) / plan.queries);
    // Three or four CTAs fit an SM. The column split count whose CTAs fill their last
    // wave best, with at least 512 and at most 65,536 columns per split and four
    // waves unless one split already exceeds that; ties go to fewer splits.
    const uint64_t slots = (plan.queries == 32 ? 4 : 3) * sms;
    const uint64_t least = (pitch + 65535) / 65536;
    uint64_t splits = least;
    double best = -1.0;
    for (uint64_t s = least; s <= std::max(most, least); ++s) {
        const uint64_t ctas = tiles * s;
        if (s > least && ctas > 4 * slots) {
            break;
        }
        const uint64_t waves = (ctas + slots - 1) / slots;
        const double fill = static_cast<double>(ctas) / static_cast<double>(waves * slots);
        if (fill > best + 1e-9) {
            best = fill;
            splits = s;
        }
    }
    plan.columns_per_split =
        static_cast<uint32_t>(round_up((pitch + splits - 1) / splits, kStageColumns));
    plan.splits =
        static_cast<uint32_t>((pitch + plan.columns_per_split - 1) / plan.columns_per_split);
    return plan;
}

void launch_fixed_scan(const FixedPlan& plan, const uint16_t* rows, uint64_t row_count,
                       const uint16_t* queries, uint64_t batch, uint64_t pitch, uint32_t* sums,
                       unsigned long long* least, const FixedQuery& f, uint32_t* candidates, int* error_flag,
                       cudaStream_t stream)
{
    const uint32_t rc = static_cast<uint32_t>(row_count);
    const uint32_t b = static_cast<uint32_t>(batch);
    const bool narrow = f.dim <= kNarrowColumns;
    const auto launch =
        plan.queries == 32
            ? (narrow ? launch_fixed_tiles<4, true> : launch_fixed_tiles<4, false>)
            : (narrow ? launch_fixed_tiles<8, true> : launch_fixed_tiles<8, false>);
    launch(plan, rows, rc, queries, b, pitch, sums, least, f, stream);
    const uint32_t tiles = (rc + kRows - 1) / kRows;
    const dim3 grid((rc + kThreads * kSelectRows - 1) / (kThreads * kSelectRows), b);
    if (plan.splits > 1) {
        fixed_upper_kernel<<<grid, kThreads, 0, stream>>>(sums, plan.splits, b, rc, f);
    }
    fixed_collect_kernel<<<plan.splits > 1 ? grid : dim3((tiles + kThreads - 1) / kThreads, b),
                           kThreads, 0, stream>>>(sums, plan.splits, b, rc, least, tiles, f,
                                                  kSplitCandidates, candidates, error_flag);
    check_cuda(cudaGetLastError(), "cannot launch the fixed-point selection kernels");
}

uint64_t fixed_tiles(uint64_t rows)
{
    return (rows + kRows - 1) / kRows;
}

}  // namespace uha
