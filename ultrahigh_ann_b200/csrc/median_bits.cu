// Certified median scan of the L1 hierarchy by row bitmaps.
//
// A row can be a query's argmin only if at least half of its p values lie
// within a threshold T of the query's (hierarchical.cu). The register-tiled
// count decides that with about four instructions per (query, row, value). Here
// every column has kSlots boundaries b_0 <= b_1 <= ... taken from its own
// values, and for each boundary a bitmap over the rows: bit = value < b. For a
// query and a column, with lo the last boundary at most y - T and hi the first
// one above y + T (both rounded outwards),
//   bitmap[hi] & ~bitmap[lo]
// holds every row whose value is within T of y, and the rows of the two boundary
// bins at most; 32 rows per word and lane. The words of the p columns are added
// bit by bit (carry-save adders, three-input logic), so a count per row and
// query stands in about nine bit planes, and one comparison per word lists the
// rows that keep at least half of the values: a superset of the rows within T,
// about 1/64 of a column's rows per value wider.
//
// The threshold is tightened before the rows are counted: exact binary32
// medians of a few spread rows give T for one chunk of 1,024 rows, the listed
// rows' medians a smaller T for more chunks, and so on to all of them, so the
// last lists hold some ten rows per query.
//
// Every row the last pass lists gets its binary32 median with its own error
// bound, and the rows whose bounds can hold the minimum are settled by the
// reference's binary64 medians: the answer, and its distance, are the
// reference CPU's. The binary64 projection of the queries
// (l1_hierarchical_projection.cpp's order) is formed first, and the binary32
// queries are its roundings, so a query value's error is its own rounding only.
//
// Measured (B200, 65,536 rows, p = 64, 4,096 queries): 0.78 ms a call against
// 5.4 ms by the binary32 passes; the last count 278 us against 2,527 us, the
// medians 330 us in all against 2,030 us (about 160 rows listed per query, 10 of
// them within the threshold), no slab of 65,536 x 4,096 distances.
#include "async_copy.cuh"
#include "common.h"
#include "hier_body.cuh"
#include "kernels.h"
#include "median64.cuh"
#include "tile_body.cuh"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>

namespace uha {
namespace {

using namespace hierbody;

constexpr uint32_t kSlots = 64;          // bitmaps per column: 62 boundaries, none, all
constexpr uint32_t kChunkWords = 32;     // one word per lane
constexpr uint32_t kChunkRows = kChunkWords * 32;
constexpr uint32_t kColumnBytes = kSlots * kChunkWords * 4;  // one column of a chunk
constexpr uint32_t kGroup = 8;           // columns per stage
constexpr uint32_t kStageBytes = kGroup * kColumnBytes;
constexpr int kCountWarps = 32;
constexpr int kCountThreads = 32 * kCountWarps;
constexpr int kWarpQueries = 4;
constexpr uint32_t kBlockQueries = kCountWarps * kWarpQueries;
// a stage: the bitmaps, then each query's offsets of the group's columns
constexpr uint32_t kOffsetBytes = kBlockQueries * kGroup * 4;
constexpr uint32_t kFullStage = kStageBytes + kOffsetBytes;
constexpr int kBoundarySample = 1024;
constexpr int kProjectQueries = 4;   // per warp of the projection kernel
constexpr int kProjectThreads = 128;  // and columns per chunk
constexpr int kProjectColumns = 8;   // columns of the projection per stage
constexpr int kProjectStages = 3;
constexpr int kThreads = 256;
// polls of a copy wait before it gives up, and the error bit it then sets
constexpr uint32_t kCopySpins = 1u << 22;
constexpr int kCopyTimeout = 16;

// ------------------------------------------------------------- index side

// One block per column: boundaries[j][1 .. kSlots - 2] = quantiles of a sample of
// the column's values (any nondecreasing values are valid), boundaries 0 and
// kSlots - 1 infinite.
__global__ void __launch_bounds__(kBoundarySample)
    boundaries_kernel(const float* __restrict__ rows, uint32_t row_count, uint32_t padded_p,
                      float* __restrict__ boundaries)
{
    __shared__ float v[kBoundarySample];
    const uint32_t j = blockIdx.x;
    const uint32_t i = threadIdx.x;
    // a row may be taken more than once
    const uint64_t row = static_cast<uint64_t>(i) * row_count / kBoundarySample;
    v[i] = rows[row * padded_p + j];
    for (uint32_t size = 2; size <= kBoundarySample; size *= 2) {
        for (uint32_t stride = size / 2; stride > 0; stride /= 2) {
            __syncthreads();
            const uint32_t o = i ^ stride;
            if (o > i) {
                const bool ascending = (i & size) == 0;
                const float a = v[i];
                const float b = v[o];
                if ((a > b) == ascending) {
                    v[i] = b;
                    v[o] = a;
                }
            }
        }
    }
    __syncthreads();
    if (i < kSlots) {
        const float inf = __int_as_float(0x7f800000);
        boundaries[j * kSlots + i] =
            i == 0 ? -inf
                   : (i == kSlots - 1 ? inf : v[i * kBoundarySample / (kSlots - 1)]);
    }
}

// grid (chunks, columns), 1,024 threads: bits[chunk][column][slot][word]; warp w
// holds rows 32 w .. 32 w + 31 of the chunk. Rows past the index have no bit.
__global__ void __launch_bounds__(kChunkRows)
    row_bits_kernel(const float* __restrict__ rows, uint32_t row_count, uint32_t padded_p,
                    uint32_t p, const float* __restrict__ boundaries, uint32_t columns,
                    uint32_t* __restrict__ bits)
{
    __shared__ uint32_t out[kSlots][kChunkWords + 1];
    const uint32_t chunk = blockIdx.x;
    const uint32_t j = blockIdx.y;
    const uint32_t row = chunk * kChunkRows + threadIdx.x;
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const bool present = j < p && row < row_count;
    const float v = present ? rows[static_cast<uint64_t>(row) * padded_p + j] : 0.f;
    for (uint32_t s = 0; s < kSlots; ++s) {
        // the last slot, +infinity, holds every row
        const uint32_t word =
            __ballot_sync(0xffffffffu, present && v < boundaries[(j < p ? j : 0) * kSlots + s]);
        if (lane == 0) {
            out[s][warp] = word;
        }
    }
    __syncthreads();
    uint32_t* to = bits + (static_cast<uint64_t>(chunk) * columns + j) * kSlots * kChunkWords;
    for (uint32_t i = threadIdx.x; i < kSlots * kChunkWords; i += kChunkRows) {
        to[i] = out[i / kChunkWords][i % kChunkWords];
    }
}

// ------------------------------------------------------------- query side

// 8 bytes copied asynchronously into shared memory, or zeros
__device__ __forceinline__ void copy8(double* to, const double* from, bool ok)
{
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(to));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(from),
                 "r"(ok ? 8 : 0)
                 : "memory");
}

// grid (query groups), kProjectThreads threads: the sampled values of the group's
// queries gathered into shared memory (with the finiteness flag) and their
// binary64 projection in the reference's order, y = sum_i x_i P_i in i order. A
// warp takes kProjectQueries queries and C coordinates per lane (lane, lane + 32,
// ...), an independent chain per query and coordinate; `blocks` warps (a power of
// two) share a query over its coordinates, the rest of the CTA's warps take more
// queries. y64[q][p]; and, where y32 is given, its binary32 rounding (zero past
// p), that rounding's error per coordinate and its maximum.
//
// Bound: shared-memory reads of the queries (a broadcast of 8 bytes costs the
// return bandwidth of 32, two cycles per query and column; C coordinates share
// it), then the FP64 pipe (two instructions per query, coordinate and column).
// A chunk's scattered reads are all in flight at once, and the next chunk's
// behind the sums: one thread per column, one query value each. The projection's
// columns, which every CTA reads at about the same time, come kProjectColumns a
// stage through shared memory, two stages ahead (register loads four columns
// ahead left the warps waiting for them). 4,096 queries x about 370 columns,
// p = 64: 120 us with one coordinate and 8 queries per thread, the gather a load
// at a time and the weights from global memory; 62 us so (184 MB of DRAM lines
// for the scattered values).
template <int C>
__global__ void __launch_bounds__(kProjectThreads)
    gather_project64_kernel(const float* __restrict__ queries, uint32_t batch, uint64_t dim,
                            const uint32_t* __restrict__ columns, uint32_t k,
                            const double* __restrict__ proj_t, uint32_t p, uint32_t blocks,
                            double* __restrict__ y64, float* __restrict__ y32,
                            uint32_t padded_p, float* __restrict__ coord_err,
                            float* __restrict__ query_err, int* error_flag)
{
    constexpr int kWarps = kProjectThreads / 32;
    constexpr int kMost = kWarps * kProjectQueries;  // queries of a CTA, at most
    extern __shared__ __align__(16) double staged[];  // kProjectStages x columns x width
    __shared__ __align__(16) double x[kMost][kProjectThreads];
    __shared__ unsigned int largest[kMost];
    const uint32_t groups = kWarps / blocks;
    const uint32_t here = groups * kProjectQueries;  // queries of this CTA
    const uint32_t q0 = blockIdx.x * here;
    const uint32_t warp = threadIdx.x / 32;
    const uint32_t lane = threadIdx.x % 32;
    const uint32_t m0 = warp / blocks * kProjectQueries;
    if (threadIdx.x < kMost) {
        largest[threadIdx.x] = 0;
    }
    float next[kMost];
    auto fetch = [&](uint32_t i0) {
        const uint32_t i = i0 + threadIdx.x;
        const uint32_t column = i < k ? columns[i] : 0;
#pragma unroll
        for (int m = 0; m < kMost; ++m) {
            next[m] = i < k && m < here && q0 + m < batch ? queries[(q0 + m) * dim + column]
                                                          : 0.f;
        }
    };
    // coordinates in rounds of 32 C blocks (one round up to 512)
    for (uint32_t j0 = 0; j0 < padded_p; j0 += 32 * C * blocks) {
        const uint32_t j = j0 + warp % blocks * 32 * C + lane;
        double acc[kProjectQueries][C];
#pragma unroll
        for (int m = 0; m < kProjectQueries; ++m) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
                acc[m][c] = 0.0;
            }
        }
        const uint32_t width = 32 * C * blocks;  // a power of two
        const uint32_t shift = __ffs(width) - 1;
        const uint32_t stages = (k + kProjectColumns - 1) / kProjectColumns;
        auto stage = [&](uint32_t at) {
            if (at < stages) {
                double* to = staged + at % kProjectStages * kProjectColumns * width;
                for (uint32_t e = threadIdx.x; e < kProjectColumns * width;
                     e += kProjectThreads) {
                    const uint32_t i = at * kProjectColumns + (e >> shift);
                    const uint32_t c = j0 + (e & (width - 1));
                    const bool ok = i < k && c < p;
                    copy8(to + e, proj_t + (ok ? static_cast<uint64_t>(i) * p + c : 0), ok);
                }
            }
            tilebody::cp_async_commit();
        };
        __syncthreads();  // the last round's stages are read
        stage(0);
        stage(1);
        fetch(0);
        const double* mine = staged + warp % blocks * 32 * C + lane;
        for (uint32_t at = 0; at < stages; ++at) {
            const uint32_t i0 = at * kProjectColumns;
            const uint32_t in_chunk = i0 % kProjectThreads;
            if (in_chunk == 0) {
                __syncthreads();
                bool bad = false;
#pragma unroll
                for (int m = 0; m < kMost; ++m) {
                    bad |= !isfinite(next[m]);
                    x[m][threadIdx.x] = static_cast<double>(next[m]);
                }
                if (bad) {
                    atomicOr(error_flag, 1);
                }
                if (i0 + kProjectThreads < k) {
                    fetch(i0 + kProjectThreads);
                }
            }
            tilebody::cp_async_wait<1>();
            // stage `at` and the chunk are there, and the stage before is read
            __syncthreads();
            stage(at + 2);
            const double* w = mine + at % kProjectStages * kProjectColumns * width;
            const uint32_t count = min(static_cast<uint32_t>(kProjectColumns), k - i0);
            auto columns_of = [&](uint32_t u) {
                double wc[C];
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    wc[c] = w[u * width + 32 * c];
                }
#pragma unroll
                for (int m = 0; m < kProjectQueries; ++m) {
                    const double v = x[m0 + m][in_chunk + u];
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        acc[m][c] = __dadd_rn(acc[m][c], __dmul_rn(v, wc[c]));
                    }
                }
            };
            if (count == kProjectColumns) {
#pragma unroll 4
                for (uint32_t u = 0; u < kProjectColumns; ++u) {
                    columns_of(u);
                }
            } else {
                for (uint32_t u = 0; u < count; ++u) {
                    columns_of(u);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < kProjectQueries; ++m) {
            const uint32_t q = q0 + m0 + m;
            float worst = 0.f;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const uint32_t at = j + 32 * c;
                if (q >= batch || at >= padded_p) {
                    continue;
                }
                const double y = at < p ? acc[m][c] : 0.0;
                if (!isfinite(y)) {
                    atomicOr(error_flag, 4);
                }
                if (at < p) {
                    y64[static_cast<uint64_t>(q) * p + at] = y;
                }
                if (y32 != nullptr) {
                    const float r = static_cast<float>(y);
                    if (!(fabsf(r) <= FLT_MAX)) {
                        // past binary32: the binary32 scan answers (or refuses)
                        atomicOr(error_flag, kCandidateOverflow);
                    }
                    // exact: y and its rounding differ by at most half an ulp
                    const float e =
                        __double2float_ru(fabs(__dsub_rn(y, static_cast<double>(r))));
                    y32[static_cast<uint64_t>(q) * padded_p + at] = r;
                    coord_err[static_cast<uint64_t>(q) * padded_p + at] = e;
                    worst = e > worst || isnan(e) ? e : worst;
                }
            }
            // the bit patterns of nonnegative values (and NaN above them) order
            // as integers
            const unsigned int most = __reduce_max_sync(0xffffffffu, __float_as_uint(worst));
            if (lane == 0) {
                atomicMax(largest + m0 + m, most);
            }
        }
    }
    __syncthreads();
    if (y32 != nullptr && threadIdx.x < here && q0 + threadIdx.x < batch) {
        query_err[q0 + threadIdx.x] = __uint_as_float(largest[threadIdx.x]);
    }
}

// What the passes share.
struct Bits {
    const float* rows;        // row_count x padded_p
    uint32_t row_count;
    uint32_t padded_p;
    uint32_t p;
    const float* queries;     // batch x padded_p
    uint32_t batch;
    const float* query_err;
    const float* coord_err;
    float row_err_max;
    float rel;
    float abs_err;
    unsigned int* min_bits;   // per query: bits of the smallest median so far
    uint32_t* counts;         // per query: rows listed
    uint32_t* listed;         // batch x list rows
    float2* medians;          // batch x list: median, its error
    uint32_t list;            // rows listed per query at most
    int* error_flag;
    bool complete;            // the pass whose lists are settled
};

// grid (queries, parts), a warp per row: the binary32 medians of the query's
// listed rows (or, for the first threshold, of `spread` rows of the index),
// their errors, and the smallest median into min_bits. A row with fewer than
// `needed` values within the query's threshold so far is not the minimum: its
// entry gets median -1 (any threshold formed from medians of rows excludes
// only such rows, so a smaller one that another warp has just set is as good).
// The test costs a row some 30 instructions, its median about 500; most listed
// rows fail it (the bitmaps' boundary bins list some ten times the rows that
// pass).
template <int PER_LANE>
__global__ void __launch_bounds__(kThreads)
    list_medians_kernel(const Bits a, uint32_t spread, uint32_t needed)
{
    const uint32_t q = blockIdx.x;
    const int lane = threadIdx.x % 32;
    const uint32_t warps = gridDim.y * (kThreads / 32);
    const uint32_t n = spread != 0 ? spread : min(a.counts[q], a.list);
    const float* y = a.queries + static_cast<uint64_t>(q) * a.padded_p;
    const float* ye = a.coord_err + static_cast<uint64_t>(q) * a.padded_p;
    uint32_t* list = a.listed + static_cast<uint64_t>(q) * a.list;
    float2* medians = a.medians + static_cast<uint64_t>(q) * a.list;
    const volatile unsigned int* best = a.min_bits + q;
    for (uint32_t i = blockIdx.y * (kThreads / 32) + threadIdx.x / 32; i < n; i += warps) {
        const uint32_t row =
            spread != 0 ? static_cast<uint32_t>(static_cast<uint64_t>(i) * a.row_count / spread)
                        : list[i];
        const float* r = a.rows + static_cast<uint64_t>(row) * a.padded_p;
        float v[PER_LANE];
        const int valid = load_abs_diffs<PER_LANE>(r, y, a.p, lane, v);
        const unsigned int found = *best;
        const float t = threshold_of(found, a.query_err[q], a.row_err_max, a.rel, a.abs_err);
        uint32_t within = 0;
#pragma unroll
        for (int e = 0; e < PER_LANE; ++e) {
            within += __popc(__ballot_sync(0xffffffffu, e < valid && v[e] <= t));
        }
        if (within < needed) {
            if (spread == 0 && lane == 0) {
                medians[i] = make_float2(-1.f, 0.f);
            }
            continue;
        }
        float lower, upper;
        warp_middles<PER_LANE>(v, valid, a.p, lower, upper);
        const float median = a.p % 2 != 0 ? upper : lower + (upper - lower) * 0.5f;
        if (spread == 0) {
            // per coordinate: the row's binary32 rounding (at most 2^-24 |r|),
            // the query's error and the rounding of r - y
            float eps[PER_LANE];
#pragma unroll
            for (int e = 0; e < PER_LANE; ++e) {
                const uint32_t j = lane + 32u * e;
                eps[e] = j < a.p ? __fadd_ru(__fadd_ru(__fmul_ru(fabsf(r[j]), 0x1p-24f), ye[j]),
                                             __fmul_ru(v[e], 0x1p-24f))
                                 : 0.f;
            }
            const float err = warp_middle_error<PER_LANE>(v, eps, valid, lower, upper);
            if (lane == 0) {
                medians[i] = make_float2(median, err);
            }
        }
        if (lane == 0 && __float_as_uint(median) < found) {
            atomicMin(a.min_bits + q, __float_as_uint(median));
        }
    }
}

// One block per query (blocks past the batch fill its last group of
// kBlockQueries): each column's two boundaries as byte offsets of their bitmaps
// (hi << 16 | lo) from the query's threshold, offsets[group of columns][query][8];
// clears the query's list.
__global__ void intervals_kernel(const Bits a, const float* __restrict__ boundaries,
                                 uint32_t columns, uint32_t* __restrict__ offsets)
{
    const uint32_t q = blockIdx.x;
    if (q >= a.batch) {
        for (uint32_t j = threadIdx.x; j < columns; j += blockDim.x) {
            offsets[(static_cast<uint64_t>(j / kGroup) * gridDim.x + q) * kGroup + j % kGroup] =
                0;  // no row
        }
        return;
    }
    if (threadIdx.x == 0) {
        a.counts[q] = 0;
    }
    const float t = median_threshold(a.min_bits, a.query_err, q, a.row_err_max, a.rel, a.abs_err);
    // a value counted within t by the binary32 |r - y| lies within t (1 + 2^-22)
    const float reach = __fmul_ru(t, 1.f + 0x1p-22f);
    for (uint32_t j = threadIdx.x; j < columns; j += blockDim.x) {
        uint32_t lo = 0;
        uint32_t hi = 0;  // columns past p: no row
        if (j < a.p) {
            const float y = a.queries[static_cast<uint64_t>(q) * a.padded_p + j];
            const float low = __fsub_rd(y, reach);
            const float high = __fadd_ru(y, reach);
            const float* b = boundaries + j * kSlots;
            // the last boundary <= low, and the first one > high (an infinite
            // reach, or a NaN, ends at none and all)
            uint32_t first = 0;
            uint32_t last = kSlots - 1;
            while (last - first > 1) {
                const uint32_t mid = (first + last) / 2;
                if (b[mid] <= low) {
                    first = mid;
                } else {
                    last = mid;
                }
            }
            lo = first;
            first = 0;
            last = kSlots - 1;
            while (last - first > 1) {
                const uint32_t mid = (first + last) / 2;
                if (b[mid] > high) {
                    last = mid;
                } else {
                    first = mid;
                }
            }
            hi = last;
        }
        offsets[(static_cast<uint64_t>(j / kGroup) * gridDim.x + q) * kGroup + j % kGroup] =
            hi * (kChunkWords * 4) << 16 | lo * (kChunkWords * 4);
    }
}

// Carry-save adder of three bit vectors: sum into s, carry returned.
__device__ __forceinline__ uint32_t carry_save(uint32_t& s, uint32_t b, uint32_t c)
{
    const uint32_t a = s;
    s = a ^ b ^ c;
    return (a & b) | (a & c) | (b & c);
}

// grid (chunks taken, groups of kBlockQueries queries): the rows of chunk
// blockIdx.x * chunk_stride that keep at least `needed` of their p values within
// the queries' intervals, appended to the queries' lists. Eight columns' bitmaps
// (64 KB) and the block's offsets for them are copied into one of two stages
// while the other is counted; a warp holds the PLANES bit planes of four
// queries, lane = word. Bound: the integer pipe, half the issue rate. Per column,
// word and query: two shared-memory reads, four address operations, one and-not
// and 1.75 + (PLANES - 3) / 4 adder operations; the adders take eight columns at
// a time (seven carry-save steps, one carry rippled into the planes from 8 up).
template <int PLANES>
__global__ void __launch_bounds__(kCountThreads, 1)
    bits_count_kernel(const Bits a, const unsigned char* __restrict__ bits, uint32_t columns,
                      const uint32_t* __restrict__ offsets, uint32_t chunk_stride,
                      uint32_t needed)
{
    extern __shared__ __align__(128) unsigned char stages[];  // 2 x kFullStage
    __shared__ uint64_t full[2];
    __shared__ uint64_t empty[2];
    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    const uint32_t chunk = blockIdx.x * chunk_stride;
    const uint32_t q0 = blockIdx.y * kBlockQueries + warp * kWarpQueries;
    const uint32_t groups = columns / kGroup;
    const unsigned char* source = bits + static_cast<uint64_t>(chunk) * columns * kColumnBytes;
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            async::mbar_init(full + s, 1);
            async::mbar_init(empty + s, kCountWarps);
        }
        async::mbar_init_fence();
    }
    __syncthreads();
    auto copy = [&](uint32_t g) {  // thread 0
        const uint32_t s = g % 2;
        async::mbar_expect_tx(full + s, kFullStage);
        async::bulk_copy_g2s(stages + s * kFullStage, source + uint64_t(g) * kStageBytes,
                             kStageBytes, full + s);
        async::bulk_copy_g2s(stages + s * kFullStage + kStageBytes,
                             offsets + (static_cast<uint64_t>(g) * gridDim.y + blockIdx.y) *
                                           (kBlockQueries * kGroup),
                             kOffsetBytes, full + s);
    };
    if (threadIdx.x == 0) {
        copy(0);
    }
    uint32_t planes[kWarpQueries][PLANES];
#pragma unroll
    for (int m = 0; m < kWarpQueries; ++m) {
#pragma unroll
        for (int b = 0; b < PLANES; ++b) {
            planes[m][b] = 0;
        }
    }
    bool ok = true;
    for (uint32_t g = 0; g < groups; ++g) {
        const uint32_t s = g % 2;
        if (threadIdx.x == 0 && g + 1 < groups) {
            // the other stage is free once every warp has counted group g - 1
            if (g == 0 || async::mbar_wait(empty + (s ^ 1u), ((g - 1) / 2) & 1u, kCopySpins)) {
                copy(g + 1);
            } else {
                atomicOr(a.error_flag, kCopyTimeout);
            }
        }
        __syncwarp();
        ok = __all_sync(0xffffffffu, async::mbar_wait(full + s, (g / 2) & 1u, kCopySpins));
        if (!ok) {
            if (lane == 0) {
                atomicOr(a.error_flag, kCopyTimeout);
            }
            break;
        }
        const unsigned char* stage = stages + s * kFullStage + lane * 4;
        const uint4* group = reinterpret_cast<const uint4*>(stages + s * kFullStage +
                                                            kStageBytes) +
                             warp * kWarpQueries * 2;
#pragma unroll
        for (int m = 0; m < kWarpQueries; ++m) {
            const uint4 w0 = group[2 * m];
            const uint4 w1 = group[2 * m + 1];
            const uint32_t w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
            uint32_t in[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const unsigned char* column = stage + c * kColumnBytes;
                in[c] = *reinterpret_cast<const uint32_t*>(column + (w[c] >> 16)) &
                        ~*reinterpret_cast<const uint32_t*>(column + (w[c] & 0xffffu));
            }
            uint32_t* x = planes[m];
            const uint32_t t0 = carry_save(x[0], in[0], in[1]);
            const uint32_t t1 = carry_save(x[0], in[2], in[3]);
            const uint32_t f0 = carry_save(x[1], t0, t1);
            const uint32_t t2 = carry_save(x[0], in[4], in[5]);
            const uint32_t t3 = carry_save(x[0], in[6], in[7]);
            const uint32_t f1 = carry_save(x[1], t2, t3);
            uint32_t carry = carry_save(x[2], f0, f1);
#pragma unroll
            for (int b = 3; b < PLANES; ++b) {
                const uint32_t next = x[b] & carry;
                x[b] ^= carry;
                carry = next;
            }
        }
        __syncwarp();
        if (lane == 0) {
            // a local arrival: the reads above are done
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                             async::smem_u32(empty + s))
                         : "memory");
        }
    }
    if (!ok) {
        // the copies this block issued land before it exits (bounded)
        if (threadIdx.x == 0) {
            for (int s = 0; s < 2; ++s) {
                async::mbar_wait(full + s, 0, kCopySpins);
                async::mbar_wait(full + s, 1, kCopySpins);
            }
        }
        return;
    }
    uint32_t keep[kWarpQueries];
    uint32_t mine = 0;  // lane m: the rows of query m
#pragma unroll
    for (int m = 0; m < kWarpQueries; ++m) {
        uint32_t above = 0;
        uint32_t equal = 0xffffffffu;
#pragma unroll
        for (int b = PLANES - 1; b >= 0; --b) {
            const uint32_t bit = (needed >> b & 1u) != 0u ? 0xffffffffu : 0u;
            above |= equal & planes[m][b] & ~bit;
            equal &= ~(planes[m][b] ^ bit);
        }
        keep[m] = q0 + m < a.batch ? above | equal : 0u;
        const uint32_t total = __reduce_add_sync(0xffffffffu, __popc(keep[m]));
        mine = lane == m ? total : mine;
    }
    uint32_t base = 0;
    if (mine != 0) {
        base = atomicAdd(a.counts + q0 + lane, mine);
        // an earlier pass only tightens the threshold: any rows do
        if (a.complete && base + mine > a.list) {
            atomicOr(a.error_flag, kCandidateOverflow);
        }
    }
#pragma unroll
    for (int m = 0; m < kWarpQueries; ++m) {
        if (__shfl_sync(0xffffffffu, mine, m) == 0) {
            continue;
        }
        uint32_t at = __shfl_sync(0xffffffffu, base, m);
        uint32_t before = __popc(keep[m]);
#pragma unroll
        for (int o = 1; o < 32; o *= 2) {
            const uint32_t other = __shfl_up_sync(0xffffffffu, before, o);
            before += lane >= o ? other : 0u;
        }
        at += before - __popc(keep[m]);
        uint32_t* list = a.listed + static_cast<uint64_t>(q0 + m) * a.list;
        for (uint32_t bitsleft = keep[m]; bitsleft != 0u; bitsleft &= bitsleft - 1u, ++at) {
            if (at < a.list) {
                list[at] = chunk * kChunkRows + lane * 32 + (__ffs(bitsleft) - 1);
            }
        }
    }
}

// One warp per query, after the last pass: the listed rows whose bounds can hold
// the minimum, settled by the reference's binary64 medians (lowest row on
// ties). A query whose list overflowed, or whose values or medians are past
// binary32, stays open.
template <int PER_LANE>
__global__ void __launch_bounds__(kThreads)
    bits_settle_kernel(const Bits a, const double* __restrict__ rows64,
                       const double* __restrict__ y64, Result* results,
                       double* exact_distances, uint32_t* replay_count)
{
    const uint32_t q = blockIdx.x * (kThreads / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    if (q >= a.batch) {
        return;
    }
    const uint32_t n = a.counts[q] <= a.list && a.query_err[q] <= FLT_MAX ? a.counts[q] : 0u;
    const float2* medians = a.medians + static_cast<uint64_t>(q) * a.list;
    const uint32_t* list = a.listed + static_cast<uint64_t>(q) * a.list;
    // |reference median - m| <= rel m + err + abs
    auto reach = [&](float2 m) {
        return __fadd_ru(__fadd_ru(__fmul_ru(a.rel, m.x), m.y), a.abs_err);
    };
    float upper = __int_as_float(0x7f800000);
    for (uint32_t i = lane; i < n; i += 32) {
        const float2 m = medians[i];
        if (m.x >= 0.f) {
            upper = fminf(upper, __fadd_ru(m.x, reach(m)));
        }
    }
    for (int o = 16; o > 0; o /= 2) {
        upper = fminf(upper, __shfl_xor_sync(0xffffffffu, upper, o));
    }
    if (!(upper <= FLT_MAX)) {
        if (lane == 0) {
            atomicOr(a.error_flag, kCandidateOverflow);
            results[q] = Result{kOpenQuery, 0.f};
            exact_distances[q] = __longlong_as_double(0x7ff8000000000000ll);
        }
        return;
    }
    const double* y = y64 + static_cast<uint64_t>(q) * a.p;
    double best = __longlong_as_double(0x7ff0000000000000ll);
    uint32_t best_row = 0xffffffffu;
    uint32_t settled = 0;
    for (uint32_t base = 0; base < n; base += 32) {
        const uint32_t i = base + lane;
        const float2 m = i < n ? medians[i] : make_float2(-1.f, 0.f);
        const uint32_t mine = i < n ? list[i] : 0;
        // (a median past binary32 is above the finite upper bound or unordered:
        // kept)
        const bool keep = m.x >= 0.f && !(__fsub_rd(m.x, reach(m)) > upper);
        for (uint32_t mask = __ballot_sync(0xffffffffu, keep); mask != 0u; mask &= mask - 1u) {
            const uint32_t row = __shfl_sync(0xffffffffu, mine, __ffs(mask) - 1);
            const double d = median64::median_in_registers<PER_LANE>(
                rows64 + static_cast<uint64_t>(row) * a.p, y, a.p, lane);
            if (d < best || (d == best && row < best_row)) {
                best = d;
                best_row = row;
            }
            ++settled;
        }
    }
    if (lane == 0) {
        results[q] = Result{best_row, static_cast<float>(best)};
        exact_distances[q] = best;
        if (settled > 1) {
            atomicAdd(replay_count, 1u);
        }
    }
}

template <int PER_LANE>
void launch_list_medians(const Bits& a, uint32_t spread, uint32_t needed, cudaStream_t stream)
{
    // eight blocks per SM in all, a warp per row
    const uint32_t parts = std::max<uint32_t>(
        1, std::min<uint32_t>(16, 8 * 148 / std::max<uint32_t>(1, a.batch)));
    list_medians_kernel<PER_LANE><<<dim3(a.batch, parts), kThreads, 0, stream>>>(a, spread,
                                                                                 needed);
    check_cuda(cudaGetLastError(), "cannot launch the list median kernel");
}

template <int PLANES>
void launch_count(const Bits& a, const unsigned char* bits, uint32_t columns,
                  const uint32_t* offsets, uint32_t chunks, uint32_t stride, uint32_t needed,
                  cudaStream_t stream)
{
    static std::once_flag once[kMaxDevices];
    std::call_once(once[current_device()], [&] {
        check_cuda(cudaFuncSetAttribute(bits_count_kernel<PLANES>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(2 * kFullStage)),
                   "cannot configure the bitmap count kernel");
    });
    const dim3 grid(chunks, (a.batch + kBlockQueries - 1) / kBlockQueries);
    bits_count_kernel<PLANES><<<grid, kCountThreads, 2 * kFullStage, stream>>>(
        a, bits, columns, offsets, stride, needed);
    check_cuda(cudaGetLastError(), "cannot launch the bitmap count kernel");
}

// The passes of a batch whose values fit PER_LANE per lane and counts PLANES
// bits.
template <int PER_LANE, int PLANES>
uint64_t launch_passes(const Bits& a, const BitsScan& s, Result* results,
                       double* exact_distances, uint32_t* replay_count, cudaStream_t stream)
{
    const uint32_t columns = bits_columns(s.p);
    const uint32_t chunks = (a.row_count + kChunkRows - 1) / kChunkRows;
    // fewer than this many values within the threshold: the row's median is
    // above it (odd p: the middle one, even p: the lower middle)
    const uint32_t needed = a.p % 2 != 0 ? a.p / 2 + 1 : a.p / 2;
    launch_list_medians<PER_LANE>(a, std::min<uint32_t>(kBitsSpread, a.row_count), needed,
                                  stream);
    uint64_t launches = 2;
    const uint32_t padded = static_cast<uint32_t>(round_up(a.batch, kBlockQueries));
    // one chunk, then eight times as many at a time, then all (up to 16 times as
    // many as the level before)
    for (uint32_t taken = 1;; taken *= 8) {
        const bool all = chunks <= (taken == 1 ? 1 : 2 * taken);
        intervals_kernel<<<padded, std::min<uint32_t>(256, columns), 0, stream>>>(
            a, s.boundaries, columns, s.offsets);
        Bits pass = a;
        pass.complete = all;
        launch_count<PLANES>(pass, static_cast<const unsigned char*>(s.bits), columns, s.offsets,
                             all ? chunks : taken, all ? 1 : chunks / taken, needed, stream);
        launch_list_medians<PER_LANE>(a, 0, needed, stream);
        launches += 3;
        if (all) {
            break;
        }
    }
    bits_settle_kernel<PER_LANE>
        <<<(a.batch + kThreads / 32 - 1) / (kThreads / 32), kThreads, 0, stream>>>(
            a, s.rows64, s.y64, results, exact_distances, replay_count);
    check_cuda(cudaGetLastError(), "cannot launch the median settlement kernel");
    return launches;
}

}  // namespace

bool bits_applies(uint64_t rows, uint64_t p)
{
    return rows >= kBitsRows && rows <= 0xffffffffull - kChunkRows && p >= 1 && p <= 256;
}

uint32_t bits_list(uint64_t rows)
{
    // The last pass lists about 160 of 65,536 rows per query at p = 64. At p = 256
    // a query far from every row can list more than 1,024 (one or so in 4,096
    // queries, whose whole call the binary32 passes then answered again: 16.4 ms
    // against 2.3), so indexes of many rows get four times the slots.
    return rows <= 16384 ? 1024 : 4096;
}

bool bits_batch(uint64_t p, uint64_t batch)
{
    // A block streams a chunk's p columns (8 KB each) whatever the queries: 2 MB
    // per level at p = 256, where up to 16 queries took 235 to 245 us against 190
    // to 240 by the binary32 passes and 64 queries 250 to 355 against 255 to 328
    // (4,096 to 20,000 rows); up to p = 64 the bitmaps were ahead from one query
    // on.
    return p <= 64 || batch * 2 >= p;
}

uint32_t bits_columns(uint64_t p)
{
    return static_cast<uint32_t>(round_up(p, kGroup));
}

uint64_t bits_bytes(uint64_t rows, uint64_t p)
{
    return (rows + kChunkRows - 1) / kChunkRows * bits_columns(p) * kColumnBytes;
}

uint64_t bits_boundaries(uint64_t p)
{
    return p * kSlots;
}

void launch_row_bits(const float* rows, uint64_t row_count, uint64_t padded_p, uint64_t p,
                     float* boundaries, void* bits, cudaStream_t stream)
{
    const uint32_t rc = static_cast<uint32_t>(row_count);
    const uint32_t pp = static_cast<uint32_t>(padded_p);
    const uint32_t columns = bits_columns(p);
    boundaries_kernel<<<static_cast<uint32_t>(p), kBoundarySample, 0, stream>>>(rows, rc, pp,
                                                                                boundaries);
    const dim3 grid((rc + kChunkRows - 1) / kChunkRows, columns);
    row_bits_kernel<<<grid, kChunkRows, 0, stream>>>(rows, rc, pp, static_cast<uint32_t>(p),
                                                     boundaries, columns,
                                                     static_cast<uint32_t*>(bits));
    check_cuda(cudaGetLastError(), "cannot launch the row bitmap kernels");
}

void launch_gather_project64(const float* queries, uint64_t batch, uint64_t dim,
                             const uint32_t* columns, uint64_t k, const double* proj_t,
                             uint64_t p, double* y64, float* y32, uint64_t padded_p,
                             float* coord_err, float* query_err, int* error_flag,
                             cudaStream_t stream)
{
    // coordinates per lane, then warps per query, by the coordinates there are
    const uint32_t each = padded_p <= 32 ? 1 : padded_p <= 64 ? 2 : 4;
    const uint32_t blocks = padded_p <= 128 ? 1 : padded_p <= 256 ? 2 : 4;
    const uint32_t here = kProjectThreads / 32 / blocks * kProjectQueries;
    const uint32_t grid = static_cast<uint32_t>((batch + here - 1) / here);
    const auto kernel = each == 1   ? gather_project64_kernel<1>
                        : each == 2 ? gather_project64_kernel<2>
                                    : gather_project64_kernel<4>;
    const size_t smem = sizeof(double) * kProjectStages * kProjectColumns * 32 * each * blocks;
    if (smem > 32 * 1024) {
        static std::once_flag once[kMaxDevices];
        std::call_once(once[current_device()], [&] {
            // the most: 4 coordinates per lane, 4 warps per query
            check_cuda(cudaFuncSetAttribute(gather_project64_kernel<4>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            static_cast<int>(sizeof(double) * kProjectStages *
                                                             kProjectColumns * 32 * 4 * 4)),
                       "cannot configure the gathering projection kernel");
        });
    }
    kernel<<<grid, kProjectThreads, smem, stream>>>(
        queries, static_cast<uint32_t>(batch), dim, columns, static_cast<uint32_t>(k), proj_t,
        static_cast<uint32_t>(p), blocks, y64, y32, static_cast<uint32_t>(padded_p), coord_err,
        query_err, error_flag);
    check_cuda(cudaGetLastError(), "cannot launch the gathering projection kernel");
}

uint64_t launch_bits_scan(const BitsScan& s, uint64_t batch, Result* results,
                          double* exact_distances, uint32_t* replay_count, int* error_flag,
                          cudaStream_t stream)
{
    const uint32_t b = static_cast<uint32_t>(batch);
    const Bits a{s.rows,
                 static_cast<uint32_t>(s.row_count),
                 static_cast<uint32_t>(s.padded_p),
                 static_cast<uint32_t>(s.p),
                 s.queries,
                 b,
                 s.query_err,
                 s.coord_err,
                 s.row_err_max,
                 s.rel,
                 s.abs_err,
                 s.min_bits,
                 s.counts,
                 s.listed,
                 s.medians,
                 bits_list(s.row_count),
                 error_flag,
                 false};
    check_cuda(cudaMemsetAsync(a.min_bits, 0xff, batch * sizeof(unsigned int), stream),
               "cannot clear median thresholds");
    if (s.p <= 32) {
        return launch_passes<1, 7>(a, s, results, exact_distances, replay_count, stream);
    }
    if (s.p <= 64) {
        return launch_passes<2, 7>(a, s, results, exact_distances, replay_count, stream);
    }
    if (s.p <= 128) {
        return launch_passes<4, 9>(a, s, results, exact_distances, replay_count, stream);
    }
    return launch_passes<8, 9>(a, s, results, exact_distances, replay_count, stream);
}

uint64_t bits_offsets(uint64_t batch, uint64_t p)
{
    return round_up(batch, kBlockQueries) * bits_columns(p);
}

}  // namespace uha
