// Certified L2 scan of larger batches on the tensor cores.
//
// The certified path needs the reference CPU's binary64 argmin, not binary32
// distances of every row: any estimate with a bounded error decides which rows
// can be the minimum, and those few are settled from the original values in
// binary64 (certify.cu). The binary32 tile scan spends two CUDA-core
// instructions per (query, row, column) on that; here the estimate is a
// contraction on the fifth-generation tensor cores.
//
// Rows and queries are centred on the index's column means c (the distance does
// not change, the products shrink) and scaled by a power of two that brings the
// rows' norms near 1 where they are far from it; each value v is split into two
// BF16 parts, v = hi + lo + rest with |lo| <= 2^-9 |v|, |rest| <= 2^-18 |v|.
// S = lo.hi + hi.lo + hi.hi estimates q.r, and
//   e = ||r||^2 - 2 S
// orders the rows of a query as the squared distance does (||q||^2 is common).
// With a = ||q||, b = ||r|| (Cauchy-Schwarz on each sum of products):
//   the parts left out (lo.lo, rest.r, q.rest)       3 * 2^-18 a b
//   the tensor core: a 64-column chunk is 12 instructions of 16 products into
//     a fresh accumulator, the 8 small ones first. Measured on the B200, one
//     instruction aligns its products and the accumulator to the largest of
//     them, keeps 2^-25 of it, adds and truncates to 24 bits: at most
//     10.5 * 2^-24 of the magnitudes added (17 truncations and the last one);
//     2^-19, three times that, is assumed (of all these terms the one that rests
//     on a measurement)                               4.1 * 2^-19 a b
//   binary32 sums of the chunks and splits           (chunks + splits) 2^-24 a b
//   the centring's rounding, the norm's, the last
//     roundings and the reference's own               2^-21 (a + b)^2
//   underflow of parts and products                   2^-60 (norms to 2^40)
// A row whose e - E exceeds some row's e + E cannot be the minimum.
//
// Bound and measurements (B200, 7,028 x 60,660): 1,024 queries, tensor pipe,
// 1.82 ms = 1,440 TFLOP/s of BF16 products against 36 ms of the binary32 tile
// scan at its issue limit; 64 queries, memory (the split rows hold as many bytes
// as the binary32 ones), 0.30 ms = 5.7 TB/s against 2.4 ms. It was the faster one
// at every measured shape (33 to 65,536 rows, 128 to 60,660 columns, 9 to 4,096
// queries), so every direct L2 batch past the streaming scan's 8 queries takes
// it; the binary32 scan answers what it cannot decide.
//
// Kernel layout (persistent, one CTA per SM, 320 or 576 threads):
//   warp 0      TMA producer: per 64-column stage the hi and lo slices of 128
//               rows and BN queries, 128-byte swizzle
//   warp 1      TMEM allocation and the MMA issuer: 12 x tcgen05.mma
//               (M=128, N=BN, K=16) per stage into one of two accumulators
//   warps 2-    tcgen05.ld of a finished accumulator into binary32 register
//               sums while the other one fills; at a tile's end the sums go to
//               the partial slab [split][query][row], or through the filter
// Every mbarrier wait is bounded; one that runs out sets bit 8 of the error
// flag, and the CTA drains its copies and instructions (bounded) and returns.
#include "async_copy.cuh"
#include "common.h"
#include "kernels.h"
#include "tensor_core.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>
#include <type_traits>

namespace uha {
namespace {

using namespace tensorcore;

constexpr uint32_t kStageColumns = 64;  // one 128-byte swizzle row of BF16
constexpr int kPrepThreads = 512;
constexpr int kSelectThreads = 256;
// rows whose mean is the centre: more do not bring the norms down further, and the
// kernel's time (one thread per column) is theirs
constexpr uint64_t kCentreRows = 128;
constexpr float kLargestNorm = 0x1p40f;
// rows per thread of the selection kernels, their loads in flight together
constexpr int kSelectRows = 8;

// records an epilogue warp stages: flushed past 64, at most 32 more at a time;
// stages of a unit whose estimates are not stored, at most
constexpr uint32_t kStagedKeys = 96;
constexpr uint32_t kFusedStages = 8;

// What the score kernel's epilogue does with its estimates (see the kernel).
enum class Score : int { slab, least, filter };

// Epilogue warps: two per TMEM lane quarter, sharing the BN columns; four on wide
// tiles that are not stored (the work per estimate is most of a short tile's
// time, and two warps per scheduler do not hide its waits).
template <int BN, Score MODE>
struct Epilogue {
    static constexpr int warps = MODE != Score::slab && BN >= 256 ? 16 : 8;
    static constexpr int threads = 64 + 32 * warps;
    static constexpr int columns = BN / (warps / 4);  // per warp
};

template <int BN, int STAGES, Score MODE>
struct SplitSmem {
    static constexpr uint32_t a_bytes = kTileRows * kSliceBytes;
    static constexpr uint32_t b_bytes = BN * kSliceBytes;
    static constexpr uint32_t stage_bytes = 2 * (a_bytes + b_bytes);
    static constexpr uint32_t tiles = STAGES * stage_bytes;
    static constexpr uint32_t barriers = (2 * STAGES + 5) * 8 + 16;
    // per epilogue warp (not slab): staged records and its columns' sides
    static constexpr uint32_t warp_bytes =
        kStagedKeys * 12 + Epilogue<BN, MODE>::columns * 8;
    static constexpr uint32_t warps_at = (tiles + barriers + 15) / 16 * 16;
    // 1024-byte alignment slack + barriers + TMEM slot + abort word
    static constexpr uint32_t total =
        1024 + warps_at + (MODE != Score::slab ? Epilogue<BN, MODE>::warps * warp_bytes : 0);
    static constexpr uint32_t tmem_cols = 2 * BN;
};

// The root of a squared norm, rounded up (the binary64 sum and root carry a
// relative error far below 1e-9).
__device__ __forceinline__ float root_up(double square)
{
    return __double2float_ru(sqrt(square) * (1.0 + 1e-9));
}

// Unsigned bits that order like the binary32 value.
__device__ __forceinline__ unsigned int ordered(float f)
{
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float from_ordered(unsigned int u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// One epilogue warp's records waiting for their places in the query lists.
struct KeyStage {
    unsigned long long key[kStagedKeys];
    uint32_t query[kStagedKeys];
};

// The staged records of one warp into the lists; one atomic per record, all of
// the warp's in flight together.
__device__ __forceinline__ void flush_keys(const KeyStage& stage, uint32_t count,
                                           const SplitQuery& sq, const SplitList& list,
                                           int lane)
{
    for (uint32_t i = lane; i < count; i += 32) {
        const uint32_t q = stage.query[i];
        const uint32_t slot = atomicAdd(sq.counts + q, 1u);
        if (slot < list.cap) {
            list.keys[static_cast<uint64_t>(q) * list.cap + slot] = stage.key[i];
        }
    }
}

// With c = 2^-21, E = rel a b + c (a + b)^2 + 2^-60. A column's (query's) sides:
// slope = (rel + 2 c) a, and what it adds to the smallest e + E,
//   e + E = (norm + c b^2) - 2 S + slope b + (c a^2 + 2^-60),
// and to its threshold tau,
//   e - E <= tau  <=>  norm - c b^2 <= 2 S + slope b + (tau + c a^2 + 2^-60).
__device__ __forceinline__ float slope_of(float a, float rel)
{
    return __fmul_ru(__fadd_ru(rel, 0x1p-20f), a);
}

__device__ __forceinline__ float own_square(float a)
{
    return __fadd_ru(__fmul_ru(0x1p-21f, __fmul_ru(a, a)), 0x1p-60f);
}

// The filter's right-hand side for one estimate, rounded up.
__device__ __forceinline__ float filter_side(float slope, float base, float b, float s)
{
    return __fmaf_ru(2.f, s, __fmaf_ru(slope, b, base));
}

// ||q|| rounded up from the query's slices.
__device__ __forceinline__ float root_of(const SplitQuery& sq, uint32_t q)
{
    double total = 0.0;
    for (uint32_t s = 0; s < sq.slices; ++s) {
        total += sq.squares[static_cast<uint64_t>(q) * sq.slices + s];
    }
    return root_up(total);
}

// The minimum over the warp of 16 values per lane: the lane's column of them.
__device__ __forceinline__ float column_minimum(float (&m)[16], int lane)
{
#pragma unroll
    for (int half = 8; half > 0; half /= 2) {
        const bool high = (lane & (2 * half)) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float mine = high ? m[i + half] : m[i];
            const float other = high ? m[i] : m[i + half];
            m[i] = fminf(mine, __shfl_xor_sync(0xffffffffu, other, 2 * half));
        }
    }
    return fminf(m[0], __shfl_xor_sync(0xffffffffu, m[0], 1));
}

// The column whose minimum column_minimum() leaves in a lane.
__device__ __forceinline__ uint32_t minimum_column(int lane)
{
    return static_cast<uint32_t>(lane / 2);
}

// One unit is a (row tile, query tile, split); the CTA takes the units blockIdx.x, blockIdx.x + gridDim.x, ...
//
// slab    partial estimates of q.r, partials[split][q][row], over the split's
//         columns; query tiles fastest, so the CTAs running together share row
//         and query tiles in L2.
// least   (one split) the smallest e + E of each query over the scored tiles
//         into its word `upper`: 16 columns' minima over a warp's rows in one
//         butterfly, then one reduction per column and warp.
// filter  (one split) the rows whose e - E is at most the query's threshold,
//         appended to its list as keys (e, row).
// Row tile t is the index's tile t * tile_stride (a stride above 1 scores
// whole tiles spread over the index).
//
// In the last two, row tiles are fastest (a query tile's sides are formed once
// per few tiles), the unit's few stages accumulate in TMEM (a wider bound than
// register sums: split_error_rel), and the epilogue takes 16 columns at a time
// from there in a rolled loop. It bounds short tiles, by waits and instruction
// fetches rather than issue: unrolled over register sums its code did not fit
// the instruction cache (22 of 36 stall cycles per issue; 65,536 x 4,096
// estimates of 64 columns took 1.51 ms, now 139 us, of which the loads
// and MMAs alone take 90 us). A group of 16 columns without a passing row costs
// two FMAs and a maximum per estimate and one vote. Passing rows are staged per
// warp and reach the lists 64 and more at a time, so the epilogue waits for an
// atomic's round trip once per many tiles.
template <int BN, int STAGES, Score MODE>
__global__ void __launch_bounds__(Epilogue<BN, MODE>::threads, 1)
    split_score_kernel(const __grid_constant__ CUtensorMap rows_map,
                       const __grid_constant__ CUtensorMap queries_map, uint32_t kblocks,
                       uint32_t kblocks_per_split, uint32_t query_tiles, uint32_t row_tiles,
                       uint32_t units, uint32_t tile_stride, uint32_t row_count, uint32_t batch,
                       float* __restrict__ partials, const SplitQuery sq,
                       const SplitList list, int* error_flag)
{
    using L = SplitSmem<BN, STAGES, MODE>;
    constexpr bool kFused = MODE != Score::slab;
    constexpr int kColumns = Epilogue<BN, MODE>::columns;  // accumulator columns per warp
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::tiles);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;  // 2
    uint64_t* acc_empty = acc_full + 2;   // 2
    uint64_t* drained = acc_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
    volatile int* aborted = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    if (warp == 0 && lane == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(acc_full + s, 1);
            mbar_init(acc_empty + s, Epilogue<BN, MODE>::warps);
        }
        mbar_init(drained, 1);
        *aborted = 0;
        async::mbar_init_fence();
        prefetch_map(&rows_map);
        prefetch_map(&queries_map);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, L::tmem_cols);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    auto give_up = [&]() {
        *aborted = 1;
        atomicOr(error_flag, kPipelineTimeout);
    };
    auto query_tile = [&](uint32_t unit) {
        return kFused ? unit / row_tiles : unit % query_tiles;
    };
    auto row_tile = [&](uint32_t unit) {
        return kFused ? unit % row_tiles : unit / query_tiles % row_tiles;
    };
    auto steps_of = [&](uint32_t unit) {
        const uint32_t begin = unit / (query_tiles * row_tiles) * kblocks_per_split;
        return min(kblocks, begin + kblocks_per_split) - begin;
    };

    if (warp == 0) {
        if (lane == 0) {
            uint32_t g = 0;  // stages issued
            for (uint32_t unit = blockIdx.x; unit < units && !*aborted; unit += gridDim.x) {
                const int32_t q0 = static_cast<int32_t>(query_tile(unit)) * BN;
                const int32_t r0 =
                    static_cast<int32_t>(row_tile(unit) * tile_stride) * kTileRows;
                const uint32_t kb =
                    unit / (query_tiles * row_tiles) * kblocks_per_split;
                const uint32_t steps = steps_of(unit);
                for (uint32_t i = 0; i < steps && !*aborted; ++i, ++g) {
                    const uint32_t s = g % STAGES;
                    if (!mbar_wait(empty + s, ((g / STAGES) & 1u) ^ 1u)) {
                        give_up();
                        break;
                    }
                    unsigned char* a = smem + s * L::stage_bytes;
                    unsigned char* b = a + 2 * L::a_bytes;
                    mbar_expect_tx(full + s, L::stage_bytes);
                    // a stage's columns are stored hi, then lo
                    const int32_t x = static_cast<int32_t>((kb + i) * 2 * kStageColumns);
                    const int32_t lo = x + static_cast<int32_t>(kStageColumns);
                    tma_load_2d(a, &rows_map, full + s, x, r0);
                    tma_load_2d(a + L::a_bytes, &rows_map, full + s, lo, r0);
                    tma_load_2d(b, &queries_map, full + s, x, q0);
                    tma_load_2d(b + L::b_bytes, &queries_map, full + s, lo, q0);
                }
            }
            if (*aborted) {
                // every issued copy lands before the CTA exits
                const uint32_t first = g > STAGES ? g - STAGES : 0;
                for (uint32_t i = first; i < g; ++i) {
                    mbar_wait(full + i % STAGES, (i / STAGES) & 1u);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = mma_idesc(false, BN);
            uint32_t g = 0;    // stages
            uint32_t turn = 0; // accumulators: one per stage, or per unit
            for (uint32_t unit = blockIdx.x; unit < units && !*aborted; unit += gridDim.x) {
                const uint32_t steps = steps_of(unit);
                for (uint32_t i = 0; i < steps && !*aborted; ++i, ++g) {
                    const uint32_t s = g % STAGES;
                    const uint32_t acc = turn % 2;
                    const bool fresh = !kFused || i == 0;
                    if ((fresh && !mbar_wait(acc_empty + acc, ((turn / 2) & 1u) ^ 1u)) ||
                        !mbar_wait(full + s, (g / STAGES) & 1u)) {
                        give_up();
                        break;
                    }
                    tc_fence_after();
                    const uint32_t base = smem_u32(smem + s * L::stage_bytes);
                    const uint64_t a_hi = sw128_desc(base);
                    const uint64_t a_lo = sw128_desc(base + L::a_bytes);
                    const uint64_t b_hi = sw128_desc(base + 2 * L::a_bytes);
                    const uint64_t b_lo = sw128_desc(base + 2 * L::a_bytes + L::b_bytes);
                    const uint32_t d = tmem + acc * BN;
                    // the small products first, so their roundings stay small;
                    // +32 bytes of K per instruction inside the swizzle atom
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; ++kk) {
                        mma_issue<false>(d, a_lo + 2 * kk, b_hi + 2 * kk, idesc,
                                         !fresh || kk != 0 ? 1u : 0u);
                    }
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; ++kk) {
                        mma_issue<false>(d, a_hi + 2 * kk, b_lo + 2 * kk, idesc, 1);
                    }
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; ++kk) {
                        mma_issue<false>(d, a_hi + 2 * kk, b_hi + 2 * kk, idesc, 1);
                    }
                    mma_commit(empty + s);
                    if (!kFused || i + 1 == steps) {
                        mma_commit(acc_full + acc);
                        ++turn;
                    }
                }
            }
            // every instruction has completed before TMEM is freed
            mma_commit(drained);
            mbar_wait(drained, 0);
        }
        __syncwarp();
    } else {
        const uint32_t quarter = static_cast<uint32_t>(warp % 4) * 32;  // TMEM lanes
        const uint32_t column0 = static_cast<uint32_t>((warp - 2) / 4) * kColumns;
        uint32_t turn = 0;
        // Waits for this turn's accumulator; warp-uniform (tcgen05.ld is executed
        // by all 32 lanes or none).
        auto accumulated = [&]() {
            const bool ok = __all_sync(0xffffffffu,
                                       mbar_wait(acc_full + turn % 2, (turn / 2) & 1u) &&
                                           !*aborted);
            if (!ok && lane == 0) {
                give_up();
            }
            tc_fence_after();
            return ok;
        };
        auto release = [&]() {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(acc_empty + turn % 2);
            }
            ++turn;
        };
        if constexpr (kFused) {
            unsigned char* mine = smem + L::warps_at + (warp - 2) * L::warp_bytes;
            // per column: slope, and the filter's base
            float2* sides = reinterpret_cast<float2*>(mine);
            KeyStage& stage = *reinterpret_cast<KeyStage*>(mine + kColumns * sizeof(float2));
            uint32_t staged = 0;
            uint32_t loaded_tile = 0xffffffffu;
            const float inf = __int_as_float(0x7f800000);
            for (uint32_t unit = blockIdx.x; unit < units; unit += gridDim.x) {
                const uint32_t scored = row_tile(unit) * kTileRows + quarter + lane;
                const uint32_t row = row_tile(unit) * tile_stride * kTileRows + quarter + lane;
                const uint32_t q0 = query_tile(unit) * BN + column0;
                // in flight behind the wait for the accumulator
                const bool row_ok = scored < row_count;
                const float b = row_ok ? sq.roots[row] : 0.f;
                // a NaN: a row past the end passes no comparison (infinity would pass
                // against an infinite side; the least pass takes whole tiles only)
                const float norm = row_ok ? sq.norms[row] : __int_as_float(0x7fffffff);
                if (query_tile(unit) != loaded_tile) {
                    loaded_tile = query_tile(unit);
                    __syncwarp();
                    for (int c = lane; c < kColumns; c += 32) {
                        float2 side = make_float2(0.f, -inf);
                        const float a = q0 + c < batch ? root_of(sq, q0 + c) : inf;
                        // a norm the bound does not cover (split_narrow_kernel
                        // reports it) lists nothing: its sides may be infinite
                        if (a <= kLargestNorm) {
                            side.x = slope_of(a, sq.rel);
                            if (MODE == Score::filter) {
                                // tau is the word plus the query's own square
                                const float own = own_square(a);
                                side.y = __fadd_ru(
                                    __fadd_ru(from_ordered(sq.upper[q0 + c]), own), own);
                            }
                        }
                        sides[c] = side;
                    }
                    __syncwarp();
                }
                if (!accumulated()) {
                    break;
                }
                // the row's side
                const float square = __fmul_ru(0x1p-21f, __fmul_ru(b, b));
                const float low = MODE == Score::filter ? __fsub_rd(norm, square)
                                                        : __fadd_ru(norm, square);
                const uint32_t from = tmem + (quarter << 16) + turn % 2 * BN + column0;
#pragma unroll 1
                for (int c0 = 0; c0 < kColumns; c0 += 16) {
                    float v[16];
                    tmem_load16(from + c0, v);
                    if (c0 + 16 == kColumns) {
                        release();
                    }
                    const float4* side2 = reinterpret_cast<const float4*>(sides + c0);
                    if constexpr (MODE == Score::least) {
#pragma unroll
                        for (int j = 0; j < 16; j += 2) {
                            const float4 l = side2[j / 2];
                            v[j] = __fmaf_ru(-2.f, v[j], __fmaf_ru(l.x, b, low));
                            v[j + 1] = __fmaf_ru(-2.f, v[j + 1], __fmaf_ru(l.z, b, low));
                        }
                        const float least = column_minimum(v, lane);
                        const uint32_t q = q0 + c0 + minimum_column(lane);
                        if (lane % 2 == 0 && q < batch) {
                            atomicMin(sq.upper + q, ordered(least));
                        }
                    } else {
                        float most = -inf;
#pragma unroll
                        for (int j = 0; j < 16; j += 2) {
                            const float4 l = side2[j / 2];
                            most = fmaxf(most, fmaxf(filter_side(l.x, l.y, b, v[j]),
                                                     filter_side(l.z, l.w, b, v[j + 1])));
                        }
                        if (!__any_sync(0xffffffffu, most >= low)) {
                            continue;
                        }
                        // the lane's passing columns, taken one per turn
                        uint32_t bits = 0;
#pragma unroll
                        for (int j = 0; j < 16; j += 2) {
                            const float4 l = side2[j / 2];
                            bits |= filter_side(l.x, l.y, b, v[j]) >= low ? 1u << j : 0u;
                            bits |= filter_side(l.z, l.w, b, v[j + 1]) >= low ? 2u << j : 0u;
                        }
                        for (uint32_t mask = __ballot_sync(0xffffffffu, bits != 0u); mask != 0u;
                             mask = __ballot_sync(0xffffffffu, bits != 0u)) {
                            if (bits != 0u) {
                                const int j = __ffs(bits) - 1;
                                bits &= bits - 1u;
                                float s = v[0];
#pragma unroll
                                for (int i = 1; i < 16; ++i) {
                                    s = i == j ? v[i] : s;
                                }
                                const uint32_t at =
                                    staged + __popc(mask & ((1u << lane) - 1u));
                                stage.query[at] = q0 + c0 + j;
                                stage.key[at] =
                                    (static_cast<unsigned long long>(
                                         __float_as_uint(__fmaf_rn(-2.f, s, norm)))
                                     << 32) |
                                    row;
                            }
                            staged += __popc(mask);
                            if (staged > kStagedKeys - 32) {
                                __syncwarp();
                                flush_keys(stage, staged, sq, list, lane);
                                __syncwarp();
                                staged = 0;
                            }
                        }
                    }
                }
            }
            if (MODE == Score::filter) {
                __syncwarp();
                flush_keys(stage, staged, sq, list, lane);
            }
        } else {
            float sum[kColumns];
            for (uint32_t unit = blockIdx.x; unit < units; unit += gridDim.x) {
#pragma unroll
                for (int c = 0; c < kColumns; ++c) {
                    sum[c] = 0.f;
                }
                const uint32_t steps = steps_of(unit);
                bool ok = true;
                for (uint32_t i = 0; i < steps; ++i) {
                    ok = accumulated();
                    if (!ok) {
                        break;
                    }
                    const uint32_t from = tmem + (quarter << 16) + turn % 2 * BN + column0;
#pragma unroll
                    for (int c = 0; c < kColumns; c += 16) {
                        float v[16];
                        tmem_load16(from + c, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            sum[c + j] = __fadd_rn(sum[c + j], v[j]);
                        }
                    }
                    release();
                }
                if (!ok) {
                    break;
                }
                const uint32_t row = row_tile(unit) * kTileRows + quarter + lane;
                const uint32_t q0 = query_tile(unit) * BN + column0;
                const uint32_t split = unit / (query_tiles * row_tiles);
                if (row < row_count) {
                    float* out = partials +
                                 (static_cast<uint64_t>(split) * batch + q0) * row_count + row;
#pragma unroll
                    for (int c = 0; c < kColumns; ++c) {
                        if (q0 + c < batch) {
                            out[static_cast<uint64_t>(c) * row_count] = sum[c];
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, L::tmem_cols);
    }
}

// --------------------------------------------------------- splitting kernels

// centre[j] = the mean of column j over `take` rows spread over the source (any
// value is valid; the mean makes the centred norms small), zeros past dim.
template <typename T>
__global__ void column_centre_kernel(const T* __restrict__ rows, uint64_t row_count,
                                     uint64_t src_pitch, uint64_t dim, uint32_t take,
                                     float* __restrict__ centre, uint64_t pitch)
{
    const uint64_t j = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    if (j >= pitch) {
        return;
    }
    double sum = 0.0;
    if (j < dim) {
#pragma unroll 8
        for (uint32_t i = 0; i < take; ++i) {
            sum += static_cast<double>(rows[row_count * i / take * src_pitch + j]);
        }
    }
    centre[j] = static_cast<float>(sum / take);
}

// What a split vector is made from: index rows (binary32, or a hierarchy's
// binary64 projected ones), dense queries, queries whose sampled columns are
// gathered (and scaled), or binary64 projected queries.
enum class SplitSource : int { rows, rows64, dense, sampled, projected };

// grid (slices, vectors): v = (source - centre) * scale (a power of two) over
// the slice's columns, split into hi and lo BF16 parts (stored as 64 hi, 64 lo,
// 64 hi, ... columns, zeros past dim), and its part of the squared norm. Query
// sources also get the preparation kernels' work: the finiteness flags and the
// prepared binary32 vector that the settlement reads (one pass over the
// queries instead of two); the first slice's thread 0 clears the query's list.
//
// Bound: memory (read 4, write 4 + 4 bytes per value); slices keep the chip
// busy when there are few vectors.
template <SplitSource SRC>
__global__ void __launch_bounds__(kPrepThreads)
    split_vectors_kernel(const SplitVectors v)
{
    constexpr bool kWide = SRC == SplitSource::projected || SRC == SplitSource::rows64;
    constexpr bool kRows = SRC == SplitSource::rows || SRC == SplitSource::rows64;
    using T = std::conditional_t<kWide, double, float>;
    __shared__ double scratch[kPrepThreads / 32];
    const uint64_t i = blockIdx.y;
    const T* in = static_cast<const T*>(v.source) + i * v.source_pitch;
    __nv_bfloat16* o = static_cast<__nv_bfloat16*>(v.out) + i * 2 * v.pitch;
    const uint64_t begin = blockIdx.x * v.slice;
    const uint64_t end = min(v.pitch, begin + v.slice);
    double acc = 0.0;
    int bad = 0;
    // four columns per thread and step; slices and pitch are multiples of 64
    for (uint64_t j = begin + 4ull * threadIdx.x; j < end; j += 4ull * blockDim.x) {
        alignas(8) __nv_bfloat16 hi[4];
        alignas(8) __nv_bfloat16 lo[4];
        T x[4];
        const float4 c = *reinterpret_cast<const float4*>(v.centre + j);
        const float cs[4] = {c.x, c.y, c.z, c.w};
        if constexpr (SRC == SplitSource::sampled) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x[e] = j + e < v.dim ? in[v.columns[j + e]] : 0.f;
                bad |= isfinite(x[e]) ? 0 : 1;
                if (v.scales != nullptr && j + e < v.dim) {
                    x[e] = __fmul_rn(x[e], v.scales[j + e]);
                    bad |= isfinite(x[e]) ? 0 : 2;
                }
            }
        } else if (!kWide && v.vector_loads) {
            // whole groups: binary32 rows are zero from dim to their pitch
            if (j < v.source_pitch) {
                const float4 f = *reinterpret_cast<const float4*>(in + j);
                x[0] = f.x;
                x[1] = f.y;
                x[2] = f.z;
                x[3] = f.w;
            } else {
                x[0] = x[1] = x[2] = x[3] = T(0);
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x[e] = j + e < v.dim ? in[j + e] : T(0);
            }
        }
        if constexpr (SRC == SplitSource::dense) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                bad |= isfinite(x[e]) ? 0 : 1;
            }
        }
        if constexpr (SRC == SplitSource::dense || SRC == SplitSource::sampled) {
            if (j < v.prepared_pitch) {  // a multiple of 4
                *reinterpret_cast<float4*>(v.prepared + i * v.prepared_pitch + j) =
                    make_float4(x[0], x[1], x[2], x[3]);
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            // the centre is 0 past dim, and so is every source there
            const T d = (x[e] - static_cast<T>(cs[e])) * static_cast<T>(v.scale);
            hi[e] = __float2bfloat16_rn(static_cast<float>(d));
            const T rest = d - static_cast<T>(__bfloat162float(hi[e]));
            lo[e] = __float2bfloat16_rn(static_cast<float>(rest));
            acc = fma(static_cast<double>(d), static_cast<double>(d), acc);
        }
        const uint64_t at = j / kStageColumns * (2 * kStageColumns) + j % kStageColumns;
        *reinterpret_cast<uint2*>(o + at) = *reinterpret_cast<const uint2*>(hi);
        *reinterpret_cast<uint2*>(o + at + kStageColumns) = *reinterpret_cast<const uint2*>(lo);
    }
    if (bad != 0) {
        atomicOr(v.error_flag, bad);
    }
    for (int s = 16; s > 0; s /= 2) {
        acc += __shfl_xor_sync(0xffffffffu, acc, s);
    }
    if (threadIdx.x % 32 == 0) {
        scratch[threadIdx.x / 32] = acc;
    }
    __syncthreads();
    if (threadIdx.x != 0) {
        return;
    }
    double total = 0.0;
    for (uint32_t w = 0; w < blockDim.x / 32; ++w) {
        total += scratch[w];
    }
    if constexpr (kRows) {
        v.norms[i] = static_cast<float>(total);
        v.roots[i] = root_up(total);
    } else {
        v.squares[i * gridDim.x + blockIdx.x] = total;
        if (blockIdx.x == 0) {
            v.counts[i] = 0;
            v.upper[i] = 0xffffffffu;
            v.done[i] = 0;
        }
    }
}

// largest[0] = the largest of the roots (their bits: nonnegative), or infinity
// bits where one is not finite.
__global__ void largest_root_kernel(const float* __restrict__ roots, uint64_t count,
                                    unsigned int* __restrict__ largest)
{
    unsigned int m = 0;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < count;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const float r = roots[i];
        m = max(m, r <= FLT_MAX ? __float_as_uint(r) : 0x7f800000u);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (threadIdx.x % 32 == 0) {
        atomicMax(largest, m);
    }
}

// ----------------------------------------------------------------- selection

// E of a row and a query (the file comment's bound).
__device__ __forceinline__ float estimate_error(float a, float b, float rel)
{
    const float sum = __fadd_ru(a, b);
    return __fadd_ru(__fadd_ru(__fmul_ru(rel, __fmul_ru(a, b)),
                               __fmul_ru(0x1p-21f, __fmul_ru(sum, sum))),
                     0x1p-60f);
}

// ||q|| of the query from its slices' parts (the whole block; synchronises).
__device__ __forceinline__ float query_root(const SplitQuery& sq, uint32_t q)
{
    __shared__ float root;
    if (threadIdx.x == 0) {
        root = root_of(sq, q);
    }
    __syncthreads();
    return root;
}

// grid (row blocks, queries): the smallest e + E over the block's rows into
// upper[q] (ordered bits); the splits' sums replace the first split's slab.
// Bound: memory (the slabs, mostly in L2); kSelectRows rows per thread in
// flight.
__global__ void __launch_bounds__(kSelectThreads)
    split_upper_kernel(float* __restrict__ partials, uint32_t splits, uint32_t batch,
                       uint32_t row_count, const SplitQuery sq)
{
    const uint32_t q = blockIdx.y;
    const float a = query_root(sq, q);
    const uint64_t stride = static_cast<uint64_t>(batch) * row_count;
    float* base = partials + static_cast<uint64_t>(q) * row_count;
    const uint32_t first = blockIdx.x * kSelectThreads * kSelectRows + threadIdx.x;
    float s[kSelectRows];
#pragma unroll
    for (int u = 0; u < kSelectRows; ++u) {
        s[u] = 0.f;
    }
    for (uint32_t sp = 0; sp < splits; ++sp) {
#pragma unroll
        for (int u = 0; u < kSelectRows; ++u) {
            const uint32_t i = first + u * kSelectThreads;
            s[u] += i < row_count ? base[sp * stride + i] : 0.f;
        }
    }
    float upper = __int_as_float(0x7f800000);
#pragma unroll
    for (int u = 0; u < kSelectRows; ++u) {
        const uint32_t i = first + u * kSelectThreads;
        if (i < row_count) {
            const float e = __fmaf_rn(-2.f, s[u], sq.norms[i]);
            upper = fminf(upper, __fadd_ru(e, estimate_error(a, sq.roots[i], sq.rel)));
            if (splits > 1) {
                base[i] = s[u];
            }
        }
    }
    const unsigned int bits = __reduce_min_sync(0xffffffffu, ordered(upper));
    if (threadIdx.x % 32 == 0) {
        atomicMin(sq.upper + q, bits);
    }
}

// grid (row blocks, queries), after split_upper_kernel over every row: the rows
// whose e - E is at most the smallest e + E, in any order, into the query's
// list. More than cap of them, or a query norm the bound does not cover (counted
// as cap + 1 rows), sets error bit kCandidateOverflow.
__global__ void __launch_bounds__(kSelectThreads)
    split_collect_kernel(const float* __restrict__ partials, uint32_t row_count,
                         const SplitQuery sq, uint32_t cap, uint32_t* __restrict__ candidates,
                         int* error_flag)
{
    const uint32_t q = blockIdx.y;
    const float a = query_root(sq, q);
    const float upper = from_ordered(sq.upper[q]);
    const float* base = partials + static_cast<uint64_t>(q) * row_count;
    const uint32_t first = blockIdx.x * kSelectThreads * kSelectRows + threadIdx.x;
    // rows and cap + 1 together stay below 2^32
    if (threadIdx.x == 0 && blockIdx.x == 0 && !(a <= kLargestNorm)) {
        atomicAdd(sq.counts + q, cap + 1);
        atomicOr(error_flag, kCandidateOverflow);
    }
    float s[kSelectRows];
#pragma unroll
    for (int u = 0; u < kSelectRows; ++u) {
        const uint32_t row = first + u * kSelectThreads;
        s[u] = row < row_count ? base[row] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kSelectRows; ++u) {
        const uint32_t row = first + u * kSelectThreads;
        if (row < row_count) {
            const float e = __fmaf_rn(-2.f, s[u], sq.norms[row]);
            if (!(__fsub_rd(e, estimate_error(a, sq.roots[row], sq.rel)) > upper)) {
                const uint32_t slot = atomicAdd(sq.counts + q, 1u);
                if (slot < cap) {
                    candidates[static_cast<uint64_t>(q) * cap + slot] = row;
                } else {
                    atomicOr(error_flag, kCandidateOverflow);
                }
            }
        }
    }
}

// One warp per query: its filtered list (keys (e, row); every row whose e - E
// can be at most the smallest e + E is in it) narrowed to the rows whose e - E
// is at most the list's smallest e + E.
__global__ void __launch_bounds__(kSelectThreads)
    split_narrow_kernel(const unsigned long long* __restrict__ keys, uint32_t list_cap,
                        uint32_t batch, const SplitQuery sq, uint32_t cap,
                        uint32_t* __restrict__ candidates, int* error_flag)
{
    const uint32_t q = blockIdx.x * (kSelectThreads / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    if (q >= batch) {
        return;
    }
    const float a = root_of(sq, q);
    const uint32_t listed = sq.counts[q];
    const uint32_t n = min(listed, list_cap);
    const unsigned long long* list = keys + static_cast<uint64_t>(q) * list_cap;
    float upper = __int_as_float(0x7f800000);
    for (uint32_t i = lane; i < n; i += 32) {
        const unsigned long long key = list[i];
        const uint32_t row = static_cast<uint32_t>(key);
        upper = fminf(upper, __fadd_ru(__uint_as_float(static_cast<uint32_t>(key >> 32)),
                                       estimate_error(a, sq.roots[row], sq.rel)));
    }
    for (int o = 16; o > 0; o /= 2) {
        upper = fminf(upper, __shfl_xor_sync(0xffffffffu, upper, o));
    }
    uint32_t kept = 0;
    for (uint32_t base = 0; base < n; base += 32) {
        const uint32_t i = base + lane;
        bool keep = false;
        uint32_t row = 0;
        if (i < n) {
            const unsigned long long key = list[i];
            row = static_cast<uint32_t>(key);
            keep = !(__fsub_rd(__uint_as_float(static_cast<uint32_t>(key >> 32)),
                               estimate_error(a, sq.roots[row], sq.rel)) > upper);
        }
        const unsigned int mask = __ballot_sync(0xffffffffu, keep);
        const uint32_t slot = kept + __popc(mask & ((1u << lane) - 1u));
        if (keep && slot < cap) {
            candidates[static_cast<uint64_t>(q) * cap + slot] = row;
        }
        kept += __popc(mask);
    }
    if (lane == 0) {
        if (listed > list_cap || kept > cap || !(a <= kLargestNorm)) {
            atomicOr(error_flag, kCandidateOverflow);
            kept = 0;  // open
        }
        sq.counts[q] = kept;
    }
}

// ------------------------------------------------------------------ host side

// The tiles a score launch covers: `tiles` of the index's, `stride` apart, of
// which `rows` rows count.
struct ScoredTiles {
    uint32_t tiles;
    uint32_t stride;
    uint32_t rows;
};

template <int BN, int STAGES, Score MODE>
void launch_split_instance(const SplitPlan& plan, const CUtensorMap& rows_map,
                           const CUtensorMap& queries_map, const ScoredTiles& t, uint64_t batch,
                           float* partials, const SplitQuery& sq, const SplitList& list,
                           int* error_flag, int sm_count, cudaStream_t stream)
{
    using L = SplitSmem<BN, STAGES, MODE>;
    auto kernel = split_score_kernel<BN, STAGES, MODE>;
    static std::once_flag once[kMaxDevices];
    std::call_once(once[current_device()], [&] {
        check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(L::total)),
                   "cannot configure the split score kernel");
    });
    const uint32_t query_tiles = static_cast<uint32_t>((batch + BN - 1) / BN);
    const uint32_t units = query_tiles * t.tiles * plan.splits;
    const uint32_t ctas = std::min<uint32_t>(units, static_cast<uint32_t>(sm_count));
    kernel<<<ctas, Epilogue<BN, MODE>::threads, L::total, stream>>>(
        rows_map, queries_map, plan.kblocks, plan.kblocks_per_split, query_tiles, t.tiles,
        units, t.stride, t.rows, static_cast<uint32_t>(batch), partials, sq, list, error_flag);
    check_cuda(cudaGetLastError(), "cannot launch the split score kernel");
}

template <Score MODE>
void launch_split_tiles(const SplitPlan& plan, const void* rows, uint64_t row_count,
                        const ScoredTiles& t, const void* queries, uint64_t batch,
                        uint64_t pitch, float* partials, const SplitQuery& sq,
                        const SplitList& list, int* error_flag, int sm_count,
                        cudaStream_t stream)
{
    // both buffers hold lowp_padded_count() vectors, so no box leaves them
    const CUtensorMap rows_map =
        make_map(rows, false, 2 * pitch, round_up(row_count, kTileRows), kTileRows);
    const CUtensorMap queries_map =
        make_map(queries, false, 2 * pitch, round_up(batch, static_cast<uint64_t>(plan.bn)),
                 static_cast<uint32_t>(plan.bn));
    switch (plan.bn) {
    case 64:
        launch_split_instance<64, 4, MODE>(plan, rows_map, queries_map, t, batch, partials, sq,
                                           list, error_flag, sm_count, stream);
        break;
    case 128:
        launch_split_instance<128, 3, MODE>(plan, rows_map, queries_map, t, batch, partials, sq,
                                            list, error_flag, sm_count, stream);
        break;
    default:
        launch_split_instance<256, 2, MODE>(plan, rows_map, queries_map, t, batch, partials, sq,
                                            list, error_flag, sm_count, stream);
        break;
    }
}

// Threads of a slice's block: four columns each, at most kPrepThreads.
uint32_t prep_threads(uint64_t slice)
{
    return static_cast<uint32_t>(
        std::min<uint64_t>(kPrepThreads, round_up((slice + 3) / 4, 32)));
}

template <typename T, SplitSource SRC>
void split_rows_typed(const T* rows, uint64_t row_count, uint64_t src_pitch, uint64_t dim,
                      void* out, uint64_t pitch, float scale, float* centre, float* norms,
                      float* roots, unsigned int* largest, cudaStream_t stream)
{
    const uint32_t take = static_cast<uint32_t>(std::min<uint64_t>(row_count, kCentreRows));
    column_centre_kernel<<<static_cast<uint32_t>((pitch + 255) / 256), 256, 0, stream>>>(
        rows, row_count, src_pitch, dim, take, centre, pitch);
    SplitVectors v{};
    v.source = rows;
    v.source_pitch = src_pitch;
    v.dim = dim;
    v.centre = centre;
    v.scale = scale;
    v.out = out;
    v.pitch = pitch;
    v.slice = pitch;
    // binary32 rows are padded to 16-byte boundaries
    v.vector_loads = SRC == SplitSource::rows;
    for (uint64_t at = 0; at < row_count; at += 65535) {
        const uint64_t count = std::min<uint64_t>(65535, row_count - at);
        v.source = rows + at * src_pitch;
        v.out = static_cast<__nv_bfloat16*>(out) + at * 2 * pitch;
        v.norms = norms + at;
        v.roots = roots + at;
        split_vectors_kernel<SRC><<<dim3(1, static_cast<uint32_t>(count)),
                                    prep_threads(v.slice), 0, stream>>>(v);
    }
    largest_root_kernel<<<64, 256, 0, stream>>>(roots, row_count, largest);
    check_cuda(cudaGetLastError(), "cannot launch the row splitting kernels");
}

uint32_t row_blocks(uint64_t rows)
{
    return static_cast<uint32_t>((rows + kSelectThreads * kSelectRows - 1) /
                                 (kSelectThreads * kSelectRows));
}

}  // namespace

uint64_t split_pitch(uint64_t dim)
{
    return round_up(dim == 0 ? 1 : dim, kStageColumns);
}

float split_largest_norm()
{
    return kLargestNorm;
}

void launch_split_rows(const float* rows, uint64_t row_count, uint64_t src_pitch, uint64_t dim,
                       void* out, uint64_t pitch, float scale, float* centre, float* norms,
                       float* roots, unsigned int* largest, cudaStream_t stream)
{
    split_rows_typed<float, SplitSource::rows>(rows, row_count, src_pitch, dim, out, pitch,
                                               scale, centre, norms, roots, largest, stream);
}

void launch_split_rows(const double* rows, uint64_t row_count, uint64_t src_pitch, uint64_t dim,
                       void* out, uint64_t pitch, float scale, float* centre, float* norms,
                       float* roots, unsigned int* largest, cudaStream_t stream)
{
    split_rows_typed<double, SplitSource::rows64>(rows, row_count, src_pitch, dim, out, pitch,
                                                  scale, centre, norms, roots, largest, stream);
}

uint32_t split_slices(uint64_t pitch, uint64_t batch)
{
    // two blocks per SM, at least 2,048 columns each
    const uint64_t want = (2 * 148 + batch - 1) / batch;
    return static_cast<uint32_t>(std::min<uint64_t>(
        {want, (pitch + 2047) / 2048, static_cast<uint64_t>(kSplitSlices)}));
}

void launch_split_queries(SplitVectors v, uint64_t batch, bool projected, cudaStream_t stream)
{
    const uint32_t slices = split_slices(v.pitch, batch);
    v.slice = round_up((v.pitch + slices - 1) / slices, kStageColumns);
    const dim3 grid(slices, static_cast<uint32_t>(batch));
    const uint32_t threads = prep_threads(v.slice);
    if (projected) {
        split_vectors_kernel<SplitSource::projected><<<grid, threads, 0, stream>>>(v);
    } else if (v.columns != nullptr) {
        split_vectors_kernel<SplitSource::sampled><<<grid, threads, 0, stream>>>(v);
    } else {
        v.vector_loads = v.source_pitch % 4 == 0 &&
                         reinterpret_cast<uintptr_t>(v.source) % 16 == 0;
        split_vectors_kernel<SplitSource::dense><<<grid, threads, 0, stream>>>(v);
    }
    check_cuda(cudaGetLastError(), "cannot launch the query splitting kernel");
}

SplitPlan split_plan(uint64_t pitch, int bn, uint64_t splits)
{
    SplitPlan plan{};
    plan.bn = bn;
    plan.kblocks = static_cast<uint32_t>(pitch / kStageColumns);
    splits = std::max<uint64_t>(1, std::min<uint64_t>(splits, plan.kblocks));
    plan.kblocks_per_split = static_cast<uint32_t>((plan.kblocks + splits - 1) / splits);
    plan.splits = (plan.kblocks + plan.kblocks_per_split - 1) / plan.kblocks_per_split;
    return plan;
}

SplitPlan plan_split(uint64_t rows, uint64_t pitch, uint64_t batch, int sm_count)
{
    const int bn = batch <= 64 ? 64 : batch <= 128 ? 128 : 256;
    const uint64_t tiles = ((batch + bn - 1) / bn) * ((rows + kTileRows - 1) / kTileRows);
    const uint64_t kblocks = pitch / kStageColumns;
    // One CTA per SM: the split count whose units fill their last wave best,
    // with at least 8 stages per split and at most 4 waves unless one split
    // already exceeds that; ties go to fewer splits.
    const uint64_t sms = static_cast<uint64_t>(sm_count > 0 ? sm_count : 148);
    const uint64_t most = std::max<uint64_t>(1, kblocks / 8);
    uint64_t splits = 1;
    double best = -1.0;
    for (uint64_t s = 1; s <= most; ++s) {
        const uint64_t units = tiles * s;
        if (s > 1 && units > 4 * sms) {
            break;
        }
        const uint64_t waves = (units + sms - 1) / sms;
        const double fill = static_cast<double>(units) / static_cast<double>(waves * sms);
        if (fill > best + 1e-9) {
            best = fill;
            splits = s;
        }
    }
    return split_plan(pitch, bn, splits);
}

std::vector<SplitPlan> split_candidates(uint64_t rows, uint64_t pitch, uint64_t batch,
                                        int sm_count)
{
    std::vector<SplitPlan> out{plan_split(rows, pitch, batch, sm_count)};
    const uint64_t kblocks = pitch / kStageColumns;
    for (int bn : {64, 128, 256}) {
        if (bn > 64 && static_cast<uint64_t>(bn) / 2 >= batch) {
            continue;  // wider than twice the batch: only padding
        }
        for (uint64_t splits : {1, 2, 3, 4, 6, 8}) {
            if (splits > 1 && splits > kblocks / 8) {
                continue;
            }
            const SplitPlan p = split_plan(pitch, bn, splits);
            bool seen = false;
            for (const SplitPlan& o : out) {
                seen = seen || (o.bn == p.bn && o.splits == p.splits);
            }
            if (!seen) {
                out.push_back(p);
            }
        }
    }
    return out;
}

float split_error_rel(const SplitPlan& plan, uint64_t row_count)
{
    // twice the file comment's bound on S (e = ||r||^2 - 2 S), 2 % above the
    // first-order sums. The filter's stages share one accumulator: every
    // instruction but the first 8 may see the whole magnitude.
    const double u = std::ldexp(1.0, -24);
    const bool filter = split_filter_applies(plan, row_count);
    const double depth =
        filter ? 2.0 : static_cast<double>(plan.kblocks_per_split) + plan.splits + 2;
    const double instructions = filter ? 12.0 * plan.kblocks - 7.9 : 4.1;
    const double s =
        3.0 * std::ldexp(1.0, -18) + instructions * std::ldexp(1.0, -19) + depth * u;
    return std::nextafter(static_cast<float>(2.0 * 1.02 * s), 1.0f);
}

void launch_split_scan(const SplitPlan& plan, const void* rows, uint64_t row_count,
                       const void* queries, uint64_t batch, uint64_t pitch, float* partials,
                       const SplitQuery& sq, uint32_t* candidates, int* error_flag,
                       int sm_count, cudaStream_t stream)
{
    const uint32_t b = static_cast<uint32_t>(batch);
    const uint32_t rc = static_cast<uint32_t>(row_count);
    launch_split_scores(plan, rows, row_count, queries, batch, pitch, partials, error_flag,
                        sm_count, stream);
    const dim3 grid(row_blocks(row_count), b);
    split_upper_kernel<<<grid, kSelectThreads, 0, stream>>>(partials, plan.splits, b, rc, sq);
    split_collect_kernel<<<grid, kSelectThreads, 0, stream>>>(
        partials, rc, sq, kSplitCandidates, candidates, error_flag);
    check_cuda(cudaGetLastError(), "cannot launch the split selection kernels");
}

void launch_split_scores(const SplitPlan& plan, const void* rows, uint64_t row_count,
                         const void* queries, uint64_t batch, uint64_t pitch, float* partials,
                         int* error_flag, int sm_count, cudaStream_t stream)
{
    const ScoredTiles all{static_cast<uint32_t>((row_count + kTileRows - 1) / kTileRows), 1,
                          static_cast<uint32_t>(row_count)};
    launch_split_tiles<Score::slab>(plan, rows, row_count, all, queries, batch, pitch, partials,
                                    SplitQuery{}, SplitList{}, error_flag, sm_count, stream);
}

bool split_filter_applies(const SplitPlan& plan, uint64_t row_count)
{
    return plan.splits == 1 && plan.kblocks <= kFusedStages && row_count >= kSplitFilterRows;
}

void launch_split_filter_scan(const SplitPlan& plan, const void* rows, uint64_t row_count,
                              const void* queries, uint64_t batch, uint64_t pitch,
                              const SplitQuery& sq, unsigned long long* keys,
                              uint32_t* candidates, int* error_flag, int sm_count,
                              cudaStream_t stream)
{
    const uint32_t b = static_cast<uint32_t>(batch);
    const SplitList list{keys, kSplitListKeys};
    // the threshold: the smallest e + E over every eighth whole tile, about
    // eight rows of a query below it (kSplitFilterRows: at least 8 such tiles)
    const uint32_t whole = static_cast<uint32_t>(row_count / kTileRows);
    const ScoredTiles some{whole / 8, 8, whole / 8 * kTileRows};
    const ScoredTiles all{static_cast<uint32_t>((row_count + kTileRows - 1) / kTileRows), 1,
                          static_cast<uint32_t>(row_count)};
    launch_split_tiles<Score::least>(plan, rows, row_count, some, queries, batch, pitch, nullptr,
                                     sq, list, error_flag, sm_count, stream);
    launch_split_tiles<Score::filter>(plan, rows, row_count, all, queries, batch, pitch, nullptr,
                                      sq, list, error_flag, sm_count, stream);
    constexpr uint32_t warps = kSelectThreads / 32;
    split_narrow_kernel<<<(b + warps - 1) / warps, kSelectThreads, 0, stream>>>(
        keys, kSplitListKeys, b, sq, kSplitCandidates, candidates, error_flag);
    check_cuda(cudaGetLastError(), "cannot launch the split selection kernels");
}

}  // namespace uha
