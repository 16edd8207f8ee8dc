// The reference's binary64 median of |row - query| for one row, by one warp
// (certify.cu's replay and the settlement of median_bits.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace uha {
namespace median64 {

// Number of j < p with |row_j - y_j| (as binary64 bits) below `bound`.
__device__ inline uint32_t count_below(const double* row, const double* y, uint64_t p,
                                unsigned long long bound, int lane)
{
    uint32_t c = 0;
    for (uint64_t j = lane; j < p; j += 32) {
        const unsigned long long bits = static_cast<unsigned long long>(
            __double_as_longlong(fabs(__dsub_rn(row[j], y[j]))));
        c += bits < bound ? 1u : 0u;
    }
    return __reduce_add_sync(0xffffffffu, c);
}

// The k-th smallest (0-based) |row_j - y_j|: binary search on the bit pattern
// (nonnegative binary64 values order like their bits).
__device__ inline double select_abs_diff(const double* row, const double* y,
                                  uint64_t p, uint32_t k, int lane)
{
    unsigned long long prefix = 0;
    for (int bit = 62; bit >= 0; --bit) {
        const unsigned long long trial = prefix | (1ull << bit);
        if (count_below(row, y, p, trial, lane) <= k) {
            prefix = trial;
        }
    }
    return __longlong_as_double(static_cast<long long>(prefix));
}

// Reference median of |r_j - y_j| with the even-p midpoint
// (hierarchical_l1_ann_index.cpp:65-99): nth_element puts the (p/2)-th
// smallest at the upper middle; the lower middle is the largest of the
// smaller half; median = lower + (upper - lower) * 0.5.
__device__ inline double replay_median(const double* row, const double* y, uint64_t p,
                                int lane)
{
    const uint32_t mid = static_cast<uint32_t>(p / 2);
    const double upper = select_abs_diff(row, y, p, mid, lane);
    if (p % 2 != 0) {
        return upper;
    }
    const double lower = select_abs_diff(row, y, p, mid - 1, lane);
    return __dadd_rn(lower, __dmul_rn(__dsub_rn(upper, lower), 0.5));
}

// The same median with the lanes' |row - y| values (p <= 32 PER_LANE) held in
// registers and the lower middle taken from the upper one (the upper middle
// itself when it occurs twice there, else the largest value below it).
template <int PER_LANE>
__device__ __forceinline__ double median_in_registers(const double* row, const double* y,
                                                      uint32_t p, int lane)
{
    // bits of the values; past p above every value
    unsigned long long v[PER_LANE];
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const uint32_t j = lane + 32u * i;
        v[i] = j < p ? static_cast<unsigned long long>(
                           __double_as_longlong(fabs(__dsub_rn(row[j], y[j]))))
                     : ~0ull;
    }
    const uint32_t mid = p / 2;
    unsigned long long upper = 0;
    for (int bit = 62; bit >= 0; --bit) {
        const unsigned long long trial = upper | (1ull << bit);
        uint32_t c = 0;
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i) {
            c += v[i] < trial ? 1u : 0u;
        }
        if (__reduce_add_sync(0xffffffffu, c) <= mid) {
            upper = trial;
        }
    }
    const double high = __longlong_as_double(static_cast<long long>(upper));
    if (p % 2 != 0) {
        return high;
    }
    uint32_t below = 0;
    unsigned long long largest = 0;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        if (v[i] < upper) {
            ++below;
            largest = v[i] > largest ? v[i] : largest;
        }
    }
    below = __reduce_add_sync(0xffffffffu, below);
    for (int o = 16; o > 0; o /= 2) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, largest, o);
        largest = other > largest ? other : largest;
    }
    const double low =
        below < mid ? high : __longlong_as_double(static_cast<long long>(largest));
    return __dadd_rn(low, __dmul_rn(__dsub_rn(high, low), 0.5));
}

}  // namespace median64
}  // namespace uha
