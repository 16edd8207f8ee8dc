// Tensor-core building blocks of the score kernels (precision.cu,
// split_scan.cu): bounded mbarrier waits, TMA tile loads, TMEM allocation,
// tcgen05.mma with 128-byte-swizzled operands, and the operands' tensor maps.
#pragma once

#include "async_copy.cuh"
#include "common.h"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <cstdint>
#include <mutex>

namespace uha {
namespace tensorcore {

constexpr int kTileRows = 128;        // UMMA M: rows per tile (TMEM lanes)
constexpr uint32_t kSliceBytes = 128; // K bytes per stage: one swizzle atom row
constexpr uint32_t kSpinLimit = 1u << 24;
constexpr int kPipelineTimeout = 8;   // error-flag bit

using async::mbar_expect_tx;
using async::mbar_init;
using async::smem_u32;

// Waits for the phase of `parity` to complete; false after kSpinLimit tries.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity)
{
    return async::mbar_wait(bar, parity, kSpinLimit);
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map,
                                            uint64_t* bar, int32_t x, int32_t y)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ void tc_fence_before()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile written by TMA
// with 128-byte swizzling: rows of 128 bytes, 8-row core groups 1024 bytes
// apart (stride byte offset), descriptor version 1, layout SWIZZLE_128B.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t smem_addr)
{
    uint64_t d = static_cast<uint64_t>((smem_addr >> 4) & 0x3fffu);
    d |= static_cast<uint64_t>(1) << 16;           // leading byte offset (16 B)
    d |= static_cast<uint64_t>(1024 >> 4) << 32;   // stride byte offset
    d |= static_cast<uint64_t>(1) << 46;           // version
    d |= static_cast<uint64_t>(2) << 61;           // 128-byte swizzle
    return d;
}

// Instruction descriptor: FP32 accumulator, A and B of the same type (BF16,
// or E4M3 for kind::f8f6f4), both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t mma_idesc(bool fp8, int n)
{
    return (1u << 4) | (fp8 ? 0u : ((1u << 7) | (1u << 10))) |
           (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(kTileRows >> 4) << 24);
}

template <bool FP8>
__device__ __forceinline__ void mma_issue(uint32_t tmem, uint64_t a, uint64_t b,
                                          uint32_t idesc, uint32_t accumulate)
{
    if constexpr (FP8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}

__device__ __forceinline__ void mma_commit(uint64_t* bar)
{
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

// Starts the load of 16 consecutive FP32 accumulator columns of this thread's
// TMEM lane into v; read v only after tmem_wait_loads() and tmem_loaded(v).
__device__ __forceinline__ void tmem_start16(uint32_t addr, float* v)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
          "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]),
          "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(addr));
}

__device__ __forceinline__ void tmem_wait_loads()
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Keeps reads of v behind the wait.
__device__ __forceinline__ void tmem_loaded(float* v)
{
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        asm volatile("" : "+f"(v[i]));
    }
}

__device__ __forceinline__ void tmem_load16(uint32_t addr, float (&v)[16])
{
    tmem_start16(addr, v);
    tmem_wait_loads();
    tmem_loaded(v);
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void prefetch_map(const CUtensorMap* map)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// By one whole warp: `columns` TMEM columns (a power of two from 32 to 512),
// their address into *slot (shared memory).
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t columns)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(slot)),
                 "r"(columns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, uint32_t columns)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(columns)
                 : "memory");
}

// ------------------------------------------------------------ host side

inline PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult status{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault,
                                    &status) == cudaSuccess &&
            status == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        } else {
            cudaGetLastError();
        }
    });
    if (fn == nullptr) {
        fail(UHA_RUNTIME_ERROR, "cuTensorMapEncodeTiled is unavailable");
    }
    return fn;
}

// 2-D tensor map over [outer][pitch] one-byte or two-byte elements, box of
// 128 bytes x box_outer with 128-byte swizzling. Callers keep every box inside
// the tensor.
inline CUtensorMap make_map(const void* base, bool fp8, uint64_t pitch, uint64_t outer,
                     uint32_t box_outer)
{
    CUtensorMap map{};
    const uint64_t elem = fp8 ? 1 : 2;
    const cuuint64_t dims[2] = {pitch, outer};
    const cuuint64_t strides[1] = {pitch * elem};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kSliceBytes / elem), box_outer};
    const cuuint32_t element_strides[2] = {1, 1};
    const CUresult r = encode_fn()(
        &map, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
        const_cast<void*>(base), dims, strides, box, element_strides,
        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        fail(UHA_RUNTIME_ERROR, "cannot describe a tensor-core operand (tensor map)");
    }
    return map;
}

}  // namespace tensorcore
}  // namespace uha
