// PTX wrappers and descriptors shared by the two prefill GEMM kernels (qmm_gemm.cu, qmm_gemm_smem.cu).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "qmm_common.cuh"

namespace qmm {

namespace {

constexpr int GEMM_BK = 64;  // K per step: 128 bytes of bf16 = one swizzle row
constexpr uint32_t GEMM_SPIN_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t g_smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void g_mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(g_smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void g_mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(g_smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void g_mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(g_smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool g_mbar_wait(uint64_t* bar, uint32_t parity)
{
    const uint32_t addr = g_smem_u32(bar);
    for (uint32_t spin = 0; spin < GEMM_SPIN_LIMIT; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) {
            return true;
        }
    }
    return false;
}

// The same for a whole converged warp, which goes on together: what follows may be a warp-wide tcgen05 instruction, and
// lanes that gave up on their own would leave the others without them.
__device__ __forceinline__ bool g_mbar_wait_warp(uint64_t* bar, uint32_t parity)
{
    return __all_sync(0xFFFFFFFFu, g_mbar_wait(bar, parity));
}

// Programmatic dependent launch: the next kernel of the stream may start its prologue; everything that earlier kernels of
// the stream wrote is visible.
__device__ __forceinline__ void g_pdl_launch_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void g_pdl_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// The same for a warp that reads nothing of the earlier kernels and only wants their end behind it: loads of weights may move
// across (with the clobber above the dequantization warps' loads were held back, 22016 x 4096 and 64 tokens 39.2 -> 39.6 us,
// 11008 x 4096 and 128 tokens 32.1 -> 33.1).
__device__ __forceinline__ void g_pdl_wait_only()
{
    asm volatile("griddepcontrol.wait;");
}

// True in one lane of a converged warp.  MMAs are issued under this and not under a lane comparison: the compiler then
// knows that their operands are uniform.
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "elect.sync _|p, 0xFFFFFFFF;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(p));
    return p != 0;
}

// 2-D tiled TMA load (no multicast): box {64 k, tokens} at element coordinates (k0, row0).
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int k0, int row0, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            g_smem_u32(dst)),
        "l"(map), "r"(k0), "r"(row0), "r"(g_smem_u32(bar))
        : "memory");
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);   // start address
    d |= (uint64_t)1 << 16;                          // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                          // descriptor version of this architecture
    d |= (uint64_t)2 << 61;                          // 128-byte swizzle
    return d;
}

// Instruction descriptor: D fp32, A and B bf16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t umma_idesc_bf16(int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(g_smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ uint32_t ldg_u32(const uint8_t* p)
{
    return __ldg(reinterpret_cast<const uint32_t*>(p));
}

__device__ __forceinline__ float h2f_bits(uint32_t bits16)
{
    return __half2float(__ushort_as_half((unsigned short)(bits16 & 0xFFFFu)));
}

// sigmoid = 1 / (1 + exp(-x)), SiLU = x * sigmoid(x) (src/LiteNN/Layer/Activation.h:20-33,52-59)
__device__ __forceinline__ float silu_mul(float g, float u)
{
    return (g * (1.0f / (1.0f + expf(-g)))) * u;
}

}  // namespace

}  // namespace qmm
