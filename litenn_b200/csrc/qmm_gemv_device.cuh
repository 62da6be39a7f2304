// Device-side building blocks of the dequant-fused matvec kernels (qmm_gemv_kernel.cuh, qmm_gemv_batch.cuh): mbarrier /
// bulk-copy PTX wrappers, the integer MMA wrappers and the batch-1 multiply routine for every block format.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "qmm_common.cuh"

namespace qmm {
namespace {

// ---- PTX helpers ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_barrier_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// Global -> shared bulk copy; `bytes` and both addresses are multiples of 16.
__device__ __forceinline__ void bulk_copy_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst_smem)),
                 "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Bounded wait for a phase of an mbarrier.  Returns false when the limit ran out
// (the caller records an error status and stops using the pipeline).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity)
{
    const uint32_t addr = smem_u32(bar);
    for (uint32_t spin = 0; spin < (1u << 22); ++spin) {
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

__device__ __forceinline__ void pdl_launch_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void pdl_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// D = A(16x32, row) * B(32x8, col, s8) with a zero C operand.
template <bool A_SIGNED>
__device__ __forceinline__ void mma_k32(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1)
{
    const int z = 0;
    if constexpr (A_SIGNED) {
        asm(
            "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(z));
    } else {
        asm(
            "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(z));
    }
}

// D = A * B + D  (k32, B s8): second half of a two-MMA block pair.
template <bool A_SIGNED>
__device__ __forceinline__ void mma_k32_acc(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                            uint32_t b0, uint32_t b1)
{
    if constexpr (A_SIGNED) {
        asm(
            "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    } else {
        asm(
            "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
}

__device__ __forceinline__ uint32_t word_of(const uint4& v, int i)
{
    return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}

__device__ __forceinline__ float half_of(const uint4& v, int b)
{
    const uint32_t w = word_of(v, b >> 1);
    return __half2float(__ushort_as_half((unsigned short)((b & 1) ? (w >> 16) : (w & 0xFFFFu))));
}

__device__ __forceinline__ uint32_t byte_of(const uint4& v, int i)
{
    return (word_of(v, i >> 2) >> (8 * (i & 3))) & 0xFFu;
}

__device__ __forceinline__ uint32_t byte_of_word(uint32_t w, int i)
{
    return (w >> (8 * i)) & 0xFFu;
}

// Batch 1: all compact records (qmm_common.cuh) staged in shared memory.
struct XShared {
    const uint8_t* base;   // [kc] records of XPK1_REC bytes
    const uint8_t* zeros;  // Q6_K: 512 zero bytes for the lanes that carry no activation row
};

// ---- batch 1 ---------------------------------------------------------------------------------
//
// With one activation row only columns 0 and 1 of an MMA would be live and the scalar
// work that follows it (combine the two digits, convert, scale) would run with three
// quarters of the lanes idle.  So four neighbouring blocks share the columns: block r of
// a group of four owns columns 2r and 2r+1.  One MMA takes k-slots 0..15 from one block and
// k-slots 16..31 from the next (for a fragment that is only a choice of registers) and its B
// operand is zero outside those blocks' columns; four MMAs, two per pair of blocks, add up in
// the same accumulators.  Lane t then folds block t of the group: one fold per four blocks, with
// every lane at work.  (Two blocks per fold left half of the lanes repeating the other half; otherwise the same
// code: 70B-shape layers, a 1024-token prompt and 64 steps, 48.1 ms against 45.7; a 7B shape, 512 tokens and 128 steps,
// 161.8 against 157.8.)

template <int FMT>
__device__ __forceinline__ void compute_chunk_m1(const uint8_t* slot, const XShared& xs, int c, int lane, float* acc)
{
    const int g = lane >> 2;
    const int t = lane & 3;
    const int role = g >> 1;  // the block of a group whose activations this lane supplies
    const uint8_t* rec = xs.base + (size_t)c * XPK1_REC;
    // Per-lane sources of the B registers: lane (g, t) feeds column g = digit g & 1 of block g >> 1; every register
    // that belongs to another block is zero.  Entry = uint2 {weights 4t.., weights 16+4t..}.  The lane loads its own entry and
    // selects; with a pointer per register, three of them to a page of zeros (as Q6_K still has them, whose entries are half
    // as large), the 40-register variants spill: pack + matvec of one row, us, Q4_0 11008 x 2304 6.04 against 5.86, 4096 x
    // 4096 5.28 and 5.15, 4096 x 14336 9.73 and 9.11; Q8_0 11008 x 2048 6.86 and 6.54; Q4_K 11008 x 8192 15.7 and 15.2.
    const uint8_t* xrow = rec + ((g & 1) * 4 + t) * 8;
    const int4* meta = reinterpret_cast<const int4*>(rec + XPK1_META);
    const uint4* qs = reinterpret_cast<const uint4*>(slot) + lane;
    const uint8_t* p1 = slot + tile_p1_offset(FMT);
    const uint8_t* p2 = slot + tile_p2_offset(FMT);
    float a0 = 0.0f, a1 = 0.0f;
    int d[4];

    if constexpr (FMT == FMT_Q6_K) {
        // the two 16-wide sub-blocks of a 32-block share one k32 MMA: sub-block j of a group of four owns columns 2j, 2j+1
        const float dg = __half2float(*reinterpret_cast<const __half*>(p2 + g * 2));
        const float dg8 = __half2float(*reinterpret_cast<const __half*>(p2 + (g + 8) * 2));
        const signed char* sc_g = reinterpret_cast<const signed char*>(p1 + g * 16) + t;
        const signed char* sc_g8 = reinterpret_cast<const signed char*>(p1 + (g + 8) * 16) + t;
        const uint8_t* x0 = role == 0 ? xrow : xs.zeros;
        const uint8_t* x1 = role == 1 ? xrow + 4 : xs.zeros;
        const uint8_t* x2 = role == 2 ? xrow + 64 : xs.zeros;
        const uint8_t* x3 = role == 3 ? xrow + 68 : xs.zeros;
        uint4 qv[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            qv[i] = qs[i * 32];
        }
#pragma unroll
        for (int quad = 0; quad < 4; ++quad) {
            uint32_t out[2][4];
#pragma unroll
            for (int rsel = 0; rsel < 2; ++rsel) {
                const int base = (quad * 2 + rsel) * 3;
                const uint32_t X = word_of(qv[(base + 0) >> 2], (base + 0) & 3);
                const uint32_t Y = word_of(qv[(base + 1) >> 2], (base + 1) & 3);
                const uint32_t Z = word_of(qv[(base + 2) >> 2], (base + 2) & 3);
                out[rsel][0] = X & 0xFCFCFCFCu;
                out[rsel][1] = Y & 0xFCFCFCFCu;
                out[rsel][2] = Z & 0xFCFCFCFCu;
                out[rsel][3] = ((X & 0x03030303u) << 6) | ((Y & 0x03030303u) << 4) | ((Z & 0x03030303u) << 2);
            }
            const int o = quad * 128;
            mma_k32<true>(d, out[0][0], out[1][0], out[0][1], out[1][1], *reinterpret_cast<const uint32_t*>(x0 + o),
                          *reinterpret_cast<const uint32_t*>(x1 + o));
            mma_k32_acc<true>(d, out[0][2], out[1][2], out[0][3], out[1][3], *reinterpret_cast<const uint32_t*>(x2 + o),
                              *reinterpret_cast<const uint32_t*>(x3 + o));
            const float xsb = __int_as_float(meta[2 * quad + (t >> 1)].z);
            const float sg = dg * (float)(int)sc_g[4 * quad];
            const float sg8 = dg8 * (float)(int)sc_g8[4 * quad];
            a0 = fmaf((float)(d[0] * 256 + d[1]), sg * xsb, a0);
            a1 = fmaf((float)(d[2] * 256 + d[3]), sg8 * xsb, a1);
        }
        acc[0] = fmaf(a0, 0.25f, acc[0]);
        acc[1] = fmaf(a1, 0.25f, acc[1]);
    } else {
        const uint8_t* mine = xrow + 64 * role;
        // this lane's block of group P is 4P + t
        const __half* dg_p = reinterpret_cast<const __half*>(p1 + g * 16) + t;
        const __half* dg8_p = reinterpret_cast<const __half*>(p1 + (g + 8) * 16) + t;
        uint32_t scw[2][2], mnw[2][2];
        float dd[2], dmin[2];
        if constexpr (FMT == FMT_Q4_K) {
#pragma unroll
            for (int rs = 0; rs < 2; ++rs) {
                const uint32_t* sp = reinterpret_cast<const uint32_t*>(p1 + (g + 8 * rs) * 12);
                const uint32_t w0 = sp[0], w1 = sp[1], w2 = sp[2];
                scw[rs][0] = w0 & 0x3F3F3F3Fu;
                mnw[rs][0] = w1 & 0x3F3F3F3Fu;
                scw[rs][1] = (w2 & 0x0F0F0F0Fu) | ((w0 >> 2) & 0x30303030u);
                mnw[rs][1] = ((w2 >> 4) & 0x0F0F0F0Fu) | ((w1 >> 2) & 0x30303030u);
                const uint32_t dm = *reinterpret_cast<const uint32_t*>(p2 + (g + 8 * rs) * 4);
                dd[rs] = __half2float(__ushort_as_half((unsigned short)(dm & 0xFFFFu)));
                dmin[rs] = __half2float(__ushort_as_half((unsigned short)(dm >> 16)));
            }
        }
        float m0 = 0.0f, m1 = 0.0f;
#pragma unroll
        for (int P = 0; P < 2; ++P) {
            const uint2 xv = *reinterpret_cast<const uint2*>(mine + P * 256), none = make_uint2(0u, 0u);
            const uint2 x0 = role == 0 ? xv : none, x1 = role == 1 ? xv : none, x2 = role == 2 ? xv : none,
                        x3 = role == 3 ? xv : none;
            const int4 mm = meta[4 * P + t];
            const float xsb = __int_as_float(mm.z);
            if constexpr (FMT == FMT_Q8_0) {
                const uint4 qa = qs[(4 * P) * 32], qb = qs[(4 * P + 1) * 32], qc = qs[(4 * P + 2) * 32], qd = qs[(4 * P + 3) * 32];
                mma_k32<true>(d, qa.x, qa.y, qb.x, qb.y, x0.x, x1.x);
                mma_k32_acc<true>(d, qa.z, qa.w, qb.z, qb.w, x0.y, x1.y);
                mma_k32_acc<true>(d, qc.x, qc.y, qd.x, qd.y, x2.x, x3.x);
                mma_k32_acc<true>(d, qc.z, qc.w, qd.z, qd.w, x2.y, x3.y);
                a0 = fmaf((float)(d[0] * 256 + d[1]), __half2float(dg_p[4 * P]) * xsb, a0);
                a1 = fmaf((float)(d[2] * 256 + d[3]), __half2float(dg8_p[4 * P]) * xsb, a1);
            } else {
                // {blk 4P w 4t.., blk 4P w 16+4t.., blk 4P+1 w 4t.., blk 4P+1 w 16+4t..} and the same of 4P+2, 4P+3
                const uint4 qa = qs[(2 * P) * 32], qb = qs[(2 * P + 1) * 32];
                mma_k32<false>(d, qa.x & 0x0F0F0F0Fu, qa.x, qa.z & 0x0F0F0F0Fu, qa.z, x0.x, x1.x);
                mma_k32_acc<false>(d, qa.y & 0x0F0F0F0Fu, qa.y, qa.w & 0x0F0F0F0Fu, qa.w, x0.y, x1.y);
                mma_k32_acc<false>(d, qb.x & 0x0F0F0F0Fu, qb.x, qb.z & 0x0F0F0F0Fu, qb.z, x2.x, x3.x);
                mma_k32_acc<false>(d, qb.y & 0x0F0F0F0Fu, qb.y, qb.w & 0x0F0F0F0Fu, qb.w, x2.y, x3.y);
                const int vg = d[0] * 256 + d[1];
                const int vg8 = d[2] * 256 + d[3] - vg;
                if constexpr (FMT == FMT_Q4_0) {
                    a0 = fmaf((float)(vg - mm.x), __half2float(dg_p[4 * P]) * xsb, a0);
                    a1 = fmaf((float)(vg8 - mm.y), __half2float(dg8_p[4 * P]) * xsb, a1);
                } else {
                    const int sh = 8 * t;  // byte t of word P
                    const float sg = dd[0] * (float)((scw[0][P] >> sh) & 0xFFu);
                    const float sg8 = dd[1] * (float)((scw[1][P] >> sh) & 0xFFu);
                    const float mg = dmin[0] * (float)((mnw[0][P] >> sh) & 0xFFu);
                    const float mg8 = dmin[1] * (float)((mnw[1][P] >> sh) & 0xFFu);
                    a0 = fmaf((float)vg, sg * xsb, a0);
                    a1 = fmaf((float)vg8, sg8 * xsb, a1);
                    const float q8 = (float)mm.x * xsb;  // 8 * sum of the block's activations, in their own units
                    m0 = fmaf(mg, q8, m0);
                    m1 = fmaf(mg8, q8, m1);
                }
            }
        }
        if constexpr (FMT == FMT_Q4_0) {
            acc[0] += a0;
            acc[1] = fmaf(a1, 0.0625f, acc[1]);
        } else if constexpr (FMT == FMT_Q8_0) {
            acc[0] += a0;
            acc[1] += a1;
        } else {
            acc[0] += fmaf(-m0, 0.125f, a0);
            acc[1] += fmaf(-m1, 0.125f, a1 * 0.0625f);
        }
    }
}

}  // namespace
}  // namespace qmm
