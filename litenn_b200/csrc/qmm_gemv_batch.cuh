// Dequant-fused skinny GEMM for decode (2..16 activation rows) on sm_100a, instantiated per block format
// (qmm_gemv_q4_0.cu, ...).  One row is qmm_gemv_kernel.cuh.
//
// The weights never become floats in memory: their quants become int8 MMA A-fragments with a few logic ops per word and meet
// the activations (16-bit quants per 32-wide block, split into a signed high and a signed low byte) on the integer
// tensor-core path.  The block sums are exact; they are folded into fp32 accumulators with the block's weight scale and the
// block's activation scale, so the accumulation across blocks is fp32 as in the reference loop (src/LiteNN/Device.h:645-658).
//
// One CTA owns one 16-row tile of the output; its warps take the 256-column K chunks of that row tile round-robin.  Every chunk
// is one contiguous packed tile (qmm_common.cuh) that a single TMA bulk copy (completion counted on an mbarrier) lands in a
// shared-memory slot, the chunk's activation record behind it.  Each warp owns DEPTH slots and refills a slot itself as soon
// as it has consumed it.  The weight copies are issued before griddepcontrol.wait, so in a chain of dependent matvecs the
// next kernel's weights stream while the previous kernel drains.
//
// Bound: instruction issue of the fold behind the MMAs at 16 rows, HBM and latency below.  The fold costs 5 instructions per weight
// row, block and pair of activation rows: the MMAs' accumulators start at float bit patterns, so their sums need no
// conversion; an MMA's eight columns are one digit of eight activation rows, so that two rows share a packed instruction.
// Against one MMA per four rows with both digits and integer arithmetic behind it (pack + matvec, us): Q4_0 4096 x 11008, 8
// rows 12.5 -> 10.5, 16 rows 19.9 -> 13.3; Q4_K 28672 x 8192, 16 rows 76.2 -> 57.6; Q8_0 4096 x 4096, 16 rows 9.8 -> 7.7;
// Q6_K 8192 x 8192, 16 rows 29.7 -> 24.4; 512 x 512 2.8..3.5 -> 2.6..3.2.
// Tried and taken back: up to 14 row tiles per CTA that share a chunk's record (a staging thread took 0.1-0.2 us per copy it
// issued; with each warp requesting its own tiles Q4_K 28672 x 8192, 16 rows 63.9, Q4_0 4096 x 11008, 8 rows 13.7).
#pragma once

#include <algorithm>
#include <mutex>

#include "qmm_gemv_device.cuh"
#include "qmm_kernels.h"

namespace qmm {

namespace {

// An accumulator that starts at the bit pattern of 1.5 * 2^31 (whose last mantissa bit is worth 256) or 1.5 * 2^23 (worth 1)
// ends as a float that is the start value plus 256 times, or one times, the integer sum.  The sums stay inside the mantissa:
// at most 32 products of 255 and 128.
constexpr int HI_BITS = 0x4F400000, LO_BITS = 0x4B400000;
constexpr float HI_LO = 3221225472.0f + 12582912.0f;  // exact

__device__ __forceinline__ uint64_t pair2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t ipair2(int a, int b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ float2 split2(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// D = A(16x32) * B(32x8, s8) + {c0, c1, c0, c1}
template <bool A_SIGNED>
__device__ __forceinline__ void mma_from(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, int c0, int c1)
{
    if constexpr (A_SIGNED) {
        asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c0), "r"(c1));
    } else {
        asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c0), "r"(c1));
    }
}

// D = A(16x16, s8) * B(16x8, s8) + {c0, c1, c0, c1}
__device__ __forceinline__ void mma16_from(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, int c0, int c1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%7,%8};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(b0), "r"(c0), "r"(c1));
}

// NM MMAs per block = ceil(rows / 4): pairs of them serve eight activation rows each (octets), an odd last one four (the quad).
// Accumulators of one row tile: rows g (0) and g + 8 (1); octet o: activation rows 8o + 2t, 8o + 2t + 1; quad: row 8 * (NM / 2) + t.
template <int NM>
struct BatchAcc {
    static constexpr int OCTETS = NM / 2 > 0 ? NM / 2 : 1;
    uint64_t o[2][OCTETS];
    float q[2];
};

// One block's activations in registers.
template <int NM>
struct BatchX {
    uint2 f[NM];     // B fragments
    float xs[NM];    // block scales: octet o: [2o], [2o + 1]; quad: [NM - 1]
    float q8[NM];    // 8 * sum of the activations, same order
};

template <int NM, bool Q8>
__device__ __forceinline__ void load_batch_x(BatchX<NM>& x, const uint8_t* rec, int b, int lane)
{
    const uint8_t* f = rec + (size_t)b * (NM * 256) + lane * (NM >= 2 ? 16 : 8);
#pragma unroll
    for (int o = 0; o < NM / 2; ++o) {  // the two MMAs of an octet lie side by side
        const uint4 v = *reinterpret_cast<const uint4*>(f + o * 512);
        x.f[2 * o] = make_uint2(v.x, v.y);
        x.f[2 * o + 1] = make_uint2(v.z, v.w);
    }
    if constexpr (NM & 1) {
        x.f[NM - 1] = *reinterpret_cast<const uint2*>(rec + (size_t)b * (NM * 256) + (NM - 1) * 256 + lane * 8);
    }
    const uint8_t* meta = rec + xpack_xq_bytes(NM) + b * 64;
    const int t = lane & 3;
#pragma unroll
    for (int k = 0; k < (Q8 ? 2 : 1); ++k) {
        float* out = k == 0 ? x.xs : x.q8;
        const uint8_t* p = meta + k * XPK_META_PLANE;
        if constexpr (NM == 4) {
            const float4 v = *reinterpret_cast<const float4*>(p + t * 16);
            out[0] = v.x, out[1] = v.y, out[2] = v.z, out[3] = v.w;
        } else {
            if constexpr (NM >= 2) {
                const float2 v = *reinterpret_cast<const float2*>(p + t * 16);
                out[0] = v.x, out[1] = v.y;
            }
            if constexpr (NM & 1) {
                out[NM - 1] = *reinterpret_cast<const float*>(p + ((t >> 1) * 4 + (NM / 2) * 2 + (t & 1)) * 4);
            }
        }
    }
}

// acc += scale of the block (row g: s0, row g + 8: s1) * activation scale * the MMAs' sums
template <int NM>
__device__ __forceinline__ void fold(BatchAcc<NM>& acc, const int (&d)[NM][4], float s0, float s1, const BatchX<NM>& x)
{
    const uint64_t minus = pair2(-HI_LO, -HI_LO);
#pragma unroll
    for (int o = 0; o < NM / 2; ++o) {
#pragma unroll
        for (int rs = 0; rs < 2; ++rs) {
            const float s = rs ? s1 : s0;
            const uint64_t v = add2(add2(ipair2(d[2 * o][2 * rs], d[2 * o][2 * rs + 1]), minus),
                                    ipair2(d[2 * o + 1][2 * rs], d[2 * o + 1][2 * rs + 1]));
            acc.o[rs][o] = fma2(v, mul2(pair2(s, s), pair2(x.xs[2 * o], x.xs[2 * o + 1])), acc.o[rs][o]);
        }
    }
    if constexpr (NM & 1) {
#pragma unroll
        for (int rs = 0; rs < 2; ++rs) {
            const float v = (__int_as_float(d[NM - 1][2 * rs]) - HI_LO) + __int_as_float(d[NM - 1][2 * rs + 1]);
            acc.q[rs] = fmaf(v, (rs ? s1 : s0) * x.xs[NM - 1], acc.q[rs]);
        }
    }
}

// acc += offset of the block's weights (row g: m0, row g + 8: m1) * sum of the block's activations
template <int NM>
__device__ __forceinline__ void fold_min(BatchAcc<NM>& acc, float m0, float m1, const BatchX<NM>& x)
{
#pragma unroll
    for (int rs = 0; rs < 2; ++rs) {
        const float m = rs ? m1 : m0;
#pragma unroll
        for (int o = 0; o < NM / 2; ++o) {
            acc.o[rs][o] = fma2(pair2(m, m), pair2(x.q8[2 * o], x.q8[2 * o + 1]), acc.o[rs][o]);
        }
        if constexpr (NM & 1) {
            acc.q[rs] = fmaf(m, x.q8[NM - 1], acc.q[rs]);
        }
    }
}

template <bool A_SIGNED, int NM>
__device__ __forceinline__ void block_mmas(int (&d)[NM][4], const uint32_t (&a)[4], const BatchX<NM>& x)
{
#pragma unroll
    for (int j = 0; j < NM; ++j) {
        const bool quad = (NM & 1) && j == NM - 1;
        const int c0 = quad || j % 2 == 0 ? HI_BITS : LO_BITS, c1 = quad ? LO_BITS : c0;
        mma_from<A_SIGNED>(d[j], a, x.f[j].x, x.f[j].y, c0, c1);
    }
}

__device__ __forceinline__ float half_lo(uint32_t w, int h)
{
    return __half2float(__ushort_as_half((unsigned short)(h ? w >> 16 : w & 0xFFFFu)));
}

// byte i of w, as 2^23 + byte
__device__ __forceinline__ float byte_f23(uint32_t w, int i)
{
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 + i));
}

// A 16 x 256 tile, resident in shared memory at `slot`, times the activations of its chunk.
template <int FMT, int NM>
__device__ __forceinline__ void batch_chunk(const uint8_t* slot, const uint8_t* rec, int lane, BatchAcc<NM>& acc)
{
    const int g = lane >> 2;
    BatchX<NM> x;
    int d[NM][4];
    if constexpr (FMT == FMT_Q4_0 || FMT == FMT_Q4_K) {
        const uint8_t* p1 = slot + tile_p1_offset(FMT);
        uint64_t dd, dmin;  // rows g and g + 8
        uint32_t sw[2][3];
        if constexpr (FMT == FMT_Q4_K) {
#pragma unroll
            for (int rs = 0; rs < 2; ++rs) {
                const uint32_t* sp = reinterpret_cast<const uint32_t*>(p1 + (g + 8 * rs) * 12);
                sw[rs][0] = sp[0];
                sw[rs][1] = sp[1];
                sw[rs][2] = sp[2];
            }
            const uint8_t* p2 = slot + tile_p2_offset(FMT);
            const float2 dm0 = __half22float2(*reinterpret_cast<const __half2*>(p2 + g * 4));
            const float2 dm1 = __half22float2(*reinterpret_cast<const __half2*>(p2 + (g + 8) * 4));
            dd = pair2(dm0.x, dm1.x * 0.0625f);                // row g + 8 is multiplied 16 times too large
            dmin = pair2(dm0.y * -0.125f, dm1.y * -0.125f);  // the offset meets 8 * the sum of the activations
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const uint4 q = *(reinterpret_cast<const uint4*>(slot) + p * 32 + lane);
            uint32_t s0, s1;
            if constexpr (FMT == FMT_Q4_0) {
                s0 = *reinterpret_cast<const uint32_t*>(p1 + g * 16 + p * 4);
                s1 = *reinterpret_cast<const uint32_t*>(p1 + (g + 8) * 16 + p * 4);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int b = 2 * p + h;
                load_batch_x<NM, FMT == FMT_Q4_K>(x, rec, b, lane);
                const uint32_t w1 = h ? q.z : q.x;  // weights 4t..   rows g | g+8
                const uint32_t w2 = h ? q.w : q.y;  // weights 16+4t..
                if constexpr (FMT == FMT_Q4_0) {
                    // 16 * (n - 8) as int8 for both rows
                    const uint32_t a[4] = {((w1 << 4) & 0xF0F0F0F0u) ^ 0x80808080u, (w1 & 0xF0F0F0F0u) ^ 0x80808080u,
                                           ((w2 << 4) & 0xF0F0F0F0u) ^ 0x80808080u, (w2 & 0xF0F0F0F0u) ^ 0x80808080u};
                    block_mmas<true, NM>(d, a, x);
                    fold<NM>(acc, d, half_lo(s0, h), half_lo(s1, h), x);
                } else {
                    const uint32_t a[4] = {w1 & 0x0F0F0F0Fu, w1 & 0xF0F0F0F0u, w2 & 0x0F0F0F0Fu, w2 & 0xF0F0F0F0u};
                    block_mmas<false, NM>(d, a, x);
                    uint32_t scw[2], mnw[2];
#pragma unroll
                    for (int rs = 0; rs < 2; ++rs) {
                        const uint32_t* w = sw[rs];
                        scw[rs] = b < 4 ? (w[0] & 0x3F3F3F3Fu) : ((w[2] & 0x0F0F0F0Fu) | ((w[0] >> 2) & 0x30303030u));
                        mnw[rs] = b < 4 ? (w[1] & 0x3F3F3F3Fu) : (((w[2] >> 4) & 0x0F0F0F0Fu) | ((w[1] >> 2) & 0x30303030u));
                    }
                    // d * scale and dmin * min are exact (11 + 6 bits)
                    const uint64_t minus = pair2(-8388608.0f, -8388608.0f);
                    const float2 sc = split2(mul2(add2(pair2(byte_f23(scw[0], b & 3), byte_f23(scw[1], b & 3)), minus), dd));
                    const float2 mn = split2(mul2(add2(pair2(byte_f23(mnw[0], b & 3), byte_f23(mnw[1], b & 3)), minus), dmin));
                    fold<NM>(acc, d, sc.x, sc.y, x);
                    fold_min<NM>(acc, mn.x, mn.y, x);
                }
            }
        }
    } else if constexpr (FMT == FMT_Q8_0) {
        const uint8_t* p1 = slot + tile_p1_offset(FMT);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            load_batch_x<NM, false>(x, rec, b, lane);
            const uint4 q = *(reinterpret_cast<const uint4*>(slot) + b * 32 + lane);
            const uint32_t a[4] = {q.x, q.y, q.z, q.w};
            block_mmas<true, NM>(d, a, x);
            const float s0 = __half2float(*reinterpret_cast<const __half*>(p1 + g * 16 + b * 2));
            const float s1 = __half2float(*reinterpret_cast<const __half*>(p1 + (g + 8) * 16 + b * 2));
            fold<NM>(acc, d, s0, s1, x);
        }
    } else {  // Q6_K: A byte = 4 * (q - 32) as int8, one k16 MMA per 16-wide sub-block
        const uint8_t* p1 = slot + tile_p1_offset(FMT);
        const uint8_t* p2 = slot + tile_p2_offset(FMT);
        const float dg = __half2float(*reinterpret_cast<const __half*>(p2 + g * 2)) * 0.25f;
        const float dg8 = __half2float(*reinterpret_cast<const __half*>(p2 + (g + 8) * 2)) * 0.25f;
        const uint4* qs = reinterpret_cast<const uint4*>(slot) + lane;
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
            // int8 scales of the four sub-blocks; + 128 makes the bytes unsigned
            const uint32_t s0 = *reinterpret_cast<const uint32_t*>(p1 + g * 16 + quad * 4) ^ 0x80808080u;
            const uint32_t s1 = *reinterpret_cast<const uint32_t*>(p1 + (g + 8) * 16 + quad * 4) ^ 0x80808080u;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                load_batch_x<NM, false>(x, rec, 2 * quad + h, lane);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int jj = 2 * h + e;
#pragma unroll
                    for (int j = 0; j < NM; ++j) {
                        const bool last = (NM & 1) && j == NM - 1;
                        const int c0 = last || j % 2 == 0 ? HI_BITS : LO_BITS, c1 = last ? LO_BITS : c0;
                        mma16_from(d[j], out[0][jj], out[1][jj], e ? x.f[j].y : x.f[j].x, c0, c1);
                    }
                    fold<NM>(acc, d, (byte_f23(s0, jj) - 8388736.0f) * dg, (byte_f23(s1, jj) - 8388736.0f) * dg8, x);
                }
            }
        }
    }
}

// Shared memory of one CTA: slots WARPS*DEPTH x (tile, that chunk's activation record) | mbarriers.  The warps' sums lie over the
// slots at the end.
template <int FMT, int NM>
struct BatchPlan {
    static constexpr int WARPS = 4;
    // a slot carries 3-9 KB of activations: a shallow ring keeps 2-3 CTAs per SM
    static constexpr int DEPTH = NM == 1 && FMT != FMT_Q8_0 ? 3 : 2;
    static constexpr int REC = xpack_copy_bytes(NM);
    static constexpr int SLOT = tile_bytes(FMT) + REC;
    static constexpr int BAR_OFF = WARPS * DEPTH * SLOT;
    static constexpr int TOTAL = BAR_OFF + WARPS * DEPTH * 8;
    static constexpr int RESIDENT = 232448 / (TOTAL + 1024);  // CTAs that an SM's shared memory holds
};

// At most 128 registers a thread: the shared memory holds no more than four CTAs, and a limit of 80 spilled (Q8_0 4096 x
// 11008, 12 rows: 18.3 us against 13.0).
template <int FMT, int NM>
__global__ void __launch_bounds__(BatchPlan<FMT, NM>::WARPS * 32, 4)
    gemv_batch_kernel(const WeightView v, const uint8_t* __restrict__ xp, float* __restrict__ y, int m, int* __restrict__ status)
{
    using Plan = BatchPlan<FMT, NM>;
    constexpr int WARPS = Plan::WARPS, DEPTH = Plan::DEPTH;
    constexpr uint32_t TILE = tile_bytes(FMT), REC = Plan::REC;
    extern __shared__ __align__(128) uint8_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kc = v.kc;
    uint8_t* slots = smem + warp * DEPTH * Plan::SLOT;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Plan::BAR_OFF) + warp * DEPTH;
    const uint8_t* src = v.tiles + ((size_t)blockIdx.x * kc + warp) * TILE;
    const uint8_t* rec_src = xp + (size_t)warp * xpack_rec_bytes(NM);
    const int chunks = warp < kc ? (kc - warp + WARPS - 1) / WARPS : 0;

    // 1. start the weight stream.  A slot's phase takes two arrivals: one with the tile's bytes, issued here, and one with
    // the record's, which can only be issued after the dependency wait.
    if (lane == 0) {
#pragma unroll
        for (int s = 0; s < DEPTH; ++s) {
            mbar_init(&bars[s], 2);
        }
        fence_barrier_init();
#pragma unroll
        for (int s = 0; s < DEPTH; ++s) {
            if (s < chunks) {
                mbar_expect_tx(&bars[s], TILE);
                bulk_copy_g2s(slots + s * Plan::SLOT, src + (size_t)s * WARPS * TILE, TILE, &bars[s]);
            }
        }
    }
    pdl_launch_dependents();
    // 2. everything below may read what earlier kernels in the stream produced
    pdl_wait();
    if (lane == 0) {
#pragma unroll
        for (int s = 0; s < DEPTH; ++s) {
            if (s < chunks) {
                mbar_expect_tx(&bars[s], REC);
                bulk_copy_g2s(slots + s * Plan::SLOT + TILE, rec_src + (size_t)s * WARPS * xpack_rec_bytes(NM), REC, &bars[s]);
            }
        }
    }
    BatchAcc<NM> acc;
#pragma unroll
    for (int rs = 0; rs < 2; ++rs) {
        acc.q[rs] = 0.0f;
#pragma unroll
        for (int o = 0; o < BatchAcc<NM>::OCTETS; ++o) {
            acc.o[rs][o] = 0ull;
        }
    }

    // 3. consume chunks as they land; refill each slot right after it has been read
    int s = 0;
    uint32_t parity = 0;
    for (int i = 0; i < chunks; ++i) {
        if (!mbar_wait(&bars[s], parity)) {
            if (lane == 0) {
                atomicExch(status, 1);
            }
            break;
        }
        uint8_t* slot = slots + s * Plan::SLOT;
        batch_chunk<FMT, NM>(slot, slot + TILE, lane, acc);
        __syncwarp();
        if (lane == 0 && i + DEPTH < chunks) {
            fence_proxy_async();  // order this warp's reads of the slot before the refill
            const size_t c = (size_t)(i + DEPTH) * WARPS;
            mbar_expect_tx(&bars[s], TILE);
            bulk_copy_g2s(slot, src + c * TILE, TILE, &bars[s]);
            mbar_expect_tx(&bars[s], REC);
            bulk_copy_g2s(slot + TILE, rec_src + c * xpack_rec_bytes(NM), REC, &bars[s]);
        }
        if (++s == DEPTH) {
            s = 0;
            parity ^= 1u;
        }
    }
    __syncthreads();

    // 4. partial sums of the warps meet in shared memory: red[warp][activation row][row]
    float* red = reinterpret_cast<float*>(smem);
    constexpr int ROWS = 4 * NM;
    const int g = lane >> 2, t = lane & 3;
    const float unit = FMT == FMT_Q4_0 ? 0.0625f : 1.0f;
#pragma unroll
    for (int rs = 0; rs < 2; ++rs) {
        float* out = red + warp * ROWS * 16 + g + 8 * rs;
#pragma unroll
        for (int o = 0; o < NM / 2; ++o) {
            const float2 w = split2(acc.o[rs][o]);
            out[(8 * o + 2 * t) * 16] = w.x * unit;
            out[(8 * o + 2 * t + 1) * 16] = w.y * unit;
        }
        if constexpr (NM & 1) {
            out[(8 * (NM / 2) + t) * 16] = acc.q[rs] * unit;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < m * 16; i += WARPS * 32) {
        const int col = i >> 4, r = i & 15;
        float sum = 0.0f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            sum += red[(w * ROWS + col) * 16 + r];
        }
        const int64_t row = (int64_t)blockIdx.x * 16 + r;
        if (row < v.n) {
            y[(int64_t)col * v.n + row] = sum;
        }
    }
}

template <int FMT, int NM>
cudaError_t launch_gemv_batch(const WeightView& w, const XPackView& xp, float* y, int m, int* status, cudaStream_t stream)
{
    using Plan = BatchPlan<FMT, NM>;
    auto kernel = gemv_batch_kernel<FMT, NM>;
    static std::mutex mu;
    static int configured[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    const int sms = sm_count_of(dev);
    if (sms < 1) {
        return cudaErrorInvalidDevice;
    }
    int smem = Plan::TOTAL;
    {
        std::lock_guard<std::mutex> lock(mu);
        // Residency cap.  The block scheduler fills an SM up to its limit before it is even with the others, so a grid that
        // could sit 7 to an SM leaves a third of the SMs with little to do (688 CTAs of the one-row kernel: 6.7 us at a limit
        // of 7, 5.2 us at 5).  The dynamic shared memory request is padded so that no SM can hold more than its even share,
        // ceil(grid / SMs), of the CTAs; where the share takes several rounds, no more than its even part per round
        // (Q8_0 8192 x 8192, 8 rows, 3.5 CTAs per SM: 18.5 us at three and one, 16.9 at two and two).
        const int share = (w.rt + sms - 1) / sms;
        const int rounds = (share + Plan::RESIDENT - 1) / Plan::RESIDENT;
        smem = std::max(smem, 232448 / ((share + rounds - 1) / rounds) - 1024 - 256);
        // the opt-in limit is a per-device function attribute; raise it only when needed
        if (dev >= 64 || configured[dev] < smem) {
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) {
                return e;
            }
            if (dev < 64) {
                configured[dev] = smem;
            }
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)w.rt);
    cfg.blockDim = dim3(Plan::WARPS * 32);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 1;
    cfg.attrs = attr;
    return cudaLaunchKernelEx(&cfg, kernel, w, xp.base, y, m, status);
}

}  // namespace

}  // namespace qmm
