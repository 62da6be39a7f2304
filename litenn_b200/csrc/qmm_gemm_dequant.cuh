// Dequantization of packed 16 x 256 tiles (qmm_common.cuh) to bf16 in registers, for the two prefill GEMM kernels: one
// lane turns its part of a 16-row x 64-column quarter into 16 registers, which is the order of tcgen05.st.16x256b
// and, two registers at a time, four neighbouring columns of a row.
#pragma once

#include "qmm_gemm_ptx.cuh"

namespace qmm {

namespace {

__device__ __forceinline__ uint4 ldg_u128(const uint8_t* p)
{
    return __ldg(reinterpret_cast<const uint4*>(p));
}

__device__ __forceinline__ uint32_t word4(const uint4& v, int i)
{
    return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}

__device__ __forceinline__ uint64_t f2_pair(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ uint32_t f2_to_bf16x2(uint64_t v)
{
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&b);
}

// Bytes 2h, 2h+1 of `w` (unsigned) as two floats 32768 + byte: the byte becomes bits 8..15 of the float
// 0x47000000, whose last mantissa bit is worth 2^-8.  One byte permute per value instead of a slow conversion;
// subtracting 32768 (+ bias) is exact.
__device__ __forceinline__ uint64_t bytes_to_f2(uint32_t w, int h)
{
    const uint32_t a = __byte_perm(w, 0x47000000u, h ? 0x7424 : 0x7404);
    const uint32_t b = __byte_perm(w, 0x47000000u, h ? 0x7434 : 0x7414);
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}

// What one lane keeps of a 16 x 256 tile: all quant words and the scales of rows g and g+8.
template <int FMT>
struct Packed {
    static constexpr int NQ = FMT == FMT_Q8_0 ? 8 : FMT == FMT_Q6_K ? 6 : 4;  // 16-byte groups of quants
    uint4 q[NQ];
};

// rows g and g+8: Q4_0/Q8_0 eight fp16 scales each; Q6_K sixteen int8 scales each; Q4_K {12 packed bytes, (d, dmin)}
template <int FMT>
struct Scales {
    uint4 s[2];
    uint32_t d;  // Q6_K: fp16 d of row g (low) and g+8 (high)
};

template <int FMT>
__device__ __forceinline__ void load_scales(Scales<FMT>& o, const uint8_t* tile, int g)
{
    const uint8_t* p1 = tile + tile_p1_offset(FMT);
    if constexpr (FMT == FMT_Q4_K) {
        const uint8_t* p2 = tile + tile_p2_offset(FMT);
#pragma unroll
        for (int rs = 0; rs < 2; ++rs) {
            const uint8_t* sp = p1 + (g + 8 * rs) * 12;
            o.s[rs] = make_uint4(ldg_u32(sp), ldg_u32(sp + 4), ldg_u32(sp + 8), ldg_u32(p2 + (g + 8 * rs) * 4));
        }
    } else {
        o.s[0] = ldg_u128(p1 + g * 16);
        o.s[1] = ldg_u128(p1 + (g + 8) * 16);
        if constexpr (FMT == FMT_Q6_K) {
            const unsigned short* p2 = reinterpret_cast<const unsigned short*>(tile + tile_p2_offset(FMT));
            o.d = (uint32_t)__ldg(p2 + g) | ((uint32_t)__ldg(p2 + g + 8) << 16);
        }
    }
}

// Loads the 16-byte groups whose last use is quarter q (all of them over q = 0..3).
template <int FMT>
__device__ __forceinline__ void load_quarter(Packed<FMT>& o, const uint8_t* tile, int q, int lane)
{
    const uint8_t* p = tile + lane * 16;
    if constexpr (FMT == FMT_Q8_0) {
        o.q[2 * q] = ldg_u128(p + (2 * q) * 512);
        o.q[2 * q + 1] = ldg_u128(p + (2 * q + 1) * 512);
    } else if constexpr (FMT == FMT_Q6_K) {
        // quarter q reads words 6q .. 6q+5
        if (q == 0) {
            o.q[0] = ldg_u128(p);
        } else if (q == 1) {
            o.q[1] = ldg_u128(p + 512);
            o.q[2] = ldg_u128(p + 2 * 512);
        } else if (q == 2) {
            o.q[3] = ldg_u128(p + 3 * 512);
        } else {
            o.q[4] = ldg_u128(p + 4 * 512);
            o.q[5] = ldg_u128(p + 5 * 512);
        }
    } else {
        o.q[q] = ldg_u128(p + q * 512);
    }
}

// Quarter q (a compile-time constant after unrolling) -> 16 registers of bf16 pairs.  The fp32 value of every weight
// has the same roundings as ggml's to_float: integers are exact, and every product is rounded once.
template <int FMT>
__device__ __forceinline__ void dequant_quarter(const Packed<FMT>& P, const Scales<FMT>& S, int q, uint32_t (&r)[16])
{
    const float base = FMT == FMT_Q4_0 ? 32776.0f : FMT == FMT_Q4_K ? 32768.0f : 32896.0f;
    const uint64_t minus = f2_pair(-base, -base);
    if constexpr (FMT == FMT_Q4_0) {
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const uint32_t w = word4(P.q[q], p);
#pragma unroll
            for (int rs = 0; rs < 2; ++rs) {
                const uint32_t n = (rs ? w >> 4 : w) & 0x0F0F0F0Fu;
                const float d = h2f_bits(word4(S.s[rs], q) >> (16 * (p >> 1)));
                const uint64_t dd = f2_pair(d, d);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    r[4 * p + 2 * rs + h] = f2_to_bf16x2(f2_mul(f2_add(bytes_to_f2(n, h), minus), dd));
                }
            }
        }
    } else if constexpr (FMT == FMT_Q8_0) {
#pragma unroll
        for (int p = 0; p < 4; ++p) {
#pragma unroll
            for (int rs = 0; rs < 2; ++rs) {
                const uint32_t n = word4(P.q[2 * q + (p >> 1)], 2 * (p & 1) + rs) ^ 0x80808080u;
                const float d = h2f_bits(word4(S.s[rs], q) >> (16 * (p >> 1)));
                const uint64_t dd = f2_pair(d, d);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    r[4 * p + 2 * rs + h] = f2_to_bf16x2(f2_mul(f2_add(bytes_to_f2(n, h), minus), dd));
                }
            }
        }
    } else if constexpr (FMT == FMT_Q4_K) {
#pragma unroll
        for (int rs = 0; rs < 2; ++rs) {
            const uint32_t w0 = S.s[rs].x, w1 = S.s[rs].y, w2 = S.s[rs].z;
            const uint32_t scw = q < 2 ? (w0 & 0x3F3F3F3Fu) : ((w2 & 0x0F0F0F0Fu) | ((w0 >> 2) & 0x30303030u));
            const uint32_t mnw = q < 2 ? (w1 & 0x3F3F3F3Fu) : (((w2 >> 4) & 0x0F0F0F0Fu) | ((w1 >> 2) & 0x30303030u));
            const float d = h2f_bits(S.s[rs].w);
            const float dmin = h2f_bits(S.s[rs].w >> 16);
            // sub-blocks 2q and 2q+1: d * scale and dmin * min are exact (11 + 6 bits)
            const uint64_t sc = f2_mul(f2_add(bytes_to_f2(scw, q & 1), minus), f2_pair(d, d));
            const uint64_t mn = f2_mul(f2_add(bytes_to_f2(mnw, q & 1), minus), f2_pair(-dmin, -dmin));
#pragma unroll
            for (int sb = 0; sb < 2; ++sb) {
                float sc1, sc2, mn1, mn2;
                asm("mov.b64 {%0, %1}, %2;" : "=f"(sc1), "=f"(sc2) : "l"(sc));
                asm("mov.b64 {%0, %1}, %2;" : "=f"(mn1), "=f"(mn2) : "l"(mn));
                const uint64_t d1 = sb ? f2_pair(sc2, sc2) : f2_pair(sc1, sc1);
                const uint64_t m1 = sb ? f2_pair(mn2, mn2) : f2_pair(mn1, mn1);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int p = 2 * sb + half;
                    const uint32_t w = word4(P.q[q], p);
                    const uint32_t n = (rs ? w >> 4 : w) & 0x0F0F0F0Fu;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        // d1 * n is exact (17 + 4 bits), so the fused form rounds once, like product and difference
                        r[4 * p + 2 * rs + h] = f2_to_bf16x2(f2_fma(f2_add(bytes_to_f2(n, h), minus), d1, m1));
                    }
                }
            }
        }
    } else {  // Q6_K: a byte is 4 * (q - 32) as int8; scaling by d * scale / 4 keeps every bit
#pragma unroll
        for (int rs = 0; rs < 2; ++rs) {
            const int w = (q * 2 + rs) * 3;
            const uint32_t X = word4(P.q[w >> 2], w & 3), Y = word4(P.q[(w + 1) >> 2], (w + 1) & 3),
                           Z = word4(P.q[(w + 2) >> 2], (w + 2) & 3);
            const float d = h2f_bits(S.d >> (16 * rs)) * 0.25f;
            const uint32_t sc = word4(S.s[rs], q) ^ 0x80808080u;
            const uint64_t s01 = f2_mul(f2_add(bytes_to_f2(sc, 0), minus), f2_pair(d, d));
            const uint64_t s23 = f2_mul(f2_add(bytes_to_f2(sc, 1), minus), f2_pair(d, d));
            float ds[4];
            asm("mov.b64 {%0, %1}, %2;" : "=f"(ds[0]), "=f"(ds[1]) : "l"(s01));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(ds[2]), "=f"(ds[3]) : "l"(s23));
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const uint32_t v = p == 0   ? X & 0xFCFCFCFCu
                                   : p == 1 ? Y & 0xFCFCFCFCu
                                   : p == 2 ? Z & 0xFCFCFCFCu
                                            : ((X & 0x03030303u) << 6) | ((Y & 0x03030303u) << 4) | ((Z & 0x03030303u) << 2);
                const uint32_t n = v ^ 0x80808080u;
                const uint64_t dd = f2_pair(ds[p], ds[p]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    r[4 * p + 2 * rs + h] = f2_to_bf16x2(f2_mul(f2_add(bytes_to_f2(n, h), minus), dd));
                }
            }
        }
    }
}

}  // namespace

}  // namespace qmm
