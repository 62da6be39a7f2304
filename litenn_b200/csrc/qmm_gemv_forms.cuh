// Which form a matvec of one row takes (qmm_gemv_kernel.cuh): its shared memory, the one-wave rule and the compiled forms.
// Host code without state; every choice is made from the format, the row tiles, the K chunks and the SM count.
#pragma once

#include <cuda_runtime.h>

#include "qmm_common.cuh"

namespace qmm {

namespace {

// Shared memory of one CTA, carved from the dynamic allocation:
//   slots  TILES*WARPS*DEPTH x tile | mbarriers (+1 for the activations) | all activation records + 512 zero bytes |
//   cross-warp reduction
template <int FMT, int WARPS, int DEPTH, int TILES>
struct SmemPlan {
    static constexpr int NW = WARPS * TILES;
    static constexpr int SLOT = tile_bytes(FMT);
    static constexpr int SLOTS_BYTES = NW * DEPTH * SLOT;
    static constexpr int BAR_OFF = SLOTS_BYTES;
    static constexpr int BAR_BYTES = (((NW * DEPTH + 1) * 8 + 15) / 16) * 16;
    static constexpr int X_OFF = BAR_OFF + BAR_BYTES;
    __host__ __device__ static constexpr int red_off(int kc) { return X_OFF + (int)xpack1_bytes(kc) + 512; }
    __host__ __device__ static constexpr int total(int kc) { return red_off(kc) + NW * 16 * 4; }
};

constexpr int GEMV_SMEM_LIMIT = 227 * 1024;

// Row tiles per CTA of the one-wave form, in whole groups of a fused form (epi_tiles), that put every tile on the chip at once,
// and whether such CTAs sit on at least four fifths of the SMs.
constexpr int gemv_wave_tiles(int rt, int group, int sms)
{
    return ((rt + sms - 1) / sms + group - 1) / group * group;
}
constexpr bool gemv_wave_fills(int rt, int group, int sms)
{
    return 5LL * rt >= 4LL * sms * gemv_wave_tiles(rt, group, sms);
}

// The longest row that the rules were measured on (28672 columns); longer ones keep the small CTAs.  Shared memory would do for
// 127 chunks (16 tiles of a 4-bit format) and more.
constexpr int GEMV_WAVE_KC = 112;

// Whether the matvec of one fp32 vector of kc chunks packs it itself, as far as the shape decides.
// One launch instead of two while every SM's copy of the vector costs less than the packing kernel and its boundary (1.1 us
// of a stream, 2.6 us of a host loop, where 1024 x 4096 falls from 7.0 to 5.2 us).  Up to 32 chunks it does, the one wave
// being also the better matvec; above, packing 11008 values takes 256 rows of Q4_0 5.5 us and not 4.4, and only Q8_0
// on one row tile per SM gains (7.5 -> 5.9).  Q8_0 beyond 16 chunks is bound by its bytes either way (28672 x 8192: 39.7
// us, 40.5 in one launch).  Of many tiles per SM only the 4-bit formats have room for enough slots.
constexpr bool gemv_packs_itself_shape(int fmt, int rt, int kc, int sms)
{
    const int tiles = gemv_wave_tiles(rt, 1, sms);
    if (kc > 32) {
        return fmt == FMT_Q8_0 && tiles == 1 && kc <= GEMV_WAVE_KC;
    }
    if (fmt == FMT_Q8_0) {
        return tiles <= (kc > 16 ? 2 : 16);
    }
    return tiles <= (fmt == FMT_Q6_K ? 16 : 28);
}

// Where the one-wave form takes a packed vector: where it was measured to be faster than the small CTAs of the forms below,
// over every format, rows of 1..112 chunks and 2..28 tiles per SM.  Small CTAs that are all resident at once and even need no
// wave of their own; how many an SM holds follows from the format's tiles and the warps that K gives them, so the lines lie
// elsewhere for each.  Streams of different weights, us each, small CTAs and one wave, on both sides of a line:
//   plain, K up to 16 chunks   two tiles per SM are one or two CTAs to an SM: 16 chunks 1.35 times, 4 chunks 0.98.
//                              Q4_0 7 tiles 6 chunks 3.6 and 2.9, 3 chunks 2.6 and 3.0; 14 tiles 16 chunks 15.0 and 15.1,
//                              16 tiles 16.7 and 18.1 (32 warps).  Q4_K 5 tiles 12 chunks 1.14 times, 7 chunks 3.8 and 4.2;
//                              5 chunks 12 tiles 1.01 times, 14 tiles 0.94.  Q6_K 6 tiles 8 chunks 1.18 times, 9 chunks 0.95.
//                              Q8_0 5 tiles 16 chunks 1.15 times, 12 chunks 6.5 and 7.2; 12 tiles 12 chunks 16.9 and 18.6
//   longer rows                Q6_K 3 tiles and more 1.2..1.5 times; 4-bit rows of up to 30 chunks three CTAs to an SM at 3
//                              tiles: 24 chunks 1.29 times with all places taken, 4.4 and 5.1 with few.  Q4_0 16 tiles 20
//                              chunks 1.05 times, 32 chunks 0.94.  Q8_0 5 tiles 1.17 times, 8 tiles 0.98, 12 tiles 0.95
//   plain, in a chain (ss_in)  small CTAs also start while the kernel before drains, which a CTA that fills its SM cannot: the
//                              line lies at nine tiles (70B-shape vocabulary 562.3 -> 558.1 us a token; with the QKV matvec in
//                              it 564.5).  Vocabularies of Q8_0: 12 chunks 1.00..1.05 times, 16..24 chunks 0.97..1.03
//   residual (n / 32 small CTAs; grids that the rounding to whole groups leaves on fewer than four fifths of the SMs gain
//                              nothing)  8192 rows, Q6_K 16 chunks 1.30 times, 32 chunks 0.97, 112 chunks 1.20; Q4_K 0.99,
//                              0.94, 1.08; 9216 rows, Q4_0 16 chunks 1.18, 12 chunks 0.98; 12288 rows, Q4_0 16 chunks 1.17, 32
//                              chunks 0.94, 80 chunks 1.12; 16384 rows, Q8_0 1.0..1.5 throughout, Q4_0 8 chunks 0.93, 12
//                              chunks 1.20, 17 chunks 0.90
//   packed gate|up             its groups of four tiles sit three to an SM: 12 tiles and fewer are one wave already (Q4_0
//                              22016 x 4096 0.98, Q6_K 0.99; Q4_K 1.06 and with 27648 rows 0.96, Q8_0 1.21 and with 9 chunks
//                              0.96).  13..16 tiles: Q4_0 16 chunks 1.12, 8 chunks 0.92; Q6_K 1.13, 1.20.  Q6_K 28 tiles 20
//                              chunks 0.95
template <int FMT, int EPI>
constexpr bool gemv_one_wave(int rt, int kc, bool chained, int sms)
{
    constexpr bool NIBBLE = tile_bytes(FMT) == 2304;
    const int tiles = gemv_wave_tiles(rt, epi_tiles(EPI), sms);
    if (kc > GEMV_WAVE_KC || tiles > (EPI == EPI_SWIGLU_PACK || (EPI == EPI_STORE && NIBBLE) ? 28 : 16)) {
        return false;
    }
    if constexpr (EPI == EPI_SWIGLU_PACK) {
        if (tiles <= 12) {
            return rt > 8 * sms && kc > 9 && (FMT == FMT_Q8_0 || (FMT == FMT_Q4_K && rt <= 11 * sms));
        }
        if (tiles <= 16) {
            return !NIBBLE || kc > (FMT == FMT_Q4_0 ? 10 : 8);
        }
        return FMT != FMT_Q6_K || tiles <= 24 || kc <= 12;
    } else if constexpr (EPI == EPI_RESID_PACK) {
        if (rt <= 2 * sms || !gemv_wave_fills(rt, epi_tiles(EPI), sms)) {
            return false;
        }
        if (tiles <= 4) {
            return kc >= 96 || (FMT == FMT_Q6_K && kc > 8 && kc <= 16) ||
                   (NIBBLE && kc > 12 && kc <= 16 && 10LL * rt >= 9LL * sms * tiles);
        }
        if (tiles <= 6) {
            return kc > 64 || (FMT != FMT_Q8_0 && kc > 8 && kc <= 16);
        }
        return !NIBBLE || (kc > 8 && (tiles > 8 || kc <= 16 || kc >= 32));
    } else {
        if (FMT == FMT_Q4_0 && tiles > 14 && ((kc > 12 && kc <= 16) || (kc > 20 && tiles <= 16))) {
            return false;
        }
        if (chained) {
            return tiles >= 9 && (FMT != FMT_Q8_0 || kc <= 12);
        }
        if (kc > 16) {
            return FMT == FMT_Q8_0   ? tiles >= (kc > 32 ? 4 : 5) && tiles <= 6
                   : FMT == FMT_Q6_K ? tiles >= 3
                                     : tiles >= 4 || (tiles == 3 && (kc > 30 || 2 * rt > 5 * sms));
        }
        if (tiles <= 2) {
            return tiles == 2 && kc >= 5;
        }
        if constexpr (FMT == FMT_Q4_0) {
            return tiles >= (kc >= 3 && kc <= 5 ? 8 : 7);
        } else if constexpr (FMT == FMT_Q4_K) {
            return tiles >= (kc <= 2 ? 6 : kc <= 5 ? 8 : kc <= 8 ? 7 : kc < 16 ? 5 : 4) &&
                   !(kc >= 3 && kc <= 5 && tiles > 12 && tiles <= 14);
        } else if constexpr (FMT == FMT_Q6_K) {
            return tiles >= (kc > 8 && kc <= 12 ? 7 : 6);
        } else {
            return tiles >= (kc == 16 ? 5 : kc == 2 || kc == 3 ? 7 : 6) && (kc <= 10 || tiles <= 8);
        }
    }
}

// Least and most K chunks with which a one-wave form of FIRST..TILES row tiles per CTA is chosen; {0, 0}: never.  The rules
// compare row tiles with multiples of the SM count, so a few fill levels of a notional chip reach every case.
struct GemvRows {
    int least, most;
};
template <int FMT, int EPI, bool XF32>
constexpr GemvRows gemv_wave_rows(int first, int tiles)
{
    constexpr int SMS = 1000, FILL[4] = {1, 501, 951, 1000};
    GemvRows r = {0, 0};
    for (int kc = 1; kc <= GEMV_WAVE_KC; ++kc) {
        bool any = false;
        for (int t = first; t <= tiles && !any; ++t) {
            for (int f = 0; f < 4 && !any; ++f) {
                const int rt = (t - 1) * SMS + FILL[f];
                any = XF32 ? gemv_packs_itself_shape(FMT, rt, kc, SMS)
                           : gemv_one_wave<FMT, EPI>(rt, kc, false, SMS) || gemv_one_wave<FMT, EPI>(rt, kc, true, SMS);
            }
        }
        if (any) {
            r.least = r.least > 0 ? r.least : kc;
            r.most = kc;
        }
    }
    return r;
}

// The one-wave form: a CTA on every SM, each with as many row tiles as that takes (ceil(tiles / SMs), up to the next
// compiled count), WARPS warps and WARPS x DEPTH slots per tile.  What bounds a matvec of many small CTAs is the last
// of its waves and, for an fp32 vector, that every CTA packs the vector again; here there is one wave and at most 148
// copies.  Measured on B200, a stream of different weights, us each, many CTAs -> one wave:
//   packed vector  Q4_0 8192 x 28672 28.9 -> 22.4, 10240 x 8192 12.4 -> 9.4, 28672 x 8192 27.4 -> 22.7, 4096 x 4096 3.8 -> 3.5;
//                  Q4_K 28672 x 8192 29.9 -> 22.6, 11008 x 4096 7.4 -> 6.7; Q6_K 28672 x 8192 35.4 -> 31.5, 14336 x 4096
//                  11.1 -> 9.7; Q8_0 11008 x 4096 11.0 -> 9.5
//   fp32 vector    (before: a kernel that packs it, then the matvec) Q4_0 1024 x 4096 4.2 -> 3.0, 14336 x 4096 9.5 -> 8.1,
//                  28672 x 8192 28.2 -> 23.9; Q4_K 14336 x 4096 10.6 -> 9.0; Q6_K 4096 x 2048 4.2 -> 3.4; Q8_0 4096 x 4096 6.0 -> 5.4
// More warps per tile shorten a short row's chain of tiles; beyond about 90 KB of slots they gain little, so the warps per
// tile fall as the tiles grow.  The shared-memory request keeps a second CTA of the same kernel off an SM: without
// it, 4096 x 8192 of Q4_K takes 7.2 us and not 5.6.
//
// Only what the rules can choose is compiled: run.form<TILES, WARPS, DEPTH>() is instantiated for those.
template <int FMT, int EPI, bool XF32, class Run>
struct GemvWave {
    int kc;
    const Run& run;
    static constexpr bool NIBBLE = tile_bytes(FMT) == 2304;

    template <int W, int D>
    struct Shape {
        static constexpr int WARPS = W, DEPTH = D;
    };

    // The first of the shapes that leaves the activations of LEAST..MOST chunks their room; the last one always does.
    template <int TILES, int LEAST, int MOST, class S, class... Less>
    cudaError_t fitting() const
    {
        using Plan = SmemPlan<FMT, S::WARPS, S::DEPTH, TILES>;
        if constexpr (sizeof...(Less) == 0 || Plan::total(MOST) <= GEMV_SMEM_LIMIT) {
            static_assert(Plan::total(MOST) <= GEMV_SMEM_LIMIT, "every row that the rules let in has a form");
            return run.template form<TILES, S::WARPS, S::DEPTH>();
        } else if constexpr (Plan::total(LEAST) > GEMV_SMEM_LIMIT) {
            return fitting<TILES, LEAST, MOST, Less...>();
        } else {
            return Plan::total(kc) <= GEMV_SMEM_LIMIT ? run.template form<TILES, S::WARPS, S::DEPTH>()
                                                      : fitting<TILES, LEAST, MOST, Less...>();
        }
    }

    // FIRST..TILES row tiles per CTA: SHORT for rows of up to KC chunks, else the first of LONG that fits.
    template <int FIRST, int TILES, int KC, class Short, class... Long>
    cudaError_t rows() const
    {
        constexpr GemvRows R = gemv_wave_rows<FMT, EPI, XF32>(FIRST, TILES);
        if constexpr (TILES % epi_tiles(EPI) != 0 || R.most == 0) {
            return cudaErrorInvalidConfiguration;  // not reached
        } else if constexpr (R.most <= KC) {
            return fitting<TILES, R.least, R.most, Short>();
        } else if constexpr (R.least > KC) {
            return fitting<TILES, R.least, R.most, Long...>();
        } else {
            return kc <= KC ? fitting<TILES, R.least, KC, Short>() : fitting<TILES, KC + 1, R.most, Long...>();
        }
    }
    template <int FIRST, int TILES, class... Long>
    cudaError_t all() const
    {
        return rows<FIRST, TILES, 0, Shape<1, 1>, Long...>();
    }

    cudaError_t launch(int tiles) const
    {
        if constexpr (EPI != EPI_SWIGLU_PACK) {
            // up to eight chunks a warp walks two tiles at most, whatever the form: fewer warps to add up
            if (tiles <= 8) {
                return tiles <= 1   ? rows<1, 1, 4, Shape<8, 1>, Shape<16, 2>>()
                       : tiles == 2 ? all<2, 2, Shape<8, 2>>()
                       : tiles == 3 ? three()
                       : tiles == 4 ? all<EPI == EPI_RESID_PACK ? 3 : 4, 4, Shape<4, 3>, Shape<4, 2>>()
                       : tiles == 5 ? all<5, 5, Shape<4, 2>, Shape<4, 1>>()
                       : tiles == 6 ? rows<EPI == EPI_RESID_PACK ? 5 : 6, 6, 8, Shape<2, 2>, Shape<4, 2>, Shape<2, 2>>()
                       : tiles == 7 ? seven()
                                    : rows<EPI == EPI_RESID_PACK ? 7 : 8, 8, 8, Shape<2, 2>, Shape<2, 3>, Shape<2, 2>>();
            }
            if (tiles <= 10) {
                return all<9, 10, Shape<2, 2>, Shape<2, 1>>();
            }
        }
        if (tiles <= 12) {
            return all<EPI == EPI_SWIGLU_PACK ? 9 : 11, 12, Shape<2, 2>, Shape<2, 1>>();
        }
        // Q6_K and Q8_0 leave room for two warps per row tile only with one slot each: one warp with three is 4 % faster.
        // So it is inside a chain for every format, as 32 warps of 64 registers leave the next kernel none (28672 x 7168
        // and three blocks, Q4_0: 227 us a token with two warps, 200 with one).
        if (tiles <= 16) {
            if constexpr (NIBBLE && EPI == EPI_STORE) {
                return tiles <= 14 ? all<13, 14, Shape<2, 2>>() : all<15, 16, Shape<2, 2>>();
            } else if constexpr (EPI == EPI_SWIGLU_PACK) {  // whole groups of four
                return all<13, 16, Shape<1, 3>, Shape<1, 2>>();
            } else {
                return tiles <= 14 ? all<13, 14, Shape<1, 3>, Shape<1, 2>>() : all<15, 16, Shape<1, 3>, Shape<1, 2>>();
            }
        }
        if constexpr (EPI == EPI_SWIGLU_PACK) {
            return tiles <= 20   ? all<17, 20, Shape<1, 2>, Shape<1, 1>>()
                   : tiles <= 24 ? all<21, 24, Shape<1, 2>, Shape<1, 1>>()
                   : tiles <= 28 ? all<25, 28, Shape<1, 2>, Shape<1, 1>>()
                                 : cudaErrorInvalidConfiguration;
        } else if constexpr (EPI == EPI_STORE && NIBBLE) {
            return tiles <= 20   ? all<17, 20, Shape<1, 2>>()
                   : tiles <= 25 ? all<21, 25, Shape<1, 2>>()
                   : tiles <= 28 ? all<26, 28, Shape<1, 2>>()
                                 : cudaErrorInvalidConfiguration;
        }
        return cudaErrorInvalidConfiguration;
    }

    cudaError_t three() const
    {
        if constexpr (XF32) {
            return kc > 4 && kc <= 8 ? fitting<3, 5, 8, Shape<8, 1>>() : all<3, 3, Shape<5, 2>>();
        } else {
            return all<3, 3, Shape<5, 2>>();
        }
    }
    cudaError_t seven() const
    {
        if constexpr (NIBBLE) {
            return rows<7, 7, 8, Shape<2, 2>, Shape<4, 2>>();
        } else {
            return rows<7, 7, 8, Shape<2, 2>, Shape<2, 3>, Shape<2, 2>>();
        }
    }
};

// The one-wave form of rt row tiles and kc chunks, where gemv_one_wave or gemv_packs_itself_shape says so.
template <int FMT, int EPI, bool XF32, class Run>
cudaError_t gemv_wave_form(int rt, int kc, int sms, const Run& run)
{
    return GemvWave<FMT, EPI, XF32, Run>{kc, run}.launch(gemv_wave_tiles(rt, epi_tiles(EPI), sms));
}

// Packed gate|up in small CTAs: four row tiles per CTA, two warps per tile with two slots each: 8 warps walk kc / 2 tiles apiece
// (8 for K = 4096) and a third of a 1376-tile gate|up weight's CTAs fit an SM together (three slots: 1 % of a 7B-shape step
// slower).  Where a long row's CTAs have an SM each, four warps per tile: two keep too few bytes in flight (8192 wide, eight
// blocks, FFN 2304 Q4_0 200 -> 182 us a token, 3584 Q4_K 227 -> 209).  One warp per tile where the activations of rows beyond
// 60000 columns leave no room for more slots.
template <int FMT, class Run>
cudaError_t gemv_small_glu_form(int rt, int kc, int sms, const Run& run)
{
    constexpr int TILES = epi_tiles(EPI_SWIGLU_PACK);
    if (kc > 16 && rt <= TILES * sms && SmemPlan<FMT, 4, 2, TILES>::total(kc) <= GEMV_SMEM_LIMIT) {
        return run.template form<TILES, 4, 2>();
    }
    if (SmemPlan<FMT, 2, 2, TILES>::total(kc) <= GEMV_SMEM_LIMIT) {
        return run.template form<TILES, 2, 2>();
    }
    return run.template form<TILES, 1, 2>();
}

}  // namespace

}  // namespace qmm
