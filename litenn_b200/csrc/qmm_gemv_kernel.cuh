// Dequant-fused GEMV for decode (one activation row) on sm_100a: the kernel template, and the per-format launcher of a
// matvec of any row count.  Each block format instantiates it in a translation
// unit of its own (qmm_gemv_q4_0.cu, ...), so the formats compile in parallel.  2..16 rows are qmm_gemv_batch.cuh.
//
// The weights never become floats in memory.  One CTA owns one 16-row tile of the
// output, or several (TILES: the fused forms' groups, and the one-wave forms of qmm_gemv_forms.cuh, which also choose
// among the small ones of gate|up); WARPS warps take the 256-column K chunks of each row tile round-robin.
// Every chunk is one contiguous packed tile (qmm_common.cuh) that a single TMA bulk
// copy (cp.async.bulk, completion counted on an mbarrier) lands in a shared-memory
// slot.  Each warp owns DEPTH slots and refills a slot itself as soon as it has
// consumed it, so the copies of a whole CTA are in flight from the first instruction
// on and HBM latency is paid once, not per chunk.  From shared memory the quants become
// int8 MMA A-fragments with two or three logic ops per word and are multiplied on the
// integer tensor-core path (mma.sync m16n8k32, s32 accumulate) with the
// activations, quantized to 16 bits per 32-wide block and split into a signed high and a
// signed low byte.  The int32 block sums are exact; they are folded into fp32 accumulators
// with the block's fp16 weight scale and the block's activation scale, so the accumulation
// across blocks is fp32 as in the reference loop (src/LiteNN/Device.h:645-658).  The only
// approximation is the 16-bit activation quantization (relative error <= 2^-16 of the
// block maximum).
//
// Kernels are launched with programmatic dependent launch: the weight copies are issued
// before griddepcontrol.wait, so in a chain of dependent matvecs the next kernel's weights
// stream while the previous kernel drains.  All packed activations come into
// shared memory with one more bulk copy.
//
// Fused forms (GemvFuse in qmm_common.cuh) let a chain of matvecs run without glue
// kernels between them: a matvec can pack its own fp32 input, apply the scalar 1/rms of an
// RMSNorm to its row sums, and write the NEXT matvec's packed input (with the residual add and the
// norm weights folded in) or silu(gate) * up from its epilogue.
#pragma once

#include <mutex>

#include "qmm_gemv_batch.cuh"
#include "qmm_gemv_device.cuh"
#include "qmm_gemv_forms.cuh"
#include "qmm_kernels.h"
#include "qmm_pack.cuh"

namespace qmm {

namespace {

// WARPS warps share one row tile; a CTA holds TILES row tiles (at least 2 for EPI_RESID_PACK: the 32 rows of
// one quantization block of the output, so the epilogue can quantize them without leaving the CTA).
// Registers decide how many CTAs an SM holds, and a batch-1 grid of 768 row tiles wants six CTAs of
// 256 threads on every SM at once (42 registers at most): the bound keeps the fp32-packing prologue
// and the fused epilogues from costing a second wave.  Plain CTAs of 128 threads are held to 64 registers, eight to an SM:
// one row of Q6_K 11008 x 2048 takes 7.29 us, 7.70 with six to an SM; Q4_0 and Q8_0 differ by 1 % at most, either way.
template <int THREADS, int EPI, int TILES, bool XF32>
constexpr int gemv_min_blocks()
{
    if (TILES > epi_tiles(EPI) || (XF32 && EPI == EPI_STORE) || EPI == EPI_RESID_PACK) {  // the one-wave forms, and few CTAs
        return 1;
    }
    if (EPI == EPI_SWIGLU_PACK) {
        return THREADS <= 256 ? 3 : 1;
    }
    return THREADS <= 128 ? 8 : THREADS <= 256 ? 6 : 3;
}

template <int FMT, int WARPS, int DEPTH, int EPI, int TILES, bool XF32>
__global__ void __launch_bounds__(WARPS * TILES * 32, gemv_min_blocks<WARPS * TILES * 32, EPI, TILES, XF32>())
    gemv_kernel(WeightView v, XPackView xp, float* __restrict__ y, int* __restrict__ status, PeerScatter ps,
                GemvFuse fu)
{
    using Plan = SmemPlan<FMT, WARPS, DEPTH, TILES>;
    constexpr int NW = WARPS * TILES;
    constexpr uint32_t TILE = tile_bytes(FMT);
    static_assert(TILES % epi_tiles(EPI) == 0, "a fused form's group of row tiles stays in one CTA");
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float s_in_sh;  // 1/rms factor of the input activations

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int wl = warp % WARPS;                                // this warp's place among its tile's warps
    const int64_t tile_row = (int64_t)blockIdx.x * TILES + warp / WARPS;  // row tile of this warp
    const int kc = v.kc;
    uint8_t* my_slots = smem + (size_t)warp * DEPTH * Plan::SLOT;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Plan::BAR_OFF);
    uint64_t* my_bars = bars + warp * DEPTH;
    uint64_t* xbar = bars + NW * DEPTH;
    const uint8_t* my_tiles = v.tiles + (size_t)tile_row * kc * TILE;
    const int n_my = (wl < kc && tile_row < v.rt) ? (kc - wl + WARPS - 1) / WARPS : 0;

    // 1. start the weight stream: the first DEPTH tiles of this warp
    if (lane == 0) {
        for (int s = 0; s < DEPTH; ++s) {
            mbar_init(&my_bars[s], 1);
        }
        if (warp == 0) {
            mbar_init(xbar, 1);
        }
        fence_barrier_init();
        for (int s = 0; s < DEPTH && s < n_my; ++s) {
            mbar_expect_tx(&my_bars[s], TILE);
            bulk_copy_g2s(my_slots + (size_t)s * Plan::SLOT, my_tiles + (size_t)(wl + s * WARPS) * TILE, TILE,
                          &my_bars[s]);
        }
    }
    if constexpr (FMT == FMT_Q6_K) {
        // zero page for the lanes that carry no activation row
        uint32_t* z = reinterpret_cast<uint32_t*>(smem + Plan::X_OFF + xpack1_bytes(kc));
        for (int i = threadIdx.x; i < 128; i += NW * 32) {
            z[i] = 0u;
        }
    }
    pdl_launch_dependents();
    // 2. everything below may read what earlier kernels in the stream produced
    pdl_wait();

    unsigned int epoch = 0;
    if constexpr (EPI == EPI_STORE || EPI == EPI_RESID_PACK) {
        if (ps.n_peers > 0) {
            epoch = (unsigned int)(*ps.pos * ps.sites + ps.site + 1);
        }
    }
    XShared xsrc;
    bool ok = true;
    float h_pre = 0.0f, w_pre = 0.0f;  // EPI_RESID_PACK: residual and norm weight of this thread's row
    uint8_t* xbase = smem + Plan::X_OFF;
    const uint32_t xbytes = (uint32_t)xpack1_bytes(kc);
    if (!XF32 && threadIdx.x == 0) {  // the thread that initialised xbar
        mbar_expect_tx(xbar, xbytes);
        bulk_copy_g2s(xbase, xp.base, xbytes, xbar);
    }
    if (warp == NW - 1) {
        // the scalar RMSNorm factor of the input: the producer left one sum of squares per 32 activations
        double t = 0.0;
        if (fu.ss_in) {
            for (int i = lane; i < fu.ss_count; i += 32) {
                t += fu.ss_in[i];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
            }
        }
        if (lane == 0) {
            s_in_sh = fu.ss_in ? (float)(1.0 / sqrt(t / (double)fu.d_in + (double)fu.eps)) : 1.0f;
        }
    }
    if constexpr (EPI == EPI_RESID_PACK) {
        if (threadIdx.x < 16 * TILES) {
            const int64_t row = (int64_t)blockIdx.x * (16 * TILES) + threadIdx.x;
            if (row < v.n) {
                h_pre = fu.h_in[row];
                w_pre = fu.norm_w[row];
            }
        }
    }
    if constexpr (XF32) {
        // pack the fp32 activations here: spans of 128, one float4 per lane, all loads of a thread issued
        // before the first is used.  Every CTA reads the same few KB: each starts at another span, so
        // that the CTAs do not all ask the same L2 lines at the same moment.
        const int nspan = (int)(v.k / 128);
        constexpr int MAXS = 4;
        const int rot = nspan > 0 ? (int)((blockIdx.x * 13u) % (unsigned)nspan) : 0;
        const float* xsrc_f = fu.x_f32;
        for (int s0 = warp; s0 < nspan; s0 += NW * MAXS) {
            float4 xv[MAXS];
#pragma unroll
            for (int i = 0; i < MAXS; ++i) {
                const int sq = s0 + i * NW;
                if (sq < nspan) {
                    const int sp = sq + rot < nspan ? sq + rot : sq + rot - nspan;
                    xv[i] = __ldcg(reinterpret_cast<const float4*>(xsrc_f) + sp * 32 + lane);
                }
            }
#pragma unroll
            for (int i = 0; i < MAXS; ++i) {
                const int sq = s0 + i * NW;
                if (sq < nspan) {
                    const int sp = sq + rot < nspan ? sq + rot : sq + rot - nspan;
                    warp_pack_span128(xv[i], xbase + (size_t)(sp >> 1) * XPK1_REC, (sp & 1) * 4);
                }
            }
        }
        for (int blk = nspan * 4 + warp; blk < kc * 8; blk += NW) {  // the ragged end, then zero blocks
            const int64_t e = (int64_t)blk * 32 + lane;
            warp_pack_block32(e < v.k ? __ldcg(xsrc_f + e) : 0.0f, xbase + (size_t)(blk >> 3) * XPK1_REC, blk & 7);
        }
    }
    __syncthreads();  // xbar initialised, zero page written, activations packed
    xsrc.base = xbase;
    xsrc.zeros = xbase + xbytes;
    if (!XF32 && !mbar_wait(xbar, 0)) {
        ok = false;
        if (lane == 0) {
            atomicExch(status, 2);
        }
    }

    float acc[2] = {0.0f, 0.0f};

    // 3. consume tiles as they land; refill each slot right after it has been read
    for (int i = 0; i < n_my; ++i) {
        const int s = i % DEPTH;
        const uint32_t parity = (uint32_t)(i / DEPTH) & 1u;
        if (ok && !mbar_wait(&my_bars[s], parity)) {
            ok = false;
            if (lane == 0) {
                atomicExch(status, 1);
            }
        }
        if (ok) {
            compute_chunk_m1<FMT>(my_slots + (size_t)s * Plan::SLOT, xsrc, wl + i * WARPS, lane, acc);
        }
        __syncwarp();
        if (ok && lane == 0 && i + DEPTH < n_my) {
            fence_proxy_async();  // order this warp's reads of the slot before the refill
            const int cn = wl + (i + DEPTH) * WARPS;
            mbar_expect_tx(&my_bars[s], TILE);
            bulk_copy_g2s(my_slots + (size_t)s * Plan::SLOT, my_tiles + (size_t)cn * TILE, TILE, &my_bars[s]);
        }
    }

    // 4. partial sums of the warps meet in shared memory: red[warp][row]
    float* red = reinterpret_cast<float*>(smem + Plan::red_off(kc));
    const int g = lane >> 2;
    const int t = lane & 3;
    // lane t folded one block of every group of four
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        acc[0] += __shfl_xor_sync(0xFFFFFFFFu, acc[0], o);
        acc[1] += __shfl_xor_sync(0xFFFFFFFFu, acc[1], o);
    }
    if (t == 0) {
        red[warp * 16 + g] = acc[0];
        red[warp * 16 + g + 8] = acc[1];
    }
    __syncthreads();
    const float s_in = s_in_sh;

    if constexpr (EPI == EPI_STORE) {
        if (threadIdx.x < 16 * TILES) {
            float sum = 0.0f;
            const int w0 = ((int)threadIdx.x >> 4) * WARPS, r = threadIdx.x & 15;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                sum += red[(w0 + w) * 16 + r];
            }
            sum *= s_in;
            const int64_t row = (int64_t)blockIdx.x * (16 * TILES) + threadIdx.x;
            if (row < v.n) {
                y[row] = sum;
                if (ps.n_peers > 0) {
#pragma unroll
                    for (int p = 0; p < QMM_MAX_PEERS; ++p) {  // over NVLink into the peer's receive buffer
                        if (p < ps.n_peers) {
                            asm volatile("st.relaxed.sys.global.v2.u32 [%0], {%1, %2};" ::"l"(ps.dst[p] + row),
                                         "r"(__float_as_uint(sum)), "r"(epoch)
                                         : "memory");
                        }
                    }
                }
            }
        }
    } else if constexpr (EPI == EPI_RESID_PACK) {
        const int64_t blk = (int64_t)blockIdx.x * (TILES / 2) + warp;  // block of 32 output rows of this warp
        if (warp < TILES / 2 && blk * 32 < v.n) {  // lane = row of the block: the warps of its tile hold the partial sums
            float sum = 0.0f;
            const int w0 = (2 * warp + (lane >> 4)) * WARPS, r = lane & 15;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                sum += red[(w0 + w) * 16 + r];
            }
            sum *= s_in;
            const int64_t row = blk * 32 + lane;
            if (ps.n_peers > 0 && row < v.n) {
                // tensor parallelism: this rank's partial goes to every peer, the peers' partials are awaited
#pragma unroll
                for (int p = 0; p < QMM_MAX_PEERS; ++p) {
                    if (p < ps.n_peers) {
                        asm volatile("st.relaxed.sys.global.v2.u32 [%0], {%1, %2};" ::"l"(ps.dst[p] + row),
                                     "r"(__float_as_uint(sum)), "r"(epoch)
                                     : "memory");
                    }
                }
                bool waiting = *reinterpret_cast<volatile int*>(ps.wait_status) == 0;
                float total = 0.0f;
                for (int r = 0; r < ps.tp_size; ++r) {
                    if (r == ps.tp_rank) {
                        total += sum;
                        continue;
                    }
                    const uint2* src = ps.recv + (size_t)r * v.n + row;
                    uint2 pk;
                    asm volatile("ld.relaxed.sys.global.v2.u32 {%0, %1}, [%2];" : "=r"(pk.x), "=r"(pk.y) : "l"(src) : "memory");
                    unsigned int spin = 0;
                    while (waiting && pk.y != epoch) {
                        if (++spin > ps.spin_limit) {
                            waiting = false;
                            atomicExch(ps.wait_status, 5);  // a peer's addend never came; the sum is incomplete
                            break;
                        }
                        asm volatile("ld.relaxed.sys.global.v2.u32 {%0, %1}, [%2];"
                                     : "=r"(pk.x), "=r"(pk.y)
                                     : "l"(src)
                                     : "memory");
                    }
                    total += __uint_as_float(pk.x);
                }
                sum = total;
            }
            const float hv = h_pre + sum;
            if (row < v.n) {
                fu.h_out[row] = hv;
                if (y) {
                    y[row] = sum;
                }
            }
            double sq = (double)hv * (double)hv;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sq += __shfl_xor_sync(0xFFFFFFFFu, sq, o);
            }
            if (lane == 0) {
                fu.ss_out[blk] = sq;
            }
            warp_pack_block32(hv * w_pre, fu.packed_out + (size_t)(blk >> 3) * XPK1_REC, (int)(blk & 7));
        }
    } else if constexpr (EPI == EPI_SWIGLU_PACK) {
        const int64_t blk = (int64_t)blockIdx.x * (TILES / 4) + warp;  // block of 32 channels of this warp
        if (warp < TILES / 4 && blk * 64 < v.n) {
            // lane = channel of the block: row tile lane / 8, tile rows lane % 8 (gate) and + 8 (up)
            const int w0 = (4 * warp + (lane >> 3)) * WARPS, r = lane & 7;
            float gate = 0.0f, up = 0.0f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                gate += red[(w0 + w) * 16 + r];
                up += red[(w0 + w) * 16 + r + 8];
            }
            gate *= s_in;
            up *= s_in;
            const int64_t ch = blk * 32 + lane;
            const float act = 2 * ch < v.n ? (gate * (1.0f / (1.0f + expf(-gate)))) * up : 0.0f;
            if (y && 2 * ch < v.n) {
                y[ch] = act;
            }
            warp_pack_block32(act, fu.packed_out + (size_t)(blk >> 3) * XPK1_REC, (int)(blk & 7));
        }
    } else {
        if (threadIdx.x < 8) {
            float gate = 0.0f, up = 0.0f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                gate += red[w * 16 + threadIdx.x];
                up += red[w * 16 + threadIdx.x + 8];
            }
            gate *= s_in;
            up *= s_in;
            const int64_t ch = (int64_t)blockIdx.x * 8 + threadIdx.x;
            if (2 * ch < v.n) {
                // sigmoid = 1 / (1 + exp(-x)), SiLU = x * sigmoid(x) (src/LiteNN/Layer/Activation.h:20-33,52-59)
                y[ch] = (gate * (1.0f / (1.0f + expf(-gate)))) * up;
            }
        }
    }
}

// Ring depth per format: 28-37 KB of tiles in flight per CTA.
template <int FMT>
struct Tune {
    static constexpr int WARPS = 4;
    static constexpr int DEPTH = FMT == FMT_Q8_0 ? 2 : 3;
};

template <int FMT, int WARPS, int DEPTH, int EPI, bool XF32, int TILES = epi_tiles(EPI)>
cudaError_t launch_gemv_xsrc(const WeightView& w, const XPackView& xp, float* y, int* status,
                             const PeerScatter& ps, const GemvFuse& fu, cudaStream_t stream)
{
    using Plan = SmemPlan<FMT, WARPS, DEPTH, TILES>;
    auto kernel = gemv_kernel<FMT, WARPS, DEPTH, EPI, TILES, XF32>;
    int smem = Plan::total(w.kc);
    if (smem > 227 * 1024) {
        return cudaErrorInvalidConfiguration;
    }
    if (w.rt % epi_tiles(EPI) != 0) {
        return cudaErrorInvalidValue;
    }
    const int grid = (w.rt + TILES - 1) / TILES;
    // Residency cap.  The block scheduler fills an SM up to its limit before it is even with the others, so
    // a grid of 688 CTAs that could sit 7 to an SM leaves a third of the SMs with little to do (measured on
    // B200: 6.7 us at a limit of 7, 5.2 us at 5 for W[11008,4096]).  The dynamic shared memory request is
    // padded so that no SM can hold more than its even share, ceil(grid / SMs), of the CTAs.
    static std::mutex mu;
    static int configured[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    {
        std::lock_guard<std::mutex> lock(mu);
        const int sms = sm_count_of(dev);
        const int share = sms > 0 ? (grid + sms - 1) / sms : 0;
        if (share >= 1 && share <= 16) {
            const int want = 232448 / share - 1024 - 256;
            smem = want > smem ? want : smem;
        }
        // the opt-in limit is a per-device function attribute; raise it only when needed
        if (dev < 0 || dev >= 64 || configured[dev] < smem) {
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) {
                return e;
            }
            if (dev >= 0 && dev < 64) {
                configured[dev] = smem;
            }
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(WARPS * TILES * 32);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 1;
    cfg.attrs = attr;
    return cudaLaunchKernelEx(&cfg, kernel, w, xp, y, status, ps, fu);
}

// Launches the form that gemv_wave_form or gemv_small_glu_form chooses.
template <int FMT, int EPI, bool XF32>
struct GemvLaunch {
    const WeightView& w;
    const XPackView& xp;
    float* y;
    int* status;
    const PeerScatter& ps;
    const GemvFuse& fu;
    cudaStream_t stream;

    template <int TILES, int WARPS, int DEPTH>
    cudaError_t form() const
    {
        return launch_gemv_xsrc<FMT, WARPS, DEPTH, EPI, XF32, TILES>(w, xp, y, status, ps, fu, stream);
    }
};

template <int FMT, int WARPS, int DEPTH, int EPI>
cudaError_t launch_gemv_variant(const WeightView& w, const XPackView& xp, float* y, int* status,
                                const PeerScatter& ps, const GemvFuse& fu, cudaStream_t stream)
{
    if constexpr (EPI == EPI_RESID_PACK) {
        if (fu.x_f32 != nullptr) {
            return launch_gemv_xsrc<FMT, WARPS, DEPTH, EPI, true>(w, xp, y, status, ps, fu, stream);
        }
    }
    if (fu.x_f32 != nullptr) {
        return cudaErrorInvalidValue;
    }
    return launch_gemv_xsrc<FMT, WARPS, DEPTH, EPI, false>(w, xp, y, status, ps, fu, stream);
}

// Batch 1: warps x ring slots by row length.
//   K of 2304..4096: eight warps with one slot each (the whole row tile is requested by the first
//   instruction, 18 KB per CTA) measured faster than four warps with three slots for every format but
//   Q8_0, whose larger tiles would leave fewer CTAs per SM.  Inside a chain (ss_in: the input's norm factor
//   comes from the kernel before) 4-bit rows take four warps with two slots: half the warps' prologues and
//   reductions, 7B-shape token with eight blocks 309.7 -> 304.9 us; on its own that form gains nothing
//   (11008 x 4096, twelve weights in turn: 92 us and 92..99).  This rule and the residual form's below together, eight
//   blocks and 128 tokens, ms without and with them, Q4_0 / Q4_K: 2304 wide 25.4 -> 24.4 / 27.6 -> 26.6, 3072 wide
//   28.1 -> 27.0 / 30.8 -> 30.1, 4096 wide 35.2 -> 34.0 / 39.6 -> 38.6, with an FFN of 14336 39.0 -> 39.2 / 44.1 -> 43.3.
//   K > 4096: with four warps a warp would walk 6-28 tiles one after the other, and in a chain of
//   dependent matvecs that walk starts only when the activations arrive; more warps per row tile
//   shorten it, as long as two CTAs still fit on an SM.
template <int FMT, int EPI>
cudaError_t launch_gemv_m1(const WeightView& w, const XPackView& xp, float* y, int* status, const PeerScatter& ps,
                           const GemvFuse& fu, cudaStream_t stream)
{
    [[maybe_unused]] constexpr int LIMIT = 113 * 1024;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    const int sms = sm_count_of(dev);
    if (sms < 1) {
        return cudaErrorInvalidDevice;
    }
    if constexpr (EPI == EPI_STORE) {
        if (fu.x_f32 != nullptr) {  // gemv_packs_itself says which
            return gemv_wave_form<FMT, EPI, true>(w.rt, w.kc, sms, GemvLaunch<FMT, EPI, true>{w, xp, y, status, ps, fu, stream});
        }
    }
    if constexpr (EPI != EPI_SWIGLU) {
        // (a tensor-parallel rank keeps the residual form that waits for its peers in small CTAs)
        if (fu.x_f32 == nullptr && !(EPI == EPI_RESID_PACK && ps.n_peers > 0) &&
            gemv_one_wave<FMT, EPI>(w.rt, w.kc, fu.ss_in != nullptr, sms)) {
            return gemv_wave_form<FMT, EPI, false>(w.rt, w.kc, sms, GemvLaunch<FMT, EPI, false>{w, xp, y, status, ps, fu, stream});
        }
    }
    if constexpr (EPI == EPI_SWIGLU_PACK) {
        if (fu.x_f32 != nullptr) {
            return cudaErrorInvalidValue;
        }
        return gemv_small_glu_form<FMT>(w.rt, w.kc, sms, GemvLaunch<FMT, EPI, false>{w, xp, y, status, ps, fu, stream});
    } else if constexpr (EPI == EPI_RESID_PACK) {
        // The residual form has two row tiles per CTA and n / 32 CTAs: 128 for a 4096-wide model, 256 for an
        // 8192-wide one.  All of them should be resident at once (a second wave of a few CTAs doubles the
        // kernel's time), so the variant is the deepest one whose shared memory lets ceil(CTAs / SMs) CTAs
        // share an SM.  8 warps per tile with three slots each walk a long row with 110 KB in flight per CTA
        // (ffn_down of the 7B shape, K = 11008: 7.1 us against 8.1 us with 16 warps x 2 slots).
        const int ctas = w.rt / 2;
        const int per_sm = (ctas + sms - 1) / sms;
        const int budget = 232448 / per_sm - 1280;
        if (w.kc > 8 && w.kc <= 16) {
            // 4-bit rows of up to 16 chunks: four warps with four slots, every tile requested at once (7B-shape step with
            // eight blocks 304.9 -> 302.5 us against eight warps with one slot)
            if constexpr (tile_bytes(FMT) == 2304) {
                if (SmemPlan<FMT, 4, 4, 2>::total(w.kc) <= budget) {
                    return launch_gemv_variant<FMT, 4, 4, EPI>(w, xp, y, status, ps, fu, stream);
                }
            }
            if constexpr (FMT != FMT_Q8_0) {
                if (SmemPlan<FMT, 8, 1, 2>::total(w.kc) <= budget) {
                    return launch_gemv_variant<FMT, 8, 1, EPI>(w, xp, y, status, ps, fu, stream);
                }
            }
        }
        if (w.kc > 16 && SmemPlan<FMT, 8, 3, 2>::total(w.kc) <= budget) {
            return launch_gemv_variant<FMT, 8, 3, EPI>(w, xp, y, status, ps, fu, stream);
        }
        if (SmemPlan<FMT, 4, 3, 2>::total(w.kc) <= budget) {
            return launch_gemv_variant<FMT, 4, 3, EPI>(w, xp, y, status, ps, fu, stream);
        }
        if (SmemPlan<FMT, 4, 2, 2>::total(w.kc) <= budget) {
            return launch_gemv_variant<FMT, 4, 2, EPI>(w, xp, y, status, ps, fu, stream);
        }
        // more than one CTA per SM wanted and nothing deeper fits: one slot per warp, the number of CTAs keeps
        // the bytes in flight up
        return launch_gemv_variant<FMT, 4, 1, EPI>(w, xp, y, status, ps, fu, stream);
    } else {
        if (w.kc > 8 && w.kc <= 16) {
            if constexpr (tile_bytes(FMT) == 2304 && EPI == EPI_STORE) {
                if (fu.ss_in != nullptr) {
                    return launch_gemv_variant<FMT, 4, 2, EPI>(w, xp, y, status, ps, fu, stream);
                }
            }
            if constexpr (FMT != FMT_Q8_0) {
                return launch_gemv_variant<FMT, 8, 1, EPI>(w, xp, y, status, ps, fu, stream);
            }
        }
        if (w.kc > 32 && SmemPlan<FMT, 16, 2, 1>::total(w.kc) <= LIMIT) {
            return launch_gemv_variant<FMT, 16, 2, EPI>(w, xp, y, status, ps, fu, stream);
        }
        if (w.kc > 16 && SmemPlan<FMT, 8, 3, 1>::total(w.kc) <= LIMIT) {
            return launch_gemv_variant<FMT, 8, 3, EPI>(w, xp, y, status, ps, fu, stream);
        }
        return launch_gemv_variant<FMT, Tune<FMT>::WARPS, Tune<FMT>::DEPTH, EPI>(w, xp, y, status, ps, fu, stream);
    }
}

template <int FMT>
cudaError_t launch_gemv_fmt(const WeightView& w, const XPackView& xp, float* y, int m, int* status,
                            const PeerScatter& ps, const GemvFuse& fu, cudaStream_t stream)
{
    if (m == 1) {
        switch (fu.mode) {
        case EPI_STORE: return launch_gemv_m1<FMT, EPI_STORE>(w, xp, y, status, ps, fu, stream);
        case EPI_RESID_PACK: return launch_gemv_m1<FMT, EPI_RESID_PACK>(w, xp, y, status, ps, fu, stream);
        case EPI_SWIGLU: return launch_gemv_m1<FMT, EPI_SWIGLU>(w, xp, y, status, ps, fu, stream);
        case EPI_SWIGLU_PACK: return launch_gemv_m1<FMT, EPI_SWIGLU_PACK>(w, xp, y, status, ps, fu, stream);
        default: return cudaErrorInvalidValue;
        }
    }
    if (fu.mode != EPI_STORE || fu.ss_in != nullptr || fu.x_f32 != nullptr || ps.n_peers > 0) {
        return cudaErrorInvalidValue;
    }
    if (m <= 4) {
        return launch_gemv_batch<FMT, 1>(w, xp, y, m, status, stream);
    }
    if (m <= 8) {
        return launch_gemv_batch<FMT, 2>(w, xp, y, m, status, stream);
    }
    if (m <= 12) {
        return launch_gemv_batch<FMT, 3>(w, xp, y, m, status, stream);
    }
    return launch_gemv_batch<FMT, 4>(w, xp, y, m, status, stream);
}

}  // namespace

}  // namespace qmm
