// Dequant-fused GEMV for decode (one activation row) on sm_100a: the kernel template, and the per-format launcher of a
// matvec of any row count.  Each block format instantiates it in a translation
// unit of its own (qmm_gemv_q4_0.cu, ...), so the formats compile in parallel.  2..16 rows are qmm_gemv_batch.cuh.
//
// The weights never become floats in memory.  One CTA owns one 16-row tile of the
// output; its warps take the 256-column K chunks of that row tile round-robin.
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

#include <atomic>
#include <mutex>

#include "qmm_gemv_batch.cuh"
#include "qmm_gemv_device.cuh"
#include "qmm_kernels.h"
#include "qmm_pack.cuh"

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
    __host__ __device__ static int red_off(int kc) { return X_OFF + (int)xpack1_bytes(kc) + 512; }
    __host__ __device__ static int total(int kc) { return red_off(kc) + NW * 16 * 4; }
};

// WARPS warps share one row tile; a CTA holds TILES row tiles (2 for EPI_RESID_PACK: the 32 rows of
// one quantization block of the output, so the epilogue can quantize them without leaving the CTA).
// Registers decide how many CTAs an SM holds, and a batch-1 grid of 768 row tiles wants six CTAs of
// 256 threads on every SM at once (42 registers at most): the bound keeps the fp32-packing prologue
// and the fused epilogues from costing a second wave.  Plain CTAs of 128 threads are held to 64 registers, eight to an SM:
// one row of Q6_K 11008 x 2048 takes 7.29 us, 7.70 with six to an SM; Q4_0 and Q8_0 differ by 1 % at most, either way.
template <int THREADS, int EPI, int TILES, bool XF32>
constexpr int gemv_min_blocks()
{
    return TILES > epi_tiles(EPI) || (XF32 && EPI == EPI_STORE) || EPI == EPI_RESID_PACK ? 1 : EPI == EPI_SWIGLU_PACK ? (THREADS <= 256 ? 3 : 1) : (THREADS <= 128 ? 8 : THREADS <= 256 ? 6 : 3);
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

// SMs of a device, 0 if it cannot be asked; asked once.
inline int sm_count_of(int dev)
{
    static std::atomic<int> known[64];
    if (dev >= 0 && dev < 64) {
        if (const int n = known[dev].load(std::memory_order_relaxed)) {
            return n;
        }
    }
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        return 0;
    }
    if (dev >= 0 && dev < 64) {
        known[dev].store(n, std::memory_order_relaxed);
    }
    return n;
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

// The one-wave form: a CTA on every SM, each with as many row tiles as that takes (ceil(tiles / SMs), up to the next
// compiled count), WARPS warps and WARPS x DEPTH slots per tile.  What bounds a matvec of many small CTAs is the last
// of its waves and, for an fp32 vector, that every CTA packs the vector again; here there is one wave and at most 148
// copies.  Measured on B200, a stream of different weights, us each, many CTAs -> one wave:
//   packed vector  Q4_0 8192 x 28672 28.9 -> 22.4, 10240 x 8192 12.4 -> 9.4, 28672 x 8192 27.4 -> 22.7, 4096 x 4096 3.8 -> 3.5;
//                  Q4_K 28672 x 8192 29.9 -> 22.6, 11008 x 4096 7.4 -> 6.7; Q6_K 28672 x 8192 35.4 -> 31.5, 14336 x 4096
//                  11.1 -> 9.7; Q8_0 11008 x 4096 11.0 -> 9.5
//   fp32 vector    (before: a kernel that packs it, then the matvec) Q4_0 1024 x 4096 4.2 -> 3.0, 14336 x 4096 9.5 -> 8.1,
//                  28672 x 8192 28.2 -> 23.9; Q4_K 14336 x 4096 10.6 -> 9.0; Q6_K 4096 x 2048 4.2 -> 3.4; Q8_0 4096 x 4096 6.0 -> 5.4
// More warps per tile shorten a short row's chain of tiles; more than about 90 KB of slots gains nothing, so the warps per
// tile fall as the tiles grow.  The shared-memory request keeps a second CTA of the same kernel off an SM: without
// it, 4096 x 8192 of Q4_K takes 7.2 us and not 5.6.  LESS: warps and depth to fall back to where long rows leave less room
// for slots; with at most GEMV_WAVE_KC chunks the last entry always fits.
template <int FMT, int EPI, bool XF32>
struct GemvWave {
    const WeightView& w;
    const XPackView& xp;
    float* y;
    int* status;
    const PeerScatter& ps;
    const GemvFuse& fu;
    cudaStream_t stream;
    static constexpr bool NIBBLE = tile_bytes(FMT) == 2304;

    template <int TILES, int WARPS, int DEPTH, int... LESS>
    cudaError_t go() const
    {
        if constexpr (TILES % epi_tiles(EPI) != 0) {
            return cudaErrorInvalidConfiguration;  // not reached: the caller rounds up to whole groups
        } else if constexpr (sizeof...(LESS) > 0) {
            if (SmemPlan<FMT, WARPS, DEPTH, TILES>::total(w.kc) > 227 * 1024) {
                return go<TILES, LESS...>();
            }
            return launch_gemv_xsrc<FMT, WARPS, DEPTH, EPI, XF32, TILES>(w, xp, y, status, ps, fu, stream);
        } else {
            return launch_gemv_xsrc<FMT, WARPS, DEPTH, EPI, XF32, TILES>(w, xp, y, status, ps, fu, stream);
        }
    }

    cudaError_t launch(int sms) const
    {
        const int tiles = gemv_wave_tiles(w.rt, epi_tiles(EPI), sms);
        if constexpr (EPI == EPI_SWIGLU_PACK) {
            if (tiles > 12) {
                return launch_many(tiles);
            }
            return go<12, 2, 2, 2, 1>();  // nine tiles at least
        } else {
            return launch_few(tiles);
        }
    }

    cudaError_t launch_few(int tiles) const
    {
        const bool small = w.kc <= 8;  // two tiles per warp at most, whatever the form: fewer warps to add up
        if constexpr (EPI == EPI_STORE) {
            if (tiles <= 1) {
                return w.kc <= 4 ? go<1, 8, 1>() : go<1, 16, 2>();
            }
            if (tiles == 2) {
                return go<2, 8, 2>();
            }
            if (tiles == 3) {
                return small && w.kc > 4 ? go<3, 8, 1>() : go<3, 5, 2>();
            }
        }
        if (tiles == 4) {
            return go<4, 4, 3, 4, 2>();
        }
        if (tiles == 5) {
            return go<5, 4, 2, 4, 1>();
        }
        if (tiles == 6) {
            return small ? go<6, 2, 2>() : go<6, 4, 2, 2, 2>();
        }
        if (tiles == 7) {
            if constexpr (NIBBLE) {
                return small ? go<7, 2, 2>() : go<7, 4, 2>();
            } else {
                return small ? go<7, 2, 2>() : go<7, 2, 3, 2, 2>();
            }
        }
        if (tiles == 8) {
            return small ? go<8, 2, 2>() : go<8, 2, 3, 2, 2>();
        }
        if (tiles <= 10) {
            return go<10, 2, 2, 2, 1>();
        }
        if (tiles <= 12) {
            return go<12, 2, 2, 2, 1>();
        }
        return launch_many(tiles);
    }

    cudaError_t launch_many(int tiles) const
    {
        // Q6_K and Q8_0 leave room for two warps per row tile only with one slot each: one warp with three is 4 % faster.
        // So it is inside a chain for every format, as 32 warps of 64 registers leave the next kernel none (28672 x 7168
        // and three blocks, Q4_0: 227 us a token with two warps, 200 with one).
        if (tiles <= 16) {
            if constexpr (NIBBLE && EPI == EPI_STORE) {
                return tiles <= 14 ? go<14, 2, 2>() : go<16, 2, 2>();
            } else {
                return tiles <= 14 ? go<14, 1, 3, 1, 2>() : go<16, 1, 3, 1, 2>();
            }
        }
        if constexpr (EPI == EPI_SWIGLU_PACK) {
            return tiles <= 20   ? go<20, 1, 2, 1, 1>()
                   : tiles <= 24 ? go<24, 1, 2, 1, 1>()
                   : tiles <= 28 ? go<28, 1, 2, 1, 1>()
                                 : cudaErrorInvalidConfiguration;
        }
        if constexpr (EPI == EPI_STORE && NIBBLE) {
            return tiles <= 20   ? go<20, 1, 2>()
                   : tiles <= 25 ? go<25, 1, 2>()
                   : tiles <= 28 ? go<28, 1, 2>()
                                 : cudaErrorInvalidConfiguration;
        }
        return cudaErrorInvalidConfiguration;
    }
};

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
bool gemv_one_wave(const WeightView& w, bool chained, int sms)
{
    constexpr bool NIBBLE = tile_bytes(FMT) == 2304;
    const int tiles = gemv_wave_tiles(w.rt, epi_tiles(EPI), sms), kc = w.kc;
    if (kc > GEMV_WAVE_KC || tiles > (EPI == EPI_SWIGLU_PACK || (EPI == EPI_STORE && NIBBLE) ? 28 : 16)) {
        return false;
    }
    if constexpr (EPI == EPI_SWIGLU_PACK) {
        if (tiles <= 12) {
            return w.rt > 8 * sms && kc > 9 && (FMT == FMT_Q8_0 || (FMT == FMT_Q4_K && w.rt <= 11 * sms));
        }
        if (tiles <= 16) {
            return !NIBBLE || kc > (FMT == FMT_Q4_0 ? 10 : 8);
        }
        return FMT != FMT_Q6_K || tiles <= 24 || kc <= 12;
    } else if constexpr (EPI == EPI_RESID_PACK) {
        if (w.rt <= 2 * sms || !gemv_wave_fills(w.rt, epi_tiles(EPI), sms)) {
            return false;
        }
        if (tiles <= 4) {
            return kc >= 96 || (FMT == FMT_Q6_K && kc > 8 && kc <= 16) ||
                   (NIBBLE && kc > 12 && kc <= 16 && 10LL * w.rt >= 9LL * sms * tiles);
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
                                     : tiles >= 4 || (tiles == 3 && (kc > 30 || 2 * w.rt > 5 * sms));
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
    constexpr int TILES = epi_tiles(EPI);
    constexpr int LIMIT = 113 * 1024;
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
            return GemvWave<FMT, EPI, true>{w, xp, y, status, ps, fu, stream}.launch(sms);
        }
    }
    if constexpr (EPI != EPI_SWIGLU) {
        // (a tensor-parallel rank keeps the residual form that waits for its peers in small CTAs)
        if (fu.x_f32 == nullptr && !(EPI == EPI_RESID_PACK && ps.n_peers > 0) &&
            gemv_one_wave<FMT, EPI>(w, fu.ss_in != nullptr, sms)) {
            return GemvWave<FMT, EPI, false>{w, xp, y, status, ps, fu, stream}.launch(sms);
        }
    }
    if constexpr (EPI == EPI_SWIGLU_PACK) {
        // four row tiles per CTA, two warps per tile with two slots each: 8 warps walk kc / 2 tiles apiece
        // (8 for K = 4096) and a third of a 1376-tile gate|up weight's CTAs fit an SM together (three slots: 1 % of a
        // 7B-shape step slower).  Where a long row's CTAs have an SM each, four warps per tile: two keep too few bytes in
        // flight (8192 wide, eight blocks, FFN 2304 Q4_0 200 -> 182 us a token, 3584 Q4_K 227 -> 209)
        if (fu.x_f32 != nullptr) {
            return cudaErrorInvalidValue;
        }
        const GemvWave<FMT, EPI, false> form{w, xp, y, status, ps, fu, stream};
        // (one warp per tile where the activations of rows beyond 60000 columns leave no room for more slots)
        return w.kc > 16 && w.rt <= TILES * sms ? form.template go<TILES, 4, 2, 2, 2, 1, 2>()
                                                : form.template go<TILES, 2, 2, 1, 2>();
    }
    if constexpr (TILES == 2) {
        // The residual form has two row tiles per CTA and n / 32 CTAs: 128 for a 4096-wide model, 256 for an
        // 8192-wide one.  All of them should be resident at once (a second wave of a few CTAs doubles the
        // kernel's time), so the variant is the deepest one whose shared memory lets ceil(CTAs / SMs) CTAs
        // share an SM.  8 warps per tile with three slots each walk a long row with 110 KB in flight per CTA
        // (ffn_down of the 7B shape, K = 11008: 7.1 us against 8.1 us with 16 warps x 2 slots).
        const int ctas = w.rt / 2;
        const int per_sm = (ctas + sms - 1) / sms;
        const int budget = 232448 / per_sm - 1280;
        // 4-bit rows of up to 16 chunks: four warps with four slots, every tile requested at once (7B-shape step with eight
        // blocks 304.9 -> 302.5 us against eight warps with one slot)
        if (tile_bytes(FMT) == 2304 && w.kc > 8 && w.kc <= 16 && SmemPlan<FMT, 4, 4, 2>::total(w.kc) <= budget) {
            return launch_gemv_variant<FMT, 4, 4, EPI>(w, xp, y, status, ps, fu, stream);
        }
        if (w.kc > 8 && w.kc <= 16 && FMT != FMT_Q8_0 && SmemPlan<FMT, 8, 1, 2>::total(w.kc) <= budget) {
            return launch_gemv_variant<FMT, 8, 1, EPI>(w, xp, y, status, ps, fu, stream);
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
    }
    if (tile_bytes(FMT) == 2304 && EPI == EPI_STORE && fu.ss_in != nullptr && w.kc > 8 && w.kc <= 16) {
        return launch_gemv_variant<FMT, 4, 2, EPI>(w, xp, y, status, ps, fu, stream);
    }
    if (w.kc > 8 && w.kc <= 16 && FMT != FMT_Q8_0) {
        return launch_gemv_variant<FMT, 8, 1, EPI>(w, xp, y, status, ps, fu, stream);
    }
    if (w.kc > 32 && SmemPlan<FMT, 16, 2, 1>::total(w.kc) <= LIMIT) {
        return launch_gemv_variant<FMT, 16, 2, EPI>(w, xp, y, status, ps, fu, stream);
    }
    if (w.kc > 16 && SmemPlan<FMT, 8, 3, TILES>::total(w.kc) <= LIMIT) {
        return launch_gemv_variant<FMT, 8, 3, EPI>(w, xp, y, status, ps, fu, stream);
    }
    return launch_gemv_variant<FMT, Tune<FMT>::WARPS, Tune<FMT>::DEPTH, EPI>(w, xp, y, status, ps, fu, stream);
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
