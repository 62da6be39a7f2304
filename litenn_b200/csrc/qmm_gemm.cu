// Prefill GEMM on the 5th-generation tensor cores (sm_100a): Y[M,N] = X[M,K] . W^T with bf16
// activations, block-quantized weights dequantized on the fly, fp32 accumulation in TMEM.
//
// The weights are the A operand and live in TMEM, the activation rows ("tokens") are the B operand
// in shared memory, so D has one weight row per TMEM lane and one token per column.  A CTA owns NB
// blocks of 128 weight rows, up to 128 tokens and a range of K.  Per 64-wide K step:
//   dequant warps   read packed tiles (qmm_common.cuh) from global memory, rebuild the exact fp32
//                   values ggml's to_float gives, round them to bf16 and store them with
//                   tcgen05.st.16x256b, whose register layout (lane 4g+t: row g and g+8, columns 2t, 2t+1)
//                   is the packed tiles' own: no shuffle, no shared memory
//   TMA warp        one 64 x tokens bf16 box of X -> shared memory (128-byte swizzle)
//   MMA warp        tcgen05.mma (kind::f16, bf16 x bf16 -> fp32, M = 128, N = tokens, K = 16), A from TMEM
// Weights never pass through shared memory, whose bandwidth (128 bytes per cycle and SM) a B operand of
// dequantized weights shares with the operand reads and the TMA writes.
// Bound: the dequant warps' instruction issue (ncu, Q4_0 22016 x 4096, 512 tokens: 65 % of the issue slots, ALU pipe 58 %,
// tensor pipe 36 %).  Q6_K 4096 x 11264, 64 tokens: 27 us here against 125 us of the shared-memory form, whose 16 dequant
// warps have two row tiles to work on; Q4_0 4096 x 4096, 512 tokens: 34.7 against 51.6.  The MMAs are issued under elect.sync: with a lane comparison in its place the same kernel took a fifth longer
// (Q4_0 4096 x 11008, 512 tokens: 94 us and 77 us).
// Every wait has an iteration limit; a CTA that gives up sets the status word, still frees its TMEM and
// returns.
#include <cuda.h>

#include <algorithm>

#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "qmm_gemm_dequant.cuh"
#include "qmm_gemm_smem.h"
#include "qmm_kernels.h"

namespace qmm {

namespace {

constexpr int GEMM_MAX_TOKENS = 128;     // B columns of one CTA
constexpr int GEMM_A_STAGES = 4;         // K steps of dequantized weights in TMEM, 32 columns per block each
constexpr int GEMM_MAX_RING = 8;         // K steps of tokens in shared memory
constexpr int GEMM_BAR_BYTES = 1024;     // barriers, in front of the ring

// D[tmem] (+)= A[tmem, 128 x 16 bf16] * B[smem descriptor, 16 x N]
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 16 rows x 32 columns (64 bf16 of K): registers 4p..4p+3 are K slice p, {row g: k 4t..4t+1, 4t+2..4t+3; row g+8: the
// same}, in lane 4g+t.
__device__ __forceinline__ void tmem_st_16x256b_x4(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// ---- the kernel -----------------------------------------------------------------------------

struct GemmArgs {
    WeightView w;
    void* y;        // [M, N] row-major, fp32 or bf16; [M, N / 2] bf16 for GEMM_OUT_SWIGLU
    int64_t m;
    int out;        // GEMM_OUT_*
    int tokens;     // B columns per CTA, a multiple of 16
    int t_tiles;    // token tiles
    int ring;       // K steps of tokens in shared memory
    int* status;
};

__device__ __forceinline__ void store_y(const GemmArgs& a, int64_t token, int64_t row, float v)
{
    if (a.out == GEMM_OUT_BF16) {
        static_cast<__nv_bfloat16*>(a.y)[token * a.w.n + row] = __float2bfloat16_rn(v);
    } else {
        static_cast<float*>(a.y)[token * a.w.n + row] = v;
    }
}

// grid = blocks x t_tiles x splits; a cluster of `splits` CTAs shares one output tile and cuts K between them.
template <int FMT, int NB>
__global__ void __launch_bounds__((8 * NB + 2) * 32, 3 - NB)
    gemm_ts_kernel(const __grid_constant__ CUtensorMap xmap, const GemmArgs args)
{
    namespace cg = cooperative_groups;
    constexpr int DW = 8 * NB;               // dequant warps: one row tile each
    constexpr uint32_t TMEM_COLS = 256 * NB;
    constexpr uint32_t D_COL = GEMM_A_STAGES * 32 * NB;  // accumulators behind the A stages
    extern __shared__ uint8_t gemm_smem_raw[];
    // the swizzle pattern is defined on absolute shared-memory addresses: 1024-byte alignment
    uint8_t* smem = gemm_smem_raw + ((1024u - (g_smem_u32(gemm_smem_raw) & 1023u)) & 1023u);
    uint64_t* full_b = reinterpret_cast<uint64_t*>(smem);  // [MAX_RING]  TMA bytes landed
    uint64_t* empty_b = full_b + GEMM_MAX_RING;            // [MAX_RING]  MMAs that read the slot have completed
    uint64_t* full_a = empty_b + GEMM_MAX_RING;            // [A_STAGES]  dequant warps done
    uint64_t* empty_a = full_a + GEMM_A_STAGES;            // [A_STAGES]  MMAs that read the stage have completed
    uint64_t* accum = empty_a + GEMM_A_STAGES;             // all MMAs completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
    uint8_t* ring = smem + GEMM_BAR_BYTES;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const WeightView& v = args.w;
    cg::cluster_group cluster = cg::this_cluster();
    const int splits = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int tile = blockIdx.x / splits;
    const int block = tile / args.t_tiles;
    const int64_t token0 = (int64_t)(tile % args.t_tiles) * args.tokens;
    const int n = args.tokens;
    const int slot_bytes = n * 128;
    // this CTA's K: whole 256-wide chunks c0..c1, in steps of 64 up to the last one that holds data
    const int c0 = (int)((long long)v.kc * rank / splits), c1 = (int)((long long)v.kc * (rank + 1) / splits);
    const int k_steps = (int)((v.k + GEMM_BK - 1) / GEMM_BK);
    const int s0 = 4 * c0, n_steps = min(4 * c1, k_steps) - s0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < GEMM_MAX_RING; ++s) {
            g_mbar_init(&full_b[s], 1);
            g_mbar_init(&empty_b[s], 1);
        }
        for (int s = 0; s < GEMM_A_STAGES; ++s) {
            g_mbar_init(&full_a[s], DW);
            g_mbar_init(&empty_a[s], 1);
        }
        g_mbar_init(accum, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == DW + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(g_smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == DW) {
        // ---- TMA producer: tokens.  Only they come from an earlier kernel; the first weights are dequantized while it drains,
        // and what is stored in the end depends on the tokens.  Every warp waits for that kernel before its first bounded wait,
        // whose limit is for this kernel's own steps ----
        if (lane == 0) {
            g_pdl_wait();
            int slot = 0;
            uint32_t phase = 1;
            for (int s = 0; s < n_steps; ++s) {
                if (s >= args.ring && !g_mbar_wait(&empty_b[slot], phase)) {
                    atomicExch(args.status, 11);
                    break;
                }
                g_mbar_expect_tx(&full_b[slot], (uint32_t)slot_bytes);
                tma_load_2d(ring + slot * slot_bytes, &xmap, (s0 + s) * GEMM_BK, (int)token0, &full_b[slot]);
                if (++slot == args.ring) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
        }
    } else if (warp == DW + 1) {
        // ---- MMA issuer: the whole warp walks the steps, one lane issues ----
        const uint32_t idesc = umma_idesc_bf16(n);
        const uint64_t desc0 = umma_smem_desc(g_smem_u32(ring));
        int slot = 0;
        uint32_t phase = 0;
        bool ok = true;
        g_pdl_wait();
        for (int s = 0; s < n_steps; ++s) {
            const int as = s % GEMM_A_STAGES;
            ok = g_mbar_wait(&full_b[slot], phase) && g_mbar_wait(&full_a[as], (uint32_t)(s / GEMM_A_STAGES) & 1u);
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok) {
                if (lane == 0) {
                    atomicExch(args.status, 12);
                }
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const uint64_t db = desc0 + (uint64_t)(slot * slot_bytes >> 4);
                const uint32_t a0 = tmem_base + (uint32_t)(as * 32 * NB);
#pragma unroll
                for (int kk = 0; kk < GEMM_BK / 16; ++kk) {
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        umma_bf16_ts(tmem_base + D_COL + (uint32_t)(b * GEMM_MAX_TOKENS), a0 + (uint32_t)(32 * b + 8 * kk),
                                     db + (uint64_t)(2 * kk), idesc, (s > 0 || kk > 0) ? 1u : 0u);
                    }
                }
                umma_commit(&empty_a[as]);  // both arrive when the MMAs above have read their operands
                umma_commit(&empty_b[slot]);
            }
            __syncwarp();
            if (++slot == args.ring) {
                slot = 0;
                phase ^= 1u;
            }
        }
        if (ok && elect_one()) {
            umma_commit(accum);
        }
        // The next kernel may start while this one stores its results.  Not earlier: its CTAs would take the places that this
        // kernel's grid leaves free, two to an SM, and leave others without (128 tokens, eight 7B-shape blocks: 1488 us without
        // overlap, 1591 with the start of this kernel as the trigger)
        g_pdl_launch_dependents();
        __syncwarp();
    } else {
        // ---- dequant producers: weights -> TMEM ----
        // a warp reaches the 32 TMEM lanes of its quadrant (warp % 4): two row tiles of a block
        const int quad = warp & 3;
        const int sub = (warp >> 2) & 1;
        const int wb = warp >> 3;
        const int rt = (block * NB + wb) * 8 + 2 * quad + sub;
        const bool has = rt < v.rt;  // rows beyond the weight: their lanes are never stored to Y
        const uint32_t a_addr = tmem_base + ((uint32_t)(32 * quad + 16 * sub) << 16) + (uint32_t)(32 * wb);
        const size_t tile_stride = tile_bytes(FMT);
        const uint8_t* wt = v.tiles + ((size_t)(has ? rt : 0) * v.kc + c0) * tile_stride;
        Packed<FMT> P;
        Scales<FMT> S, SN;
        if (c0 < c1) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                load_quarter<FMT>(P, wt, q, lane);
            }
            load_scales<FMT>(S, wt, lane >> 2);
        }
        SN = S;
        bool ok = true;
        int s = 0;
        static_assert(GEMM_A_STAGES == 4, "a chunk's four K steps fill the stages");
        for (int c = c0; c < c1 && ok; ++c) {
            const bool more = c + 1 < c1;
            const uint8_t* next = wt + tile_stride;
            if (more) {
                load_scales<FMT>(SN, next, lane >> 2);
            }
            if (c + 3 < c1 && lane * 128 < (int)tile_stride) {  // three chunks ahead into L2
                asm volatile("prefetch.global.L2 [%0];" ::"l"(wt + 3 * tile_stride + lane * 128));
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (s < n_steps && ok) {
                    uint32_t r[16];
                    dequant_quarter<FMT>(P, S, q, r);
                    if (more) {  // the registers just read are free: refill them from the next tile
                        load_quarter<FMT>(P, next, q, lane);
                    }
                    const int as = s % GEMM_A_STAGES;
                    if (q == 0 && c == c0 + 1) {  // s == GEMM_A_STAGES: stages are reused from here on
                        g_pdl_wait_only();
                    }
                    if (s >= GEMM_A_STAGES && !g_mbar_wait_warp(&empty_a[as], (uint32_t)(s / GEMM_A_STAGES - 1) & 1u)) {
                        if (lane == 0) {
                            atomicExch(args.status, 13);
                        }
                        ok = false;
                    }
                    if (ok) {
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (has) {
                            tmem_st_16x256b_x4(a_addr + (uint32_t)(as * 32 * NB), r);
                        }
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            g_mbar_arrive(&full_a[as]);
                        }
                    }
                    ++s;
                }
            }
            S = SN;
            wt = next;
        }

        // ---- epilogue: D has one weight row per lane, one token per column ----
        g_pdl_wait();
        if (!g_mbar_wait_warp(accum, 0)) {
            if (lane == 0) {
                atomicExch(args.status, 14);
            }
        } else {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int units = NB * (n / 16);
            for (int u = warp >> 2; u < units; u += 2 * NB) {
                const int b = u / (n / 16), col0 = (u % (n / 16)) * 16;
                uint32_t acc[16];
                __syncwarp();
                tmem_ld_32x32b_x16(tmem_base + ((uint32_t)(32 * quad) << 16) + D_COL + (uint32_t)(b * GEMM_MAX_TOKENS + col0),
                                   acc);
                const int row_in = 32 * quad + lane;
                if (NB == 1 && splits > 1) {  // partial sums [token][128 rows] in the ring, whose last reader is done
                    float* part = reinterpret_cast<float*>(ring);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        part[(col0 + i) * 128 + row_in] = __uint_as_float(acc[i]);
                    }
                } else if (args.out == GEMM_OUT_SWIGLU) {
                    // lanes 8..15 of a row tile hold up for the gates of lanes 0..7: the two swap every other token
                    const int64_t row = (int64_t)(block * NB + b) * 128 + row_in;
                    const bool up_lane = (lane & 8) != 0;
                    const int64_t ch = (row >> 4) * 8 + (row & 7);
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        const float mine = __uint_as_float(up_lane ? acc[i + 1] : acc[i]);
                        const float other = __shfl_xor_sync(0xFFFFFFFFu, __uint_as_float(up_lane ? acc[i] : acc[i + 1]), 8);
                        const int64_t token = token0 + col0 + i + (up_lane ? 1 : 0);
                        if (token < args.m && row < v.n) {
                            static_cast<__nv_bfloat16*>(args.y)[token * (v.n >> 1) + ch] =
                                __float2bfloat16_rn(up_lane ? silu_mul(other, mine) : silu_mul(mine, other));
                        }
                    }
                } else {
                    const int64_t row = (int64_t)(block * NB + b) * 128 + row_in;
                    if (row < v.n) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const int64_t token = token0 + col0 + i;
                            if (token < args.m) {
                                store_y(args, token, row, __uint_as_float(acc[i]));
                            }
                        }
                    }
                }
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == DW + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
    if constexpr (NB == 1) {
        if (splits > 1) {
            // The TMEM is free before the CTAs wait for one another.  Each sums its share of the tokens over the
            // ranks' partials, always in rank order.
            cluster.sync();
            const int per = n / splits;  // n is a multiple of 16, splits 2, 4 or 8
            const float* own = reinterpret_cast<const float*>(ring);
            auto total = [&](int col, int row_in) {
                float sum = 0.0f;
                for (int r = 0; r < splits; ++r) {
                    sum += cluster.map_shared_rank(own, r)[col * 128 + row_in];
                }
                return sum;
            };
            if (args.out == GEMM_OUT_SWIGLU) {
                for (int i = threadIdx.x; i < per * 64; i += (DW + 2) * 32) {
                    const int col = rank * per + (i >> 6), ch = i & 63, row_in = (ch >> 3) * 16 + (ch & 7);
                    const int64_t token = token0 + col, row = (int64_t)block * 128 + row_in;
                    if (token < args.m && row < v.n) {
                        static_cast<__nv_bfloat16*>(args.y)[token * (v.n >> 1) + (int64_t)block * 64 + ch] =
                            __float2bfloat16_rn(silu_mul(total(col, row_in), total(col, row_in + 8)));
                    }
                }
            } else {
                for (int i = threadIdx.x; i < per * 128; i += (DW + 2) * 32) {
                    const int col = rank * per + (i >> 7), row_in = i & 127;
                    const int64_t token = token0 + col, row = (int64_t)block * 128 + row_in;
                    if (token < args.m && row < v.n) {
                        store_y(args, token, row, total(col, row_in));
                    }
                }
            }
            cluster.sync();  // a peer may still read this CTA's partials
        }
    }
}


// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(p);
        }
    }
    return fn;
}

template <int FMT, int NB>
cudaError_t launch_gemm_nb(const CUtensorMap& xmap, const GemmArgs& args, const GemmPlan& plan, cudaStream_t stream)
{
    auto kernel = gemm_ts_kernel<FMT, NB>;
    static bool configured[64] = {};
    constexpr int LIMIT = 204 * 1024;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LIMIT);
        if (e != cudaSuccess) {
            return e;
        }
        if (dev >= 0 && dev < 64) {
            configured[dev] = true;
        }
    }
    if (plan.smem > LIMIT) {
        return cudaErrorInvalidConfiguration;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)plan.grid);
    cfg.blockDim = dim3((8 * NB + 2) * 32);
    cfg.dynamicSmemBytes = (size_t)plan.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)plan.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, xmap, args);
}

template <int FMT>
cudaError_t launch_gemm_fmt(const CUtensorMap& xmap, const GemmArgs& args, const GemmPlan& plan, cudaStream_t stream)
{
    return plan.nb == 2 ? launch_gemm_nb<FMT, 2>(xmap, args, plan, stream)
                        : launch_gemm_nb<FMT, 1>(xmap, args, plan, stream);
}

}  // namespace

GemmPlan gemm_form(const WeightView& w, int64_t m, int sm_count, int nb, int tokens, int splits)
{
    GemmPlan p = {};
    if (nb == 0) {
        p.groups = gemm_smem_groups(w.rt, m, sm_count);
        p.grid = (int)((m + 255) / 256) * p.groups;
        return p;
    }
    p.nb = nb;
    p.tokens = tokens;
    p.t_tiles = (int)((m + tokens - 1) / tokens);
    p.splits = splits;
    p.grid = (w.rt + 8 * nb - 1) / (8 * nb) * p.t_tiles * splits;
    const int room = nb == 2 ? 200 * 1024 : 110 * 1024;
    p.ring = std::min(GEMM_MAX_RING, room / (tokens * 128));
    const int part_bytes = splits > 1 ? tokens * 128 * 4 : 0;
    p.smem = 1024 /*alignment*/ + GEMM_BAR_BYTES + std::max(p.ring * tokens * 128, part_bytes);
    // One CTA per SM, also where the kernel before still holds some SMs.  Clusters of four and eight leave SMs of a GPC
    // over: 15 clusters of eight fit a B200 this way (Q4_0, K = 4096, 48 rows: 9.0 us for 120 CTAs, 15.2 for 128 and 9.5 for
    // 136 at two to an SM), so beyond 13/16 of the SMs they may share.
    if (nb == 1 && p.grid <= (splits >= 4 ? sm_count * 13 / 16 : sm_count)) {
        p.smem = std::max(p.smem, 116 * 1024);
    }
    return p;
}

// Three shapes of CTA, and the one with the least estimated time wins.
//   NB = 2    one CTA per SM, each token tile read once for 256 weight rows
//   NB = 1    two CTAs per SM; cuts finer and can split K over a cluster: few tokens or few weight rows
//   shared memory (qmm_gemm_smem.cu)   one dequantization per 256 tokens instead of 128: many tokens, where the
//             dequantization is what the other two spend their time on
// The estimates are microseconds on a B200: waves of CTAs x steps of 64 columns x time per step, plus a start-up per
// wave, fitted to 100 (weight, token count) pairs from 512 x 1024 to 8192 x 28672 and 17 to 1999 tokens, over which the
// choice costs 2 % against the best of all shapes.  Some of them (us): Q4_0 4096 x 4096, 64 tokens: NB = 1 with K split
// in four 14.7, shared memory 43.3; 1024 tokens: NB = 2 45.2, shared memory 57.4; 1999 tokens: NB = 2 85.6, shared
// memory 71.8.  Q6_K 8192 x 28672, 128 tokens: NB = 1 90.8, shared memory 327; 1024 tokens: 588 and 444.
//
// keep_order asks for the shared-memory form with the K offsets it has always started from.  They follow from the weight,
// the number of 256-token groups and the SM count, so the order of a row's sums is fixed for a given product on a given
// GPU, not for a weight; the other two forms start elsewhere and add the K splits of a tile, which changes the last bits.
GemmPlan plan_gemm(const WeightView& w, int64_t m, int sm_count, bool keep_order)
{
    GemmPlan best = gemm_form(w, m, sm_count, 0, 0, 1);
    const int64_t steps = (w.k + GEMM_BK - 1) / GEMM_BK;
    const auto waves = [](int64_t ctas, int64_t slots) { return (double)((ctas + slots - 1) / slots); };
    const double tiles_per_cta = (double)((w.rt + best.groups - 1) / best.groups);
    double best_cost = waves(best.grid, sm_count) * (4.0 * w.kc * (0.57 + 0.026 * tiles_per_cta) + 9.2);
    if (keep_order) {
        return best;
    }
    const int64_t min_tiles = (m + GEMM_MAX_TOKENS - 1) / GEMM_MAX_TOKENS;
    for (int64_t tt = min_tiles; tt <= min_tiles + 1; ++tt) {
        const int64_t tokens = ((m + tt - 1) / tt + 15) / 16 * 16;
        const int64_t t_tiles = (m + tokens - 1) / tokens;
        const double fill = (double)tokens / GEMM_MAX_TOKENS;
        for (int nb = 1; nb <= 2; ++nb) {
            const int64_t tiles = ((w.rt + 8 * nb - 1) / (8 * nb)) * t_tiles;
            for (int splits = 1; splits <= (nb == 1 ? 8 : 1) && splits <= w.kc; splits *= 2) {
                const int64_t ctas = tiles * splits;
                double cost;
                if (nb == 2) {
                    cost = waves(ctas, sm_count) * (steps * (0.481 + 0.15 * fill) + 7.1);
                } else {
                    // two CTAs per SM; a last round that leaves most SMs with one runs its steps faster
                    const double st = (double)((steps + splits - 1) / splits);
                    const double paired = st * (0.615 + 0.104 * fill) + 6.7, alone = st * (0.385 + 0.034 * fill) + 6.7;
                    const int64_t rounds = ctas / (2 * sm_count), rest = ctas % (2 * sm_count);
                    cost = rounds * paired + (rest > sm_count ? paired : rest > 0 ? alone : 0.0) + (splits > 1 ? 4.2 : 0.0);
                }
                if (cost < best_cost) {
                    best_cost = cost;
                    best = gemm_form(w, m, sm_count, nb, (int)tokens, splits);
                }
            }
        }
    }
    return best;
}

cudaError_t launch_gemm_bf16(const WeightView& w, const void* x_bf16, void* y, int64_t m, int out, bool keep_order,
                             int sm_count, int* status, cudaStream_t stream, const char** why)
{
    return launch_gemm_plan(plan_gemm(w, m, sm_count, keep_order), w, x_bf16, y, m, out, keep_order, status, stream, why);
}

cudaError_t launch_gemm_plan(const GemmPlan& plan, const WeightView& w, const void* x_bf16, void* y, int64_t m, int out,
                             bool keep_order, int* status, cudaStream_t stream, const char** why)
{
    *why = nullptr;
    EncodeTiledFn encode = encode_tiled_fn();
    if (!encode) {
        *why = "cuTensorMapEncodeTiled is not available from the driver";
        return cudaErrorNotSupported;
    }
    if ((reinterpret_cast<uintptr_t>(x_bf16) & 15u) != 0 || (w.k % 8) != 0) {
        *why = "activations must be 16-byte aligned with a row length that is a multiple of 8";
        return cudaErrorInvalidValue;
    }
    if (out == GEMM_OUT_SWIGLU && (w.n % 16 != 0 || (reinterpret_cast<uintptr_t>(y) & 15u) != 0)) {
        *why = "a gate|up product needs whole 16-row tiles and a 16-byte aligned result";
        return cudaErrorInvalidValue;
    }
    CUtensorMap xmap;
    const cuuint64_t dims[2] = {(cuuint64_t)w.k, (cuuint64_t)m};
    const cuuint64_t strides[1] = {(cuuint64_t)w.k * 2};
    const cuuint32_t box[2] = {(cuuint32_t)GEMM_BK, (cuuint32_t)(plan.groups > 0 ? GEMM_SMEM_BOX_ROWS : plan.tokens)};
    const cuuint32_t estr[2] = {1u, 1u};
    const CUresult cr = encode(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x_bf16), dims, strides, box,
                               estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) {
        *why = "cuTensorMapEncodeTiled rejected the activation tensor";
        return cudaErrorInvalidValue;
    }
    if (plan.groups > 0) {
        return launch_gemm_smem(w, xmap, y, m, out, plan.groups, keep_order, status, stream);
    }
    GemmArgs args;
    args.w = w;
    args.y = y;
    args.m = m;
    args.out = out;
    args.tokens = plan.tokens;
    args.t_tiles = plan.t_tiles;
    args.ring = plan.ring;
    args.status = status;
    switch (w.fmt) {
    case FMT_Q4_0: return launch_gemm_fmt<FMT_Q4_0>(xmap, args, plan, stream);
    case FMT_Q8_0: return launch_gemm_fmt<FMT_Q8_0>(xmap, args, plan, stream);
    case FMT_Q4_K: return launch_gemm_fmt<FMT_Q4_K>(xmap, args, plan, stream);
    case FMT_Q6_K: return launch_gemm_fmt<FMT_Q6_K>(xmap, args, plan, stream);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace qmm
