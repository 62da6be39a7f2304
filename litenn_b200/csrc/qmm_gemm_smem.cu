// The prefill GEMM (qmm_gemm.cu) for many tokens: the dequantized weights go through shared memory as the B operand, so
// one dequantization serves 256 tokens instead of 128.
//
// One CTA owns up to 256 activation rows (two 128-row UMMA tiles) and a contiguous group
// of up to 16 row tiles of the weight (n <= 256 output features); its accumulators fill
// 2 x n <= 512 TMEM columns, so every weight tile is dequantized once per CTA and reused
// for all its activation rows.  Per 64-wide K step:
//   warp 0          TMA: two 128x64 bf16 boxes of X -> shared memory (128-byte swizzle)
//   warps 2..17     read the packed weight tiles (qmm_common.cuh) from global memory,
//                   rebuild the exact fp32 values ggml's to_float gives, round them to bf16
//                   and store them as the K-major, 128-byte-swizzled B tile
//   warp 1          tcgen05.mma (kind::f16, bf16 x bf16 -> fp32, M=128, N=n, K=16) x 4 x 2,
//                   then tcgen05.commit to hand the stage back
// A 3-stage mbarrier ring decouples the three roles.  At the end warps 2..17 read the
// accumulators with tcgen05.ld and write Y.  Every wait has an iteration limit; a CTA
// that gives up sets the status word, still frees its TMEM and returns.
// Bound: latency.  No unit is near its limit (ncu, Q4_0 12288 x 4096, 1999 tokens: tensor pipe 51 %, memory pipes 50 %,
// issue 41 %); the dequant warps wait for packed words and scales, and three stages do not hide it.  Q4_K 14336 x 4096,
// 512 tokens takes 71 us (850 TFLOP/s).  It took 94 us when every value went through an integer conversion of its own and
// the MMAs were issued under a lane comparison instead of elect.sync.
#include <algorithm>

#include "qmm_gemm_dequant.cuh"
#include "qmm_gemm_smem.h"
#include "qmm_kernels.h"

namespace qmm {

namespace {

constexpr int GEMM_STAGES = 3;
constexpr int GEMM_A_TILE_BYTES = 128 * 128;   // 128 rows x 64 bf16
constexpr int GEMM_A_STAGE_BYTES = 2 * GEMM_A_TILE_BYTES;
constexpr int GEMM_B_STAGE_BYTES = 256 * 128;  // up to 256 weight rows x 64 bf16
constexpr int GEMM_STAGE_BYTES = GEMM_A_STAGE_BYTES + GEMM_B_STAGE_BYTES;
constexpr int GEMM_DEQ_WARPS = 16;
constexpr int GEMM_THREADS = (2 + GEMM_DEQ_WARPS) * 32;
constexpr int GEMM_SMEM_BYTES = GEMM_STAGES * GEMM_STAGE_BYTES + 1024 /*alignment*/ + 256 /*barriers*/;

// Same with a non-suspending probe: used by single elected threads that sit on the critical
// path of the stage hand-over (a suspended try_wait wakes up late).
__device__ __forceinline__ bool g_mbar_poll(uint64_t* bar, uint32_t parity)
{
    const uint32_t addr = g_smem_u32(bar);
    for (uint32_t spin = 0; spin < (GEMM_SPIN_LIMIT << 4); ++spin) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
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

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                          uint32_t accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Byte offset of element (row, k) of a K-major tile with 128-byte rows and 128-byte swizzle:
// the 16-byte chunk index is XORed with the row index modulo 8.
__device__ __forceinline__ uint32_t swz128(int row, int k)
{
    const uint32_t chunk = (uint32_t)(k >> 3) ^ (uint32_t)(row & 7);
    return (uint32_t)row * 128u + chunk * 16u + (uint32_t)(k & 7) * 2u;
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// Rows (16*rl + g) and (16*rl + g + 8), 64 columns, of the B tile.
__device__ __forceinline__ void store_quarter(const uint32_t (&r)[16], uint8_t* btile, int rl, int lane)
{
    const int row0 = 16 * rl + (lane >> 2), t = lane & 3;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
#pragma unroll
        for (int rs = 0; rs < 2; ++rs) {
            *reinterpret_cast<uint2*>(btile + swz128(row0 + 8 * rs, 16 * p + 4 * t)) =
                make_uint2(r[4 * p + 2 * rs], r[4 * p + 2 * rs + 1]);
        }
    }
}

// ---- the kernel -----------------------------------------------------------------------------

struct GemmArgs {
    WeightView w;
    void* y;            // [M, N] row-major, fp32 or bf16; [M, N / 2] bf16 for GEMM_OUT_SWIGLU
    int64_t m;
    int out;            // GEMM_OUT_*
    int groups_per_tg;  // CTAs that share one group of 256 activation rows
    int* status;
};


// EXACT: the K offset at which a CTA starts may lie inside a chunk, which is the order of K that results of keep_order
// calls have; the other form starts at whole chunks and walks them without tests (Q4_K 14336 x 4096, 512 tokens: 73 us
// against 78).
template <int FMT, bool EXACT>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap xmap, const GemmArgs args)
{
    extern __shared__ uint8_t gemm_smem_raw[];
    // the swizzle pattern is defined on absolute shared-memory addresses: 1024-byte alignment
    uint8_t* smem = gemm_smem_raw + ((1024u - (g_smem_u32(gemm_smem_raw) & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + GEMM_STAGES * GEMM_STAGE_BYTES);
    uint64_t* full_a = bars;                    // [STAGES]  TMA bytes landed
    uint64_t* full_b = bars + GEMM_STAGES;      // [STAGES]  dequant warps done
    uint64_t* empty = bars + 2 * GEMM_STAGES;   // [STAGES]  MMAs that read the stage have completed
    uint64_t* accum = bars + 3 * GEMM_STAGES;   // all MMAs completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * GEMM_STAGES + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const WeightView& v = args.w;
    const int tg = blockIdx.x / args.groups_per_tg;
    const int gi = blockIdx.x % args.groups_per_tg;
    const int rt0 = (int)((long long)v.rt * gi / args.groups_per_tg);
    const int rt1 = (int)((long long)v.rt * (gi + 1) / args.groups_per_tg);
    const int R = rt1 - rt0;        // row tiles of this CTA, 1..16
    const int n = R * 16;           // UMMA N
    const int64_t row_base = (int64_t)tg * 256;
    const int ntt = (args.m - row_base) > 128 ? 2 : 1;
    const int n_stages = EXACT ? (int)((v.k + GEMM_BK - 1) / GEMM_BK) : 4 * v.kc;  // columns past K are zero on both sides
    // CTAs that share activation rows start at different K offsets, so they do not all ask L2 for the same lines at the
    // same moment.
    const int k_rot = EXACT ? (int)((long long)n_stages * gi / args.groups_per_tg)
                            : 4 * (int)((long long)v.kc * gi / args.groups_per_tg);

    if (threadIdx.x == 0) {
        for (int s = 0; s < GEMM_STAGES; ++s) {
            g_mbar_init(&full_a[s], 1);
            g_mbar_init(&full_b[s], GEMM_DEQ_WARPS);
            g_mbar_init(&empty[s], 1);
        }
        g_mbar_init(accum, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        // 512 columns: two accumulators of up to 256 columns each
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(g_smem_u32(tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---- TMA producer: activations.  Only they come from an earlier kernel; the first weights are dequantized while it
        // drains, and what is stored in the end depends on the activations.  Every warp waits for that kernel before its first
        // bounded wait, whose limit is for this kernel's own steps ----
        if (lane == 0) {
            g_pdl_wait();
            for (int s = 0; s < n_stages; ++s) {
                const int slot = s % GEMM_STAGES;
                if (s >= GEMM_STAGES && !g_mbar_poll(&empty[slot], (uint32_t)(s / GEMM_STAGES - 1) & 1u)) {
                    atomicExch(args.status, 11);
                    break;
                }
                uint8_t* a = smem + (size_t)slot * GEMM_STAGE_BYTES;
                g_mbar_expect_tx(&full_a[slot], (uint32_t)(ntt * GEMM_A_TILE_BYTES));
                const int ks = (s + k_rot) % n_stages;
                tma_load_2d(a, &xmap, ks * GEMM_BK, (int)row_base, &full_a[slot]);
                if (ntt == 2) {
                    tma_load_2d(a + GEMM_A_TILE_BYTES, &xmap, ks * GEMM_BK, (int)row_base + 128, &full_a[slot]);
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer: the whole warp walks the stages, one lane issues ----
        const uint32_t idesc = umma_idesc_bf16(n);
        bool ok = true;
        g_pdl_wait();
        for (int s = 0; s < n_stages; ++s) {
            const int slot = s % GEMM_STAGES;
            const uint32_t parity = (uint32_t)(s / GEMM_STAGES) & 1u;
            ok = g_mbar_wait(&full_a[slot], parity) && g_mbar_wait(&full_b[slot], parity);
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok) {
                if (lane == 0) {
                    atomicExch(args.status, 12);
                }
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const uint64_t da = umma_smem_desc(g_smem_u32(smem + (size_t)slot * GEMM_STAGE_BYTES));
                const uint64_t db = da + (uint64_t)(GEMM_A_STAGE_BYTES >> 4);
#pragma unroll
                for (int kk = 0; kk < GEMM_BK / 16; ++kk) {
                    for (int tt = 0; tt < ntt; ++tt) {
                        umma_bf16(tmem_base + (uint32_t)tt * 256u, da + (uint64_t)(tt * (GEMM_A_TILE_BYTES >> 4) + 2 * kk),
                                  db + (uint64_t)(2 * kk), idesc, (s > 0 || kk > 0) ? 1u : 0u);
                    }
                }
                umma_commit(&empty[slot]);  // arrives when the MMAs above have read their operands
            }
            __syncwarp();
        }
        if (ok && elect_one()) {
            umma_commit(accum);
        }
        g_pdl_launch_dependents();  // the next kernel may start while this one stores its results
        __syncwarp();
    } else {
        // ---- dequant producers: weights -> bf16 B tile ----
        const int dw = warp - 2;  // 0..15: row tile dw of this CTA
        const bool has0 = dw < R;
        const size_t tile_stride = tile_bytes(FMT);
        const uint8_t* t0 = v.tiles + ((size_t)(rt0 + (has0 ? dw : 0)) * v.kc) * tile_stride;
        Packed<FMT> P;
        Scales<FMT> S, SN;
        // The walk starts inside chunk c_rot at quarter q_rot and ends with the quarters of that chunk it left out.
        const int c_rot = k_rot >> 2, q_rot = EXACT ? k_rot & 3 : 0;
        const int walk = v.kc + (q_rot > 0 ? 1 : 0);
        const uint8_t* wt = t0 + (size_t)c_rot * tile_stride;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            load_quarter<FMT>(P, wt, q, lane);
        }
        load_scales<FMT>(S, wt, lane >> 2);
        SN = S;
        bool ok = true;
        int s = 0;
        for (int i = 0; i < walk && ok; ++i) {
            const int chunk = (i + c_rot) % v.kc;
            const bool more = i + 1 < walk;
            const uint8_t* next = t0 + (size_t)((i + 1 + c_rot) % v.kc) * tile_stride;
            if (more) {
                load_scales<FMT>(SN, next, lane >> 2);
            }
            if (i + 3 < v.kc && lane * 128 < (int)tile_stride) {  // three chunks ahead into L2
                asm volatile("prefetch.global.L2 [%0];" ::"l"(t0 + (size_t)((i + 3 + c_rot) % v.kc) * tile_stride + lane * 128));
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool mine = !EXACT || ((i == 0 ? q >= q_rot : i < v.kc || q < q_rot) && 4 * chunk + q < n_stages);
                if (mine) {
                    uint32_t r[16];
                    dequant_quarter<FMT>(P, S, q, r);
                    const int slot = s % GEMM_STAGES;
                    if (s == GEMM_STAGES) {
                        g_pdl_wait_only();
                    }
                    if (ok && s >= GEMM_STAGES) {
                        // lane 0 probes, the others wait for it at the warp barrier
                        bool landed = true;
                        if (lane == 0) {
                            landed = g_mbar_poll(&empty[slot], (uint32_t)(s / GEMM_STAGES - 1) & 1u);
                        }
                        ok = __shfl_sync(0xFFFFFFFFu, landed, 0);
                        if (!ok && lane == 0) {
                            atomicExch(args.status, 13);
                        }
                    }
                    if (ok) {
                        if (has0) {
                            store_quarter(r, smem + (size_t)slot * GEMM_STAGE_BYTES + GEMM_A_STAGE_BYTES, dw, lane);
                        }
                        // make the generic-proxy stores visible to the tensor core (async proxy), then signal
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            g_mbar_arrive(&full_b[slot]);
                        }
                    }
                    ++s;
                }
                if (more) {  // the registers of this quarter are free: refill them from the next tile
                    load_quarter<FMT>(P, next, q, lane);
                }
            }
            S = SN;
        }

        // ---- epilogue: a warp reaches TMEM lanes 32*(warp%4).., four warps share them by columns ----
        g_pdl_wait();
        if (!g_mbar_wait_warp(accum, 0)) {
            if (lane == 0) {
                atomicExch(args.status, 14);
            }
        } else {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int quad = warp & 3;
            const bool y_aligned = (reinterpret_cast<uintptr_t>(args.y) & 15u) == 0;  // a caller's y may be any element
            for (int tt = 0; tt < ntt; ++tt) {
                const int64_t row = row_base + 128 * tt + 32 * quad + lane;
                for (int c0 = 32 * (dw >> 2); c0 < n; c0 += 128) {
                    uint32_t acc[32];
                    tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(32 * quad) << 16) + (uint32_t)(tt * 256 + c0), acc);
                    if (row < args.m) {
                        const int64_t col0 = (int64_t)rt0 * 16 + c0;
                        // 8 columns at a time: 16-byte (bf16) or 2 x 16-byte (fp32) stores when
                        // base and row pitch keep them aligned, scalar stores elsewhere and at ragged edges
                        if (args.out == GEMM_OUT_SWIGLU) {
                            // a row tile's 16 columns are 8 gates and their 8 ups
                            __nv_bfloat16* yo = static_cast<__nv_bfloat16*>(args.y) + row * (v.n >> 1) + (col0 >> 1);
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                if (c0 + 16 * j < n && col0 + 16 * j < v.n) {
                                    uint32_t o[4];
#pragma unroll
                                    for (int i = 0; i < 4; ++i) {
                                        const int e = 16 * j + 2 * i;
                                        o[i] = pack_bf16x2(
                                            silu_mul(__uint_as_float(acc[e]), __uint_as_float(acc[e + 8])),
                                            silu_mul(__uint_as_float(acc[e + 1]), __uint_as_float(acc[e + 9])));
                                    }
                                    *reinterpret_cast<uint4*>(yo + 8 * j) = make_uint4(o[0], o[1], o[2], o[3]);
                                }
                            }
                        } else if (args.out == GEMM_OUT_BF16) {
                            __nv_bfloat16* yo = static_cast<__nv_bfloat16*>(args.y) + row * v.n + col0;
                            const bool vec = y_aligned && (v.n & 7) == 0;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                if (vec && c0 + 8 * j + 8 <= n && col0 + 8 * j + 8 <= v.n) {
                                    uint4 o;
                                    o.x = pack_bf16x2(__uint_as_float(acc[8 * j + 0]), __uint_as_float(acc[8 * j + 1]));
                                    o.y = pack_bf16x2(__uint_as_float(acc[8 * j + 2]), __uint_as_float(acc[8 * j + 3]));
                                    o.z = pack_bf16x2(__uint_as_float(acc[8 * j + 4]), __uint_as_float(acc[8 * j + 5]));
                                    o.w = pack_bf16x2(__uint_as_float(acc[8 * j + 6]), __uint_as_float(acc[8 * j + 7]));
                                    *reinterpret_cast<uint4*>(yo + 8 * j) = o;
                                } else {
#pragma unroll
                                    for (int i = 8 * j; i < 8 * j + 8; ++i) {
                                        if (col0 + i < v.n && c0 + i < n) {
                                            yo[i] = __float2bfloat16_rn(__uint_as_float(acc[i]));
                                        }
                                    }
                                }
                            }
                        } else {
                            float* yo = static_cast<float*>(args.y) + row * v.n + col0;
                            const bool vec = y_aligned && (v.n & 3) == 0;
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                if (vec && c0 + 4 * j + 4 <= n && col0 + 4 * j + 4 <= v.n) {
                                    *reinterpret_cast<uint4*>(yo + 4 * j) =
                                        make_uint4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
                                } else {
#pragma unroll
                                    for (int i = 4 * j; i < 4 * j + 4; ++i) {
                                        if (col0 + i < v.n && c0 + i < n) {
                                            yo[i] = __uint_as_float(acc[i]);
                                        }
                                    }
                                }
                            }
                        }
                    }
                }
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}


template <int FMT, bool EXACT>
cudaError_t launch_smem_exact(const CUtensorMap& xmap, const GemmArgs& args, int grid, cudaStream_t stream)
{
    auto kernel = gemm_tcgen05_kernel<FMT, EXACT>;
    static bool configured[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        return e;
    }
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM_BYTES);
        if (e != cudaSuccess) {
            return e;
        }
        if (dev >= 0 && dev < 64) {
            configured[dev] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = GEMM_SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, xmap, args);
}

template <int FMT>
cudaError_t launch_smem_fmt(const CUtensorMap& xmap, const GemmArgs& args, int grid, bool keep_order, cudaStream_t stream)
{
    return keep_order ? launch_smem_exact<FMT, true>(xmap, args, grid, stream)
                      : launch_smem_exact<FMT, false>(xmap, args, grid, stream);
}

}  // namespace

int gemm_smem_groups(int rt, int64_t m, int sm_count)
{
    const int tgs = (int)((m + 255) / 256);
    return std::min(std::max(sm_count / tgs, (rt + 15) / 16), rt);
}

cudaError_t launch_gemm_smem(const WeightView& w, const CUtensorMap& xmap, void* y, int64_t m, int out, int groups,
                             bool keep_order, int* status, cudaStream_t stream)
{
    GemmArgs args;
    args.w = w;
    args.y = y;
    args.m = m;
    args.out = out;
    args.groups_per_tg = groups;
    args.status = status;
    const int grid = (int)((m + 255) / 256) * groups;
    switch (w.fmt) {
    case FMT_Q4_0: return launch_smem_fmt<FMT_Q4_0>(xmap, args, grid, keep_order, stream);
    case FMT_Q8_0: return launch_smem_fmt<FMT_Q8_0>(xmap, args, grid, keep_order, stream);
    case FMT_Q4_K: return launch_smem_fmt<FMT_Q4_K>(xmap, args, grid, keep_order, stream);
    case FMT_Q6_K: return launch_smem_fmt<FMT_Q6_K>(xmap, args, grid, keep_order, stream);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace qmm
