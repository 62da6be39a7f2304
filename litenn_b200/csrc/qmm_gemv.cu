// Activation packing for the integer-MMA matvec and the dispatch of a matvec to the block
// format's kernels (qmm_gemv_kernel.cuh, instantiated per format in qmm_gemv_<format>.cu).
#include <atomic>

#include "qmm_gemv_device.cuh"
#include "qmm_gemv_forms.cuh"
#include "qmm_kernels.h"
#include "qmm_pack.cuh"

namespace qmm {

namespace {

// Quantize x to 16 bits per (row, 32-wide block) and store it in B-fragment order
// (qmm_common.cuh).  grid (kc, ncp), 128 threads: warp w handles activation row 4*blockIdx.y + w
// of chunk blockIdx.x, lane L its columns 8L..8L+7 (block L >> 2).
__global__ void __launch_bounds__(128) pack_x_kernel(const float* __restrict__ x, int m, int64_t k, int ncp,
                                                     int compact, uint8_t* __restrict__ out)
{
    pdl_launch_dependents();  // the matvec that follows may start fetching its weights
    pdl_wait();               // x may come from the previous kernel; the buffer may still be read by it
    const int c = blockIdx.x;
    const int j = blockIdx.y;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int row = 4 * j + warp;

    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int64_t col = (int64_t)c * 256 + 8 * lane + i;
        v[i] = (row < m && col < k) ? x[(int64_t)row * k + col] : 0.0f;
    }
    if (compact) {
        if (warp == 0) {
            warp_pack_chunk(v, out + (size_t)c * XPK1_REC);
        }
        return;
    }
    // lane L holds one fragment word of each digit twice: activations 8L..8L+3 and 8L+4..8L+7 of block L >> 2
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        amax = fmaxf(amax, fabsf(v[i]));
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    const float inv = amax > 0.0f ? 32639.0f / amax : 0.0f;
    uint32_t hw[2] = {0u, 0u}, lw[2] = {0u, 0u};
    int bsum = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        int hi, lo;
        bsum += quant16(v[i], inv, hi, lo);
        hw[i >> 2] |= (uint32_t)(hi & 0xFF) << (8 * (i & 3));
        lw[i >> 2] |= (uint32_t)(lo & 0xFF) << (8 * (i & 3));
    }
    bsum += __shfl_xor_sync(0xFFFFFFFFu, bsum, 1);
    bsum += __shfl_xor_sync(0xFFFFFFFFu, bsum, 2);
    uint8_t* rec = out + (size_t)c * xpack_rec_bytes(ncp);
    const int b = lane >> 2, part = lane & 3;
    const int t0 = 2 * (part & 1), half = part >> 1;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        *xpack_word(rec, ncp, row, b, 0, t0 + i, half) = hw[i];
        *xpack_word(rec, ncp, row, b, 1, t0 + i, half) = lw[i];
    }
    if (part == 0) {
        xpack_meta(rec, ncp, row, b, bsum, amax);
    }
}

// Inverse of the compact packing, for verification: x[i] = xs * (256*hi + lo).
__global__ void unpack_x_kernel(const uint8_t* __restrict__ packed, int64_t k, float* __restrict__ x)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k; i += (int64_t)gridDim.x * blockDim.x) {
        const uint8_t* rec = packed + (size_t)(i >> 8) * XPK1_REC;
        const int b = (int)(i >> 5) & 7, e = (int)i & 31;
        const int half = e >> 4, t = (e & 15) >> 2, byte = e & 3;
        const uint32_t* xq = reinterpret_cast<const uint32_t*>(rec + b * 64);
        const int hi = (int)(signed char)((xq[(0 * 4 + t) * 2 + half] >> (8 * byte)) & 0xFFu);
        const int lo = (int)(signed char)((xq[(1 * 4 + t) * 2 + half] >> (8 * byte)) & 0xFFu);
        const float xs = __int_as_float(reinterpret_cast<const int4*>(rec + XPK1_META)[b].z);
        x[i] = xs * (float)(256 * hi + lo);
    }
}

__device__ __forceinline__ uint32_t bf16_bits(float x)  // round to nearest even; keeps infinities and NaN
{
    const uint32_t u = __float_as_uint(x);
    return ((u & 0x7F800000u) == 0x7F800000u ? u : u + 0x7FFFu + ((u >> 16) & 1u)) >> 16;
}

// fp32 -> bf16, for fp32 callers of the prefill GEMM.  Bound by memory latency: VEC takes sixteen bytes per load, which
// needs an aligned x (77 rows of 11008 with the product that follows: 32.8 us with single elements, 30.7 with four).
template <bool VEC>
__global__ void __launch_bounds__(256) f32_to_bf16_kernel(const float* __restrict__ x, int64_t count,
                                                          unsigned short* __restrict__ out)
{
    pdl_launch_dependents();
    pdl_wait();  // x may come from the previous kernel; the buffer may still be read by it
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    if constexpr (VEC) {
        for (int64_t i = first; i < count / 4; i += step) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(x) + i);
            reinterpret_cast<uint2*>(out)[i] =
                make_uint2(bf16_bits(v.x) | (bf16_bits(v.y) << 16), bf16_bits(v.z) | (bf16_bits(v.w) << 16));
        }
    } else {
        for (int64_t i = first; i < count; i += step) {
            out[i] = (unsigned short)bf16_bits(__ldcg(x + i));
        }
    }
}

}  // namespace

cudaError_t launch_f32_to_bf16(const float* x, int64_t count, void* out_bf16, cudaStream_t stream)
{
    unsigned short* out = static_cast<unsigned short*>(out_bf16);
    const bool vec = count % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0 &&
                     (reinterpret_cast<uintptr_t>(out_bf16) & 7u) == 0;
    const int64_t blocks = ((vec ? count / 4 : count) + 255) / 256;
    const unsigned grid = (unsigned)(blocks < 4096 ? blocks : 4096);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, vec ? f32_to_bf16_kernel<true> : f32_to_bf16_kernel<false>, x, count, out);
}

cudaError_t launch_pack_x(const float* x, int m, int64_t k, int kc, uint8_t* out, cudaStream_t stream)
{
    const int ncp = xpack_ncp(m);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)kc, (unsigned)ncp);
    cfg.blockDim = dim3(128);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, pack_x_kernel, x, m, k, ncp, m == 1 ? 1 : 0, out);
}

cudaError_t launch_unpack_x(const uint8_t* packed, int64_t k, float* x, cudaStream_t stream)
{
    unpack_x_kernel<<<(unsigned)((k + 255) / 256), 256, 0, stream>>>(packed, k, x);
    return cudaGetLastError();
}

int sm_count_of(int dev)
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

// Never where y lies over x: CTAs that are done store y while others still read x.  The packing kernel reads all of x first.
bool gemv_packs_itself(const WeightView& w, const float* x, const float* y, int sm_count)
{
    const uintptr_t x0 = reinterpret_cast<uintptr_t>(x), x1 = x0 + (uintptr_t)w.k * sizeof(float);
    const uintptr_t y0 = reinterpret_cast<uintptr_t>(y), y1 = y0 + (uintptr_t)w.n * sizeof(float);
    if (x0 < y1 && y0 < x1) {
        return false;
    }
    if ((x0 & 15u) != 0 || w.k % 32 != 0 || sm_count < 1) {  // x is read 16 bytes at a time
        return false;
    }
    return gemv_packs_itself_shape(w.fmt, w.rt, w.kc, sm_count);
}

cudaError_t launch_gemv_fused(const WeightView& w, const XPackView& xp, float* y, int m, int* status,
                              const PeerScatter& ps, const GemvFuse& fu, cudaStream_t stream)
{
    if ((ps.n_peers > 0 || fu.mode != EPI_STORE || fu.ss_in != nullptr || fu.x_f32 != nullptr) && m != 1) {
        return cudaErrorInvalidValue;
    }
    if (ps.n_peers > 0 && fu.mode != EPI_STORE &&
        !(fu.mode == EPI_RESID_PACK && ps.recv != nullptr && ps.wait_status != nullptr && ps.tp_size == ps.n_peers + 1)) {
        return cudaErrorInvalidValue;  // only the residual form also finishes the sum over the ranks
    }
    if ((fu.mode == EPI_RESID_PACK && w.n % 32 != 0) || (fu.mode == EPI_SWIGLU && w.n % 16 != 0) ||
        (fu.mode == EPI_SWIGLU_PACK && (w.n % 64 != 0 || fu.packed_out == nullptr)) || (fu.x_f32 && w.k % 32 != 0)) {
        return cudaErrorInvalidValue;
    }
    switch (w.fmt) {
    case FMT_Q4_0: return launch_gemv_q4_0(w, xp, y, m, status, ps, fu, stream);
    case FMT_Q8_0: return launch_gemv_q8_0(w, xp, y, m, status, ps, fu, stream);
    case FMT_Q4_K: return launch_gemv_q4_k(w, xp, y, m, status, ps, fu, stream);
    case FMT_Q6_K: return launch_gemv_q6_k(w, xp, y, m, status, ps, fu, stream);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_gemv(const WeightView& w, const XPackView& xp, float* y, int m, int* status, cudaStream_t stream)
{
    const PeerScatter none = {};
    const GemvFuse plain = {};
    return launch_gemv_fused(w, xp, y, m, status, none, plain, stream);
}

}  // namespace qmm
