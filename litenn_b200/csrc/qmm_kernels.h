// Host-callable launchers of the CUDA kernels (internal to the library).
#pragma once

#include "qmm_layout.cuh"

namespace qmm {

cudaError_t launch_repack(int fmt, const RawSource& src, int rt, int kc, uint8_t* tiles, int sm_count,
                          cudaStream_t stream);
cudaError_t launch_dequant_packed(const WeightView& v, float* out, int sm_count, cudaStream_t stream);
cudaError_t launch_dequant_raw(int fmt, const uint8_t* payload, int64_t n, int64_t k, float* out, int sm_count,
                               cudaStream_t stream);

// Quantize and pack x[m,k] (fp32) for the integer-MMA GEMV into `out`
// (xpack1_bytes(kc) bytes for m == 1, else xpack_bytes(kc, xpack_ncp(m))).
cudaError_t launch_pack_x(const float* x, int m, int64_t k, int kc, uint8_t* out, cudaStream_t stream);
// Compact (m == 1) packed activations back to fp32 [k]; verification aid.
cudaError_t launch_unpack_x(const uint8_t* packed, int64_t k, float* x, cudaStream_t stream);

// y[m,n] = x · Wᵀ from a packed weight and packed activations (launch_pack_x first).
// `status` points at a device int that a kernel sets non-zero if a bounded wait ran out.
cudaError_t launch_gemv(const WeightView& w, const XPackView& xp, float* y, int m, int* status, cudaStream_t stream);
// Batch 1 only when ps.n_peers > 0 (also scatters the result to the peers, PeerScatter) or when
// `fu` asks for an input RMSNorm factor or a fused epilogue (GemvFuse); both in qmm_common.cuh.
cudaError_t launch_gemv_fused(const WeightView& w, const XPackView& xp, float* y, int m, int* status,
                              const PeerScatter& ps, const GemvFuse& fu, cudaStream_t stream);
// SMs of a device, 0 if it cannot be asked; asked once.
int sm_count_of(int dev);
// Whether gate|up of a decode chain writes its product packed (EPI_SWIGLU_PACK, groups of four row tiles per CTA) or as fp32
// from CTAs of one tile each (EPI_SWIGLU), which ffn_down then packs itself.  Packed costs less, but a long row (kc > 16) of
// few tiles is bound by how many SMs read it: eight blocks, us a token, fp32 form and packed: 8192 wide, FFN 1024 Q4_0 154 and
// 185, 1792 Q4_0 170 and 193, Q6_K 199 and 216; 2304 (288 tiles) Q4_0 180 and 200, with more warps per tile 182; Q6_K 239
// and 229, with more warps 212; 3584 Q4_0 220 and 213.  12288 wide, FFN 1536 Q4_0 217 and 264, 2304 Q4_K 290 and 304.
constexpr bool gemv_swiglu_packs(int rt, int kc, int sms)
{
    return kc <= 16 || 4LL * rt > 7LL * sms;
}
// Whether the matvec of one fp32 vector is one launch that packs x itself (launch_gemv_fused with fu.x_f32 and EPI_STORE).
bool gemv_packs_itself(const WeightView& w, const float* x, const float* y, int sm_count);
// per-format instantiations (qmm_gemv_<format>.cu)
cudaError_t launch_gemv_q4_0(const WeightView& w, const XPackView& xp, float* y, int m, int* status,
                             const PeerScatter& ps, const GemvFuse& fu, cudaStream_t stream);
cudaError_t launch_gemv_q8_0(const WeightView& w, const XPackView& xp, float* y, int m, int* status,
                             const PeerScatter& ps, const GemvFuse& fu, cudaStream_t stream);
cudaError_t launch_gemv_q4_k(const WeightView& w, const XPackView& xp, float* y, int m, int* status,
                             const PeerScatter& ps, const GemvFuse& fu, cudaStream_t stream);
cudaError_t launch_gemv_q6_k(const WeightView& w, const XPackView& xp, float* y, int m, int* status,
                             const PeerScatter& ps, const GemvFuse& fu, cudaStream_t stream);

// fp32 -> bf16, round to nearest even.
cudaError_t launch_f32_to_bf16(const float* x, int64_t count, void* out_bf16, cudaStream_t stream);

// Prefill GEMM on tcgen05: y[m,n] = x_bf16[m,k] · Wᵀ.  On a configuration error `*why` explains it.
//   GEMM_OUT_SWIGLU  the rows are interleaved gate|up (EPI_SWIGLU, qmm_common.cuh): y[m, n / 2] = bf16(silu(gate) * up);
//                    n a multiple of 16, y 16-byte aligned
//   keep_order       sums in the shared-memory form's order of K for this m, also where another form is faster
constexpr int GEMM_OUT_F32 = 0, GEMM_OUT_BF16 = 1, GEMM_OUT_SWIGLU = 2;
cudaError_t launch_gemm_bf16(const WeightView& w, const void* x_bf16, void* y, int64_t m, int out, bool keep_order,
                             int sm_count, int* status, cudaStream_t stream, const char** why);

// How launch_gemm_bf16 cuts one product: NB blocks of 128 weight rows and `tokens` activation rows per CTA, `splits` CTAs
// along K; or, with groups > 0, the shared-memory kernel with that many CTAs per 256 tokens.
struct GemmPlan {
    int nb, tokens, t_tiles, splits, ring, grid, smem, groups;
};
GemmPlan plan_gemm(const WeightView& w, int64_t m, int sm_count, bool keep_order);
// The plan of one form, for plan_gemm and for tests that walk every form: nb 1 or 2 with `tokens` a multiple of 16 up to
// 128 and splits 1, 2, 4 or 8 up to the weight's K chunks (nb 2: 1); nb 0 is the shared-memory form.
GemmPlan gemm_form(const WeightView& w, int64_t m, int sm_count, int nb, int tokens, int splits);
cudaError_t launch_gemm_plan(const GemmPlan& plan, const WeightView& w, const void* x_bf16, void* y, int64_t m, int out,
                             bool keep_order, int* status, cudaStream_t stream, const char** why);

}  // namespace qmm
