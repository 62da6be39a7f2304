// The prefill attention kernels with fp32 results, for the tests: the library's own source with the other output type.
#include "../../litenn_b200/csrc/llama_kernels.cu"

extern "C" int attn_prefill_f32(int head_dim, const float* qkv, int m, int pos0, int n_heads, int n_kv, int max_seq,
                                const void* cache_k, const void* cache_v, float* ctx, int rows_max, void* stream)
{
    return (int)qmm::attn_prefill(qkv, m, pos0, n_heads, n_kv, head_dim, max_seq, static_cast<const __half*>(cache_k),
                                  static_cast<const __half*>(cache_v), ctx, rows_max, static_cast<cudaStream_t>(stream));
}
