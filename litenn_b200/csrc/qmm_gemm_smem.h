// The shared-memory form of the prefill GEMM (qmm_gemm_smem.cu), dispatched by qmm_gemm.cu.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "qmm_common.cuh"

namespace qmm {

constexpr int GEMM_SMEM_BOX_ROWS = 128;  // token rows of its tensor map's box

// CTAs that share one group of 256 tokens: one wave over the SMs, at most 16 row tiles each.
int gemm_smem_groups(int rt, int64_t m, int sm_count);
cudaError_t launch_gemm_smem(const WeightView& w, const CUtensorMap& xmap, void* y, int64_t m, int out, int groups,
                             bool keep_order, int* status, cudaStream_t stream);

}  // namespace qmm
