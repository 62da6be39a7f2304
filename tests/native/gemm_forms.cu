// Lets the tests ask which form of the prefill GEMM a product takes and run one form of their choice: the plan functions of
// qmm_kernels.h behind a C interface, linked against libqmm_b200.so.
#include "../../litenn_b200/csrc/qmm_internal.h"
#include "../../litenn_b200/csrc/qmm_kernels.h"

using namespace qmm;

extern "C" {

// out = {nb, tokens, t_tiles, splits, groups} of the plan for an [n, k] weight; needs no GPU
void gemm_plan_of(int64_t n, int64_t k, int64_t m, int sm_count, int keep_order, int* out)
{
    WeightView w = {};
    w.n = n;
    w.k = k;
    w.rt = (int)((n + 15) / 16);
    w.kc = (int)((k + 255) / 256);
    const GemmPlan p = plan_gemm(w, m, sm_count, keep_order != 0);
    out[0] = p.nb;
    out[1] = p.tokens;
    out[2] = p.t_tiles;
    out[3] = p.splits;
    out[4] = p.groups;
}

// One form (gemm_form's nb, tokens and splits) on the weight's device; the launch's CUDA error code
int gemm_run_form(const qmm_weight* weight, const void* x_bf16, void* y, int64_t m, int out, int nb, int tokens, int splits,
                  int keep_order, void* stream)
{
    WeightView w;
    int dev = 0, sms = 0, *status = nullptr;
    if (qmm_internal_weight_view(weight, &w) || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        qmm_internal_status_word(dev, &status)) {
        return -1;
    }
    if (nb < 0 || nb > 2 || (nb > 0 && (tokens < 16 || tokens > 128 || tokens % 16 != 0)) || splits < 1 || splits > w.kc ||
        splits > (nb == 1 ? 8 : 1) || (splits & (splits - 1)) != 0) {
        return -2;
    }
    const char* why = nullptr;
    return (int)launch_gemm_plan(gemm_form(w, m, sms, nb, tokens, splits), w, x_bf16, y, m, out, keep_order != 0, status,
                                 static_cast<cudaStream_t>(stream), &why);
}

}  // extern "C"
