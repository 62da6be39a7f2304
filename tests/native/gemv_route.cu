// Lets the tests ask how a matvec of one fp32 vector is launched: the rules of qmm_kernels.h behind a C interface, linked
// against libqmm_b200.so.
#include "../../litenn_b200/csrc/qmm_kernels.h"

using namespace qmm;

extern "C" {

// Whether y = W[n, k] * x is one launch; x and y are addresses that nothing reads
int gemv_one_launch(int fmt, int64_t n, int64_t k, uint64_t x, uint64_t y, int sm_count)
{
    WeightView w = {};
    w.fmt = fmt;
    w.n = n;
    w.k = k;
    w.rt = (int)((n + 15) / 16);
    w.kc = (int)((k + 255) / 256);
    return gemv_packs_itself(w, reinterpret_cast<const float*>(x), reinterpret_cast<const float*>(y), sm_count) ? 1 : 0;
}

// Whether gate|up of `channels` channels writes its product packed
int swiglu_packs(int channels, int64_t k, int sm_count)
{
    return gemv_swiglu_packs((channels + 7) / 8, (int)((k + 255) / 256), sm_count) ? 1 : 0;
}

}  // extern "C"
