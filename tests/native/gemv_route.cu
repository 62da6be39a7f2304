// Lets the tests ask how a matvec of one row is launched: the rules of qmm_kernels.h and qmm_gemv_kernel.cuh behind a C
// interface, linked against libqmm_b200.so.
#include "../../litenn_b200/csrc/qmm_gemv_kernel.cuh"

using namespace qmm;

namespace {

WeightView shape(int fmt, int64_t n, int64_t k)
{
    WeightView w = {};
    w.fmt = fmt;
    w.n = n;
    w.k = k;
    w.rt = (int)((n + 15) / 16);
    w.kc = (int)((k + 255) / 256);
    return w;
}

template <int FMT>
bool one_wave(int epi, const WeightView& w, bool chained, int sms)
{
    return epi == EPI_RESID_PACK    ? gemv_one_wave<FMT, EPI_RESID_PACK>(w, chained, sms)
           : epi == EPI_SWIGLU_PACK ? gemv_one_wave<FMT, EPI_SWIGLU_PACK>(w, chained, sms)
                                    : gemv_one_wave<FMT, EPI_STORE>(w, chained, sms);
}

}  // namespace

extern "C" {

// Whether a packed vector takes the one-wave form; epi as in qmm_common.cuh
int gemv_takes_one_wave(int fmt, int epi, int64_t n, int64_t k, int chained, int sm_count)
{
    const WeightView w = shape(fmt, n, k);
    return fmt == FMT_Q4_0   ? one_wave<FMT_Q4_0>(epi, w, chained != 0, sm_count)
           : fmt == FMT_Q8_0 ? one_wave<FMT_Q8_0>(epi, w, chained != 0, sm_count)
           : fmt == FMT_Q4_K ? one_wave<FMT_Q4_K>(epi, w, chained != 0, sm_count)
                             : one_wave<FMT_Q6_K>(epi, w, chained != 0, sm_count);
}

// Whether y = W[n, k] * x is one launch; x and y are addresses that nothing reads
int gemv_one_launch(int fmt, int64_t n, int64_t k, uint64_t x, uint64_t y, int sm_count)
{
    const WeightView w = shape(fmt, n, k);
    return gemv_packs_itself(w, reinterpret_cast<const float*>(x), reinterpret_cast<const float*>(y), sm_count) ? 1 : 0;
}

// Whether gate|up of `channels` channels writes its product packed
int swiglu_packs(int channels, int64_t k, int sm_count)
{
    return gemv_swiglu_packs((channels + 7) / 8, (int)((k + 255) / 256), sm_count) ? 1 : 0;
}

}  // extern "C"
