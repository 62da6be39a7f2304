// Lets the tests ask how a matvec of one row is launched: the rules of qmm_kernels.h and qmm_gemv_forms.cuh behind a C
// interface, linked against libqmm_b200.so.
#include <algorithm>
#include <map>
#include <set>
#include <tuple>

#include "../../litenn_b200/csrc/qmm_gemv_forms.cuh"
#include "../../litenn_b200/csrc/qmm_kernels.h"

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
    return epi == EPI_RESID_PACK    ? gemv_one_wave<FMT, EPI_RESID_PACK>(w.rt, w.kc, chained, sms)
           : epi == EPI_SWIGLU_PACK ? gemv_one_wave<FMT, EPI_SWIGLU_PACK>(w.rt, w.kc, chained, sms)
                                    : gemv_one_wave<FMT, EPI_STORE>(w.rt, w.kc, chained, sms);
}

// Stands where the library launches: notes the chosen form, and in `compiled` every form that was instantiated.
template <int FMT, int EPI, bool XF32>
struct Note {
    int* out;
    static std::set<std::tuple<int, int, int>>& compiled()
    {
        static std::set<std::tuple<int, int, int>> forms;
        return forms;
    }
    template <int TILES, int WARPS, int DEPTH>
    struct Known {
        static inline const bool yes = compiled().insert({TILES, WARPS, DEPTH}).second;
    };
    template <int TILES, int WARPS, int DEPTH>
    cudaError_t form() const
    {
        out[0] = TILES;
        out[1] = WARPS;
        out[2] = DEPTH;
        out[3] = Known<TILES, WARPS, DEPTH>::yes ? 1 : 0;
        return cudaSuccess;
    }
};

// The form of one shape, or -1 where the one-wave form is not taken
template <int FMT, int EPI, bool XF32>
int choose(int rt, int kc, bool chained, int sms, int* out)
{
    const bool taken = XF32 ? gemv_packs_itself_shape(FMT, rt, kc, sms) : gemv_one_wave<FMT, EPI>(rt, kc, chained, sms);
    return taken ? (int)gemv_wave_form<FMT, EPI, XF32>(rt, kc, sms, Note<FMT, EPI, XF32>{out}) : -1;
}

// Walks rows and chunks; returns how many compiled forms no shape reached, -1 if a chosen form does not fit or covers too little
template <int FMT, int EPI, bool XF32>
int walk(int sms)
{
    auto forms = Note<FMT, EPI, XF32>::compiled();
    for (int rt = 1; rt <= 29 * sms; ++rt) {
        for (int kc = 1; kc <= 130; ++kc) {
            for (int chained = 0; chained < (EPI == EPI_STORE && !XF32 ? 2 : 1); ++chained) {
                int out[4] = {};
                const int rc = choose<FMT, EPI, XF32>(rt, kc, chained != 0, sms, out);
                if (rc == -1) {
                    continue;
                }
                const int nw = out[0] * out[1], slots = nw * out[2] * tile_bytes(FMT);
                const int smem = slots + (nw * out[2] + 1) * 8 + kc * XPK1_REC + 512 + nw * 64;
                if (rc != 0 || (int64_t)out[0] * sms < rt || out[0] % epi_tiles(EPI) != 0 || nw > 32 || smem > GEMV_SMEM_LIMIT ||
                    !Note<FMT, EPI, XF32>::compiled().count({out[0], out[1], out[2]})) {
                    return -1;
                }
                forms.erase({out[0], out[1], out[2]});
            }
        }
    }
    return (int)forms.size();
}

// Smallest shapes that reach each form, {TILES, WARPS, DEPTH, rt, kc, chained} each: one of any length and one whose warps refill
// every slot; returns their number
template <int FMT, int EPI, bool XF32>
int shapes(int sms, int* out, int room)
{
    std::map<std::tuple<int, int, int, bool>, std::tuple<int64_t, int, int, int>> best;
    for (int rt = epi_tiles(EPI); rt <= 29 * sms; rt += epi_tiles(EPI)) {
        for (int kc = 1; kc <= GEMV_WAVE_KC; ++kc) {
            for (int chained = 0; chained < (EPI == EPI_STORE && !XF32 ? 2 : 1); ++chained) {
                int f[4] = {};
                if (choose<FMT, EPI, XF32>(rt, kc, chained != 0, sms, f) != 0) {
                    continue;
                }
                for (int refilled = 0; refilled < (kc >= 2 * f[1] * f[2] ? 2 : 1); ++refilled) {
                    auto& b = best[{f[0], f[1], f[2], refilled != 0}];
                    if (std::get<0>(b) == 0 || std::get<0>(b) > (int64_t)rt * kc) {
                        b = {(int64_t)rt * kc, rt, kc, chained};
                    }
                }
            }
        }
    }
    int n = 0;
    for (const auto& [form, shape] : best) {
        if (n < room) {
            const int row[6] = {std::get<0>(form), std::get<1>(form), std::get<2>(form),
                                std::get<1>(shape), std::get<2>(shape), std::get<3>(shape)};
            std::copy(row, row + 6, out + 6 * n++);
        }
    }
    return n;
}

template <int FMT>
int shapes_of(int epi, bool xf32, int sms, int* out, int room)
{
    return xf32                     ? shapes<FMT, EPI_STORE, true>(sms, out, room)
           : epi == EPI_RESID_PACK  ? shapes<FMT, EPI_RESID_PACK, false>(sms, out, room)
           : epi == EPI_SWIGLU_PACK ? shapes<FMT, EPI_SWIGLU_PACK, false>(sms, out, room)
                                    : shapes<FMT, EPI_STORE, false>(sms, out, room);
}

template <int FMT>
int walk_format(int epi, bool xf32, int sms)
{
    return xf32                     ? walk<FMT, EPI_STORE, true>(sms)
           : epi == EPI_RESID_PACK  ? walk<FMT, EPI_RESID_PACK, false>(sms)
           : epi == EPI_SWIGLU_PACK ? walk<FMT, EPI_SWIGLU_PACK, false>(sms)
                                    : walk<FMT, EPI_STORE, false>(sms);
}

}  // namespace

extern "C" {

// One-wave forms that are compiled and that no shape takes, of one format and epilogue; -1: a shape has no fitting form
int gemv_wave_forms_unreached(int fmt, int epi, int xf32, int sm_count)
{
    return fmt == FMT_Q4_0   ? walk_format<FMT_Q4_0>(epi, xf32 != 0, sm_count)
           : fmt == FMT_Q8_0 ? walk_format<FMT_Q8_0>(epi, xf32 != 0, sm_count)
           : fmt == FMT_Q4_K ? walk_format<FMT_Q4_K>(epi, xf32 != 0, sm_count)
                             : walk_format<FMT_Q6_K>(epi, xf32 != 0, sm_count);
}

int gemv_wave_shapes(int fmt, int epi, int xf32, int sm_count, int* out, int room)
{
    return fmt == FMT_Q4_0   ? shapes_of<FMT_Q4_0>(epi, xf32 != 0, sm_count, out, room)
           : fmt == FMT_Q8_0 ? shapes_of<FMT_Q8_0>(epi, xf32 != 0, sm_count, out, room)
           : fmt == FMT_Q4_K ? shapes_of<FMT_Q4_K>(epi, xf32 != 0, sm_count, out, room)
                             : shapes_of<FMT_Q6_K>(epi, xf32 != 0, sm_count, out, room);
}

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
