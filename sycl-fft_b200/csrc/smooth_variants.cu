// Instantiations of the size-specialised kernels of the 7-smooth lengths (smooth_catalog.h). Compiled once per
// SFB_SMOOTH_PART and SFB_SMOOTH_SUB (every third entry of the part), so that the parts build in parallel and load
// separately (kernel_set.hpp); with SFB_SMOOTH_RUN the run-on forms of a part's plain columns instead.
#include <type_traits>

#include "smooth_catalog.h"
#include "smooth_kernel.cuh"
#include "smooth_launch.hpp"

#define SFB_CAT2(a, b) a##b
#define SFB_CAT(a, b) SFB_CAT2(a, b)

namespace sfb {
namespace {

template <class T, int N, int TPL, int KIND, int W, int PADS, int PITCH, int FEAT, int MAXT, int MINB, int... Rs>
struct Entry {
    // the entry itself where `take`, else nullptr
    template <bool take>
    static const void* plain() {
        if constexpr (take)
            return reinterpret_cast<const void*>(&fft_smooth_kernel<T, N, TPL, KIND, W, PADS, PITCH, FEAT, MAXT, MINB, Rs...>);
        else return nullptr;
    }
    // its run-on form (plain columns of more than two lines per tile: smooth_runs_on)
    static const void* run() {
        if constexpr (KIND == kSmoothCC && FEAT == 0 && W > 2)
            return reinterpret_cast<const void*>(
                &fft_smooth_kernel<T, N, TPL, KIND, W, PADS, PITCH, kSmoothRun, MAXT, MINB, Rs...>);
        else return nullptr;
    }
};

}  // namespace

#define SFB_ENTRY(DBL, KIND, FEAT, N, TPL, W, PADS, PITCH, MAXT, MINB, ...) \
    Entry<std::conditional_t<(DBL) != 0, double, float>, N, TPL, KIND, W, PADS, PITCH, FEAT, MAXT, MINB, __VA_ARGS__>
#ifdef SFB_SMOOTH_RUN
#define SFB_NAME SFB_CAT(smooth_run_part_, SFB_SMOOTH_PART)
#define SFB_X(ID, DBL, KIND, FEAT, N, TPL, W, PADS, PITCH, MAXT, MINB, ...) \
    {ID, SFB_ENTRY(DBL, KIND, FEAT, N, TPL, W, PADS, PITCH, MAXT, MINB, __VA_ARGS__)::run()},
#else
#define SFB_NAME SFB_CAT(SFB_CAT(smooth_part_, SFB_SMOOTH_PART), SFB_CAT(_, SFB_SMOOTH_SUB))
#define SFB_X(ID, DBL, KIND, FEAT, N, TPL, W, PADS, PITCH, MAXT, MINB, ...) \
    {ID, SFB_ENTRY(DBL, KIND, FEAT, N, TPL, W, PADS, PITCH, MAXT, MINB, __VA_ARGS__)::plain<(ID) % 3 == SFB_SMOOTH_SUB>()},
#endif

const SmoothKernel* SFB_NAME(int* count) {
    static const SmoothKernel kernels[] = {SFB_CAT(SFB_SMOOTH_PART_, SFB_SMOOTH_PART)(SFB_X)};
    *count = static_cast<int>(sizeof(kernels) / sizeof(kernels[0]));
    return kernels;
}

}  // namespace sfb
