// Instantiations of the size-specialised kernels of the 7-smooth lengths (smooth_catalog.h), compiled
// once per SFB_SMOOTH_PART so that the parts build in parallel.
#include <type_traits>

#include "smooth_catalog.h"
#include "smooth_kernel.cuh"
#include "smooth_launch.hpp"

#define SFB_CAT2(a, b) a##b
#define SFB_CAT(a, b) SFB_CAT2(a, b)

namespace sfb {

const SmoothKernel* SFB_CAT(smooth_part_, SFB_SMOOTH_PART)(int* count) {
    static const SmoothKernel kernels[] = {
#define SFB_X(ID, DBL, KIND, FEAT, N, TPL, W, PADS, PITCH, MAXT, MINB, ...)                                       \
    {ID, reinterpret_cast<const void*>(&fft_smooth_kernel<std::conditional_t<(DBL) != 0, double, float>, N, TPL, \
                                                          KIND, W, PADS, PITCH, FEAT, MAXT, MINB, __VA_ARGS__>)},
        SFB_CAT(SFB_SMOOTH_PART_, SFB_SMOOTH_PART)(SFB_X)
#undef SFB_X
    };
    *count = static_cast<int>(sizeof(kernels) / sizeof(kernels[0]));
    return kernels;
}

// The run-on form of a plain column entry with more than two lines per tile (of two, a tile of one column
// would be half idle: contiguous lines), nullptr for the others.
template <class T, int N, int TPL, int KIND, int W, int PADS, int PITCH, int FEAT, int MAXT, int MINB, int... Rs>
static const void* run_on() {
    if constexpr (KIND == kSmoothCC && FEAT == 0 && W > 2)
        return reinterpret_cast<const void*>(
            &fft_smooth_kernel<T, N, TPL, KIND, W, PADS, PITCH, kSmoothRun, MAXT, MINB, Rs...>);
    else return nullptr;
}

const SmoothKernel* SFB_CAT(smooth_run_part_, SFB_SMOOTH_PART)(int* count) {
    static const SmoothKernel kernels[] = {
#define SFB_X(ID, DBL, KIND, FEAT, N, TPL, W, PADS, PITCH, MAXT, MINB, ...) \
    {ID, run_on<std::conditional_t<(DBL) != 0, double, float>, N, TPL, KIND, W, PADS, PITCH, FEAT, MAXT, MINB, __VA_ARGS__>()},
        SFB_CAT(SFB_SMOOTH_PART_, SFB_SMOOTH_PART)(SFB_X)
#undef SFB_X
    };
    *count = static_cast<int>(sizeof(kernels) / sizeof(kernels[0]));
    return kernels;
}

}  // namespace sfb
