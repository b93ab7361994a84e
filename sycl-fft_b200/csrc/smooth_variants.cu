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

}  // namespace sfb
