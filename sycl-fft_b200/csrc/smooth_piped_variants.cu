// Instantiations of the copy-engine-pipelined 7-smooth kernels (smooth_piped_catalog.h), compiled once per
// SFB_SPIPED_PART so that the parts build in parallel.
#include "smooth_launch.hpp"
#include "smooth_piped.cuh"
#include "smooth_piped_catalog.h"

#define SFB_CAT2(a, b) a##b
#define SFB_CAT(a, b) SFB_CAT2(a, b)

namespace sfb {

const SmoothKernel* SFB_CAT(smooth_piped_part_, SFB_SPIPED_PART)(int* count) {
    static const SmoothKernel kernels[] = {
#define SFB_X(ID, DBL, KIND, FEAT, N, TPL, W, PADS, PITCH, MAXT, MINB, ...) \
    {ID, reinterpret_cast<const void*>(&fft_smooth_piped_kernel<float, N, TPL, PADS, PITCH, FEAT, MAXT, MINB, __VA_ARGS__>)},
        SFB_CAT(SFB_SPIPED_PART_, SFB_SPIPED_PART)(SFB_X)
#undef SFB_X
    };
    *count = static_cast<int>(sizeof(kernels) / sizeof(kernels[0]));
    return kernels;
}

}  // namespace sfb
