// Instantiations of the Bluestein and Rader pass kernels (conv_catalog.h), compiled once per SFB_CONV_PART.
#include <type_traits>

#include "conv_catalog.h"
#include "conv_kernel.cuh"
#include "conv_launch.hpp"

#define SFB_CAT2(a, b) a##b
#define SFB_CAT(a, b) SFB_CAT2(a, b)

namespace sfb {
namespace {

// Features by 4 * rader + kind: fused single pass, forward columns, row convolution, inverse columns.
constexpr int kConvFeat[8] = {kFeatPremul | kFeatConv | kFeatPostmul, kFeatPremul | kFeatTw4,
                              kFeatConv | kFeatTw4 | kFeatTw4Conj, kFeatPostmul,
                              kFeatGather | kFeatConv | kFeatScatter | kFeatRaderDC, kFeatGather | kFeatTw4,
                              kFeatConv | kFeatTw4 | kFeatTw4Conj | kFeatRaderDC, kFeatScatter};

}  // namespace

const ConvKernel* SFB_CAT(conv_part_, SFB_CONV_PART)(int* count) {
    static const ConvKernel kernels[] = {
#define SFB_X(ID, DBL, KIND, RADER, N, TPL, W, PADS, PITCH, MAXT, MINB, COST, ...)                                           \
    {ID, reinterpret_cast<const void*>(                                                                                 \
             &fft_conv_kernel<std::conditional_t<(DBL) != 0, double, float>, N, TPL, (KIND) == 1 || (KIND) == 3, W, PADS, \
                              PITCH, kConvFeat[(RADER) * 4 + (KIND)], MAXT, MINB, __VA_ARGS__>)},
        SFB_CAT(SFB_CONV_PART_, SFB_CONV_PART)(SFB_X)
#undef SFB_X
    };
    *count = static_cast<int>(sizeof(kernels) / sizeof(kernels[0]));
    return kernels;
}

}  // namespace sfb
