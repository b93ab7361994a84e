// Instantiations of the Bluestein and Rader pass kernels (conv_catalog.h), compiled once per SFB_CONV_PART and
// SFB_CONV_SUB (every other entry of the part), as in smooth_variants.cu.
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

template <bool take, class T, int KIND, int RADER, int N, int TPL, int W, int PADS, int PITCH, int MAXT, int MINB, int... Rs>
const void* kernel() {
    if constexpr (take)
        return reinterpret_cast<const void*>(&fft_conv_kernel<T, N, TPL, KIND == 1 || KIND == 3, W, PADS, PITCH,
                                                              kConvFeat[RADER * 4 + KIND], MAXT, MINB, Rs...>);
    else return nullptr;
}

}  // namespace

const ConvKernel* SFB_CAT(SFB_CAT(conv_part_, SFB_CONV_PART), SFB_CAT(_, SFB_CONV_SUB))(int* count) {
    static const ConvKernel kernels[] = {
#define SFB_X(ID, DBL, KIND, RADER, N, TPL, W, PADS, PITCH, MAXT, MINB, COST, ...)                                          \
    {ID, kernel<(ID) % 2 == SFB_CONV_SUB, std::conditional_t<(DBL) != 0, double, float>, KIND, RADER, N, TPL, W, PADS, PITCH, \
                MAXT, MINB, __VA_ARGS__>()},
        SFB_CAT(SFB_CONV_PART_, SFB_CONV_PART)(SFB_X)
#undef SFB_X
    };
    *count = static_cast<int>(sizeof(kernels) / sizeof(kernels[0]));
    return kernels;
}

}  // namespace sfb
