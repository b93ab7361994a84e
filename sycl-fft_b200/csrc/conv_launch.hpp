// Host entry into the Bluestein and Rader pass kernels of conv_catalog.h (conv_variants.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "fixed_kernel.cuh"
#include "planner.hpp"

namespace sfb {

// Launches a catalog entry; p carries the pass (its table p.tw: the rows of smooth_twiddles over the entry's radices,
// then, for convolutions, over their reverse), the tile geometry (w, col_tiles) is set here.
cudaError_t launch_conv(const ConvEntry& e, FixedParams p, int64_t n_outer, int sms, const void* in, void* out,
                        cudaStream_t stream);

// Loads the kernel, so that its first launch need not.
cudaError_t prepare_conv(const ConvEntry& e);

struct ConvKernel {
    int id;
    const void* fn;
};

}  // namespace sfb
