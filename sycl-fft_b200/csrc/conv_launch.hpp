// Host entry into the Bluestein and Rader pass kernels of conv_catalog.h (conv_variants.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "fixed_kernel.cuh"
#include "planner.hpp"

namespace sfb {

// Launches a catalog entry; p carries the pass (its table p.tw: conv_twiddles), the tile geometry (w,
// col_tiles) is set here.
cudaError_t launch_conv(const ConvEntry& e, FixedParams p, int64_t n_outer, int sms, const void* in, void* out,
                        cudaStream_t stream);

struct ConvKernel {
    int id;
    const void* fn;
};

}  // namespace sfb
