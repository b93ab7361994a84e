// Host entry into the size-specialised kernels of the 7-smooth lengths (smooth_variants.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "planner.hpp"
#include "smooth_kernel.cuh"

namespace sfb {

// Launches a catalog entry over n_outer outer indices; p.n_cols, its strides and tables are set by
// the caller, the tile geometry (w, col_tiles) here.
cudaError_t launch_smooth(const SmoothEntry& e, SmoothParams p, int64_t n_outer, int sms, const void* in, void* out,
                          cudaStream_t stream);

// One kernel of a compiled part of the catalog.
struct SmoothKernel {
    int id;
    const void* fn;
};

}  // namespace sfb
