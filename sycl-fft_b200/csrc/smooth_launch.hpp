// Host entry into the size-specialised kernels of the 7-smooth lengths (smooth_variants.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "planner.hpp"
#include "smooth_kernel.cuh"
#include "smooth_piped.cuh"

namespace sfb {

// Launches a catalog entry over n_outer outer indices; p.n_cols, its strides and tables are set by
// the caller, the tile geometry (w, col_tiles) here.
cudaError_t launch_smooth(const SmoothEntry& e, SmoothParams p, int64_t n_outer, int sms, const void* in, void* out,
                          cudaStream_t stream);

// Runs p.n_cols whole lines on a smooth_piped_catalog.h kernel; buffers and input pitch are multiples of 16
// bytes. `status` is set to 1 when a copy is not there after `wait_polls` polls.
cudaError_t launch_smooth_piped(const SmoothEntry& e, const SmoothParams& p, int sms, int* status, long long wait_polls,
                                const void* in, void* out, cudaStream_t stream);

// Loads the kernel that a pass of this size takes (the pipelined form), so that its first launch need not.
cudaError_t prepare_smooth(const SmoothEntry& e, int64_t n_cols, int64_t n_outer);
cudaError_t prepare_smooth_piped(const SmoothEntry& e);

// One kernel of a compiled part of the catalog (nullptr: in another object of the part).
struct SmoothKernel {
    int id;
    const void* fn;
};

}  // namespace sfb
