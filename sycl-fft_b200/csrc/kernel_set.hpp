// Kernels of a catalog compiled in parts, and their launch: lookup by id, shared-memory opt-in once per
// kernel and device.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <climits>
#include <cstdint>
#include <vector>

namespace sfb {

class KernelSet {
public:
    template <class Kernel>
    void add(const Kernel* (*part)(int*)) {
        int n = 0;
        const Kernel* k = part(&n);
        for (int i = 0; i < n; ++i) {
            if (static_cast<size_t>(k[i].id) >= fn_.size()) fn_.resize(k[i].id + 1, nullptr);
            fn_[k[i].id] = k[i].fn;
        }
    }
    void finish() { ready_ = std::vector<std::atomic<unsigned char>>(fn_.size() * kMaxDevices); }

    // smem: this launch's dynamic shared memory; smem_max: the most any launch of the kernel takes.
    cudaError_t launch(int id, int64_t grid, int threads, size_t smem, size_t smem_max, void** args, cudaStream_t stream) {
        if (id < 0 || static_cast<size_t>(id) >= fn_.size() || !fn_[id]) return cudaErrorInvalidDeviceFunction;
        if (grid <= 0 || grid > INT_MAX) return cudaErrorInvalidConfiguration;
        if (smem > 48 * 1024) {
            int dev = 0;
            cudaError_t err = cudaGetDevice(&dev);
            if (err != cudaSuccess) return err;
            if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
            std::atomic<unsigned char>& ready = ready_[static_cast<size_t>(id) * kMaxDevices + dev];
            if (!ready.load(std::memory_order_acquire)) {
                err = cudaFuncSetAttribute(fn_[id], cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_max));
                if (err != cudaSuccess) return err;
                ready.store(1, std::memory_order_release);
            }
        }
        return cudaLaunchKernel(fn_[id], dim3(static_cast<unsigned>(grid)), dim3(static_cast<unsigned>(threads)), args, smem,
                                stream);
    }

private:
    static constexpr int kMaxDevices = 64;
    std::vector<const void*> fn_;                    // by catalog id
    std::vector<std::atomic<unsigned char>> ready_;  // [id * kMaxDevices + device]: shared memory opted in
};

// Lines per block of a whole-line kernel: the catalog's, fewer while that leaves SMs without a block.
inline int lines_per_block(int w, int64_t lines, int sms) {
    while (w > 1 && (lines + w - 1) / w < sms) w = (w + 1) / 2;
    return w;
}

}  // namespace sfb
