// Kernels of a catalog compiled in parts, and their launch: lookup by id, loading and shared-memory opt-in once
// per kernel and device.
//
// A kernel is loaded on its first use, and with the first of an object file its index: 3.1 ms for files of 140
// kernels, 1.1 ms of 50 (B200, driver 580). The files are therefore small, and a plan loads its kernels when it is
// made (prepare): its first execute, of 3000 float points for instance, takes 0.1 ms instead of 3.3.
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
            if (k[i].fn) fn_[k[i].id] = k[i].fn;
        }
    }
    void finish() { ready_ = std::vector<std::atomic<unsigned char>>(fn_.size() * kMaxDevices); }

    // Loads the kernel on the current device and opts it into smem_max, the most any launch of it takes.
    cudaError_t prepare(int id, size_t smem_max) {
        if (id < 0 || static_cast<size_t>(id) >= fn_.size() || !fn_[id]) return cudaErrorInvalidDeviceFunction;
        int dev = 0;
        cudaError_t err = cudaGetDevice(&dev);
        if (err != cudaSuccess) return err;
        if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
        std::atomic<unsigned char>& ready = ready_[static_cast<size_t>(id) * kMaxDevices + dev];
        if (ready.load(std::memory_order_acquire)) return cudaSuccess;
        if (smem_max > 48 * 1024) {
            err = cudaFuncSetAttribute(fn_[id], cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_max));
        } else {
            cudaFuncAttributes attr;
            err = cudaFuncGetAttributes(&attr, fn_[id]);
        }
        if (err == cudaSuccess) ready.store(1, std::memory_order_release);
        return err;
    }

    // smem: this launch's dynamic shared memory; smem_max: the most any launch of the kernel takes.
    cudaError_t launch(int id, int64_t grid, int threads, size_t smem, size_t smem_max, void** args, cudaStream_t stream) {
        if (id < 0 || static_cast<size_t>(id) >= fn_.size() || !fn_[id]) return cudaErrorInvalidDeviceFunction;
        if (grid <= 0 || grid > INT_MAX) return cudaErrorInvalidConfiguration;
        if (smem > 48 * 1024) {
            const cudaError_t err = prepare(id, smem_max);
            if (err != cudaSuccess) return err;
        }
        return cudaLaunchKernel(fn_[id], dim3(static_cast<unsigned>(grid)), dim3(static_cast<unsigned>(threads)), args, smem,
                                stream);
    }

private:
    static constexpr int kMaxDevices = 64;
    std::vector<const void*> fn_;                    // by catalog id
    std::vector<std::atomic<unsigned char>> ready_;  // [id * kMaxDevices + device]: loaded, shared memory opted in
};

// Lines per block of a whole-line kernel: the catalog's, fewer while that leaves SMs without a block.
inline int lines_per_block(int w, int64_t lines, int sms) {
    while (w > 1 && (lines + w - 1) / w < sms) w = (w + 1) / 2;
    return w;
}

}  // namespace sfb
