// Launch of the size-specialised kernels of the 7-smooth lengths: kernel lookup, shared-memory
// opt-in and tile geometry.
#include <atomic>
#include <climits>
#include <vector>

#include "smooth_catalog.h"
#include "smooth_launch.hpp"

namespace sfb {

#define SFB_EACH_PART(F) F(0) F(1) F(2) F(3) F(4) F(5) F(6) F(7) F(8) F(9) F(10) F(11) F(12) F(13) F(14) F(15) \
    F(16) F(17) F(18) F(19) F(20) F(21) F(22) F(23)
static_assert(SFB_SMOOTH_PARTS == 24, "SFB_EACH_PART lists the parts");

#define SFB_DECL(P) const SmoothKernel* smooth_part_##P(int* count);
SFB_EACH_PART(SFB_DECL)
#undef SFB_DECL

namespace {

constexpr int kMaxDevices = 64;

struct Kernels {
    std::vector<const void*> fn;                   // by catalog id
    std::vector<std::atomic<unsigned char>> ready;  // [id * kMaxDevices + device]: shared memory opted in
    Kernels() {
        auto add = [&](const SmoothKernel* (*part)(int*)) {
            int n = 0;
            const SmoothKernel* k = part(&n);
            for (int i = 0; i < n; ++i) {
                if (static_cast<size_t>(k[i].id) >= fn.size()) fn.resize(k[i].id + 1, nullptr);
                fn[k[i].id] = k[i].fn;
            }
        };
#define SFB_ADD(P) add(smooth_part_##P);
        SFB_EACH_PART(SFB_ADD)
#undef SFB_ADD
        ready = std::vector<std::atomic<unsigned char>>(fn.size() * kMaxDevices);
    }
};

Kernels& kernels() {
    static Kernels k;
    return k;
}

}  // namespace

cudaError_t launch_smooth(const SmoothEntry& e, SmoothParams p, int64_t n_outer, int sms, const void* in, void* out,
                          cudaStream_t stream) {
    Kernels& ks = kernels();
    if (e.id < 0 || static_cast<size_t>(e.id) >= ks.fn.size() || !ks.fn[e.id]) return cudaErrorInvalidDeviceFunction;
    p.w = e.w;
    int threads = e.maxt;
    if (e.kind == kSmoothKK) {
        // fewer lines per block while that leaves SMs without one
        while (p.w > 1 && (p.n_cols + p.w - 1) / p.w < sms) p.w = (p.w + 1) / 2;
        threads = (p.w * e.tpl + 31) / 32 * 32;
    }
    p.col_tiles = (p.n_cols + p.w - 1) / p.w;
    const int64_t grid = n_outer * p.col_tiles;
    if (grid <= 0 || grid > INT_MAX) return cudaErrorInvalidConfiguration;
    const size_t cs = e.dbl ? 16 : 8;
    const size_t smem = static_cast<size_t>(p.w) * e.pitch * cs;
    if (smem > 48 * 1024) {
        int dev = 0;
        cudaError_t err = cudaGetDevice(&dev);
        if (err != cudaSuccess) return err;
        if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
        std::atomic<unsigned char>& ready = ks.ready[static_cast<size_t>(e.id) * kMaxDevices + dev];
        if (!ready.load(std::memory_order_acquire)) {
            err = cudaFuncSetAttribute(ks.fn[e.id], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(static_cast<size_t>(e.w) * e.pitch * cs));
            if (err != cudaSuccess) return err;
            ready.store(1, std::memory_order_release);
        }
    }
    void* args[] = {&p, const_cast<void**>(&in), &out};
    return cudaLaunchKernel(ks.fn[e.id], dim3(static_cast<unsigned>(grid)), dim3(static_cast<unsigned>(threads)), args, smem,
                            stream);
}

}  // namespace sfb
