// Persistent, copy-engine-pipelined form of smooth_kernel.cuh for long contiguous lines.
//
// Of the long lines one or two blocks fit an SM, by their shared memory or (radices above 16) by their
// registers, and a plain kernel alternates load -> exchanges -> store with the HBM idle during the
// exchanges. Here each CTA is persistent and owns two buffers: a copy buffer, filled by the bulk-copy engine
// (cp.async.bulk, completion on an mbarrier) with the next line as it is in HBM, and a work buffer for the
// exchanges. The first stage reads the copy buffer into registers and writes the work buffer; right after
// it, the copy engine is told to fetch the following line into the copy buffer, so that load hides behind
// the remaining stages, and the last stage's stores drain during the next line. R2C lines take the same
// road: their input is the half-length complex line.
//
// Taken by the even lengths that timed at least 5% below the plain kernel (56 of 228; 128 MB of lines: 1.16x
// complex, 1.15x R2C; 12544 points 80 -> 66 us), where there are more lines than SMs: the first line of a CTA
// hides behind nothing. Pipelined over plain time, the 56 entries at 38 line counts: from 149 to 444 lines 0.82 to
// 1.19, 0.99 in the geometric mean (a half-full last round costs either form more or less), from 445 lines 0.91, from
// 1185 0.90. A higher line would cost the lengths that gain from the first line on (12544 points: 0.87 at 180 lines)
// what it gives the others (12096: 1.14). R2C 26880 x 4096: 307 -> 249 to 253 us, bound by the exchanges of one CTA
// per SM (three stages and the pairs' pass: issue 52%, load/store data pipe 54%, DRAM 36%). Shorter lines mostly
// lose: two copy buffers per SM displace blocks.
//
// Waits on the copy are bounded: after Q.wait_polls polls the CTA records a timeout in the
// plan's status word, lets the copy it gave up on land (bounded again by kSpinLimit, so no
// copy into its shared memory outlives it) and stops (all threads agree through a barrier
// first).
#pragma once

#include <cuda_runtime.h>

#include "async_util.cuh"
#include "smooth_kernel.cuh"

namespace sfb {

struct SmoothPipedParams {
    SmoothParams s;         // n_cols lines; in_cs * sizeof(C) is a multiple of 16
    int* status = nullptr;  // set to 1 if a copy wait timed out
    long long wait_polls = kSpinLimit;  // polls before a copy wait gives up
};

constexpr uint32_t kLineChunks = 4;  // bulk copies per line

template <class T, int N, int TPL, int PADS, int PITCH, int FEAT, int R0, int... Rest>
__device__ __forceinline__ void smooth_piped_first(SmoothCtx<T>& X) {
    smooth_stage<T, N, TPL, kSmoothKK, 1, PADS, PITCH, FEAT, 1, 0, R0, true, false>(X);
}

// The stages after the first.
template <class T, int N, int TPL, int PADS, int PITCH, int FEAT, int R0, int... Rest>
__device__ __forceinline__ void smooth_piped_rest(SmoothCtx<T>& X) {
    smooth_stages<T, N, TPL, kSmoothKK, 1, PADS, PITCH, FEAT, R0, smooth_tw_entries(R0), false, Rest...>(X);
    if constexpr (FEAT & kSmoothPost) smooth_post<T, N, TPL, PADS, PITCH>(X);
}

// Dynamic shared memory of a float line: copy buffer, work buffer, barrier.
constexpr int64_t smooth_piped_smem(int n, int pitch) { return (int64_t(n) + pitch) * 8 + 16; }

// grid <= lines; block = MAXT threads (TPL rounded up to whole warps).
template <class T, int N, int TPL, int PADS, int PITCH, int FEAT, int MAXT, int MINB, int... Rs>
__global__ void __launch_bounds__(MAXT, MINB)
    fft_smooth_piped_kernel(const __grid_constant__ SmoothPipedParams Q, const cplx<T>* in, cplx<T>* out) {
    using C = cplx<T>;
    constexpr uint32_t kLineBytes = N * sizeof(C);
    constexpr uint32_t kChunk = kLineBytes / kLineChunks / 16 * 16, kLast = kLineBytes - (kLineChunks - 1) * kChunk;
    static_assert(kLineBytes % 16 == 0 && sizeof...(Rs) >= 2 && (FEAT & ~kSmoothPost) == 0, "whole lines of 16-byte multiples");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SmoothParams& P = Q.s;
    C* const copy = reinterpret_cast<C*>(smem_raw);
    uint64_t* const bar = reinterpret_cast<uint64_t*>(smem_raw + kLineBytes + PITCH * sizeof(C));
    const int t = threadIdx.x;

    SmoothCtx<T> X;
    X.sm = copy + N;
    X.gin = copy;
    X.tw = static_cast<const C*>(P.tw);
    X.real_tw = static_cast<const C*>(P.real_tw);
    X.t_in = X.t_out = t;
    X.w_in = X.w_out = 0;
    X.in_ok = X.out_ok = X.act_in = X.act_out = t < TPL;
    X.in_ks = X.out_ks = 1;
    X.in_sy = P.conj_in ? T(-1) : T(1);
    X.sx = static_cast<T>(P.scale);
    X.sy = P.conj_out ? -X.sx : X.sx;

    auto fetch = [&](int64_t line) {
        mbar_expect_tx(bar, kLineBytes);
        const unsigned char* src = reinterpret_cast<const unsigned char*>(in + line * P.in_cs);
#pragma unroll
        for (uint32_t c = 0; c < kLineChunks; ++c)
            bulk_g2s(smem_raw + c * kChunk, src + c * kChunk, c + 1 < kLineChunks ? kChunk : kLast, bar);
    };
    if (t == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (blockIdx.x < P.n_cols) fetch(blockIdx.x);
    }
    __syncthreads();

    uint32_t parity = 0;
    for (int64_t line = blockIdx.x; line < P.n_cols; line += gridDim.x) {
        const bool ok = mbar_wait_bounded(bar, parity, Q.wait_polls);
        if (__syncthreads_or(!ok)) {
            if (t == 0) {
                report_status(Q.status, 1);
                // the only copy in flight is the one given up on: let it land before the
                // shared memory is released
                mbar_wait_bounded(bar, parity, kSpinLimit);
            }
            __syncthreads();
            return;
        }
        parity ^= 1u;
        X.gout = out + line * P.out_cs;
        smooth_piped_first<T, N, TPL, PADS, PITCH, FEAT, Rs...>(X);  // ends with a barrier: the copy buffer is consumed
        const int64_t next = line + gridDim.x;
        if (t == 0 && next < P.n_cols) {
            fence_proxy_async();  // order the generic reads of the copy buffer before the copy
            fetch(next);
        }
        smooth_piped_rest<T, N, TPL, PADS, PITCH, FEAT, Rs...>(X);
        __syncthreads();  // the work buffer is free for the next line's first stage
    }
}

}  // namespace sfb
