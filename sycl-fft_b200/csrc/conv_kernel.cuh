// Passes of the convolution transforms (Bluestein, Rader) on the building blocks of smooth_kernel.cuh. The
// hooks are those of fixed_kernel.cuh (FixedParams and its kFeat bits):
//
//   load : zero padding and chirp pre-multiply, or the Rader gather;
//   mid  : spectrum multiply between two FFTs (kFeatConv), and the Rader bin-0 term;
//   store: four-step twiddle, chirp post-multiply with truncation, or the Rader scatter.
//
// A convolution runs its second FFT on the reversed radix sequence: the last stage of the first FFT
// leaves element j + r * N/R of the spectrum in the registers of the thread whose first butterfly of the
// second FFT reads exactly those, so the spectrum multiply and that butterfly follow in registers, and
// one exchange of the 2S - 1 of an S-stage pair falls away (row convolutions of 256 points, float, 16.8 M
// points: 77 -> 66 us; double, 8.4 M points: 80 -> 64 us).
//
// What bounds it: exchanges and issue slots (convolution kernels run at 100 to 270 G points/s in float, HBM
// would allow about 400; the 65537-point rows: issue 77%, load/store data pipe 71%), the Rader gather and scatter the
// 32-byte sectors their 8- or 16-byte accesses take (65537 points x 256, float: 109 and 103 us of 285 to 298).
// Convolution lengths are chosen by the passes' timed cost per point (conv_catalog.h): the smallest length is often
// slower than one a little longer (double 28927: 210 x 288 = 60480 points 227 us, 64 x 960 = 61440 points 192 us).
// Against the kernels of bluestein_catalog.h, 106 primes from 11 to 65537 at 32 MB: 1.24x float, 1.13x double
// (geometric means; none slower).
#pragma once

#include <cuda_runtime.h>

#include "fixed_kernel.cuh"
#include "smooth_kernel.cuh"

namespace sfb {

template <class T>
struct ConvCtx {
    using C = cplx<T>;
    C* row;  // this thread's line in shared memory
    const C* gin;
    C* gout;
    const C* tw;
    int t;
    bool act, ok;
    int64_t in_ks, out_ks;
    T scale;
    bool conj_in, conj_out, conj_mid, flip_in, flip_out;
    int sel;
    const C *tw4_hi, *tw4_lo;
    int tw4_shift;
    T tw4_sy;
    const C *premul, *postmul, *pw;
    int g_k, in_len, out_len;
    const int *perm_in, *perm_out;
    const int* sidx;  // MODEC scatter: this column's entries of perm_out in shared memory, element k at k * W
    const C* gline;
    C* gline_out;
    const C* rx;
    C* ry;
    T dc_scale;
    bool dc_flip_in, dc_flip_out;
};

// The first stage's elements j + r * NR.
template <int FEAT, bool MODEC, int R, int NR, class T, class C>
__device__ __forceinline__ void conv_load(ConvCtx<T>& X, int j, C* v) {
    if constexpr (FEAT & kFeatGather) {
        // all indices first, then all gathers: one round trip each
        int src[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int g = (j + r * NR) * X.g_k + X.sel;
            src[r] = X.ok && g < X.in_len ? __ldg(X.perm_in + g) : -1;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            v[r] = cmake<C>(T(0), T(0));
            if (src[r] >= 0) v[r] = X.gline[src[r]];
            if (X.flip_in != X.conj_in) v[r].y = -v[r].y;
        }
    } else if constexpr (FEAT & kFeatPremul) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int k = j + r * NR, g = k * X.g_k + X.sel;
            C a = cmake<C>(T(0), T(0));
            if (X.ok && g < X.in_len) {
                a = X.gin[MODEC ? static_cast<int64_t>(k) * X.in_ks : k];
                if (X.flip_in) a.y = -a.y;
                a = cmul(a, __ldg(X.premul + g));
                if (X.conj_in) a.y = -a.y;
            }
            v[r] = a;
        }
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int k = j + r * NR;
            C a = cmake<C>(T(0), T(0));
            if (X.ok) a = X.gin[MODEC ? static_cast<int64_t>(k) * X.in_ks : k];
            if (X.conj_in) a.y = -a.y;
            v[r] = a;
        }
    }
}

// The last stage's outputs k = j + r * NR.
template <int FEAT, bool MODEC, int W, int R, int NR, class T, class C>
__device__ __forceinline__ void conv_store(ConvCtx<T>& X, int j, C* u) {
    if (!X.ok) return;
    if constexpr (FEAT & kFeatTw4) {
        SmoothCtx<T> Y;
        Y.sel = X.sel;
        Y.tw4_hi = X.tw4_hi;
        Y.tw4_lo = X.tw4_lo;
        Y.tw4_shift = X.tw4_shift;
        Y.tw4_sy = X.tw4_sy;
        smooth_tw4<R, NR>(u, Y, j);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int k = j + r * NR, g = k * X.g_k + X.sel;
        C a = u[r];
        if (X.conj_out) a.y = -a.y;
        if constexpr (FEAT & kFeatPostmul) {
            if (g >= X.out_len) continue;
            a = cmul(a, __ldg(X.postmul + g));
        }
        if constexpr (FEAT & kFeatScatter) {
            if (g >= X.out_len) continue;
        }
        a.x *= X.scale;
        a.y *= X.scale;
        if constexpr (FEAT & (kFeatPostmul | kFeatScatter)) {
            if (X.flip_out) a.y = -a.y;
        }
        if constexpr ((FEAT & kFeatScatter) && MODEC) X.gline_out[X.sidx[k * W]] = a;
        else if constexpr (FEAT & kFeatScatter) X.gline_out[__ldg(X.perm_out + g)] = a;
        else X.gout[MODEC ? static_cast<int64_t>(k) * X.out_ks : k] = a;
    }
}

// Spectrum multiply of the values k = j + r * NR (and the Rader bin-0 term at k = 0 of row 0).
template <int FEAT, int R, int NR, class T, class C>
__device__ __forceinline__ void conv_mid(ConvCtx<T>& X, int j, C* u) {
    C dc = cmake<C>(T(0), T(0));
    if constexpr (FEAT & kFeatRaderDC) {
        if (X.sel == 0 && j == 0 && X.ok) {
            dc = X.rx[0];
            if (X.dc_flip_in) dc.y = -dc.y;
            C y0 = cmake<C>((dc.x + u[0].x) * X.dc_scale, (dc.y + u[0].y) * X.dc_scale);
            if (X.dc_flip_out) y0.y = -y0.y;
            X.ry[0] = y0;
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        u[r] = cmul(u[r], __ldg(X.pw + j + r * NR));
        if constexpr (FEAT & kFeatRaderDC) {
            if (r == 0) {
                u[0].x += dc.x;
                u[0].y += dc.y;
            }
        }
        if (X.conj_mid) u[r].y = -u[r].y;
    }
}

// One radix-R stage; MID: the last stage of the first FFT of a convolution, followed by the spectrum
// multiply and the first butterfly of the second FFT.
template <class T, int N, int TPL, bool MODEC, int W, int PADS, int FEAT, int NS, int TWOFF, int R, bool FIRST, bool LAST,
          bool MID>
__device__ __forceinline__ void conv_stage(ConvCtx<T>& X) {
    using C = cplx<T>;
    constexpr int NR = N / R, NB = (NR + TPL - 1) / TPL, PAD = PADS ? 1 << PADS : 1;
    constexpr bool EXACT = (NR % TPL) == 0, LIN_IN = PADS == 0 || NR % PAD == 0;
    C v[NB * R];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int j = X.t + i * TPL;
        if (X.act && (EXACT || i + 1 < NB || j < NR)) {
            if constexpr (FIRST) {
                conv_load<FEAT, MODEC, R, NR>(X, j, &v[i * R]);
            } else if constexpr (LIN_IN) {
                const C* p = X.row + smooth_idx<PADS>(j);
#pragma unroll
                for (int r = 0; r < R; ++r) v[i * R + r] = p[r * (NR + (PADS ? NR / PAD : 0))];
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) v[i * R + r] = X.row[smooth_idx<PADS>(j + r * NR)];
            }
        }
    }
    if constexpr (!FIRST && !LAST) __syncthreads();
    // the indices this thread's own copies brought (conv_fetch_scatter)
    if constexpr (LAST && MODEC && (FEAT & kFeatScatter)) cp_async_commit_wait_all();
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int j = X.t + i * TPL;
        if (X.act && (EXACT || i + 1 < NB || j < NR)) {
            C* u = &v[i * R];
            const int jm = LAST || MID ? j : j % NS;
            if constexpr (NS > 1) smooth_twiddle<R, NS>(u, X.tw + TWOFF, jm);
            dft<R, T>(u);
            if constexpr (LAST) {
                conv_store<FEAT, MODEC, W, R, NR>(X, j, u);
            } else {
                constexpr int NSO = MID ? 1 : NS;  // the second FFT starts over at Ns = 1
                if constexpr (MID) {
                    conv_mid<FEAT, R, NR>(X, j, u);
                    dft<R, T>(u);
                }
                const int base = MID ? j * R : (j - jm) * R + jm;
                if constexpr (PADS == 0 || NSO % PAD == 0 || (R * NSO <= PAD && PAD % (R * NSO) == 0)) {
                    C* p = X.row + smooth_idx<PADS>(base);
#pragma unroll
                    for (int r = 0; r < R; ++r) p[r * NSO + (PADS ? (r * NSO) / PAD : 0)] = u[r];
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) X.row[smooth_idx<PADS>(base + r * NSO)] = u[r];
                }
            }
        }
    }
    if constexpr (!LAST) __syncthreads();
}

// Stages IDX.. of the sequence R[0..S-1]; CONV: then the second FFT over R[S-1], .., R[0].
template <int S>
struct ConvRadices {
    int r[S];
};

template <class T, int N, int TPL, bool MODEC, int W, int PADS, int FEAT, int NS, int TWOFF, int IDX, int... Rs>
__device__ __forceinline__ void conv_forward(ConvCtx<T>& X) {
    constexpr int S = sizeof...(Rs);
    constexpr ConvRadices<S> seq{{Rs...}};
    constexpr int R = seq.r[IDX];
    constexpr bool CONV = (FEAT & kFeatConv) != 0, END = IDX == S - 1;
    conv_stage<T, N, TPL, MODEC, W, PADS, FEAT, NS, TWOFF, R, IDX == 0, END && !CONV, END && CONV>(X);
    if constexpr (!END)
        conv_forward<T, N, TPL, MODEC, W, PADS, FEAT, NS * R, TWOFF + NS * smooth_tw_entries(R), IDX + 1, Rs...>(X);
}

// Second FFT, stages after its first: IDX counts down.
template <class T, int N, int TPL, bool MODEC, int W, int PADS, int FEAT, int NS, int TWOFF, int IDX, int... Rs>
__device__ __forceinline__ void conv_backward(ConvCtx<T>& X) {
    constexpr int S = sizeof...(Rs);
    constexpr ConvRadices<S> seq{{Rs...}};
    constexpr int R = seq.r[IDX];
    conv_stage<T, N, TPL, MODEC, W, PADS, FEAT, NS, TWOFF, R, false, IDX == 0, false>(X);
    if constexpr (IDX > 0)
        conv_backward<T, N, TPL, MODEC, W, PADS, FEAT, NS * R, TWOFF + NS * smooth_tw_entries(R), IDX - 1, Rs...>(X);
}

// The column's scatter indices perm_out[k * g_k + c], asynchronously into shared memory while the stages
// run; each thread fetches the ones its own last stage stores through, so no barrier is needed.
template <int N, int TPL, int W, int... Rs, class T>
__device__ __forceinline__ void conv_fetch_scatter(ConvCtx<T>& X, int* sidx) {
    constexpr int S = sizeof...(Rs);
    constexpr ConvRadices<S> seq{{Rs...}};
    constexpr int R = seq.r[S - 1], NR = N / R;
    if (X.ok)
        for (int j = X.t; j < NR; j += TPL)
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int k = j + r * NR, g = k * X.g_k + X.sel;
                if (g < X.out_len) cp_async4(sidx + k * W, X.perm_out + g);
            }
    cp_async_commit_only();
    X.sidx = sidx;
}

// Table entries of the sequence (the second FFT's table follows the first's).
template <int NS>
__host__ __device__ constexpr int conv_table() { return 0; }
template <int NS, int R, int... Rest>
__host__ __device__ constexpr int conv_table() { return NS * smooth_tw_entries(R) + conv_table<NS * R, Rest...>(); }

// grid: MODEC n_outer * col_tiles blocks of round_up(W * TPL, 32), else tiles of w lines, block >= w * TPL;
// dynamic smem: lines * PITCH complex values, column scatters also N * W ints.
template <class T, int N, int TPL, bool MODEC, int W, int PADS, int PITCH, int FEAT, int MAXT, int MINB, int... Rs>
__global__ void __launch_bounds__(MAXT, MINB)
    fft_conv_kernel(const __grid_constant__ FixedParams P, const cplx<T>* in, cplx<T>* out) {
    using C = cplx<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* sm = reinterpret_cast<C*>(smem_raw);
    ConvCtx<T> X;
    X.tw = static_cast<const C*>(P.tw);
    X.scale = static_cast<T>(P.scale);
    X.conj_in = P.conj_in != 0;
    X.conj_out = P.conj_out != 0;
    X.conj_mid = P.conj_mid != 0;
    X.flip_in = P.flip_in != 0;
    X.flip_out = P.flip_out != 0;
    X.premul = static_cast<const C*>(P.premul);
    X.postmul = static_cast<const C*>(P.postmul);
    X.g_k = P.g_k;
    X.in_len = P.in_len;
    X.out_len = P.out_len;
    X.perm_in = P.perm_in;
    X.perm_out = P.perm_out;
    X.tw4_hi = static_cast<const C*>(P.tw4_hi);
    X.tw4_lo = static_cast<const C*>(P.tw4_lo);
    X.tw4_shift = P.tw4_shift;
    // the store conjugates after the twiddle: conj(u) * w = conj(u * conj(w))
    X.tw4_sy = (((FEAT & kFeatTw4Conj) != 0) != X.conj_out) ? T(-1) : T(1);
    X.in_ks = P.in_ks;
    X.out_ks = P.out_ks;
    const int tid = threadIdx.x;
    if constexpr (MODEC) {
        const int w = tid % W;
        X.t = tid / W;
        X.act = X.t < TPL;
        const int64_t tile = blockIdx.x;
        const int64_t o = tile / P.col_tiles;
        const int64_t c = (tile - o * P.col_tiles) * W + w;
        X.ok = X.act && c < P.n_cols;
        X.sel = static_cast<int>(c);
        X.row = sm + w * PITCH;
        X.gin = in + o * P.in_hi + c;
        X.gout = out + o * P.out_hi + c;
        X.gline = in + o * P.in_hi;
        X.gline_out = out + o * P.out_hi;
        if constexpr (FEAT & kFeatScatter)
            conv_fetch_scatter<N, TPL, W, Rs...>(X, reinterpret_cast<int*>(sm + W * PITCH) + w);
    } else {
        const int w = tid / TPL;
        X.t = tid - w * TPL;
        X.act = w < P.w;
        const int64_t c = static_cast<int64_t>(blockIdx.x) * P.w + w;
        X.ok = X.act && c < P.n_cols;
        X.row = sm + w * PITCH;
        X.gin = in + c * P.in_pitch;
        X.gout = out + c * P.out_pitch;
        X.gline = X.gin;
        X.gline_out = X.gout;
        X.sel = P.rows > 1 ? static_cast<int>(c % P.rows) : 0;
        if constexpr (FEAT & kFeatRaderDC) {
            if constexpr (FEAT & kFeatGather) {  // the whole line: its own scale and flips
                X.rx = X.gin;
                X.ry = X.gout;
                X.dc_scale = X.scale;
                X.dc_flip_in = X.flip_in;
                X.dc_flip_out = X.flip_out;
            } else {  // row c of the three-pass form is row c % rows of line c / rows
                const int64_t o = c / P.rows;
                X.rx = static_cast<const C*>(P.dc_x) + o * P.dc_x_pitch;
                X.ry = static_cast<C*>(P.dc_y) + o * P.dc_y_pitch;
                X.dc_scale = static_cast<T>(P.dc_scale);
                X.dc_flip_in = P.dc_flip_in != 0;
                X.dc_flip_out = P.dc_flip_out != 0;
            }
        }
    }
    if constexpr (FEAT & kFeatConv) X.pw = static_cast<const C*>(P.pointwise) + static_cast<int64_t>(X.sel) * P.pw_stride;
    conv_forward<T, N, TPL, MODEC, W, PADS, FEAT, 1, 0, 0, Rs...>(X);
    if constexpr (FEAT & kFeatConv) {
        constexpr int S = sizeof...(Rs);
        constexpr ConvRadices<S> seq{{Rs...}};
        constexpr int R = seq.r[S - 1], OFF = conv_table<1, Rs...>() + smooth_tw_entries(R);
        conv_backward<T, N, TPL, MODEC, W, PADS, FEAT, R, OFF, S - 2, Rs...>(X);
    }
}

}  // namespace sfb
