// Size-specialised pass kernels of the 7-smooth lengths (smooth_catalog.h): the Stockham register /
// shared-memory scheme of fixed_kernel.cuh, with length, radices, threads per line and shared-memory rows
// fixed at compile time, for every length instead of a list of powers of two, and with
//
//  * a thread mapping per side. "K": lanes walk the elements of a line (element stride 1), "C": lanes walk W
//    adjacent lines (line stride 1). KK whole contiguous lines, CC strided columns, CK columns stored as
//    rows and KC rows stored as columns (the transposed store of a four-step's rows). The mapping turns at
//    the first (CK) or the last (KC) exchange, so a layout change costs no shared-memory trip of its own.
//  * radices 6, 9, 10, 12, 14 and 15 next to the powers of two and 3, 5, 7, so that lengths with odd
//    factors take three or four stages instead of five to seven; an odd radix first where there is one:
//    its exchange then falls in distinct banks without padding, which saves the padding's address
//    arithmetic in every stage (3000 points x 16384, bare launches on one card: [8, 15, 5, 5] padded 196 us,
//    [15, 8, 5, 5] without 166 us).
//  * float radices to 32 at up to 128 registers a thread: 256 to 1024 points in two stages, longer lines in
//    three. Shared-memory traffic and barriers fall with every exchange, and the values in flight per SM rise.
//    [15, 8, 5, 5] -> [25, 10, 12] in the same launches: 166 -> 160 us; 810 x 840 four-step [9, 9, 10] and
//    [15, 4, 14] -> [27, 30] and [30, 28]: 680400 x 64 360 -> 310 to 326 us; 1024 columns -> rows [16, 8, 8] ->
//    [32, 32]: 240 -> 209 to 224 us (ranges: several cards). 869 of the 1820 float entries, those that gained at
//    least 1.5%: 1.15x (geometric mean). Packed two-value additions (add.f32x2) in their place gave nothing: the
//    exchanges, not the arithmetic, fill the time.
//  * up to 16 values a thread in double too, at 128 registers and half the threads: the same bytes in
//    flight with one exchange less (2048 points: [8, 8, 8, 4] 180 us, [16, 16, 8] 168 us per 1.07 GB).
//
// What bounds it: HBM for the lines up to about 2000 points (4.9 to 6.4 of the 6.5 TB/s copy rate), the issue slots
// and exchanges of the longer ones (3000 points: issue 67%, load/store data pipe 64%, DRAM 56%; 4096: 63, 61 and
// 64%), one or two blocks of the longest of which fill an SM. Times per execute on B200 against the runtime-length
// kernels: 3000 x 16384 float 338 -> 155 to 161 us, 680400 x 64 float (810 x 840 four-step) 640 -> 316 to 326 us,
// 840 x 1200 x 4 float 101 -> 34 us; complex<double> 65536 x 512 (256 x 256) 402 to 421 -> 341 to 357 us against
// fixed_kernel.cuh. The catalog's 680 whole-line lengths: 2.06x (geometric mean, 64 MB), columns of 64-column arrays
// 1.9x (354 lengths), four-steps to 2^20 1.78x (619 lengths), real lines 2.4x (681); none of them slower.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "butterfly.cuh"
#include "pass_params.h"

namespace sfb {

struct SmoothParams {
    int64_t n_cols = 1;     // lines per outer index
    int64_t col_tiles = 1;  // ceil(n_cols / w)
    int w = 1;              // lines per CTA (KK; the other mappings use the compile-time W)
    int run_cols = 0;       // kSmoothRun: columns per outer index; n_cols then counts the lines of all outer indices
    int64_t in_hi = 0, in_cs = 0, in_ks = 1;     // element (o, c, k) at o * hi + c * cs + k * ks
    int64_t out_hi = 0, out_cs = 0, out_ks = 1;  // (K sides: ks = 1; C sides: cs = 1)
    const void* tw = nullptr;  // stage twiddles (smooth_tw_entries)
    int conj_in = 0, conj_out = 0;
    double scale = 1.0;
    // four-step column pass (CC): output k of column c times W_L^(k*c) = hi[m >> shift] * lo[m & mask]
    const void* tw4_hi = nullptr;
    const void* tw4_lo = nullptr;
    int tw4_shift = 0, tw4_conj = 0;
    const void* real_tw = nullptr;  // W_2N^k, k = 0..N (real transforms of length 2N)
};

// Twiddles of one butterfly, u[r] *= w^r with w = W_(Ns*R)^jm. The table holds w, w^2, w^4 and w^8 for every
// jm (rows of Ns entries, so lanes read them coalesced) and the other powers take at most two products: the error of a
// full table (3000 points: 1.2e-7, 1.7e-7 from the powers of w alone) for 1% (4096 points, three stages of 16) to 7%
// (3000 points as [15, 8, 5, 5]) more time than the powers alone, where a full table's R - 1 loads took another 4%.
template <int R, int NS, class C>
__device__ __forceinline__ void smooth_twiddle(C* u, const C* __restrict__ tw, int jm) {
    const C w1 = __ldg(tw + jm);
    u[1] = cmul(u[1], w1);
    if constexpr (R > 2) {
        const C w2 = __ldg(tw + NS + jm);
        u[2] = cmul(u[2], w2);
        if constexpr (R > 3) u[3] = cmul(u[3], cmul(w2, w1));
        if constexpr (R > 4) {
            const C w4 = __ldg(tw + 2 * NS + jm);
            u[4] = cmul(u[4], w4);
            if constexpr (R > 5) u[5] = cmul(u[5], cmul(w4, w1));
            if constexpr (R > 6) {
                const C w6 = cmul(w4, w2);
                u[6] = cmul(u[6], w6);
                if constexpr (R > 7) u[7] = cmul(u[7], cmul(w6, w1));
            }
            if constexpr (R > 8) {
                const C w8 = __ldg(tw + 3 * NS + jm);
                u[8] = cmul(u[8], w8);
                if constexpr (R > 9) u[9] = cmul(u[9], cmul(w8, w1));
                if constexpr (R > 10) u[10] = cmul(u[10], cmul(w8, w2));
                if constexpr (R > 11) u[11] = cmul(u[11], cmul(cmul(w8, w2), w1));
                if constexpr (R > 12) {
                    const C w12 = cmul(w8, w4);
                    u[12] = cmul(u[12], w12);
                    if constexpr (R > 13) u[13] = cmul(u[13], cmul(w12, w1));
                    if constexpr (R > 14) u[14] = cmul(u[14], cmul(w12, w2));
                    if constexpr (R > 15) u[15] = cmul(u[15], cmul(cmul(w12, w2), w1));
                }
            }
        }
    }
}

// Radices above 16: the power 4h + s is one product of the rows w^(4h) and w^s (s = 1, 2, 3), so that no power
// is more than one product away from the table and few of them are live beside the values. Over 43 lengths
// from 324 to 10^6 points the errors against FP64 are 0.9 to 1.04 times those of full tables (products
// of w, w^2, w^4, w^8 and w^16: 1.6e-7 against 1.4e-7 at one length).
template <int R, int NS, class C>
__device__ __forceinline__ void smooth_twiddle_wide(C* u, const C* __restrict__ tw, int jm) {
    const C w1 = __ldg(tw + jm), w2 = __ldg(tw + NS + jm), w3 = __ldg(tw + 2 * NS + jm);
    u[1] = cmul(u[1], w1);
    u[2] = cmul(u[2], w2);
    u[3] = cmul(u[3], w3);
#pragma unroll
    for (int h = 1; 4 * h < R; ++h) {
        const C b = __ldg(tw + (2 + h) * NS + jm);
        u[4 * h] = cmul(u[4 * h], b);
        if (4 * h + 1 < R) u[4 * h + 1] = cmul(u[4 * h + 1], cmul(b, w1));
        if (4 * h + 2 < R) u[4 * h + 2] = cmul(u[4 * h + 2], cmul(b, w2));
        if (4 * h + 3 < R) u[4 * h + 3] = cmul(u[4 * h + 3], cmul(b, w3));
    }
}

template <int PADS>
__device__ __forceinline__ int smooth_idx(int k) {
    if constexpr (PADS == 0) return k;
    else return k + (k >> PADS);
}

template <class T>
struct SmoothCtx {
    using C = cplx<T>;
    C* sm;          // tile base in shared memory
    const C* gin;   // this thread's line in the input (first-stage mapping)
    C* gout;        // and in the output (last-stage mapping)
    const C* tw;
    int t_in, w_in, t_out, w_out;  // lane of the line, line of the tile, under the two mappings
    bool in_ok, out_ok;            // the line exists
    bool act_in, act_out;          // the thread belongs to a line
    int64_t in_ks, out_ks;
    T in_sy, sx, sy;               // input conjugation, output scale
    int sel;
    const C *tw4_hi, *tw4_lo;
    int tw4_shift;
    T tw4_sy;
    const C* real_tw;
};

// Four-step twiddles of one butterfly's outputs k = j + r * NR of column c: W^(k*c) = W^(j*c) * s^r with
// s = W^(NR*c). s, s^2, s^4, s^8 come from the two-level table (one lookup each per thread: they do not
// depend on j), the products form a binary tree, so an output is at most four roundings away from
// the table and the scattered table reads are 1 + 4 / NB per butterfly instead of R.
template <class T, class C = cplx<T>>
__device__ __forceinline__ C smooth_tw4_at(const SmoothCtx<T>& X, int m) {
    C q = cmul(__ldg(X.tw4_hi + (m >> X.tw4_shift)), __ldg(X.tw4_lo + (m & ((1 << X.tw4_shift) - 1))));
    q.y *= X.tw4_sy;
    return q;
}

template <int R, int NR, class T, class C>
__device__ __forceinline__ void smooth_tw4(C* u, const SmoothCtx<T>& X, int j) {
    C q[R < 8 ? R : 8];
    q[0] = smooth_tw4_at(X, j * X.sel);
#pragma unroll
    for (int b = 1; b < 8 && b < R; b *= 2) {
        const C s = smooth_tw4_at(X, b * NR * X.sel);
#pragma unroll
        for (int r = b; r < 2 * b && r < R; ++r) q[r] = cmul(q[r - b], s);
    }
#pragma unroll
    for (int r = 0; r < R && r < 8; ++r) u[r] = cmul(u[r], q[r]);
    if constexpr (R > 8) {
        const C s = smooth_tw4_at(X, 8 * NR * X.sel);
        C t = s;
#pragma unroll
        for (int r = 8; r < R; ++r) {
            if (r == 16) t = smooth_tw4_at(X, 16 * NR * X.sel);
            if (r == 24) t = cmul(t, s);
            u[r] = cmul(u[r], cmul(q[r & 7], t));
        }
    }
}

// KIND: the mapping pair; a stage's reads and writes use the mapping of its phase. Shared memory
// holds one row of PITCH elements per line, one padding element per 2^PADS (0: none).
template <class T, int N, int TPL, int KIND, int W, int PADS, int PITCH, int FEAT, int NS, int TWOFF, int R, bool FIRST,
          bool LAST>
__device__ __forceinline__ void smooth_stage(SmoothCtx<T>& X) {
    using C = cplx<T>;
    constexpr int NR = N / R;
    constexpr int NB = (NR + TPL - 1) / TPL;
    constexpr bool EXACT = (NR % TPL) == 0;
    // the mapping of this stage: KC turns before its last stage, CK after its first
    constexpr bool INMAP = KIND == kSmoothKC ? !LAST : FIRST || KIND == kSmoothKK || KIND == kSmoothCC;
    constexpr bool CMAP = KIND == kSmoothCC || (KIND == kSmoothCK && FIRST) || (KIND == kSmoothKC && LAST);
    constexpr int PAD = PADS ? (1 << PADS) : 1;
    constexpr bool LIN_IN = PADS == 0 || NR % PAD == 0;
    const int t = INMAP ? X.t_in : X.t_out;
    const int w = INMAP ? X.w_in : X.w_out;
    const bool act = INMAP ? X.act_in : X.act_out;
    C* const row = X.sm + w * PITCH;
    C v[NB * R];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int j = t + i * TPL;
        if (act && (EXACT || i + 1 < NB || j < NR)) {
            if constexpr (FIRST && !(FEAT & kSmoothPre)) {
                if (X.in_ok) {
                    const C* g = CMAP ? X.gin + (int64_t)j * X.in_ks : X.gin + j;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        C a = CMAP ? g[(int64_t)(r * NR) * X.in_ks] : g[r * NR];
                        a.y *= X.in_sy;
                        v[i * R + r] = a;
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) v[i * R + r] = cmake<C>(T(0), T(0));
                }
            } else if constexpr (LIN_IN) {
                const C* p = row + smooth_idx<PADS>(j);
#pragma unroll
                for (int r = 0; r < R; ++r) v[i * R + r] = p[r * (NR + (PADS ? NR / PAD : 0))];
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) v[i * R + r] = row[smooth_idx<PADS>(j + r * NR)];
            }
        }
    }
    if constexpr ((!FIRST || (FEAT & kSmoothPre)) && !LAST) __syncthreads();
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int j = t + i * TPL;
        if (act && (EXACT || i + 1 < NB || j < NR)) {
            C* u = &v[i * R];
            const int jm = LAST ? j : j % NS;
            if constexpr (NS > 1 && R > 16) smooth_twiddle_wide<R, NS>(u, X.tw + TWOFF, jm);
            else if constexpr (NS > 1) smooth_twiddle<R, NS>(u, X.tw + TWOFF, jm);
            dft<R, T>(u);
            if constexpr (LAST && (FEAT & kSmoothPost)) {
                // over the elements this thread read; the bins are formed from pairs after a barrier
#pragma unroll
                for (int r = 0; r < R; ++r) row[smooth_idx<PADS>(j + r * NR)] = u[r];
            } else if constexpr (LAST) {
                if (X.out_ok) {
                    if constexpr (FEAT & kSmoothTw4) smooth_tw4<R, NR>(u, X, j);
                    C* g = CMAP ? X.gout + (int64_t)j * X.out_ks : X.gout + j;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        C a = u[r];
                        a.x *= X.sx;
                        a.y *= X.sy;
                        if constexpr (CMAP) g[(int64_t)(r * NR) * X.out_ks] = a;
                        else g[r * NR] = a;
                    }
                }
            } else {
                const int base = (j - jm) * R + jm;
                if constexpr (PADS == 0 || NS % PAD == 0 || (R * NS <= PAD && PAD % (R * NS) == 0)) {
                    C* p = row + smooth_idx<PADS>(base);
#pragma unroll
                    for (int r = 0; r < R; ++r) p[r * NS + (PADS ? (r * NS) / PAD : 0)] = u[r];
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) row[smooth_idx<PADS>(base + r * NS)] = u[r];
                }
            }
        }
    }
    if constexpr (!LAST) __syncthreads();
}

template <class T, int N, int TPL, int KIND, int W, int PADS, int PITCH, int FEAT, int NS, int TWOFF, bool FIRST, int R,
          int... Rest>
__device__ __forceinline__ void smooth_stages(SmoothCtx<T>& X) {
    constexpr bool LAST = sizeof...(Rest) == 0;
    smooth_stage<T, N, TPL, KIND, W, PADS, PITCH, FEAT, NS, TWOFF, R, FIRST, LAST>(X);
    if constexpr (!LAST)
        smooth_stages<T, N, TPL, KIND, W, PADS, PITCH, FEAT, NS * R, TWOFF + NS * smooth_tw_entries(R), false, Rest...>(
            X);
}

// Real transforms: bins k and N - k of each line from its spectrum in shared memory, and the reverse. One
// thread takes the pair, so each value moves once and the two bins share their arithmetic; the loads of a
// group of pairs are issued before the first is used.
template <class T, int N, int TPL, int PADS, int PITCH>
__device__ __forceinline__ void smooth_post(SmoothCtx<T>& X) {
    using C = cplx<T>;
    constexpr int NP = N / 2 + 1, G = 4;
    __syncthreads();
    if (!X.out_ok) return;
    const T half = T(0.5) * X.sx;
    const C* row = X.sm + X.w_out * PITCH;
    for (int k0 = X.t_out; k0 < NP; k0 += G * TPL) {
        C a[G], c[G], w[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int k = k0 + g * TPL, kk = N - k;
            if (k < NP) {
                w[g] = __ldg(X.real_tw + k);
                a[g] = row[smooth_idx<PADS>(k)];
                c[g] = row[smooth_idx<PADS>(k == 0 ? 0 : kk)];
            }
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int k = k0 + g * TPL, kk = N - k;
            if (k < NP) {
                real_post_both(a[g], c[g], w[g], half);
                X.gout[k] = a[g];
                if (kk != k) X.gout[kk] = c[g];
            }
        }
    }
}

template <class T, int N, int TPL, int PADS, int PITCH>
__device__ __forceinline__ void smooth_pre(SmoothCtx<T>& X) {
    using C = cplx<T>;
    constexpr int NP = N / 2 + 1, G = sizeof(T) == 4 ? 6 : 4;
    C* row = X.sm + X.w_in * PITCH;
    if (X.act_in) {
        for (int k0 = X.t_in; k0 < NP; k0 += G * TPL) {
            C a[G], c[G], w[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int k = k0 + g * TPL;
                a[g] = c[g] = w[g] = cmake<C>(T(0), T(0));
                if (k < NP && X.in_ok) {
                    a[g] = X.gin[k];
                    c[g] = X.gin[N - k];
                    w[g] = __ldg(X.real_tw + k);
                }
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int k = k0 + g * TPL, kk = N - k;
                if (k < NP) {
                    if (k == 0) a[g].y = c[g].y = T(0);  // bins 0 and N of a real signal are real
                    real_pre_both(a[g], c[g], w[g]);
                    a[g].y *= X.in_sy;
                    c[g].y *= X.in_sy;
                    row[smooth_idx<PADS>(k)] = a[g];
                    if (kk != k && k > 0) row[smooth_idx<PADS>(kk)] = c[g];
                }
            }
        }
    }
    __syncthreads();
}

// grid = n_outer * col_tiles; KK: block >= w * TPL, other mappings: block = round_up(W * TPL, 32);
// dynamic smem: lines * PITCH complex values.
template <class T, int N, int TPL, int KIND, int W, int PADS, int PITCH, int FEAT, int MAXT, int MINB, int... Rs>
__global__ void __launch_bounds__(MAXT, MINB)
    fft_smooth_kernel(const __grid_constant__ SmoothParams P, const cplx<T>* in, cplx<T>* out) {
    using C = cplx<T>;
    static_assert(!(FEAT & (kSmoothPost | kSmoothPre)) || KIND == kSmoothKK, "whole contiguous lines");
    static_assert(!(FEAT & kSmoothRun) || (KIND == kSmoothCC && FEAT == kSmoothRun), "plain columns");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmoothCtx<T> X;
    X.sm = reinterpret_cast<C*>(smem_raw);
    X.tw = static_cast<const C*>(P.tw);
    X.in_sy = P.conj_in ? T(-1) : T(1);
    X.sx = static_cast<T>(P.scale);
    // output conjugation: the sign of the imaginary part's scale, and of the four-step twiddle
    // (conj(u) * w = conj(u * conj(w)))
    X.sy = P.conj_out ? -X.sx : X.sx;
    X.in_ks = P.in_ks;
    X.out_ks = P.out_ks;
    X.real_tw = static_cast<const C*>(P.real_tw);
    const int tid = threadIdx.x;
    constexpr bool CIN = KIND == kSmoothCC || KIND == kSmoothCK, COUT = KIND == kSmoothCC || KIND == kSmoothKC;
    const int lines = KIND == kSmoothKK ? P.w : W;
    X.w_in = CIN ? tid % W : tid / TPL;
    X.t_in = CIN ? tid / W : tid - X.w_in * TPL;
    X.w_out = COUT ? tid % W : tid / TPL;
    X.t_out = COUT ? tid / W : tid - X.w_out * TPL;
    X.act_in = CIN ? X.t_in < TPL : X.w_in < lines;
    X.act_out = COUT ? X.t_out < TPL : X.w_out < lines;
    const int64_t tile = blockIdx.x;
    const int64_t o = KIND == kSmoothKK ? 0 : tile / P.col_tiles;
    const int64_t c0 = (tile - o * P.col_tiles) * lines;
    const int64_t ci = (KIND == kSmoothKK ? tile * lines : c0) + X.w_in;
    const int64_t co = (KIND == kSmoothKK ? tile * lines : c0) + X.w_out;
    X.in_ok = X.act_in && ci < P.n_cols;
    X.out_ok = X.act_out && co < P.n_cols;
    if constexpr (FEAT & kSmoothRun) {
        const RunLine l = smooth_run_line(static_cast<uint32_t>(ci), static_cast<uint32_t>(P.run_cols));
        X.gin = in + l.o * P.in_hi + l.c;
        X.gout = out + l.o * P.out_hi + l.c;
    } else {
        X.gin = in + o * P.in_hi + (CIN ? ci : ci * P.in_cs);
        X.gout = out + o * P.out_hi + (COUT ? co : co * P.out_cs);
    }
    if constexpr (FEAT & kSmoothTw4) {
        X.sel = static_cast<int>(co);
        X.tw4_hi = static_cast<const C*>(P.tw4_hi);
        X.tw4_lo = static_cast<const C*>(P.tw4_lo);
        X.tw4_shift = P.tw4_shift;
        X.tw4_sy = (P.tw4_conj != P.conj_out) ? T(-1) : T(1);
    }
    if constexpr (FEAT & kSmoothPre) smooth_pre<T, N, TPL, PADS, PITCH>(X);
    smooth_stages<T, N, TPL, KIND, W, PADS, PITCH, FEAT, 1, 0, true, Rs...>(X);
    if constexpr (FEAT & kSmoothPost) smooth_post<T, N, TPL, PADS, PITCH>(X);
}

}  // namespace sfb
