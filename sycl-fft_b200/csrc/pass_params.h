// One "pass" of the B200 FFT provider: a batch of line FFTs executed by a single
// kernel launch, with everything a pass needs fused into its load and store.
//
// A pass sees its data as lines. Line (o, c) has elements k = 0..n-1 at
//   addr = (o / d) * hi + (o % d) * lo + c * cs + k * ks          (in complex units)
// separately for the input and the output layout. A CTA owns one tile: a fixed
// outer index o and `w` consecutive columns c. The FFT along k is a Stockham
// autosort sequence of radix-R stages held in registers, exchanging through
// shared memory between stages.
//
// Fused extras (all optional):
//   load : zero padding (element index g >= in_len reads 0), pre-multiply by a table
//          indexed by g, conjugation (inverse transforms run as conj-FFT-conj);
//   mid  : point-wise multiply by a table, conjugation, and a second FFT (Bluestein
//          convolution in one kernel);
//   store: conjugation, the four-step twiddle W_N^(sign*k*sel), post-multiply by a
//          table indexed by g, the normalization scale, truncation (g >= out_len is
//          not written).
// The element index is g = k * g_k + sel with sel = 0, c, (o % sel_d) or (c % sel_d).
//
// This header is plain C++ so host planning code and device code share it.
#pragma once

#include <cstdint>

namespace sfb {

constexpr int kMaxStages = 16;

enum : int { kModeK = 0, kModeC = 1 };         // thread mapping / coalesced dimension
// Thread mappings of smooth_kernel.cuh, input side then output side: K lanes walk a line's elements
// (element stride 1), C lanes walk adjacent lines (line stride 1).
enum : int { kSmoothKK = 0, kSmoothCC = 1, kSmoothCK = 2, kSmoothKC = 3 };
// Features of a smooth_kernel.cuh instantiation: four-step twiddle on the store; real transforms of length
// 2N, bins formed after the last stage (R2C) or read before the first (C2R); columns whose tiles run on across
// outer indices (not in the catalog: the second form of its plain column entries, smooth_runs_on).
enum : int { kSmoothTw4 = 1, kSmoothPost = 2, kSmoothPre = 4, kSmoothRun = 8 };
// Rows of a radix-R stage's twiddle table in smooth_kernel.cuh: W^(r*jm) for r = 1, 2, 4, 8 below R; above
// radix 16 for r = 1, 2, 3, 4, 8, 12, .. below R.
#if defined(__CUDACC__)
__host__ __device__
#endif
constexpr int smooth_tw_entries(int R) { return R > 16 ? 3 + (R - 1) / 4 : R > 8 ? 4 : R > 4 ? 3 : R > 2 ? 2 : 1; }
inline int smooth_tw_power(int R, int q) { return R <= 16 ? 1 << q : q < 3 ? q + 1 : 4 * (q - 2); }  // of row q
// Column tiles of smooth_kernel.cuh over arrays narrower than a tile (the first axis of [500, 2]): a tile takes its
// W lines from several outer indices, line l being column l % cols of outer index l / cols. One tile per outer
// index leaves W - cols of W lanes idle, which made two columns slower than the runtime-length kernel. 48 MB
// arrays on B200, runtime-length / one tile per outer index / run on: double 375 x 2 69 / 98 / 57 us, float
// 175 x 2 170 / 208 / 122 us; geometric means over the 177 lengths of each precision, of the runtime-length
// kernel's time and of the idle lanes': 2 columns 1.5x and 1.33x, 3 columns 1.5x and 1.16x, 6 columns 1.8x and 1.06x.
struct RunLine {
    int64_t o, c;
};
#if defined(__CUDACC__)
__host__ __device__
#endif
inline RunLine smooth_run_line(uint32_t l, uint32_t cols) { return {l / cols, l % cols}; }
inline bool smooth_runs_on(int kind, int feat, int w, int64_t n_cols, int64_t n_outer) {
    return kind == kSmoothCC && feat == 0 && w > 2 && n_cols < w && n_outer > 1 && n_outer * n_cols <= INT32_MAX;
}
enum : int { kSelNone = 0, kSelCol = 1, kSelOuterLo = 2, kSelColMod = 3 };

struct LineLayout {
    int64_t hi = 0, lo = 0, d = 1, cs = 0, ks = 1;
};

struct StageSeq {
    int nstages = 0;
    int radix[kMaxStages] = {};
    int ns[kMaxStages] = {};      // product of the radices before this stage
    int tw_off[kMaxStages] = {};  // offset of this stage's twiddles in `tw` (complex units)
    const void* tw = nullptr;     // per stage: [ns][radix-1] of exp(-2 pi i r j / (ns*radix))
};

struct PassParams {
    int n = 1;           // FFT length along k
    int tpl = 1;         // threads per line
    int w = 1;           // lines (columns) per CTA tile
    int mode = kModeK;   // kModeK: threads walk k; kModeC: threads walk columns
    int pitch = 0;       // shared-memory line pitch (kModeK) in complex units
    int pad_shift = 31;  // shared-memory padding: one element per 2^pad_shift
    int64_t n_outer = 1, n_cols = 1, col_tiles = 1, tiles = 1;
    LineLayout in, out;

    // element index g = k * g_k + sel
    int64_t g_k = 1;
    int sel_mode = kSelNone;
    int64_t sel_d = 1;
    int64_t in_len = 0;   // input elements with g >= in_len read as zero
    int64_t out_len = 0;  // outputs with g >= out_len are not stored

    const void* premul = nullptr;     // [in_len] multiplied on load (indexed by g)
    int conj_in = 0;
    StageSeq fft1;
    const void* pointwise = nullptr;  // multiplied after fft1, indexed k + sel * pw_stride
    int64_t pw_stride = 0;
    int conj_mid = 0;
    StageSeq fft2;                    // nstages == 0: no second FFT
    int conj_out = 0;
    const void* tw4_hi = nullptr;     // four-step twiddle W^(m) = hi[m >> shift] * lo[m & mask]
    const void* tw4_lo = nullptr;
    int tw4_shift = 0;
    int tw4_sign = 0;                 // 0: off; -1 / +1: exponent sign
    const void* postmul = nullptr;    // indexed by g on store
    double scale = 1.0;
    int store_via_smem = 0;           // transpose through shared memory before storing
    // Direction override of a whole plan (conj(F(conj x))): conjugate the raw input before
    // the pre-multiply and the final value after the post-multiply and scale. Used instead of
    // conj_in / conj_out by passes that carry premul / postmul tables (Bluestein), where the
    // plan's own conjugations sit between the FFTs and the chirp products.
    int flip_in = 0, flip_out = 0;
    // Rader passes: int32 permutations of the line (load element g from perm_in[g], store
    // element g to perm_out[g], both relative to the line start)
    const void* perm_in = nullptr;
    const void* perm_out = nullptr;
    // Size-specialised four-step row pass: row l (= o*ts_rows + k1) stored at
    // (l / ts_rows) * ts_line + l % ts_rows + k * ts_rows.
    int64_t ts_rows = 0, ts_line = 0;
};

}  // namespace sfb
