// The line map of column tiles that run on across outer indices (smooth_run_line, smooth_runs_on of
// pass_params.h) -- TEST INFRASTRUCTURE ONLY.
#include "../../sycl-fft_b200/csrc/pass_params.h"

using namespace sfb;

// The (outer, column) pairs of every lane of every tile, in tile order; returns their count, or -1 where the
// tiles end with the columns.
extern "C" int64_t narrow_lines(int kind, int feat, int w, int64_t n_cols, int64_t n_outer, int64_t* o, int64_t* c) {
    if (!smooth_runs_on(kind, feat, w, n_cols, n_outer)) return -1;
    const int64_t lines = n_outer * n_cols, tiles = (lines + w - 1) / w;
    int64_t n = 0;
    for (int64_t tile = 0; tile < tiles; ++tile)
        for (int lane = 0; lane < w; ++lane) {
            const int64_t l = tile * w + lane;
            if (l >= lines) continue;
            const RunLine r = smooth_run_line(static_cast<uint32_t>(l), static_cast<uint32_t>(n_cols));
            o[n] = r.o;
            c[n++] = r.c;
        }
    return n;
}
