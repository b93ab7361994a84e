// Host emulation of the size-specialised kernels of the 7-smooth lengths (smooth_kernel.cuh) and of the
// Bluestein and Rader passes (conv_kernel.cuh) -- TEST INFRASTRUCTURE ONLY. Plans come from the product
// planner; every thread of every block of a smooth_catalog.h or conv_catalog.h pass is then stepped through the kernel's own index arithmetic in FP64: the two thread
// mappings, the padded shared-memory rows, the stage twiddle tables and the global strides. Each access is
// checked against its buffer, and each shared-memory word against being written twice, or read before it
// is written, between two barriers.
#include <algorithm>
#include <complex>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../sycl-fft_b200/csrc/planner.hpp"

using cd = std::complex<double>;
using namespace sfb;

namespace {

struct Span {
    const char* name;
    std::vector<cd> v;
    cd& at(int64_t i) {
        if (i < 0 || i >= static_cast<int64_t>(v.size()))
            throw std::runtime_error(std::string(name) + " index " + std::to_string(i) + " outside " + std::to_string(v.size()));
        return v[i];
    }
};

// The product of the kernel's twiddle rows that gives w^r (rows w, w^2, w^4, w^8; above radix 16 w, w^2, w^3
// and w^4, w^8, w^12, ..).
cd power(const std::vector<cd>& tw, int64_t off, int ns, int jm, int r, int R = 16) {
    cd w = 1.0;
    if (R > 16) {
        if (r % 4) w *= tw[off + int64_t(r % 4 - 1) * ns + jm];
        if (r / 4) w *= tw[off + int64_t(2 + r / 4) * ns + jm];
        return w;
    }
    for (int q = 0; (1 << q) <= r; ++q)
        if (r & (1 << q)) w *= tw[off + int64_t(q) * ns + jm];
    return w;
}

void run_smooth(const PlanSpec& plan, const PassSpec& ps, Span& src, Span& dst, int w_lines) {
    const SmoothEntry& e = *smooth_entry(ps.smooth_id);
    const PassParams& p = ps.p;
    const auto& tw = plan.tables[ps.tables.smooth];
    int64_t n_outer = p.n_outer, n_cols = p.n_cols, in_hi = p.in.hi, out_hi = p.out.hi, out_cs = p.out.cs, out_ks = p.out.ks;
    if (p.ts_rows > 0) {
        n_outer = p.n_cols / p.ts_rows;
        n_cols = p.ts_rows;
        in_hi = p.ts_rows * p.in.cs;
        out_hi = p.ts_line;
        out_cs = 1;
        out_ks = p.ts_rows;
    }
    const bool cin = e.kind == kSmoothCC || e.kind == kSmoothCK, cout = e.kind == kSmoothCC || e.kind == kSmoothKC;
    const int w = e.kind == kSmoothKK ? w_lines : e.w;
    const int threads = e.kind == kSmoothKK ? (w * e.tpl + 31) / 32 * 32 : e.maxt;
    const int64_t col_tiles = (n_cols + w - 1) / w;
    if (threads > e.maxt) throw std::runtime_error("block larger than the launch bound");
    for (int64_t tile = 0; tile < n_outer * col_tiles; ++tile) {
        const int64_t o = e.kind == kSmoothKK ? 0 : tile / col_tiles;
        const int64_t c0 = e.kind == kSmoothKK ? tile * w : (tile - o * col_tiles) * w;
        std::vector<cd> sm(static_cast<size_t>(w) * e.pitch);
        std::vector<char> written(sm.size(), 0);
        struct Out { int64_t at; cd v; };
        std::vector<Out> out;
        int ns = 1;
        int64_t off = 0;
        for (int s = 0; s < e.nstages; ++s) {
            const bool first = s == 0, last = s == e.nstages - 1;
            const int R = e.radices[s], nr = e.n / R, nb = (nr + e.tpl - 1) / e.tpl;
            const bool inmap = e.kind == kSmoothKC ? !last : first || e.kind == kSmoothKK || e.kind == kSmoothCC;
            const bool lanes_c = inmap ? cin : cout;
            std::vector<cd> next(sm.size());
            std::vector<char> nw(sm.size(), 0);
            for (int tid = 0; tid < threads; ++tid) {
                const int wl = lanes_c ? tid % w : tid / e.tpl;
                const int t = lanes_c ? tid / w : tid - wl * e.tpl;
                const bool act = lanes_c ? t < e.tpl : wl < w;
                if (!act) continue;
                const int64_t c = c0 + wl;
                auto cell = [&](int k) {
                    const int64_t i = int64_t(wl) * e.pitch + (e.pads ? k + (k >> e.pads) : k);
                    if (k < 0 || k >= e.n || i >= int64_t(sm.size()) || (wl + 1 < w && i >= int64_t(wl + 1) * e.pitch))
                        throw std::runtime_error("shared-memory index outside its row");
                    return i;
                };
                for (int i = 0; i < nb; ++i) {
                    const int j = t + i * e.tpl;
                    if (j >= nr) continue;
                    cd v[32], u[32];
                    for (int r = 0; r < R; ++r) {
                        const int k = j + r * nr;
                        if (first) {
                            v[r] = c < n_cols ? src.at(o * in_hi + c * p.in.cs + k * p.in.ks) : 0.0;
                            if (p.conj_in) v[r] = std::conj(v[r]);
                        } else {
                            if (!written[cell(k)]) throw std::runtime_error("shared memory read before it is written");
                            v[r] = sm[cell(k)];
                        }
                    }
                    const int jm = last ? j : j % ns;
                    if (jm >= ns) throw std::runtime_error("twiddle index outside its stage");
                    for (int r = 1; r < R; ++r)
                        if (ns > 1) v[r] *= power(tw, off, ns, jm, r, R);
                    for (int q = 0; q < R; ++q) {
                        u[q] = 0.0;
                        for (int r = 0; r < R; ++r) u[q] += v[r] * cis_neg(int64_t(q) * r, R);
                    }
                    for (int r = 0; r < R; ++r) {
                        if (!last) {
                            const int64_t at = cell((j - jm) * R + jm + r * ns);
                            if (nw[at]) throw std::runtime_error("shared memory written twice");
                            nw[at] = 1;
                            next[at] = u[r];
                            continue;
                        }
                        if (c >= n_cols) continue;
                        const int64_t k = j + int64_t(r) * nr;
                        cd a = u[r];
                        if (p.tw4_sign != 0) {
                            const int64_t m = k * c, mask = (int64_t(1) << p.tw4_shift) - 1;
                            cd q = plan.tables[ps.tables.tw4_hi][m >> p.tw4_shift] * plan.tables[ps.tables.tw4_lo][m & mask];
                            if ((p.tw4_sign > 0) != (p.conj_out != 0)) q = std::conj(q);
                            a *= q;
                        }
                        if (p.conj_out) a = std::conj(a);
                        out.push_back({o * out_hi + c * out_cs + k * out_ks, a * p.scale});
                    }
                }
            }
            sm.swap(next);
            written.swap(nw);
            off += int64_t(ns) * smooth_tw_entries(R);
            ns *= R;
        }
        // a block reads its tile before it writes it, and tiles are disjoint
        for (const Out& x : out) dst.at(x.at) = x.v;
    }
}

// A Bluestein or Rader pass on its conv_catalog.h kernel (conv_kernel.cuh). `dc`: the axis input and output
// of the Rader bin-0 term between the column passes, their line pitches and the outputs' scale.
struct BinZero {
    Span *x = nullptr, *y = nullptr;
    int64_t x_pitch = 0, y_pitch = 0;
    double scale = 1.0;
};

void run_conv(const PlanSpec& plan, const PassSpec& ps, Span& src, Span& dst, int w_lines, const BinZero& dc) {
    const ConvEntry& e = *conv_entry(ps.conv_id);
    const PassParams& p = ps.p;
    const auto& tw = plan.tables[ps.tables.smooth];
    auto table = [&](int id) -> const std::vector<cd>* { return id < 0 ? nullptr : &plan.tables[id]; };
    const auto *premul = table(ps.tables.premul), *postmul = table(ps.tables.postmul), *pw = table(ps.tables.pointwise);
    const auto *hi = table(ps.tables.tw4_hi), *lo = table(ps.tables.tw4_lo);
    const auto* perm_in = ps.tables.perm_in < 0 ? nullptr : &plan.index_tables[ps.tables.perm_in];
    const auto* perm_out = ps.tables.perm_out < 0 ? nullptr : &plan.index_tables[ps.tables.perm_out];
    const bool cols = e.kind == kBlueColsFwd || e.kind == kBlueColsInv;
    const bool conv = e.kind == kBlueFused || e.kind == kBlueRowsConv;
    const int w = cols ? e.w : std::min(w_lines > 0 ? w_lines : e.w, e.w);
    const int threads = cols ? e.maxt : (w * e.tpl + 31) / 32 * 32;
    const int64_t col_tiles = (p.n_cols + w - 1) / w;
    const int64_t outer = cols ? p.n_outer : 1;
    std::vector<int> seq(e.radices, e.radices + e.nstages);
    if (conv)  // the second FFT's first butterfly follows the spectrum multiply in registers
        for (int s = e.nstages - 2; s >= 0; --s) seq.push_back(e.radices[s]);
    const int stages = static_cast<int>(seq.size());
    for (int64_t tile = 0; tile < outer * col_tiles; ++tile) {
        const int64_t o = tile / col_tiles, c0 = (tile - o * col_tiles) * w;
        std::vector<cd> sm(static_cast<size_t>(w) * e.pitch);
        std::vector<char> written(sm.size(), 0);
        struct Out { int64_t at; cd v; };
        std::vector<Out> out;
        int ns = 1;
        int64_t off = 0;
        for (int s = 0; s < stages; ++s) {
            const bool first = s == 0, last = s == stages - 1, mid = conv && s == e.nstages - 1;
            const int R = seq[s], nr = e.n / R, nb = (nr + e.tpl - 1) / e.tpl;
            std::vector<cd> next(sm.size());
            std::vector<char> nw(sm.size(), 0);
            for (int tid = 0; tid < threads; ++tid) {
                const int wl = cols ? tid % w : tid / e.tpl, t = cols ? tid / w : tid - wl * e.tpl;
                if (cols ? t >= e.tpl : wl >= w) continue;
                const int64_t c = c0 + wl;
                const bool ok = c < p.n_cols;
                const int64_t rows = p.sel_mode == kSelColMod ? p.sel_d : 1;
                const int64_t sel = cols ? c : rows > 1 ? c % rows : 0;
                const int64_t ib = cols ? o * p.in.hi + c : c * p.in.cs, ob = cols ? o * p.out.hi + c : c * p.out.cs;
                const int64_t il = cols ? o * p.in.hi : ib, ol = cols ? o * p.out.hi : ob;
                const int64_t iks = cols ? p.in.ks : 1, oks = cols ? p.out.ks : 1;
                auto cell = [&](int k) {
                    const int64_t i = int64_t(wl) * e.pitch + (e.pads ? k + (k >> e.pads) : k);
                    if (k < 0 || k >= e.n || i >= int64_t(sm.size()) || (wl + 1 < w && i >= int64_t(wl + 1) * e.pitch))
                        throw std::runtime_error("shared-memory index outside its row");
                    return i;
                };
                auto dft = [&](cd* v) {
                    cd u[32];
                    for (int q = 0; q < R; ++q) {
                        u[q] = 0.0;
                        for (int r = 0; r < R; ++r) u[q] += v[r] * cis_neg(int64_t(q) * r, R);
                    }
                    std::copy(u, u + R, v);
                };
                for (int i = 0; i < nb; ++i) {
                    const int j = t + i * e.tpl;
                    if (j >= nr) continue;
                    cd v[32];
                    for (int r = 0; r < R; ++r) {
                        const int k = j + r * nr;
                        if (!first) {
                            if (!written[cell(k)]) throw std::runtime_error("shared memory read before it is written");
                            v[r] = sm[cell(k)];
                            continue;
                        }
                        const int64_t g = k * p.g_k + sel;
                        v[r] = 0.0;
                        if (!ok || g >= p.in_len) continue;
                        v[r] = perm_in ? src.at(il + perm_in->at(g)) : src.at(ib + k * iks);
                        if (premul) v[r] *= premul->at(g);
                        if (p.conj_in) v[r] = std::conj(v[r]);
                    }
                    const int jm = last || mid ? j : j % ns;
                    for (int r = 1; r < R; ++r)
                        if (ns > 1) v[r] *= power(tw, off, ns, jm, r);
                    dft(v);
                    if (mid) {
                        cd x0 = 0.0;
                        if (ps.rader && sel == 0 && j == 0 && ok) {
                            const bool whole = perm_in != nullptr;
                            const int64_t line = c / rows;
                            x0 = whole ? src.at(ib) : dc.x->at(line * dc.x_pitch);
                            const cd y0 = (x0 + v[0]) * (whole ? p.scale : dc.scale);
                            if (whole) out.push_back({ob, y0});
                            else dc.y->at(line * dc.y_pitch) = y0;
                        }
                        for (int r = 0; r < R; ++r) {
                            v[r] *= pw->at(j + r * nr + sel * p.pw_stride);
                            if (r == 0) v[0] += x0;
                            if (p.conj_mid) v[r] = std::conj(v[r]);
                        }
                        dft(v);
                    }
                    for (int r = 0; r < R; ++r) {
                        if (!last) {
                            const int64_t at = mid ? cell(j * R + r) : cell((j - jm) * R + jm + r * ns);
                            if (nw[at]) throw std::runtime_error("shared memory written twice");
                            nw[at] = 1;
                            next[at] = v[r];
                            continue;
                        }
                        const int64_t k = j + int64_t(r) * nr, g = k * p.g_k + sel;
                        if (!ok || g >= p.out_len) continue;
                        cd a = v[r];
                        if (p.conj_out) a = std::conj(a);
                        if (p.tw4_sign != 0) {
                            const int64_t m = k * sel;
                            const cd q = hi->at(m >> p.tw4_shift) * lo->at(m & ((int64_t(1) << p.tw4_shift) - 1));
                            a *= p.tw4_sign > 0 ? std::conj(q) : q;
                        }
                        if (postmul) a *= postmul->at(g);
                        out.push_back({perm_out ? ol + perm_out->at(g) : ob + k * oks, a * p.scale});
                    }
                }
            }
            sm.swap(next);
            written.swap(nw);
            off += int64_t(ns) * smooth_tw_entries(R);
            ns *= R;
            if (mid) {
                off += smooth_tw_entries(R);  // the second table's first stage
                ns = R;
            }
        }
        for (const Out& x : out) dst.at(x.at) = x.v;
    }
}

void fail(char* err, size_t cap, const char* what) {
    std::strncpy(err, what, cap - 1);
    err[cap - 1] = 0;
}

int run_plan(const PlanRequest& req, const double* in, int64_t in_len, double* out, int64_t out_len, int w_lines, char* err,
             size_t cap) {
    try {
        const PlanSpec plan = make_plan(req);
        Span input{"input", {}}, output{"output", {}}, scratch{"scratch", {}};
        input.v.resize(in_len);
        output.v.resize(out_len);
        scratch.v.resize(plan.scratch_elements);
        for (int64_t i = 0; i < in_len; ++i) input.v[i] = cd(in[2 * i], in[2 * i + 1]);
        for (int64_t i = 0; i < out_len; ++i) output.v[i] = cd(out[2 * i], out[2 * i + 1]);
        if (req.in_place) output.v = input.v;
        auto buf = [&](Buf b) -> Span& {
            return b == Buf::Scratch ? scratch : b == Buf::Input && !req.in_place ? input : output;
        };
        for (size_t i = 0; i < plan.passes.size(); ++i) {
            const PassSpec& ps = plan.passes[i];
            if (ps.conv_id >= 0) {
                BinZero dc;
                if (ps.rader_dc)
                    dc = {&buf(ps.rader_src), &output, plan.passes[i - 1].p.in.hi, plan.passes[i + 1].p.out.hi,
                          plan.passes[i + 1].p.scale};
                run_conv(plan, ps, buf(ps.src), buf(ps.dst), w_lines, dc);
                continue;
            }
            if (ps.smooth_id < 0) return 2;
            const int top = smooth_entry(ps.smooth_id)->w;
            run_smooth(plan, ps, buf(ps.src), buf(ps.dst), w_lines > 0 ? std::min(w_lines, top) : top);
        }
        for (int64_t i = 0; i < out_len; ++i) {
            out[2 * i] = output.v[i].real();
            out[2 * i + 1] = output.v[i].imag();
        }
        return 0;
    } catch (const std::exception& e) {
        fail(err, cap, e.what());
        return 1;
    }
}

}  // namespace

// A contiguous batch-major plan all of whose passes are smooth_catalog.h or conv_catalog.h kernels (2: one is
// not). w_lines:
// lines per block of whole-line passes (0: the catalog's).
extern "C" int smooth_run(int dbl, int dir, int norm, int in_place, unsigned rank, const uint64_t* shape, uint64_t batch,
                          int w_lines, const double* in, double* out, char* err, size_t cap) {
    PlanRequest req;
    req.dbl = dbl != 0;
    req.direction = dir;
    req.normalization = norm;
    req.in_place = in_place != 0;
    req.shape.assign(shape, shape + rank);
    req.batch = batch;
    int64_t n = static_cast<int64_t>(batch);
    for (unsigned k = 0; k < rank; ++k) n *= static_cast<int64_t>(shape[k]);
    return run_plan(req, in, n, out, n, w_lines, err, cap);
}

// A strided one-dimensional plan (PlanRequest::strided_line).
extern "C" int smooth_run_line(int dbl, int dir, int norm, int in_place, uint64_t n, uint64_t batch, const int64_t* cs_ks,
                               const double* in, int64_t in_len, double* out, int64_t out_len, char* err, size_t cap) {
    PlanRequest req;
    req.dbl = dbl != 0;
    req.direction = dir;
    req.normalization = norm;
    req.in_place = in_place != 0;
    req.shape = {n};
    req.batch = batch;
    req.strided_line = true;
    req.line_in.cs = cs_ks[0];
    req.line_in.ks = cs_ks[1];
    req.line_out.cs = cs_ks[2];
    req.line_out.ks = cs_ks[3];
    return run_plan(req, in, in_len, out, out_len, 0, err, cap);
}
