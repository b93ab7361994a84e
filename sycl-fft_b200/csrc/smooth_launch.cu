// Launch of the size-specialised kernels of the 7-smooth lengths (smooth_catalog.h) and of the Bluestein
// and Rader passes (conv_catalog.h).
#include "conv_catalog.h"
#include "conv_launch.hpp"
#include "kernel_set.hpp"
#include "smooth_catalog.h"
#include "smooth_launch.hpp"

namespace sfb {

#define SFB_EACH_PART(F) F(0) F(1) F(2) F(3) F(4) F(5) F(6) F(7) F(8) F(9) F(10) F(11) F(12) F(13) F(14) F(15) \
    F(16) F(17) F(18) F(19) F(20) F(21) F(22) F(23)
static_assert(SFB_SMOOTH_PARTS == 24, "SFB_EACH_PART lists the parts");
#define SFB_EACH_CONV_PART(F) F(0) F(1) F(2) F(3) F(4) F(5) F(6) F(7)
static_assert(SFB_CONV_PARTS == 8, "SFB_EACH_CONV_PART lists the parts");

// a part of smooth_catalog.h is compiled in three objects and one of its run-on forms, one of conv_catalog.h in two
#define SFB_DECL(P)                                       \
    const SmoothKernel* smooth_part_##P##_0(int* count);  \
    const SmoothKernel* smooth_part_##P##_1(int* count);  \
    const SmoothKernel* smooth_part_##P##_2(int* count);  \
    const SmoothKernel* smooth_run_part_##P(int* count);
SFB_EACH_PART(SFB_DECL)
#undef SFB_DECL
#define SFB_EACH_SPIPED_PART(F) F(0) F(1) F(2) F(3)
#define SFB_DECL(P) const SmoothKernel* smooth_piped_part_##P(int* count);
SFB_EACH_SPIPED_PART(SFB_DECL)
#undef SFB_DECL
#define SFB_DECL(P) const ConvKernel* conv_part_##P##_0(int* count); const ConvKernel* conv_part_##P##_1(int* count);
SFB_EACH_CONV_PART(SFB_DECL)
#undef SFB_DECL

namespace {

KernelSet& smooth_kernels() {
    static KernelSet* k = [] {
        auto* s = new KernelSet;
#define SFB_ADD(P) s->add(smooth_part_##P##_0); s->add(smooth_part_##P##_1); s->add(smooth_part_##P##_2);
        SFB_EACH_PART(SFB_ADD)
#undef SFB_ADD
        s->finish();
        return s;
    }();
    return *k;
}

KernelSet& smooth_run_kernels() {
    static KernelSet* k = [] {
        auto* s = new KernelSet;
#define SFB_ADD(P) s->add(smooth_run_part_##P);
        SFB_EACH_PART(SFB_ADD)
#undef SFB_ADD
        s->finish();
        return s;
    }();
    return *k;
}

KernelSet& smooth_piped_kernels() {
    static KernelSet* k = [] {
        auto* s = new KernelSet;
#define SFB_ADD(P) s->add(smooth_piped_part_##P);
        SFB_EACH_SPIPED_PART(SFB_ADD)
#undef SFB_ADD
        s->finish();
        return s;
    }();
    return *k;
}

KernelSet& conv_kernels() {
    static KernelSet* k = [] {
        auto* s = new KernelSet;
#define SFB_ADD(P) s->add(conv_part_##P##_0); s->add(conv_part_##P##_1);
        SFB_EACH_CONV_PART(SFB_ADD)
#undef SFB_ADD
        s->finish();
        return s;
    }();
    return *k;
}

// The most dynamic shared memory a launch of the entry takes.
size_t smooth_smem(const SmoothEntry& e) { return static_cast<size_t>(e.w) * e.pitch * (e.dbl ? 16 : 8); }
size_t conv_smem(const ConvEntry& e) { return static_cast<size_t>(e.w) * e.pitch * (e.dbl ? 16 : 8) + conv_index_bytes(e); }

}  // namespace

cudaError_t prepare_smooth(const SmoothEntry& e, int64_t n_cols, int64_t n_outer) {
    return (smooth_runs_on(e.kind, e.feat, e.w, n_cols, n_outer) ? smooth_run_kernels() : smooth_kernels())
        .prepare(e.id, smooth_smem(e));
}

cudaError_t prepare_smooth_piped(const SmoothEntry& e) {
    return smooth_piped_kernels().prepare(e.id, static_cast<size_t>(smooth_piped_smem(e.n, e.pitch)));
}

cudaError_t prepare_conv(const ConvEntry& e) { return conv_kernels().prepare(e.id, conv_smem(e)); }

cudaError_t launch_smooth(const SmoothEntry& e, SmoothParams p, int64_t n_outer, int sms, const void* in, void* out,
                          cudaStream_t stream) {
    const size_t line = static_cast<size_t>(e.pitch) * (e.dbl ? 16 : 8);
    p.w = e.w;
    int threads = e.maxt;
    if (e.kind == kSmoothKK) {
        p.w = lines_per_block(e.w, p.n_cols, sms);
        threads = (p.w * e.tpl + 31) / 32 * 32;
    }
    const bool run = smooth_runs_on(e.kind, e.feat, e.w, p.n_cols, n_outer);
    if (run) {
        p.run_cols = static_cast<int>(p.n_cols);
        p.n_cols *= n_outer;
        n_outer = 1;
    }
    p.col_tiles = (p.n_cols + p.w - 1) / p.w;
    void* args[] = {&p, const_cast<void**>(&in), &out};
    return (run ? smooth_run_kernels() : smooth_kernels())
        .launch(e.id, n_outer * p.col_tiles, threads, p.w * line, smooth_smem(e), args, stream);
}

cudaError_t launch_smooth_piped(const SmoothEntry& e, const SmoothParams& p, int sms, int* status, long long wait_polls,
                                const void* in, void* out, cudaStream_t stream) {
    SmoothPipedParams q;
    q.s = p;
    q.status = status;
    q.wait_polls = wait_polls;
    const size_t smem = static_cast<size_t>(smooth_piped_smem(e.n, e.pitch));
    const int64_t ctas = static_cast<int64_t>(sms) * e.minb;
    void* args[] = {&q, const_cast<void**>(&in), &out};
    return smooth_piped_kernels().launch(e.id, p.n_cols < ctas ? p.n_cols : ctas, e.maxt, smem, smem, args, stream);
}

cudaError_t launch_conv(const ConvEntry& e, FixedParams p, int64_t n_outer, int sms, const void* in, void* out,
                        cudaStream_t stream) {
    const size_t line = static_cast<size_t>(e.pitch) * (e.dbl ? 16 : 8);
    p.w = e.w;
    int threads = e.maxt;
    if (e.kind == kBlueFused || e.kind == kBlueRowsConv) {
        p.w = lines_per_block(e.w, p.n_cols, sms);
        threads = (p.w * e.tpl + 31) / 32 * 32;
        n_outer = 1;
    }
    p.col_tiles = (p.n_cols + p.w - 1) / p.w;
    const size_t extra = conv_index_bytes(e);
    void* args[] = {&p, const_cast<void**>(&in), &out};
    return conv_kernels().launch(e.id, n_outer * p.col_tiles, threads, p.w * line + extra, conv_smem(e), args, stream);
}

}  // namespace sfb
