// pipe_f32.cu -- the pipelined launches of the FP32 streaming kernel
// (sw2d_pipe.cuh): several iterations per cooperative launch.  Compiled as
// step_f32.cu is: the same bits.
#include "sw2d_launch.h"
#include "sw2d_pipe.cuh"
#include "sw2d_stream_builds.h"

namespace sw2d {

// The forms of a build: uniform rain and the storm as the build unrolls them, those
// with the sources with the row loop not unrolled (pipe_unroll): unrolled by 2, build 0 with both
// the storm and the sources spilled 492 bytes (412 with the sources alone), which in
// strips of more than a few rows cost more than the pipelining saves; not unrolled
// it spills 28 (16).  The storm alone spills 24 unrolled, 52 not (24.6 against 25.7
// us at 701 x 1237).  us per iteration, one form for all of them unrolled by 2
// against these, 701 x 1237 / 1500 x 1500: storm 55.5 / 115 -> 24.6 / 50.0, sources
// 54.7 / 108 -> 26.6 / 51.0, both 59.9 / 120 -> 27.4 / 55.5, storm and rain factors
// 61.7 / 134 -> 28.2 / 56.6.
cudaError_t prepare_stream_pipe(int variant) {
#define SW2D_PF(nw, mb, un, w, f) ((const void *)stream_pipe_kernel<nw, mb, pipe_unroll(un, f), w, f>)
#define SW2D_P(id, nw, mb, un)                                                                         \
    if (variant == id) {                                                                               \
        const void *k[6] = {SW2D_PF(nw, mb, un, false, kFormUniform), SW2D_PF(nw, mb, un, false, kFormStorm),      \
                            SW2D_PF(nw, mb, un, false, kFormSources), SW2D_PF(nw, mb, un, false, kFormAny),        \
                            SW2D_PF(nw, mb, un, true, kFormUniform), SW2D_PF(nw, mb, un, true, kFormAny)};         \
        for (const void *f : k) {                                                                      \
            cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout,    \
                                                 kStreamCarveoutPercent);                              \
            if (e != cudaSuccess) return e;                                                            \
        }                                                                                              \
        return cudaSuccess;                                                                            \
    }
    SW2D_STREAM_VARIANTS(SW2D_P)
#undef SW2D_P
#undef SW2D_PF
    return cudaErrorInvalidValue;
}

// Resident CTAs per SM of the build's pipelined form (every form of a build
// has the same register budget and shared memory).
int stream_pipe_ctas_per_sm(int variant) {
    if (variant == kTmaVariant) variant = 0;  // the TMA build has no pipelined form: build 0's
    int n = 0;
#define SW2D_PO(id, nw, mb, un)                                                                          \
    if (variant == id &&                                                                                 \
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stream_pipe_kernel<nw, mb, un, false, kFormUniform>, nw * 32, 0) != \
            cudaSuccess)                                                                                 \
        n = 0;
    SW2D_STREAM_VARIANTS(SW2D_PO)
#undef SW2D_PO
    return n;
}

int stream_pipe_max_iters() { return kPipeMaxIters; }
int stream_pipe_min_strip() { return kPipeMinStrip; }

// The plan kernel, then one cooperative launch of K iterations.
cudaError_t launch_stream_pipe(int variant, int nblocks, int tiles_w, int strip_h, int units, const GridDesc &G,
                               const ForcingDesc &F, const StateBufs<float> &S, const Thr<float> &T, Clock *clk,
                               const Control *ctl, int slot, Plan *plans, unsigned *words, unsigned *flags, int K,
                               cudaStream_t st) {
    const int strips = (G.rows + strip_h - 1) / strip_h;  // the shortest strip has rows / strips rows
    if (K < 1 || K > kPipeMaxIters || (strips > 1 && G.rows / strips < kPipeMinStrip)) return cudaErrorInvalidValue;
    pipe_plan_kernel<<<1, ((K + 31) / 32) * 32, 0, st>>>(G, F, clk, ctl, slot, plans, words, flags, units, K);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const StreamShape sh = stream_shape(G.rows, tiles_w, strip_h, units, true, 0);
    PipeDesc P;
    P.plans = plans;
    P.words = words;
    P.flags = flags;
    const bool rainw = S.rainw != nullptr;
    const int form = stream_form(F.rain_kind == RAIN_STORM, G.n_src > 0, rainw);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;  // every unit resident: the waits between units end
    attr[0].val.cooperative = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(nblocks);
    // unused: with the uniform form's own 96 bytes a CTA ran 512^2 in 18.3 us per
    // iteration, with 1 KB (or 4 KB) in 16.7; the step kernels (1 KB of their own)
    // do not change with more
    lc.dynamicSmemBytes = 1024;
    lc.stream = st;
    lc.attrs = attr;
    lc.numAttrs = 1;
    if (variant == kTmaVariant) variant = 0;
#define SW2D_PK(nw, mb, un, w, f) \
    return cudaLaunchKernelEx(&lc, stream_pipe_kernel<nw, mb, pipe_unroll(un, f), w, f>, G, F, S, T, clk, ctl, slot, sh, P)
#define SW2D_PL(id, nw, mb, un)                                              \
    if (variant == id) {                                                     \
        lc.blockDim = dim3(nw * 32);                                         \
        if (rainw && form == kFormAny) SW2D_PK(nw, mb, un, true, kFormAny);  \
        if (rainw) SW2D_PK(nw, mb, un, true, kFormUniform);                  \
        if (form == kFormAny) SW2D_PK(nw, mb, un, false, kFormAny);          \
        if (form == kFormStorm) SW2D_PK(nw, mb, un, false, kFormStorm);      \
        if (form == kFormSources) SW2D_PK(nw, mb, un, false, kFormSources);  \
        SW2D_PK(nw, mb, un, false, kFormUniform);                            \
    }
    SW2D_STREAM_VARIANTS(SW2D_PL)
#undef SW2D_PL
#undef SW2D_PK
    return cudaErrorInvalidValue;
}

}  // namespace sw2d
