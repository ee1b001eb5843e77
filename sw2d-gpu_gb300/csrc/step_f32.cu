// step_f32.cu -- FP32 instantiations (fast math: FMA contraction,
// approximate division, square root and power).  Accuracy is checked against
// the FP64 oracle with stated tolerances, not bit for bit.
#define SW2D_REAL float
#include "sw2d_launch_impl.cuh"
#include "sw2d_stream.cuh"
#include "sw2d_stream_builds.h"

namespace sw2d {

cudaError_t prepare_step(int th, int tw) {
    if (th == 16 && tw == 32) return detail::step_prepare<float, 16, 32, 256>();
    if (th == 32 && tw == 32) return detail::step_prepare<float, 32, 32, 256>();
    if (th == 16 && tw == 64) return detail::step_prepare<float, 16, 64, 256>();
    return cudaErrorInvalidValue;
}

cudaError_t launch_step(int th, int tw, int nblocks, const GridDesc &G, const ForcingDesc &F,
                        const StateBufs<float> &S, const Thr<float> &T, Clock *clk, const Control *ctl, int slot,
                        cudaStream_t st) {
    if (th == 16 && tw == 32) return detail::step_launch<float, 16, 32, 256>(nblocks, G, F, S, T, clk, ctl, slot, st);
    if (th == 32 && tw == 32) return detail::step_launch<float, 32, 32, 256>(nblocks, G, F, S, T, clk, ctl, slot, st);
    if (th == 16 && tw == 64) return detail::step_launch<float, 16, 64, 256>(nblocks, G, F, S, T, clk, ctl, slot, st);
    return cudaErrorInvalidValue;
}

int stream_out_cols() { return kStreamOut; }

// Build 6: the shape of build 0 with its rows staged in shared memory by TMA
// (stream_step_tma_kernel), for uniform forcing; the other forcing forms run
// build 0 (the same arithmetic, the same bits).
constexpr size_t kTmaSmem = (size_t)2 * kTmaStages * kTmaStageBytes;

int stream_variants() { return 7; }

int stream_warps(int variant) {
    if (variant == kTmaVariant) return 2;
#define SW2D_W(id, nw, mb, un) \
    if (variant == id) return nw;
    SW2D_STREAM_VARIANTS(SW2D_W)
#undef SW2D_W
    return 4;
}

cudaError_t prepare_stream_step(int variant) {
    if (variant == kTmaVariant) {
        cudaError_t e = cudaFuncSetAttribute(stream_step_tma_kernel<2, 10, 2>,
                                             cudaFuncAttributePreferredSharedMemoryCarveout,
                                             (int)cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        e = cudaFuncSetAttribute(stream_step_tma_kernel<2, 10, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kTmaSmem);
        if (e != cudaSuccess) return e;
        variant = 0;  // the build the other forcing forms run
    }
    // the default build's forms for short strips
    if (variant == 0) {
        const void *k[5] = {(const void *)stream_step_kernel<2, 10, 2, false, kFormUniform, true>,
                            (const void *)stream_step_kernel<2, 10, 2, false, kFormStorm, true>,
                            (const void *)stream_step_kernel<2, 10, 2, false, kFormSources, true>,
                            (const void *)stream_step_kernel<2, 10, 2, false, kFormAny, true>,
                            (const void *)stream_step_kernel<2, 10, 2, true, kFormUniform, true>};
        for (int i = 0; i < 5; i++) {
            cudaError_t e = cudaFuncSetAttribute(k[i], cudaFuncAttributePreferredSharedMemoryCarveout,
                                                 kStreamCarveoutPercent);
            if (e != cudaSuccess) return e;
        }
    }
#define SW2D_P(id, nw, mb, un)                                                                            \
    if (variant == id) {                                                                               \
        const void *k[6] = {(const void *)stream_step_kernel<nw, mb, un, false, kFormUniform, false>,         \
                            (const void *)stream_step_kernel<nw, mb, un, false, kFormStorm, false>,           \
                            (const void *)stream_step_kernel<nw, mb, un, false, kFormSources, false>,         \
                            (const void *)stream_step_kernel<nw, mb, un, false, kFormAny, false>,             \
                            (const void *)stream_step_kernel<nw, mb, un, true, kFormUniform, false>,          \
                            (const void *)stream_step_kernel<nw, mb, un, true, kFormAny, false>};             \
        for (int i = 0; i < 6; i++) {                                                                  \
            cudaError_t e = cudaFuncSetAttribute(k[i], cudaFuncAttributePreferredSharedMemoryCarveout, \
                                                 kStreamCarveoutPercent);                             \
            if (e != cudaSuccess) return e;                                                            \
        }                                                                                              \
        return prepare_stream_pipe(id);                                                                \
    }
    SW2D_STREAM_VARIANTS(SW2D_P)
#undef SW2D_P
    return cudaErrorInvalidValue;
}

const char *stream_variant_name(int variant) {
    if (variant == kTmaVariant) return "stream_step_tma_kernel<2,10,2>";
#define SW2D_N(id, nw, mb, un) \
    if (variant == id) return "stream_step_kernel<" #nw "," #mb "," #un ">";
    SW2D_STREAM_VARIANTS(SW2D_N)
#undef SW2D_N
    return "stream_step_kernel<?>";
}

std::string stream_build_name(int variant, int strip_h, bool storm, bool sources, bool rainw, bool pipelined,
                              std::string *form) {
    static const char *const names[4] = {"uniform", "storm", "sources", "any"};
    const int f = stream_form(storm, sources, rainw);
    *form = names[f];
    if (variant == kTmaVariant && (pipelined || rainw || f != kFormUniform)) variant = 0;
    if (!pipelined) {
        if (stream_skips(variant, strip_h, f, rainw)) *form += "+skip";
        return stream_variant_name(variant);
    }
#define SW2D_N(id, nw, mb, un)                                                            \
    if (variant == id)                                                                    \
        return "stream_pipe_kernel<" #nw "," #mb "," + std::to_string(pipe_unroll(un, f)) + ">";
    SW2D_STREAM_VARIANTS(SW2D_N)
#undef SW2D_N
    return "stream_pipe_kernel<?>";
}

int stream_ctas_per_sm(int variant) {
    int n = 0;
    if (variant == kTmaVariant)
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stream_step_tma_kernel<2, 10, 2>, 64, kTmaSmem) ==
                       cudaSuccess
                   ? n
                   : 0;
#define SW2D_O(id, nw, mb, un)                                                                           \
    if (variant == id &&                                                                                 \
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stream_step_kernel<nw, mb, un, false, kFormUniform, false>, nw * 32, 0) != \
            cudaSuccess)                                                                                 \
        n = 0;
    SW2D_STREAM_VARIANTS(SW2D_O)
#undef SW2D_O
    return n;
}

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry points (no link
// against the driver library)
EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// Tensor map of one plane of the pitched layout, frame included, from its
// cell-(0,0) pointer: dimensions (pitch, plane rows), boxes of one row.
bool plane_map(CUtensorMap *m, const void *cell00, int rows, int pitch, bool u8) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn || !cell00) return false;
    const size_t es = u8 ? 1 : 4;
    char *base = (char *)cell00 - origin_for(pitch) * es;
    cuuint64_t dims[2] = {(cuuint64_t)pitch, (cuuint64_t)(plane_for(rows, pitch) / pitch)};
    cuuint64_t strides[1] = {(cuuint64_t)pitch * es};
    cuuint32_t box[2] = {(cuuint32_t)(u8 ? kTmaBoxM : kTmaBoxF), 1u};
    cuuint32_t estr[2] = {1u, 1u};
    return fn(m, u8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box,
              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

cudaError_t launch_stream_step(int variant, int nblocks, int tiles_w, int strip_h, int units, int skew,
                               const GridDesc &G, const ForcingDesc &F, const StateBufs<float> &S,
                               const Thr<float> &T, Clock *clk, const Control *ctl, int slot, cudaStream_t st) {
    const StreamShape sh = stream_shape(G.rows, tiles_w, strip_h, units, false, skew);
    const bool rainw = S.rainw != nullptr;
    const int form = stream_form(F.rain_kind == RAIN_STORM, G.n_src > 0, rainw);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(nblocks);
    lc.dynamicSmemBytes = 0;
    lc.stream = st;
    lc.attrs = attr;
    lc.numAttrs = 1;
    if (variant == kTmaVariant) {
        if (!rainw && form == kFormUniform) {
            TmaMaps M;
            std::memset(&M, 0, sizeof(M));
            bool ok = true;
            for (int b = 0; b < 2; b++)
                ok = ok && plane_map(&M.h[b], S.h[b], G.rows, G.pitch, false) &&
                     plane_map(&M.um[b], S.um[b], G.rows, G.pitch, false) &&
                     plane_map(&M.vn[b], S.vn[b], G.rows, G.pitch, false) &&
                     plane_map(&M.r[b], S.hr[b], G.rows, G.pitch, false);
            ok = ok && plane_map(&M.dzx, S.dzx, G.rows, G.pitch, false) &&
                 plane_map(&M.dzy, S.dzy, G.rows, G.pitch, false) && plane_map(&M.m, S.mask, G.rows, G.pitch, true);
            if (S.nman) ok = ok && plane_map(&M.n, S.nman, G.rows, G.pitch, false);
            if (!ok) return cudaErrorInvalidValue;
            lc.blockDim = dim3(64);
            lc.dynamicSmemBytes = kTmaSmem;
            return cudaLaunchKernelEx(&lc, stream_step_tma_kernel<2, 10, 2>, G, F, S, T, clk, ctl, slot, sh, M);
        }
        variant = 0;
    }
#define SW2D_LK(nw, mb, un, rw, fm, sk) \
    return cudaLaunchKernelEx(&lc, stream_step_kernel<nw, mb, un, rw, fm, sk>, G, F, S, T, clk, ctl, slot, sh)
    // Short strips leave out the warm-up rows' unread stages (SKIP), in the default
    // build.  us per iteration without / with, rows per strip in brackets: uniform
    // 13.5 / 12.6 (1), 15.1 / 14.2 (2), 16.7 / 16.2 (4), 17.3 / 17.2 (6), but 18.9 /
    // 19.0 (8), 21.9 / 22.1 (10), 73.3 / 76.8 (52); storm 13.5 / 12.6 (1), 31.4 / 31.0
    // (13), 78.2 / 81.4 (52); sources 17.3 / 15.5 (1), 40.2 / 39.4 (13), 93.6 / 95.1
    // (52); rain factors 14.1 / 13.4 (1), 33.2 / 33.0 (13), 39.2 / 39.6 (16), 98 / 103
    // (52).
    if (stream_skips(variant, strip_h, form, rainw)) {
        lc.blockDim = dim3(64);
        if (rainw) SW2D_LK(2, 10, 2, true, kFormUniform, true);
        if (form == kFormStorm) SW2D_LK(2, 10, 2, false, kFormStorm, true);
        if (form == kFormSources) SW2D_LK(2, 10, 2, false, kFormSources, true);
        if (form == kFormAny) SW2D_LK(2, 10, 2, false, kFormAny, true);
        SW2D_LK(2, 10, 2, false, kFormUniform, true);
    }
#define SW2D_L(id, nw, mb, un)                                                      \
    if (variant == id) {                                                            \
        lc.blockDim = dim3(nw * 32);                                                \
        if (rainw && form == kFormAny) SW2D_LK(nw, mb, un, true, kFormAny, false);  \
        if (rainw) SW2D_LK(nw, mb, un, true, kFormUniform, false);                  \
        if (form == kFormStorm) SW2D_LK(nw, mb, un, false, kFormStorm, false);      \
        if (form == kFormSources) SW2D_LK(nw, mb, un, false, kFormSources, false);  \
        if (form == kFormAny) SW2D_LK(nw, mb, un, false, kFormAny, false);          \
        SW2D_LK(nw, mb, un, false, kFormUniform, false);                            \
    }
    SW2D_STREAM_VARIANTS(SW2D_L)
#undef SW2D_L
#undef SW2D_LK
    return cudaErrorInvalidValue;
}

}  // namespace sw2d
