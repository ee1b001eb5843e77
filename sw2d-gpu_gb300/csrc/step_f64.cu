// step_f64.cu -- FP64 kernels.  Compiled with --fmad=false: every
// multiply and add rounds separately, as in the serial oracle and in the
// reference built without contraction, which makes the FP64 path
// bit-reproducible against them wherever no transcendental is involved.
#define SW2D_REAL double
#include "sw2d_launch_impl.cuh"
#include "sw2d_step64.cuh"

namespace sw2d {

// Fills this translation unit's tables of the deterministic log/exp (on the
// legacy stream, waited for: the handles' own streams do not order with it).
cudaError_t init_det_tables() {
    pow_tables_kernel<<<2 * kPowN / 256, 256>>>();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(0);
}

// Builds of the step kernel: (tile rows, tile columns, threads, minimum
// resident CTAs per SM).  16 x 32 runs two CTAs of 512 threads per SM, whose
// stages overlap: 313 us per iteration on a 1013 x 900 catchment, 447 with one
// CTA of 768 (the stages then wait at each other's barriers), 358 with one CTA on
// a 32 x 32 tile (less halo, same wait); 256 to 448 threads are within 3 %.
//
// The smaller tiles are for grids that would leave SMs without a CTA: a tile's
// work runs on one SM, so a grid is cut into the smallest tiles that still give
// one CTA per SM (step64_tile).  Measured with the first form of the kernel, us
// per iteration, tiles 4x8 / 4x16 / 8x16 / 8x32 / 16x32: 64 x 64 23.8 / 27.0 /
// 30.3 / 42.3 / 53.5; 117 x 131 48.8 / 42.8 / 34.5 / 47.5 / 60.2; 256 x 256 159 /
// 106 / 79 / 72 / 69.5; 512 x 512 593 / 327 / 261 / 225 / 185 (the halo costs 2.3
// times the faces of the tile at 4 x 8, 1.4 at 16 x 32); the final form runs 18.9,
// 23.2, 43 and 106 on the tile the rule takes.  With one CTA per SM more threads
// shorten the stages: 8 x 16 23.2 with 512 against 26.9 with 256, 8 x 32 30.6 with
// 768 against 34.2 with 384.
#define SW2D_STEP64_TILES(X) \
    X(16, 32, 512, 2) X(8, 32, 768, 1) X(8, 16, 512, 1) X(4, 16, 256, 1) X(4, 8, 256, 1)

bool step64_tile_supported(int th, int tw) {
#define SW2D_S64(h, w, nt, mb) \
    if (th == h && tw == w) return true;
    SW2D_STEP64_TILES(SW2D_S64)
#undef SW2D_S64
    return false;
}

// The smallest tile with at most one CTA per SM, 16 x 32 beyond.
void step64_tile(int rows, int cols, int sms, int *th, int *tw) {
    *th = 16;
    *tw = 32;
    long long best = 16 * 32;
#define SW2D_D64(h, w, nt, mb)                                                                       \
    if (h * w < best && (long long)((rows + h - 1) / h) * ((cols + w - 1) / w) <= sms) {             \
        best = h * w;                                                                                \
        *th = h;                                                                                     \
        *tw = w;                                                                                     \
    }
    SW2D_STEP64_TILES(SW2D_D64)
#undef SW2D_D64
}

cudaError_t prepare_step64(int th, int tw) {
    const cudaError_t e = init_det_tables();
    if (e != cudaSuccess) return e;
#define SW2D_P64(h, w, nt, mb)                                                                                  \
    if (th == h && tw == w) {                                                                                   \
        const cudaError_t e2 = cudaFuncSetAttribute(step64_kernel<h, w, nt, mb>,                                \
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize,                \
                                                    (int)Step64Shape<h, w>::smem(nt / 32));                    \
        if (e2 != cudaSuccess) return e2;                                                                       \
        return cudaFuncSetAttribute(step64_kernel<h, w, nt, mb>, cudaFuncAttributePreferredSharedMemoryCarveout, \
                                    (int)cudaSharedmemCarveoutMaxShared);                                       \
    }
    SW2D_STEP64_TILES(SW2D_P64)
#undef SW2D_P64
    return cudaErrorInvalidValue;
}

cudaError_t launch_step64(int th, int tw, int nblocks, int sms, const GridDesc &G, const ForcingDesc &F,
                          const StateBufs<double> &S, const Thr<double> &T, const double *gnx, const double *gny,
                          Clock *clk, const Control *ctl, int slot, cudaStream_t st) {
    Step64Extra X;
    X.gnx = gnx;
    X.gny = gny;
    X.gn = G.sd.g * G.sd.manning * G.sd.manning;
    X.thf = (float)T.ge_th;
    X.dx = known_divisor(G.sd.dx);
    X.dy = known_divisor(G.sd.dy);
    // a programmatic dependent of the launch before it (step64_kernel, stage 0)
    // where one CTA per SM holds the grid: 53.5 against 55.9 us on 64 x 64.  With
    // more, the early CTAs crowd the SMs that drain first (256 CTAs of 8 x 32:
    // 91 against 72 us).
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = nblocks <= sms ? 1 : 0;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(nblocks);
    lc.stream = st;
    lc.attrs = attr;
    lc.numAttrs = 1;
#define SW2D_L64(h, w, nt, mb)                                                                             \
    if (th == h && tw == w) {                                                                              \
        lc.blockDim = dim3(nt);                                                                            \
        lc.dynamicSmemBytes = Step64Shape<h, w>::smem(nt / 32);                                            \
        return cudaLaunchKernelEx(&lc, step64_kernel<h, w, nt, mb>, G, F, S, T, X, clk, ctl, slot);        \
    }
    SW2D_STEP64_TILES(SW2D_L64)
#undef SW2D_L64
    return cudaErrorInvalidValue;
}

cudaError_t launch_pack_gn(const double *n, int rows, int cols, int pitch, double g, double *gnx, double *gny,
                           cudaStream_t st) {
    pack_gn_kernel<<<detail::grid_for((long long)rows * cols, 256), 256, 0, st>>>(n, rows, cols, pitch, g, gnx, gny);
    return cudaGetLastError();
}

}  // namespace sw2d
