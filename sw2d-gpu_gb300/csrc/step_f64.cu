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
// stages overlap: 312 us per iteration on a 1013 x 900 catchment, 447 with one
// CTA of 768 (the stages then wait at each other's barriers), 358 with one CTA on
// a 32 x 32 tile (less halo, same wait); 256 to 448 threads are within 3 %.
//
// A tile's work runs on one SM, and an iteration takes as long as the SM with the
// most of it: a grid of one CTA per SM, or of two, is cut into the smallest tiles
// that still leave it so (step64_tile).  us per iteration, tiles 16x32 / 14x32 /
// 12x32 / 10x32 / 8x32 / 6x32, the one that the rule takes in brackets:
//   140 x 160  40.1 /  38.3  /  33.9  /  32.3  / 30.4 / (26.4)
//   180 x 256  42.1 /  40.5  /  38.2  / (34.1) / 55.6 /  49.4
//   200 x 256  43.6 /  40.2  / (38.4) /  55.3  / 56.6 /  50.0
//   256 x 256  44.3 / (42.4) /  62.4  /  59.7  / 58.3 /  69.8
// and, where two CTAs of 512 per SM hold the grid, 16x32 / 14x32: 256 x 512 63.5 /
// (57.2), 270 x 480 60.6 / (57.2), 256 x 370 59.2 / (54.8), 270 x 300 55.6 /
// (54.4); with few more CTAs of 16 x 32 than SMs most of these run alone, and
// 14 x 32 is the slower: 256 x 300 (160 CTAs) (48.4) / 51.9, 656 x 128 (164) (45.0)
// / 47.2; from 170 on it is the faster or within 4 % (672 x 128, 130 x 700).  The
// narrow tiles, 8x16 / 4x16 / 4x8: 64 x 64 21.7 / 20.1 / (18.6), 80 x 100 22.2 /
// (20.6) / 20.9, 117 x 131 (23.0) / 25.9 / 37.5.  Beyond two CTAs per SM the halo
// decides (4 x 8 has 2.3 faces for each one of the tile, 14 x 32 1.5, 16 x 32
// 1.4): 16x32 / 14x32 300 x 500 63.0 / 83.9, 400 x 400 79.2 / 82.5, 1013 x 900
// 312 / 334.  With one CTA per SM more threads shorten the stages: 8 x 16 23.2
// with 512 against 26.9 with 256, 8 x 32 30.6 with 768 against 34.2 with 384,
// 10 x 32 33.1 with 768 against 34.8 with 512; 14 x 32 and 16 x 32 are the
// exception (41.7 with 768 against 40.6 on 256 x 256, 43.5 against 42.3 on 230 x
// 300: the next launch's CTAs, which start early, then no longer fit beside them).
#define SW2D_STEP64_TILES(X)                                                                        \
    X(16, 32, 512, 2) X(14, 32, 512, 2) X(12, 32, 768, 1) X(10, 32, 768, 1) X(8, 32, 768, 1)        \
    X(6, 32, 512, 1) X(8, 16, 512, 1) X(4, 16, 256, 1) X(4, 8, 256, 1)

// The general build, for every grid of a handle that needs it: the largest tile.
#define SW2D_STEP64_GENERAL step64_kernel<16, 32, 512, 2, true>

bool step64_general(double ge_th, double gt_evmin, double g) {
    // th = 0 and EV_WL_min < 0 are no positive constants; the FP32 estimates of the
    // wave speeds hold for depths from 1e-20 m on and an ordinary g (a discharge that
    // FP32 flushes to zero is then below their margin)
    return !(ge_th >= 1e-20) || !(gt_evmin > 0.0) || !(g >= 1e-10 && g <= 1e10);
}

bool step64_tile_supported(int th, int tw) {
#define SW2D_S64(h, w, nt, mb) \
    if (th == h && tw == w) return true;
    SW2D_STEP64_TILES(SW2D_S64)
#undef SW2D_S64
    return false;
}

std::string step64_build_name(int th, int tw, bool general) {
    if (general) return "step64_kernel<16,32,512,2,general>";
#define SW2D_S64(h, w, nt, mb) \
    if (th == h && tw == w) return "step64_kernel<" #h "," #w "," #nt "," #mb ">";
    SW2D_STEP64_TILES(SW2D_S64)
#undef SW2D_S64
    return "step64_kernel<?>";
}

// The smallest tile whose CTAs all have an SM to themselves; else the smallest of
// which all are resident where two run per SM, if 16 x 32 would give more than a
// twelfth of the SMs a second one; else 16 x 32.
void step64_tile(int rows, int cols, int sms, int *th, int *tw) {
    auto ctas = [&](int h, int w) { return (long long)((rows + h - 1) / h) * ((cols + w - 1) / w); };
    *th = 16;
    *tw = 32;
    int best = 16 * 32;
#define SW2D_D64(h, w, nt, mb)                                        \
    if (h * w < best && mb >= per_sm && ctas(h, w) <= per_sm * sms) { \
        best = h * w;                                                 \
        *th = h;                                                      \
        *tw = w;                                                      \
    }
    int per_sm = 1;
    SW2D_STEP64_TILES(SW2D_D64)
    if (best < 16 * 32 || ctas(16, 32) <= sms + sms / 12) return;
    per_sm = 2;
    SW2D_STEP64_TILES(SW2D_D64)
#undef SW2D_D64
}

namespace {

template <class Kernel>
cudaError_t prepare_build(Kernel *k, size_t smem) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
}

}  // namespace

cudaError_t prepare_step64(int th, int tw, bool general) {
    const cudaError_t e = init_det_tables();
    if (e != cudaSuccess) return e;
    if (general) return prepare_build(SW2D_STEP64_GENERAL, Step64Shape<16, 32>::smem(16));
#define SW2D_P64(h, w, nt, mb) \
    if (th == h && tw == w) return prepare_build(step64_kernel<h, w, nt, mb>, Step64Shape<h, w>::smem(nt / 32));
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
    X.overlapped = nblocks <= sms;
    attr[0].val.programmaticStreamSerializationAllowed = X.overlapped ? 1 : 0;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(nblocks);
    lc.stream = st;
    lc.attrs = attr;
    lc.numAttrs = 1;
    if (step64_general(T.ge_th, T.gt_evmin, G.sd.g)) {
        if (th != 16 || tw != 32) return cudaErrorInvalidValue;
        lc.blockDim = dim3(512);
        lc.dynamicSmemBytes = Step64Shape<16, 32>::smem(16);
        return cudaLaunchKernelEx(&lc, SW2D_STEP64_GENERAL, G, F, S, T, X, clk, ctl, slot);
    }
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

cudaError_t launch_pack_static_gn(const double *z, const double *n, int rows, int cols, int pitch, double nodata,
                                  double g, double *zout, uint8_t *mask, double *gnx, double *gny, cudaStream_t st) {
    const dim3 block(32, 8), grid((cols + 31) / 32, (unsigned)((rows + 7) / 8 < 65535 ? (rows + 7) / 8 : 65535));
    pack_static_gn_kernel<<<grid, block, 0, st>>>(z, n, rows, cols, pitch, nodata, g, zout, mask, gnx, gny);
    return cudaGetLastError();
}

}  // namespace sw2d
