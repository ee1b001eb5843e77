// sw2d_stream_builds.h -- the builds of the FP32 streaming kernel and the launch
// shape, shared by its one-iteration launches (step_f32.cu) and its pipelined
// ones (pipe_f32.cu).
#pragma once

#include <cstring>
#include <numeric>

#include "sw2d_stream.cuh"

namespace sw2d {

namespace {

// The launch shape: ceil(rows / strip_h) strips, split evenly or with the
// heights skewed (strip_rows); for the pipelined launches the units go to
// warps in a scattered order (a multiplier near 0.618 units, coprime with
// units).
StreamShape stream_shape(int rows, int tiles_w, int strip_h, int units, bool scatter, int skew) {
    StreamShape sh;
    std::memset(&sh, 0, sizeof(sh));
    sh.tiles_w = tiles_w;
    sh.strips = (rows + strip_h - 1) / strip_h;
    sh.units = units;
    sh.perm = 1;
    sh.skew = skew;
    if (scatter && units > 2) {
        int p = (int)(units * 0.6180339887498949);
        if (p < 1) p = 1;
        while (std::gcd(p, units) != 1) p++;
        sh.perm = p;
    }
    return sh;
}

}  // namespace

// Shared-memory share of the L1/shared split for the streaming kernel, in
// percent.  Each CTA needs only a few KB (source slots and the reduction, plus
// the 1 KB the system reserves), but asking for the largest L1 left room for
// just 2-3 CTAs per SM and capped the occupancy of the smaller-CTA builds.
constexpr int kStreamCarveoutPercent = 25;

// Builds of the streaming kernel the autotuner chooses from: (id, warps per
// CTA, minimum resident CTAs per SM -- which sets the register budget: 20
// warps per SM fit 96 registers, 16 fit 128, 24 fit 80 --, unrolling of the
// row loop).  Build 0 is the default.
#define SW2D_STREAM_VARIANTS(X) \
    X(0, 2, 10, 2) X(1, 2, 10, 1) X(2, 4, 5, 2) X(3, 8, 2, 1) X(4, 8, 2, 2) X(5, 12, 2, 1)

// Build 6 (step_f32.cu) has no pipelined form: its launches run build 0's.
constexpr int kTmaVariant = 6;

// Attributes of a build's pipelined forms (pipe_f32.cu)
cudaError_t prepare_stream_pipe(int variant);

// The form that carries the forcing that is set and, but with rain factors, no other.
inline int stream_form(bool storm, bool sources, bool rainw) {
    if (rainw) return storm || sources ? kFormAny : kFormUniform;
    return storm ? (sources ? kFormAny : kFormStorm) : (sources ? kFormSources : kFormUniform);
}

// Whether strips of strip_h rows run the form's SKIP build (launch_stream_step).
inline bool stream_skips(int variant, int strip_h, int form, bool rainw) {
    return variant == 0 && !(rainw && form == kFormAny) && strip_h <= (form == kFormUniform && !rainw ? 6 : 13);
}

// The unrolling of a form's pipelined row loop in a build that unrolls by `un`
// (prepare_stream_pipe).
constexpr int pipe_unroll(int un, int form) { return form == kFormSources || form == kFormAny ? 1 : un; }

}  // namespace sw2d
