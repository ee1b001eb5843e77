// sw2d_step64.cuh -- the FP64 step kernel: one iteration of the reference
// loop (SW2D-GPU_linux/src/SW2D-GPU.cu:1256-1336) on a TH x TW tile per CTA.
//
// Same decomposition, halo and clock bookkeeping as step_kernel
// (sw2d_device.cuh: 4 halo cells north and west, 3 south and east, the CFL
// bound of the new state known when the launch ends), and the same bits as the
// serial oracle: every product, sum, quotient and root below is the correctly
// rounded one of the reference's expression.  What differs is what it costs.
// The kernel is bound by the FP64 pipe (2 results per SM and cycle, 1/64 of
// FP32; 83 % busy in step_kernel, about 520 FP64 instructions per cell), so
// work is taken off that pipe:
//
//   * an upwinded flux is formed once and read by the two faces it separates
//     (step_kernel formed it for each), the bed+depth sum once per cell, and
//     g n^2 of a face once per handle (the planes gnx, gny);
//   * halves and quarters ride on exact powers of two folded into dt2/dx,
//     dt2/dy and dt2 (the scaled product rounds as the unscaled one);
//   * divisions, roots and the friction power's polynomials run in integer
//     arithmetic (sw2d_f64math.cuh: a 53-bit result and its exact remainder),
//     divisions by dx and dy with a reciprocal kept per handle;
//   * what a face needs differs from face to face, and an FP64 instruction
//     holds the pipe 64 cycles for 1 lane as for 32: faces and fluxes are
//     sorted into lists first, and a cell's final depth is its provisional one
//     where nothing changed it;
//   * threshold and sign tests, clamps and maxima are integer comparisons of
//     the bits;
//   * the CFL bound is a maximum: an FP32 estimate of every face's wave speed
//     finds the few faces that can hold the CTA's maximum, and only those are
//     evaluated in FP64;
//   * rain and evaporation are counted per cell and multiplied once per CTA
//     where they are uniform; sums that are zero in a whole warp are skipped.
//
// The scaled products differ from the unscaled ones only where one of them leaves the
// normal range: below 1e-300 (by a subnormal), or above 4e307, a quarter of the largest
// number (a run that grows without bound is reported an iteration or two earlier).
// Halving on the exponent instead is exact there too, and took 5.0 against 4.8 ms on
// the 256 x 512 channel and 10.9 against 10.0 on 1013 x 900.
#pragma once

#include "sw2d_device.cuh"
#include "sw2d_f64math.cuh"

namespace sw2d {

// Tables of the friction power, filled by pow_tables_kernel (with those of the
// plain det_log / det_exp) before the first use (init_det_tables).
static __device__ PowTables g_pow_tab;

static __global__ void pow_tables_kernel() {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    det_tables_entry(t);
    if (t < 128) {
        const double c = 1.0 + (double)t * 0.0078125;
        g_pow_tab.inv[t] = 1.0 / c;
        g_pow_tab.logc[t] = det_log_series(c);
    }
    if (t < 64)
        g_pow_tab.exp2j[t] =
            det_exp_series((double)t * (0x1.62e42p-1 / 64.0) + (double)t * (0x1.fdf473de6af28p-22 / 64.0));
    if (t < 2 * kPowE) {
        const double e = (double)(t - kPowE);
        g_pow_tab.ehi[t] = e * 0x1.62e42p-1;
        g_pow_tab.elo[t] = e * 0x1.fdf473de6af28p-22;
    }
    if (t < 2 * kPowN) {
        const double n = (double)(t - kPowN);
        g_pow_tab.nhi[t] = n * (0x1.62e42p-1 / 64.0);
        g_pow_tab.nlo[t] = n * (0x1.fdf473de6af28p-22 / 64.0);
    }
}

// The friction power for what the integer form does not cover (d_pow43_int).
static __device__ __noinline__ double pow43_rest(double x) {
    bool ok;
    const double r = d_pow43_fast(x, &g_pow_tab, &ok);
    return ok ? r : det_exp(1.3333330 * det_log(x));
}

__device__ __forceinline__ double pow43(double x) {
    bool ok;
    const double r = d_pow43_int(x, &g_pow_tab, &ok);
    return ok ? r : pow43_rest(x);
}

// set_static with a Manning raster: bed, active mask (pack_static_kernel) and g n^2
// of every face, with the face's n the mean of its two cells' (the order of g * rn *
// rn in cu:196, cu:313); faces at the domain edge are never read.  Bound by the FP64
// pipe (8 operations a cell are 55 us at 2048 x 2048) but where neighbours are alike.
// set_static with a kernel of its own for g n^2 / this way: 64 x 64 27 / 22 us, 2048 x
// 2048 504 / 448 with land-use patches, 503 / 517 with every cell drawn by itself (an n
// plane alone, without the face products, took 445).
static __global__ void pack_static_gn_kernel(const double *__restrict__ z, const double *__restrict__ n, int rows,
                                             int cols, int pitch, double nodata, double g, double *__restrict__ zout,
                                             uint8_t *__restrict__ mask, double *__restrict__ gnx,
                                             double *__restrict__ gny) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cols) return;
    const unsigned lanes = __activemask();  // a warp's lanes share their row
    for (int i = blockIdx.y * blockDim.y + threadIdx.y; i < rows; i += gridDim.y * blockDim.y) {
        const size_t k = (size_t)i * cols + j, gp = (size_t)i * pitch + j;
        const double zv = z[k], nv = n[k], na = i > 0 ? n[k - cols] : nv, nw = j > 0 ? n[k - 1] : nv;
        mask[gp] = zv != nodata ? 1 : 0;
        zout[gp] = zv;
        const bool x = d_bits(na) != d_bits(nv), y = d_bits(nw) != d_bits(nv);
        double gx = 0.0, gy = 0.0;
        if (__any_sync(lanes, !x || !y)) gx = gy = g * nv * nv;  // both cells alike: most of a land-use raster
        if (__any_sync(lanes, x)) {
            const double r = d_half(nv + na);
            if (x) gx = g * r * r;
        }
        if (__any_sync(lanes, y)) {
            const double r = d_half(nv + nw);
            if (y) gy = g * r * r;
        }
        gnx[gp] = gx;
        gny[gp] = gy;
    }
}

// FP64 planes of the step kernel that step_kernel does not have: g n^2 of the
// x-face north of a cell and of the y-face west of it (nullptr: scalar n).
struct Step64Extra {
    const double *gnx, *gny;
    double gn;          // g n^2 of the scalar n
    KnownDivisor dx, dy;
    float thf;          // T.ge_th in FP32
    bool overlapped;    // launched as a programmatic dependent
};

constexpr int kStep64Arrays = 13;

// Work lists of one CTA: the faces (new discharges), and per warp the fluxes they read.
template <int TH, int TW>
struct Step64Shape {
    static constexpr int kFaces = 2 * (TH + 4) * (TW + 4);
    static constexpr int kFluxList = 192;  // entries of a warp's list of fluxes: a block's 128 and a remainder
    static constexpr size_t smem(int warps) {
        return (size_t)(TH + 7) * (TW + 7) * (kStep64Arrays * sizeof(double) + 3) +
               (size_t)(kFaces + warps * kFluxList) * sizeof(uint16_t) + 16;
    }
};
// List entries: the element of the tile, and for a face its direction and rule,
// for a flux its kind.
constexpr unsigned kItemY = 1u << 13, kItemRule = 14, kItemKind = 14, kItemElem = kItemY - 1;

// Appends `item` of the lanes with `keep` to a list in shared memory (one
// atomic per warp); every lane of a converged warp calls it.
__device__ __forceinline__ void append(uint16_t *list, int *count, bool keep, unsigned item, int lane) {
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (!bal) return;
    int base = 0;
    if (lane == 0) base = atomicAdd(count, __popc(bal));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (keep) list[base + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)item;
}

// The same downwards from `end`.
__device__ __forceinline__ void append_back(uint16_t *end, int *count, bool keep, unsigned item, int lane) {
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (!bal) return;
    int base = 0;
    if (lane == 0) base = atomicAdd(count, __popc(bal));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (keep) *(end - (base + __popc(bal & ((1u << lane) - 1u)))) = (uint16_t)item;
}

// GENERAL: for thresholds that the bit comparisons and the FP32 estimates do not
// cover (step64_general).
template <int TH, int TW, int NT, int MINB, bool GENERAL = false>
__global__ void __launch_bounds__(NT, MINB)
    step64_kernel(const GridDesc G, const ForcingDesc F, const StateBufs<double> S, const Thr<double> T,
                  const Step64Extra X, Clock *__restrict__ clk, const Control *__restrict__ ctl, const int slot) {
    constexpr int HN = 4;
    constexpr int RH = TH + 7, RW = TW + 7, RN = RH * RW;
    constexpr int NW = NT / 32;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *s_h = reinterpret_cast<double *>(smem_raw);
    double *s_z = s_h + RN;
    double *s_eta = s_z + RN;   // depth + bed
    double *s_umo = s_eta + RN;  // old um, later the corrected new um
    double *s_vno = s_umo + RN;
    double *s_uu = s_vno + RN;   // face velocities; s_uu later holds the provisional depth
    double *s_vv = s_uu + RN;
    double *s_fx = s_vv + RN;    // upwinded fluxes (times 4): of um through the cell, ...
    double *s_cu = s_fx + RN;    // ... of um through the corner west of the x-face,
    double *s_cv = s_cu + RN;    // of vn through the corner north of the y-face,
    double *s_fy = s_cv + RN;    // of vn through the cell
    double *s_rum = s_fy + RN;   // new um before the dry-cell fix
    double *s_rvn = s_rum + RN;
    constexpr int kFaces = Step64Shape<TH, TW>::kFaces;
    static_assert(RN <= (int)kItemElem, "list entries are 16 bits wide");
    uint16_t *s_face = reinterpret_cast<uint16_t *>(s_rvn + RN);  // momentum faces from the front, weir faces from the back
    uint16_t *s_flux = s_face + kFaces;  // one list per warp
    uint8_t *s_m = reinterpret_cast<uint8_t *>(s_flux + NW * Step64Shape<TH, TW>::kFluxList);
    uint8_t *s_tx = s_m + RN, *s_ty = s_tx + RN;  // 1: the x- / y-face takes the momentum equation
    uint8_t *s_dry = s_tx;  // after stage 2: the cell is active and dry after the provisional update
    double *s_hs = s_uu;

    __shared__ double s_red[NW][B_N];
    __shared__ int s_cnt[NW][2];
    __shared__ double s_k[9];  // dt2/dx and dt2/dy by 4, by 2, dt2 by 2, rr0 and rr1 times pct_hi, pct_lo
    __shared__ int s_n[2];  // lengths of the face lists: momentum, weir
    __shared__ unsigned s_est;
    __shared__ unsigned long long s_cm;
    __shared__ int s_nloc;
    __shared__ int s_srcp[kMaxLocalSources];
    __shared__ double s_srcq0[kMaxLocalSources], s_srcq1[kMaxLocalSources];
    __shared__ int s_wcnt[NW];

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int slot_out = slot == 2 ? 0 : slot + 1;
    const int slot_nx = slot == 0 ? 2 : slot - 1;
    const int rows = G.rows, cols = G.cols, pitch = G.pitch;
    const int ti = blockIdx.x / G.tiles_w, tj = blockIdx.x - ti * G.tiles_w;
    const int I0 = ti * TH - HN, J0 = tj * TW - HN;  // global index of smem (0,0)

    // ---- stage 0: stage the tile + halo in shared memory --------------------
    // Launched as a programmatic dependent of the previous iteration (X.overlapped:
    // at most one CTA per SM), the static fields are read while that one drains,
    // then its completion (and the visibility of its writes) is waited for.
    // Otherwise they are read with the state, after the plan: the launches of a
    // replay past the end time then load nothing (an advance of one iteration and
    // 47 such: 4.52 -> 3.84 ms at 2048 x 2048, 1.25 -> 1.05 at 1024 x 1024).
    auto stage_static = [&](int idx) {
        const int r = idx / RW, c = idx - (idx / RW) * RW;
        const int gi = I0 + r, gj = J0 + c;
        const bool in = (unsigned)gi < (unsigned)rows && (unsigned)gj < (unsigned)cols;
        const size_t gp = (size_t)gi * pitch + gj;
        s_z[idx] = in ? S.z[gp] : 0.0;
        s_m[idx] = in ? S.mask[gp] : (uint8_t)0;
        s_tx[idx] = s_ty[idx] = 0;
    };
    if (X.overlapped)
        for (int idx = tid; idx < RN; idx += NT) stage_static(idx);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const Clock &ci = clk[slot];
    const Plan &pl = ci.plan;

    if (!pl.run) {  // nothing to do: carry the state's clock forward
        if (blockIdx.x == 0 && wid == 0) carry_slot_deferred_warp(lane, clk, slot, slot_out, slot_nx);
        return;
    }

    const int buf = ci.buf;
    const double *__restrict__ Hin = S.h[buf];
    const double *__restrict__ Uin = S.um[buf];
    const double *__restrict__ Vin = S.vn[buf];
    double *__restrict__ Hout = S.h[1 - buf];
    double *__restrict__ Uout = S.um[1 - buf];
    double *__restrict__ Vout = S.vn[1 - buf];

    const LaunchScalars<double> LS = pl.d;
    const double dt2 = LS.dt2;
    const double dx = G.sd.dx, dy = G.sd.dy, g = G.sd.g;
    const unsigned long long gt_th = d_bits(T.gt_th), ge_th = d_bits(T.ge_th);
    const unsigned long long gt_ev = d_bits(T.gt_evmin);
    // x >= th and x > EV_WL_min: on the bits where the constant is positive
    auto wet = [&](double x) { return GENERAL ? x >= T.ge_th : d_ge_pos(x, ge_th); };
    auto above_ev = [&](double x) { return GENERAL ? x >= T.gt_evmin : d_ge_pos(x, gt_ev); };

    for (int idx = tid; idx < RN; idx += NT) {
        const int r = idx / RW, c = idx - (idx / RW) * RW;
        const int gi = I0 + r, gj = J0 + c;
        const bool in_r = (unsigned)gi < (unsigned)rows, in_c = (unsigned)gj < (unsigned)cols;
        const size_t gp = (size_t)gi * pitch + gj;
        const double h = in_r && in_c ? Hin[gp] : 0.0;
        if (!X.overlapped) stage_static(idx);
        s_h[idx] = h;
        s_eta[idx] = h + s_z[idx];  // this thread's own s_z
        s_umo[idx] = ((unsigned)gi <= (unsigned)rows && in_c) ? Uin[gp] : 0.0;
        s_vno[idx] = (in_r && (unsigned)gj <= (unsigned)cols) ? Vin[gp] : 0.0;
    }
    // per-launch products, one lane each
    if (wid == NW - 1 && lane < 9) {
        const double a = lane < 4 ? (lane & 1 ? LS.dt2dy : LS.dt2dx) : (lane == 4 ? dt2 : (lane < 7 ? LS.rr0 : LS.rr1));
        const double b = lane < 2 ? 0.25 : (lane < 5 ? 0.5 : (lane & 1 ? G.sd.pct_hi : G.sd.pct_lo));
        s_k[lane] = a * b;
    }
    if (tid == 0) {
        s_nloc = 0;
        s_n[0] = s_n[1] = 0;
        s_est = 0u;
        s_cm = 0ull;
    }
    // point sources inside this tile's provisional-depth region, kept in
    // list order so that a later source on the same cell wins (cu:545)
    if (G.n_src > 0) {
        __syncthreads();
        const double area = G.dx * G.dy;
        for (int base = 0; base < G.n_src; base += NT) {
            const int s = base + tid;
            bool in = false;
            int p = 0;
            if (s < G.n_src) {
                const int cell = F.src_cell[s];
                const int gi = cell / cols, gj = cell - (cell / cols) * cols;
                const int r = gi - I0, c = gj - J0;
                in = (r >= 2 && r < TH + 5 && c >= 2 && c < TW + 5);
                p = r * RW + c;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, in);
            if (lane == 0) s_wcnt[wid] = __popc(bal);
            __syncthreads();
            if (in) {
                int off = s_nloc;
                for (int w = 0; w < wid; w++) off += s_wcnt[w];
                off += __popc(bal & ((1u << lane) - 1u));
                if (off < kMaxLocalSources) {
                    s_srcp[off] = p;
                    s_srcq0[off] = source_rate(F, G.n_src, s, pl.t0, area);
                    s_srcq1[off] = source_rate(F, G.n_src, s, pl.t1, area);
                } else {
                    atomicOr(&clk[slot_out].status, (unsigned)ST_TOO_MANY_LOCAL_SOURCES);
                }
            }
            __syncthreads();
            if (tid == 0) {
                int tot = s_nloc;
                for (int w = 0; w < NW; w++) tot += s_wcnt[w];
                s_nloc = tot < kMaxLocalSources ? tot : kMaxLocalSources;
            }
            __syncthreads();  // s_wcnt is rewritten by the next chunk
        }
    }
    __syncthreads();

    const double *__restrict__ W = S.rainw;  // spatial rain factors (extension) or nullptr
    const int nloc = s_nloc;
    const double pct_hi = G.sd.pct_hi, pct_lo = G.sd.pct_lo;
    const bool storm = F.rain_kind == RAIN_STORM;

    // ---- stage 1: face velocities (cu:363-453) ------------------------------
    for (int idx = tid; idx < RN; idx += NT) {
        const int r = idx / RW, c = idx - (idx / RW) * RW;
        const int gi = I0 + r, gj = J0 + c;
        const double h = s_h[idx];
        if (r >= 1) {
            double hm;
            if (gi == rows) hm = s_h[idx - RW];
            else if (gi == 0) hm = h;
            else hm = d_half(h + s_h[idx - RW]);
            const double q = s_umo[idx];  // (at rest the division is left out; with th = 0 it may be 0 / 0)
            s_uu[idx] = wet(hm) && (GENERAL || !d_is_zero(q)) ? d_div(q, hm) : 0.0;
        }
        if (c >= 1) {
            double hn;
            if (gj == cols) hn = s_h[idx - 1];
            else if (gj == 0) hn = h;
            else hn = d_half(h + s_h[idx - 1]);
            const double q = s_vno[idx];
            s_vv[idx] = wet(hn) && (GENERAL || !d_is_zero(q)) ? d_div(q, hn) : 0.0;
        }
    }

    // ---- stage 1a: what each face does (cu:116-165, cu:232-282) --------------
    // A warp's FP64 instruction costs the same for 1 as for 32 lanes, and on a
    // thin film over steep ground dry-bed rules and momentum alternate from face
    // to face, so the faces are sorted into a list for each first.
    constexpr int FH = TH + 4, FW = TW + 4, FN = FH * FW;  // faces: rows/cols [2, TH+6) x [2, TW+6)
    for (int b0 = wid * 32; b0 < FN; b0 += NT) {
        const int k = b0 + lane;
        const int r = 2 + k / FW, c = 2 + (k - (k / FW) * FW);
        const int p = r * RW + c;
        const int gi = I0 + r, gj = J0 + c;
        int rule_x = 0, rule_y = 0;  // 1, 2, 3: dry-bed rules, 4: momentum, 0: no flow
        const bool in = k < FN && (unsigned)gi <= (unsigned)rows && (unsigned)gj < (unsigned)cols;
        if (in) {
            const double hb = s_h[p], zb = s_z[p], eb = s_eta[p];
            const bool b_act = s_m[p] != 0, b_wet = d_ge_pos(hb, gt_th), b_ge = wet(hb);
            // cell "a" (north / west) of the face; p is "b"
            auto rule_of = [&](int pa) -> int {
                const double ha = s_h[pa];
                const bool a_wet = d_ge_pos(ha, gt_th);
                if (!(b_act && s_m[pa] && (a_wet || b_wet))) return 0;
                if (d_lt(eb, s_z[pa])) return a_wet ? 1 : 0;   // cu:130: b's surface below a's bed
                if (d_lt(s_eta[pa], zb)) return b_wet ? 2 : 0;  // cu:138
                // cu:149: exactly one side strictly wet; false for NaN
                const bool a_dry = !wet(ha) && !d_is_nan(ha);
                const bool b_dry = !b_ge && !d_is_nan(hb);
                return (b_wet && a_dry) || (b_dry && a_wet) ? 3 : 4;
            };
            if (gi > 0 && gi < rows) rule_x = rule_of(p - RW);
            // free outfall (extension): the weir formula of rule 1
            else if (gi == rows && G.south_open && s_m[p - RW] && d_ge_pos(s_h[p - RW], gt_th)) rule_x = 1;
            if (gj > 0 && gi < rows) rule_y = rule_of(p - 1);
        }
        if (k < FN) {
            s_tx[p] = rule_x == 4;
            s_ty[p] = rule_y == 4;
            if (rule_x == 0) s_rum[p] = 0.0;
            if (rule_y == 0) s_rvn[p] = 0.0;
        }
        append(s_face, &s_n[0], rule_x == 4, p, lane);
        append(s_face, &s_n[0], rule_y == 4, p | kItemY, lane);
        append_back(s_face + kFaces - 1, &s_n[1], rule_x >= 1 && rule_x <= 3, p | (rule_x << kItemRule), lane);
        append_back(s_face + kFaces - 1, &s_n[1], rule_y >= 1 && rule_y <= 3, p | kItemY | (rule_y << kItemRule), lane);
    }
    __syncthreads();

    // ---- stage 1b: upwinded fluxes (cu:172-190, cu:289-307), each once ------
    // vel (o + s) / 2 + |vel| (s - o) / 2 with vel = (v + w) / 2 is a quarter of
    // (v + w) (o + s) + |v + w| (s - o); for every flux the second factor is
    // (lower-index value) - (higher-index value) of the discharge.
    //   kind 0: fx[p], of um through cell p, between the x-faces p and p + RW
    //   kind 1: cv[p], of vn through the corner between the y-faces p - RW and p
    //   kind 2: cu[p], of um through the corner between the x-faces p - 1 and p
    //   kind 3: fy[p], of vn through cell p, between the y-faces p and p + 1
    // each read by the two faces it lies between where they take the momentum
    // equation (s_tx and s_ty are 0 outside the faces above).
    // A warp lists the needed ones of its own elements and forms them from that
    // list, so nothing waits for the other warps' lists. This, and the surface
    // elevations formed while staging (no barrier between the velocities and the
    // face rules), took two of the tile's barriers out: 321 -> 318 us an
    // iteration at 1024 x 1024, 106.3 -> 104.5 at 512 x 512, 43.3 -> 42.3 at 256 x 256.
    constexpr int EW = TW + 5, EN = (TH + 5) * EW;  // higher-index faces: rows/cols [2, TH+7) x [2, TW+7)
    uint16_t *list = s_flux + wid * Step64Shape<TH, TW>::kFluxList;
    int n_flux = 0;
    auto form_fluxes = [&](int n) {
        __syncwarp();
        for (int i = lane; i < n; i += 32) {
            const int it = list[i], kind = it >> kItemKind, e = it & ((1 << kItemKind) - 1);
            const int oq = kind < 2 ? -RW : -1, ov = kind == 0 || kind == 2 ? -RW : -1;
            const double *v = kind < 2 ? s_uu : s_vv, *q = kind == 0 || kind == 2 ? s_umo : s_vno;
            double *out = kind == 0 ? s_fx - RW : kind == 1 ? s_cv : kind == 2 ? s_cu : s_fy - 1;
            const double qb = q[e], qa = q[e + oq], vel = v[e] + v[e + ov];
            out[e] = vel * (qa + qb) + fabs(vel) * (qa - qb);
        }
        __syncwarp();
    };
    for (int b0 = wid * 32; b0 < EN; b0 += NT) {
        const int k = b0 + lane, e = (2 + k / EW) * RW + 2 + (k - (k / EW) * EW);
        bool need[4] = {false, false, false, false};
        if (k < EN) {
            const bool x = s_tx[e] != 0, y = s_ty[e] != 0;
            need[0] = x || s_tx[e - RW];
            need[1] = y || s_ty[e - RW];
            need[2] = x || s_tx[e - 1];
            need[3] = y || s_ty[e - 1];
            // (with th = 0 a velocity may be 0 / 0 where there is no discharge)
            const bool u0 = !GENERAL && d_is_zero(s_umo[e]), v0 = !GENERAL && d_is_zero(s_vno[e]);
            if (need[0] && u0 && d_is_zero(s_umo[e - RW])) s_fx[e - RW] = 0.0, need[0] = false;
            if (need[1] && v0 && d_is_zero(s_vno[e - RW])) s_cv[e] = 0.0, need[1] = false;
            if (need[2] && u0 && d_is_zero(s_umo[e - 1])) s_cu[e] = 0.0, need[2] = false;
            if (need[3] && v0 && d_is_zero(s_vno[e - 1])) s_fy[e - 1] = 0.0, need[3] = false;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const unsigned bal = __ballot_sync(0xffffffffu, need[q]);
            if (need[q]) list[n_flux + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)(e | (q << kItemKind));
            n_flux += __popc(bal);
        }
        if (n_flux > Step64Shape<TH, TW>::kFluxList - 128) {  // room for another block's
            const int whole = n_flux & ~31;
            form_fluxes(whole);
            if (lane < n_flux - whole) list[lane] = list[whole + lane];
            n_flux -= whole;
            __syncwarp();
        }
    }
    form_fluxes(n_flux);
    __syncthreads();

    // ---- stage 2: new face discharges (cu:98-354) ---------------------------
    const double qdx = s_k[0], qdy = s_k[1];  // with the fluxes' quarters
    const double hdx = s_k[2], hdy = s_k[3], hdt2 = s_k[4];
    const int n_mom = s_n[0], n_weir = s_n[1];
    const int mom_chunks = (n_mom + 31) / 32, chunks = mom_chunks + (n_weir + 31) / 32;
    for (int ch = wid; ch < chunks; ch += NW) {
        if (ch < mom_chunks) {
            const int i = ch * 32 + lane;
            if (i >= n_mom) continue;
            const int it = s_face[i], p = it & kItemElem;
            const bool isx = !(it & kItemY);
            const int r = p / RW, pa = isx ? p - RW : p - 1;
            const int gi = I0 + r, gj = J0 + p - r * RW;
            const double ha = s_h[pa], hb = s_h[p], za = s_z[pa], eb = s_eta[p];
            const double mo = isx ? s_umo[p] : s_vno[p];
            const double hsum = hb + ha, hm = d_half(hsum);
            // gravity (cu:166, cu:283): g hm (dt2/dx) (hb + zb - ha - za)
            const double u13 = g * hsum * (isx ? hdx : hdy) * (eb - ha - za);
            // convection along i and along j (cu:172-190, cu:289-307)
            const double *f1 = isx ? s_fx + p : s_cv + p + RW;
            const double *f2 = isx ? s_cu + p + 1 : s_fy + p;
            double a1 = qdx * (f1[0] - f1[-RW]), a2 = qdy * (f2[0] - f2[-1]);
            if (!isx && gi == 0) a1 = 0.0;  // cu:289-291
            if (isx && gj == 0) a2 = 0.0;   // cu:178-180
            const double rest = -a1 - a2 - u13;
            // friction (cu:194-199, cu:311-316): zero only when hm <= th or n == 0
            const double gn = X.gnx ? (isx ? X.gnx : X.gny)[(size_t)gi * pitch + gj] : X.gn;
            double q;
            if ((d_ge_pos(hm, gt_th) || d_is_nan(hm)) && !d_is_zero(gn)) {
                const double *t = isx ? s_vv + p : s_uu + p;
                const int o1 = isx ? 1 : RW, o2 = isx ? -RW : -1;
                const double t4 = t[0] + t[o1] + t[o2] + t[o1 + o2];  // 4 times vva / uua
                const double own = isx ? s_uu[p] : s_vv[p];
                const double speed = d_sqrt(d_fma(t4 * t4, 0.0625, own * own));
                const double x = hdt2 * d_div(gn * speed, pow43(hm));
                q = d_div((1.00 - x) * mo + rest, 1.00 + x);  // cu:203, cu:320
            } else {
                q = mo + rest;
            }
            (isx ? s_rum : s_rvn)[p] = q;
        } else {
            // dry-bed rules (cu:130-159, cu:247-276) and the outfall: a
            // coefficient times depth times sqrt(g depth) or sqrt(2 g depth)
            const int i = (ch - mom_chunks) * 32 + lane;
            if (i >= n_weir) continue;
            const int it = s_face[kFaces - 1 - i], rule = it >> kItemRule, p = it & kItemElem;
            const bool isx = !(it & kItemY);
            const int pa = isx ? p - RW : p - 1;
            const double ha = s_h[pa], hb = s_h[p];
            double d = rule == 1 ? ha : hb, w = rule == 1 ? 0.5440 : -0.544;
            if (rule == 3) {
                const double ea = s_eta[pa], eb = s_eta[p], za = s_z[pa], zb = s_z[p];
                d = fmax(eb, ea) - fmax(zb, za);
                w = d_ge_pos(hb, gt_th) ? -0.350 : 0.350;  // cu:151-154
            }
            (isx ? s_rum : s_rvn)[p] = w * d * d_sqrt((rule == 3 ? 2.00 * g : g) * d);
        }
    }
    __syncthreads();

    // storm rain at a cell centre; the centre (sx, sy) is per launch
    const double storm_amp = G.sd.storm_amp, storm_2s2 = G.sd.storm_2s2;
    auto storm_rate = [&](int gi, int gj, bool on, double sx, double sy) -> double {
        if (!on) return 0.0;
        const double x = ((double)gj + 0.5) * dx - sx;
        const double y = ((double)gi + 0.5) * dy - sy;
        return storm_amp * det_exp(-(x * x + y * y) / storm_2s2);
    };
    // ho - dt2 ((us - un) / dx + (ve - vw) / dy - ql - rr pct + evapo) (cu:654),
    // the terms that are zero everywhere left out; rp = rr pct
    const bool any_ev0 = !d_is_zero(LS.ev0), any_ev1 = !d_is_zero(LS.ev1);
    auto balance = [&](double ho, double un, double us, double vw, double ve, double ql, double rp, double evapo,
                       bool any_ev) -> double {
        double s = d_div_known(us - un, X.dx) + d_div_known(ve - vw, X.dy);
        if (nloc) s = s - ql;
        s = s - rp;
        if (any_ev) s = s + evapo;
        return ho - dt2 * s;
    };
    const bool uniform = !storm && !W;

    // ---- stage 3: provisional depth with forcing at t (cu:1278-1288) -------
    const double rp0_hi = s_k[5], rp0_lo = s_k[6];
    constexpr int PH = TH + 3, PW = TW + 3;  // rows/cols [2, TH+5) x [2, TW+5)
    for (int k = tid; k < PH * PW; k += NT) {
        const int r = 2 + k / PW, c = 2 + (k - (k / PW) * PW);
        const int p = r * RW + c;
        double hraw = 0.0;
        bool dry = false;
        if (s_m[p]) {
            const double ho = s_h[p];
            const bool hi = above_ev(ho);
            double ql = 0.0;
            for (int q = 0; q < nloc; q++)
                if (s_srcp[q] == p) ql = s_srcq0[q];
            double rp = hi ? rp0_hi : rp0_lo;
            if (!uniform) {
                double rr = storm ? storm_rate(I0 + r, J0 + c, pl.storm_on0, LS.sx0, LS.sy0) : LS.rr0;
                if (W) rr = rr * W[(size_t)(I0 + r) * pitch + (J0 + c)];
                rp = rr * (hi ? pct_hi : pct_lo);
            }
            hraw = balance(ho, s_rum[p], s_rum[p + RW], s_rvn[p], s_rvn[p + 1], ql, rp, hi ? LS.ev0 : 0.0, any_ev0);
            dry = !wet(d_clamp0(hraw));  // cu:657
        }
        s_hs[p] = hraw;
        s_dry[p] = dry;
    }
    __syncthreads();

    // ---- stage 4: dry-cell fix per face (cu:695-725) + final depth ----------
    // corrected face at p (a: the other cell's element): zero if it drains a dry
    // cell (a zero stays one, a NaN too); hit: a face of the cell was corrected
    auto fix = [&](double q, int p, int a, bool &hit) -> double {
        const bool drains = s_dry[(int)d_hi(q) < 0 ? p : a] != 0;
        if (!drains || d_is_zero(q) || d_is_nan(q)) return q;
        hit = true;
        return 0.0;
    };
    // With the same forcing at t and t + dt and none of its faces corrected, a
    // cell's final depth is the provisional one: the same operands.
    const bool steady = uniform && nloc == 0 && d_bits(LS.rr0) == d_bits(LS.rr1) && d_bits(LS.ev0) == d_bits(LS.ev1);
    const double rp1_hi = s_k[7], rp1_lo = s_k[8];
    float *s_hf = reinterpret_cast<float *>(s_fx);  // the fluxes are done with: FP32 depths for stage 5
    int n_hi = 0, n_lo = 0;  // active owned cells above / not above EV_WL_min
    double b_rain = 0.0, b_src = 0.0, b_out = 0.0, b_clamp = 0.0;
    bool bad = false;
    constexpr int OH = TH + 1, OW = TW + 1;  // rows/cols [3, TH+4) x [3, TW+4)
    for (int k = tid; k < OH * OW; k += NT) {
        const int r = 3 + k / OW, c = 3 + (k - (k / OW) * OW);
        const int p = r * RW + c;
        const int gi = I0 + r, gj = J0 + c;
        bool hit = false;
        const double un = fix(s_rum[p], p, p - RW, hit), us = fix(s_rum[p + RW], p + RW, p, hit);
        const double vw = fix(s_rvn[p], p, p - 1, hit), ve = fix(s_rvn[p + 1], p + 1, p, hit);
        double hv = 0.0, hraw = 0.0;
        const bool act = s_m[p] != 0;
        bool hi = false;
        double ql = 0.0, rp = 0.0;
        if (act) {
            const double ho = s_h[p];
            hi = above_ev(ho);
            for (int q = 0; q < nloc; q++)
                if (s_srcp[q] == p) ql = s_srcq1[q];
            rp = hi ? rp1_hi : rp1_lo;
            if (!uniform) {
                double rr = storm ? storm_rate(gi, gj, pl.storm_on1, LS.sx1, LS.sy1) : LS.rr1;
                if (W) rr = rr * W[(size_t)gi * pitch + gj];
                rp = rr * (hi ? pct_hi : pct_lo);
            }
            if (steady && !hit) hraw = s_hs[p];
            else hraw = balance(ho, un, us, vw, ve, ql, rp, hi ? LS.ev1 : 0.0, any_ev1);
            hv = d_clamp0(hraw);
        }
        s_h[p] = hv;  // the new depth; only this thread reads s_h[p] in this stage
        s_umo[p] = un;
        s_vno[p] = vw;
        if (r == TH + 3) s_umo[p + RW] = us;
        if (c == TW + 3) s_vno[p + 1] = ve;
        s_hf[p] = d_abs_float(hv);
        const bool core = r >= HN && c >= HN && r < TH + HN && c < TW + HN && gi < rows && gj < cols;
        if (core) {
            const size_t gp = (size_t)gi * pitch + gj;
            Hout[gp] = hv;
            Uout[gp] = un;
            Vout[gp] = vw;
            if (gi == rows - 1) {
                Uout[gp + pitch] = us;
                b_out += us;
            }
            if (act) {
                if (hi) n_hi++;
                else n_lo++;
                if (!uniform) b_rain += rp;
                if (nloc) b_src += ql;
                if (d_lt_zero(hraw)) b_clamp -= hraw;
            }
            if (!d_is_finite(hv) || !d_is_finite(un) || !d_is_finite(vw)) bad = true;
        }
    }
    __syncthreads();

    // ---- stage 5: CFL bound of the new state over the owned faces ----------
    // An FP32 estimate of |q / h| + sqrt(g h), within 2^-18 of the FP64 value,
    // is formed for every owned face between active cells (and the open south
    // faces).  The CTA's largest estimate among the faces certainly deeper than
    // th, less that margin, is a bar below the exact maximum: only faces whose
    // estimate reaches it are evaluated in FP64.  Estimates are compared as bits, so
    // that one beyond FP32 (infinite or 0 x infinity, in a run that grows without
    // bound) is the largest; it makes no bar.  GENERAL evaluates every face.
    const float gf = G.sf.g, thf = X.thf;
    auto faces = [&](auto &&visit) {
        for (int k = tid; k < TH * TW; k += NT) {
            const int r = HN + k / TW, c = HN + (k - (k / TW) * TW);
            const int p = r * RW + c;
            const int gi = I0 + r, gj = J0 + c;
            if (gi >= rows || gj >= cols || !s_m[p]) continue;
            if (gi > 0 && s_m[p - RW]) visit(s_umo[p], p, p - RW);
            if (gi == rows - 1 && G.south_open) visit(s_umo[p + RW], p, p);
            if (gj > 0 && s_m[p - 1]) visit(s_vno[p], p, p - 1);
        }
    };
    auto estimate = [&](double q, int p0, int p1, float &hm) -> unsigned {
        hm = 0.5f * (s_hf[p0] + s_hf[p1]);
        return __float_as_uint(__fdividef(d_abs_float(q), hm) + __fsqrt_rn(gf * hm));
    };
    constexpr float kMargin = 1.f / 131072.f;
    constexpr unsigned kInfinite = 0x7f800000u;
    unsigned sure = 0u, est = 0u;  // over faces certainly / possibly deeper than th
    if (!GENERAL)
        faces([&](double q, int p0, int p1) {
            float hm;
            const unsigned e = estimate(q, p0, p1, hm);
            if (hm >= thf * (1.f + kMargin)) sure = max(sure, e);
            if (hm >= thf * (1.f - kMargin)) est = max(est, e);
        });
    const unsigned wmax = __reduce_max_sync(0xffffffffu, sure);
    if (lane == 0 && wmax) atomicMax(&s_est, wmax);
    const bool any_bad = __syncthreads_or(bad);
    const unsigned bar = s_est < kInfinite ? __float_as_uint(__uint_as_float(s_est) * (1.f - kMargin)) : 0u;
    if (est >= bar) {
        // a face with the values of the thread's last one (still water of one
        // depth) is not evaluated again
        unsigned long long cm = 0ull, seen_q = 1ull, seen_0 = 0ull, seen_1 = 0ull;
        faces([&](double q, int p0, int p1) {
            if (!GENERAL) {
                float hf;
                if (estimate(q, p0, p1, hf) < bar || !(hf >= thf * (1.f - kMargin))) return;
            }
            const double h0 = s_h[p0], h1 = s_h[p1];
            if ((d_bits(q) << 1) == seen_q && d_bits(h0) == seen_0 && d_bits(h1) == seen_1) return;
            seen_q = d_bits(q) << 1;
            seen_0 = d_bits(h0);
            seen_1 = d_bits(h1);
            const double hm = 0.50 * (h0 + h1);
            if (!wet(hm)) return;
            const double v = (d_is_zero(q) ? 0.0 : fabs(d_div(q, hm))) + d_sqrt(g * hm);
            if (!d_is_nan(v)) cm = d_bits(v) > cm ? d_bits(v) : cm;
        });
        if (cm) atomicMax(&s_cm, cm);
    }

    // ---- block reductions, one atomic per quantity --------------------------
    n_hi = __reduce_add_sync(0xffffffffu, n_hi);
    n_lo = __reduce_add_sync(0xffffffffu, n_lo);
    double vals[4] = {b_rain, b_src, b_out, b_clamp};
#pragma unroll
    for (int q = 0; q < 4; q++) {
        double v = vals[q];
        if (__any_sync(0xffffffffu, !d_is_zero(v))) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        vals[q] = v;
    }
    if (lane == 0) {
        s_red[wid][0] = vals[0];
        s_red[wid][1] = vals[1];
        s_red[wid][2] = vals[2];
        s_red[wid][3] = vals[3];
        s_cnt[wid][0] = n_hi;
        s_cnt[wid][1] = n_lo;
    }
    __syncthreads();
    // warp 0 takes what the last CTA of the launch needs to its ticket, warp 1
    // the budgets, which only the next launch reads
    if (wid == 0) {
        if (lane == 0) accumulate_cmax(clk[slot_out], blockIdx.x % kBuckets, d_from_bits(s_cm), any_bad);
        finish_cta_deferred_warp(lane, clk, slot, slot_out, slot_nx, pl, *ctl, G, F);
    } else if (tid == 32) {
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        int c_hi = 0, c_lo = 0;
        for (int w = 0; w < NW; w++) {
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (!d_is_zero(s_red[w][q])) acc[q] += s_red[w][q];
            c_hi += s_cnt[w][0];
            c_lo += s_cnt[w][1];
        }
        if (uniform) acc[0] = counted_rate(c_hi, rp1_hi) + counted_rate(c_lo, rp1_lo);
        const double area = G.dx * G.dy;
        const double scale = pl.d.dt2 * area;
        double v[B_N];
        v[B_RAIN] = acc[0] * scale;
        v[B_SRC] = acc[1] * scale;
        v[B_EV] = counted_rate(c_hi, LS.ev1) * scale;
        v[B_OUT] = acc[2] * pl.d.dt2 * G.dy;
        v[B_CLAMP] = acc[3] * area;
        accumulate_budgets(clk[slot_out], blockIdx.x % kBuckets, v);
    }
}

}  // namespace sw2d
