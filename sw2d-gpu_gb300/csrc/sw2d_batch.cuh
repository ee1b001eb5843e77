// sw2d_batch.cuh -- many scenarios of uneven size advanced by one persistent
// FP32 launch per iteration.
//
// Each scenario keeps its own state, static fields, forcing, CFL time step
// and clock (three rotating slots, as a single-scenario handle).  The work of
// one launch is the list of (scenario, column tile, row strip) units of every
// scenario in the batch, the longest first; each warp of a fixed grid of CTAs
// starts on the unit of its own index and pulls further ones from a queue head
// (one atomic each), so scenarios of 64 x 64 and 2048 x 2048 cells share the GPU
// without load imbalance.  A scenario's units take a ticket when they finish; the
// last one finalises that scenario's clock slot (time, CFL bound, the plan of its
// next iteration), whose budgets the first one of the next launch folds -- no warp
// ever waits.
//
// The unit table, its length and the scenario descriptors live in device
// memory, so the CUDA graph of launches stays valid while scenarios are
// admitted and retired between replays.  A scenario whose plan says "stop"
// (end time reached) costs one queue entry per unit and launch until it is
// retired.
#pragma once

#include "sw2d_stream_unit.cuh"

namespace sw2d {

// Compact per-scenario status for the host, written by the finaliser.
struct ScenarioStatus {
    double t;
    long long steps;
    int running;     // the next iteration will run (end time not reached)
    int nonfinite;
    unsigned status;
    int pad;
};

struct ScenarioDev {
    GridDesc G;
    ForcingDesc F;
    Thr<float> T;
    Control ctl;
    float *h[2], *um[2], *vn[2], *hr[2];  // hr: depth remainders (compensated depth)
    const float *z, *dzx, *dzy, *nman;  // elevation, bed differences across faces, Manning n
    const uint8_t *mask;
    Clock *clk;                // three slots
    ScenarioStatus *status;    // this scenario's entry of the batch status array
    int tiles_w, strip_h, nunits, pad;
};

struct BatchHeader {
    int n_units;               // length of the unit table
    int pad;
    unsigned int head[3];      // queue heads, one per launch parity
    unsigned int pad2;
};

struct BatchDev {
    ScenarioDev *scen;
    const int2 *units;         // (scenario slot, unit index within the scenario)
    BatchHeader *hdr;
};

__device__ inline void write_status(const Clock &c, ScenarioStatus *st) {
    st->t = c.t;
    st->steps = c.steps;
    st->running = c.plan.run;
    st->nonfinite = (int)c.nonfinite;
    st->status = c.status;
}

// Reads the cache lines of a scenario's descriptor into L1 (one line per lane).
__device__ __forceinline__ void prefetch_scenario(const ScenarioDev *S, int lane) {
    if (lane * 128 < (int)sizeof(ScenarioDev))
        asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char *>(S) + lane * 128));
}

template <int NWARP, int MINB, int UNR>
__global__ void __launch_bounds__(NWARP * 32, MINB) batch_step_kernel(const BatchDev B, const int slot) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int slot_out = slot == 2 ? 0 : slot + 1;
    const int slot_nx = slot == 0 ? 2 : slot - 1;
    // Every warp starts on a unit of its own and pulls further ones from the
    // queue.  With at most one unit per warp the units are dealt out across the
    // CTAs first, so that they spread over the SMs.
    const int warps = (int)gridDim.x * NWARP, n_units = B.hdr->n_units;
    unsigned u = n_units <= warps ? wid * gridDim.x + blockIdx.x : blockIdx.x * NWARP + wid;
    int2 ue = make_int2(0, 0);
    if (u < (unsigned)n_units) {
        ue = B.units[u];
        prefetch_scenario(B.scen + ue.x, lane);
    }
    // Launched as a programmatic dependent of the previous iteration: the unit
    // table and the descriptors are the host's, but the queue head, every
    // scenario's state and clock are that grid's, so wait until it has completed
    // and its writes are visible, then let the next iteration's grid be
    // scheduled; its CTAs wait here the same way
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (blockIdx.x == 0 && threadIdx.x == 0) B.hdr->head[slot_out] = 0u;  // queue of the next launch
    while (u < (unsigned)n_units) {
        const ScenarioDev &S = B.scen[ue.x];
        const Clock &ci = S.clk[slot];
        const int run = ci.plan.run;
        StreamAcc A;
        acc_clear(A);
        if (run) {
            StreamView V;
            const int b = ci.buf;
            V.rows = S.G.rows;
            V.cols = S.G.cols;
            V.pitch = S.G.pitch;
            V.south_open = S.G.south_open;
            V.Hin = S.h[b];
            V.Uin = S.um[b];
            V.Vin = S.vn[b];
            V.DZX = S.dzx;
            V.DZY = S.dzy;
            V.Rin = S.hr[b];
            V.Rout = S.hr[1 - b];
            V.Nin = S.nman;
            V.Min = S.mask;
            V.Win = nullptr;  // batched scenarios rain uniformly
            V.Hout = S.h[1 - b];
            V.Uout = S.um[1 - b];
            V.Vout = S.vn[1 - b];
            V.GS = S.G.sf;
            V.T = S.T;
            V.LS = ci.plan.f;
            V.storm = S.F.rain_kind == RAIN_STORM;
            V.on0 = ci.plan.storm_on0;
            V.on1 = ci.plan.storm_on1;
            V.n_src = S.G.n_src;
            V.F = &S.F;
            V.t0 = ci.plan.t0;
            V.t1 = ci.plan.t1;
            V.dx = S.G.dx;
            V.dy = S.G.dy;
            const int ct = ue.y % S.tiles_w, rs = ue.y / S.tiles_w;
            // batched scenarios take neither a storm nor point sources nor rain
            // factors (sw2d_batch_add accepts none), so the uniform-forcing unit
            const int r0 = rs * S.strip_h;
            stream_unit<UNR, false, kFormUniform>(V, ct, r0, min(r0 + S.strip_h, V.rows), lane, nullptr, nullptr,
                                                  nullptr, nullptr, A);
            warp_reduce_acc<false, kFormUniform>(A);
            if (lane == 0) accumulate_cmax(S.clk[slot_out], ue.y % kBuckets, (double)A.cm, A.bad);
            // the budgets, one per lane (B_RAIN .. B_CLAMP; no sources here): FP64
            // operations have long latencies and this warp is on the way to its ticket
            if (lane < B_N && lane != B_SRC) {
                const LaunchScalars<float> &L = ci.plan.f;
                const double area = S.G.dx * S.G.dy, dt2 = ci.plan.d.dt2;
                const float rate = lane == B_RAIN ? L.rr1 * S.G.sf.pct_hi : (lane == B_EV ? L.ev1 : 0.f);
                const float rate_lo = lane == B_RAIN ? L.rr1 * S.G.sf.pct_lo : 0.f;
                const float sum = lane == B_OUT ? A.out : (lane == B_CLAMP ? A.clamp : 0.f);
                const double per = lane == B_CLAMP ? area : dt2 * (lane == B_OUT ? S.G.dy : area);
                const double v = (double)sum + counted_rate(A.n_hi, rate) + counted_rate(A.n_act - A.n_hi, rate_lo);
                if (v != 0.0) atomicAdd(&S.clk[slot_out].stepb[lane][ue.y % kBuckets], v * per);
            }
        }
        // the scenario's first unit to finish folds the budgets of the previous
        // iteration, its last finalises this one (finish_cta_deferred_warp)
        unsigned ticket = 0u;
        if (lane == 0) {
            __threadfence();
            ticket = atomicAdd(&S.clk[slot_out].done_blocks, 1u);
        }
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        if (run && ticket == 0u) fold_slot_warp(lane, S.clk[slot_nx], S.clk[slot]);
        if (ticket == (unsigned)S.nunits - 1u) {
            __threadfence();
            if (run)
                finalize_slot_deferred_warp(lane, ci, S.clk[slot_out], S.clk[slot_nx], ci.plan, S.ctl, S.G, S.F);
            else
                carry_slot_deferred_warp(lane, S.clk, slot, slot_out, slot_nx);
            __syncwarp();
            if (lane == 0) write_status(S.clk[slot_out], S.status);
        }
        // the next unit: the queue starts behind the warps' own
        if (n_units <= warps) break;
        unsigned k = 0;
        if (lane == 0) k = atomicAdd(&B.hdr->head[slot], 1u);
        u = (unsigned)warps + __shfl_sync(0xffffffffu, k, 0);
        if (u < (unsigned)n_units) ue = B.units[u];
        __syncwarp();
    }
}

}  // namespace sw2d
