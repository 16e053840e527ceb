// Fused surface-flow step: one launch = one accepted step of HydroPol2D_Main_While.m
// :403-782 (rain + Green-Ampt + clamp, local-inertial fluxes, draining limiter,
// continuity, outlet sink, running maximum / arrival time, CFL reductions, and the
// timestep refresh + clock advance, done by the next launch of a grid and by the last CTA to
// finish an ensemble member).
//
// Warp-streaming layout.  Each warp owns a strip of 32*CPL columns (CPL = 1 or 2 cells per
// lane; cell h of lane L sits at column CPL L + h), of which all but two columns on each side
// are its output, and walks down a block of rows.  The draining limiter makes a cell's new
// depth depend on cells two away (face <- donor scale <- donor's four faces <- their far
// cells); in x those neighbours come from other lanes by warp shuffles (hence the
// two-column apron on each side), in y from a rolling window of registers that holds the
// previous two rows.  Per row a lane does, for each of its cells: hydrology of (r, j), the
// x face (r, j) and y face (r-1|r, j), the donor scale of (r-1, j), the limited faces of
// row r-1 and the continuity / outlet / maxima / CFL of row r-2.  No CTA barrier inside the
// row loop.
//
// Memory: a cell is two 16-byte records -- the static {dz_x, dz_y, n^2, meta} and the
// state {h, q_x, q_y, dmax} -- read and one state record written.  A strip's records of one
// row are contiguous, so one 1-D bulk copy (TMA) brings each record row into a per-warp
// ring of shared-memory stages, counted in bytes by the stage's mbarrier; the rows after
// row k are in flight while row k is computed.
//
// Dry rows: a vote per row tells whether the strip's depths are all zero after the
// hydrology.  Faces and limiter are skipped when rows r-2..r are dry, continuity and CFL
// when rows r-3..r-1 are, and a row r with rows r-3..r dry (deep-dry) only writes row r-2's
// zero depth and fluxes and its running maximum; each shortcut stores exactly what the
// full computation would.
//
// CFL reductions: the step needs max(speed) and, over non-stagnant cells, max of the wave
// celerity sqrt(g*depth).  Because IEEE sqrt is correctly rounded and monotone, max of
// sqrt(x_i) equals sqrt(max x_i) exactly, so the kernel reduces speed^2 and g*depth and
// takes one square root at the end; the stagnant test speed < 0.01 becomes
// speed^2 < stag_s2 with stag_s2 the smallest value whose rounded root reaches 0.01.
//
// The state is double-buffered (StepScalars::cur selects the read side), so a CUDA graph
// of many launches needs no host involvement, and a launch after the end of the
// simulation is a no-op that leaves the buffers and the clock alone.
#pragma once

#include "hp2d_device.cuh"

namespace hp2d {

#ifndef HP2D_STAGES
#define HP2D_STAGES 4
#endif
constexpr int kStages = HP2D_STAGES;   // shared-memory ring depth of the row pipeline
#ifndef HP2D_ROW_UNROLL
#define HP2D_ROW_UNROLL 1
#endif
constexpr int kRowUnroll = HP2D_ROW_UNROLL;   // row-loop unroll (register renaming of the window)
// Phase (F) without a per-lane branch around each cell's body (stores and reductions masked
// instead), so that the CPL cells interleave: 3 % faster on the plain instantiations (60-minute
// dam-break 115.5 vs 111.8 GCUPS when it was introduced); the Green-Ampt + rain-map instantiation,
// at its register cap, ran 20.3 vs 21.2 with it and keeps the branch.
// What a row of wet cells costs is its instructions (wet 2048^2, 73 us a step: 61 % of the issue
// slots, 11.6 warp instructions a cell, DRAM at 40 %), so what only some rows need is
// decided once per row by a vote: the grid's edges, outlet and gauge cells, arrivals, dry flags.  A
// lane's two cells are neighbours (one shuffle an exchange), columns and rows outside the grid are
// records whose faces are closed, no face carries a flag, and a cell's two faces share one FP32x2
// instruction (faces_open, faces_update).
template <int INF, bool MAP> constexpr bool kFlatF = INF == 0 && !MAP;

// dynamic shared memory of k_fused_step: per warp kStages x (2 records x 32*CPL cells)
template <typename R, int CPL = 1> constexpr size_t fused_smem_bytes(int nt) {
    return size_t(nt / 32) * kStages * 64 * CPL * sizeof(typename Vec<R>::V4);
}

template <typename R> struct FusedArgs {
    using V4 = typename Vec<R>::V4;
    using V2 = typename Vec<R>::V2;
    int ny, nx;
    int n_strips, rows_per_warp, n_warps_total;
    double res;
    double tol_mm, thr_mm;
    double t_end;                // routing_time + min_time_step/60 [min]
    double min_dt, max_dt, inc, tsc, alfa_min, alfa_max;
    double inv_inc, inv_tsc, inv_res;   // correctly rounded reciprocals (div_by)
    R k_const[4];                // StepConsts' inv_dx, g, tol, thr
    R map_sy, map_sx;            // rain map cells per grid cell
    int flag_timestep, adaptive, flag_critical, outlet_type, ga;   // ga: infiltration on (either model)
    int scheme;                  // flag_numerical_scheme: 1 Bates, 2 s-upwind, 3 s-centred
    unsigned int wait_polls;     // polls of a row-copy wait before it gives up (HP2D_TIMEOUT)
    int own_r0, own_r1;          // rows whose cells enter the CFL maxima, ledgers and checks (a
                                 // row slab's own rows; the others are halo rows of other slabs)
    unsigned int n_ctas;
    R stag_s2;
    const V4* stat;
    V4* st0; V4* st1;            // state records, double buffer
    V2* gs0; V2* gs1;            // soil records, double buffer
    const SoilClass<R>* classes;       // Green-Ampt classes
    const SoilClassVG<R>* classes_vg;  // van Genuchten classes
    VGGlobals<R> vg;
    const int32_t* outlet_cells; const R* outlet_coef; int n_outlets;
    R* hf3; R* qo;
    R* arrival;
    RainDesc rain;
    InflowDesc<R> inflow;
    RecordDesc<R> rec;
    StructDesc<R> strct;         // reservoir / control structures (n = 0: none)
    R* vmax; R* hzmax;           // velocity / hazard maxima [m/s], [m^2/s] (null: not tracked)
    // [2][n_strips][dry_rows]: 1 when a deep-dry row of the strip wrote its records into state
    // buffer b; the same row deep-dry again two steps later would write identical values
    // (null: off; dry_rows is ny rounded up to a multiple of 4, rows_per_warp <= 128 and a
    // multiple of 4, so that a warp reads its rows' flags as one word per lane)
    unsigned char* dryflag;
    int dry_rows;
    int tile_nx;                 // tiles per row of tiles (hp2d_tile.cuh); 0: strips
    int tile_rpt;                // rows per thread of the tile step
    unsigned tile_grid;          // CTAs of the tile step's launch at most
    StepScalars* sc;
    StepPrep<R>* prep;           // [2] the step's rain, prepared by the step before
    StepAcc* acc;                // [4] accumulators (see StepAcc); sc is [2] in the same rotation
};

// refreshing_timestep.m:94-134, :315-359 in three parts, so that the quotients q_adv = res / max(vmax,
// 1e-10), q_wave = alfa_min res / cmax and the last one by the increment can be formed elsewhere
__device__ __host__ inline double finalize_new(double vmax, double cmax, double q_adv, double q_wave, double alfa_min,
                                               double alfa_max, double max_dt, int flag_timestep) {
    double dt_adv;
    if (vmax > 0) {
        dt_adv = q_adv;
        double tsf = fmax(alfa_max - 2.0 * fmax(vmax - 5.0, 0.0), alfa_min);
        dt_adv = fmin(dt_adv * tsf, max_dt);
    } else {
        dt_adv = max_dt;
    }
    double dt_wave = cmax > 0 ? q_wave : max_dt;
    double nw = flag_timestep == 1 ? fmin(dt_adv, dt_wave) : dt_wave;
    if (isnan(nw) || isinf(nw)) nw = max_dt;
    return nw;
}
__device__ __host__ inline double finalize_snap(double q_inc, double min_dt, double max_dt, double inc) {
    double tcr = fmax(inc * floor(q_inc), min_dt);
    return fmin(tcr, max_dt);
}
__device__ __host__ inline double finalize_dt(double vmax, double cmax, double res, double alfa_min,
                                              double alfa_max, double min_dt, double max_dt, double inc,
                                              int flag_timestep) {
    const double nw = finalize_new(vmax, cmax, 1.0 * res / fmax(vmax, 1e-10), (alfa_min * res) / cmax, alfa_min,
                                   alfa_max, max_dt, flag_timestep);
    return finalize_snap(nw / inc, min_dt, max_dt, inc);
}

// compensated (Kahan) running sum: s + c tracks the exact sum of the added terms to about one
// rounding of the state precision, however many terms (the library builds without contraction,
// so the compensation is not folded away)
template <typename R> struct Kahan {
    R s = R(0), c = R(0);
    __device__ __forceinline__ void add(R x) {
        const R y = x - c;
        const R t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ double value() const { return double(s) - double(c); }
    __device__ __forceinline__ bool any() const { return s != R(0) || c != R(0); }
};

template <typename R> __device__ __forceinline__ R warp_max(R v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ unsigned long long warp_max_u(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename R> __device__ __forceinline__ R bits_to(unsigned long long b);
template <> __device__ __forceinline__ float bits_to<float>(unsigned long long b) { return __uint_as_float((unsigned)b); }
template <> __device__ __forceinline__ double bits_to<double>(unsigned long long b) { return __longlong_as_double((long long)b); }

// Neighbour exchange across a warp's strip of 32*CPL columns (cell h of lane L sits at
// column CPL L + h): value of the cell to the right / to the left, one shuffle each.
template <typename R, int CPL>
__device__ __forceinline__ void right_of(const R (&v)[CPL], R (&out)[CPL], int lane) {
    out[CPL - 1] = __shfl_down_sync(0xffffffffu, v[0], 1);
    if (CPL == 2) out[0] = v[CPL - 1];
}
template <typename R, int CPL>
__device__ __forceinline__ void left_of(const R (&v)[CPL], R (&out)[CPL], int lane) {
    out[0] = __shfl_up_sync(0xffffffffu, v[CPL - 1], 1);
    if (CPL == 2) out[CPL - 1] = v[0];
}

// resident CTAs per SM the register budget is sized for (float: 8 x 128 threads)
#ifndef HP2D_MINB_F32
#define HP2D_MINB_F32 8
#endif
#ifndef HP2D_MINB_F32_PAIR
#define HP2D_MINB_F32_PAIR 4
#endif
template <typename R, int CPL = 1> struct FusedOcc { static constexpr int minb = CPL == 1 ? HP2D_MINB_F32 : HP2D_MINB_F32_PAIR; };
template <int CPL> struct FusedOcc<double, CPL> { static constexpr int minb = CPL == 1 ? 3 : 2; };

// One CTA-sized work item of the fused step: warps blk*NT/32 .. of the grid described by
// `a`.  k_fused_step runs item blockIdx.x of one grid; k_ens_step runs items of many grids
// pulled from a queue.  Every thread of the CTA calls it; it may return early for all of
// them together.  Returns false when a row copy timed out (the CTA must stop using its
// shared-memory ring).
// INF: infiltration model (0 none, 1 Green-Ampt, 2 van Genuchten); MAP: rain from coarse
// maps (else a uniform rate); INFL: inflow hydrographs present (the grids without them do not
// carry the lookup); SCH: 0 Bates faces, 1 the schemes with numerical diffusion
// (flag_numerical_scheme 2 or 3, a.scheme), whose faces also read the previous fluxes of the
// neighbouring faces of the same direction
// The depth d_tot a step hands to its fluxes at each control structure's reservoir cell --
// phase (A) of that cell restated: rain, infiltration, inflow, clamps, from the state and
// soil records `st`/`gs` the step starts from -- then the structures' transfers (one thread,
// in structure order).  The end of a step runs it for the next step; k_struct_prime for
// the first step of a call.
template <typename R, int INF, bool MAP, bool INFL>
__device__ __noinline__ void structure_prepare(const FusedArgs<R>& a, const RainStep<R>& rs, bool skip,
                                               const StepConsts<R>& K, const typename Vec<R>::V4* st,
                                               const typename Vec<R>::V2* gs, int tid, int nt, double time_step) {
    for (int i = tid; i < a.strct.n; i += nt) {
        const int c = a.strct.slot_cell[a.strct.slot[3 * i]];
        const int r = c / a.nx, j = c % a.nx;
        R hh = st[c].x;
        const R rr = MAP ? rs.at(a.rain, r, j, a.ny, a.nx) : rs.depth;
        hh = hh + rr;
        const unsigned meta = meta_bits(a.stat[c].w);
        if (INF) {
            const unsigned scl = meta & 255u;
            if (scl != 255u) {
                R Ic = gs[c].x, Tc = gs[c].y;
                if (INF == 1) green_ampt(hh, Ic, Tc, a.classes[scl], K);
                else vg_infiltration(hh, Ic, Tc, a.classes_vg[scl], a.vg, K);
            }
        }
        if (INFL) add_inflow(a.inflow, meta, hh);
        if (!skip && hh < R(1e-9)) hh = R(0);
        if (hh < R(0)) hh = R(0);
        a.strct.hres[i] = hh;
    }
    __syncthreads();
    if (tid == 0) structure_transfers(a.strct, time_step, a.res * a.res);
}

// The clock of a step, as its launch finds it once the step before has ended.
struct StepNow {
    double t_min, time_step, dts;        // [min], [min], [s]
    double rain_a, rain_b, t_prev;
    double tcr, vm, time_save;           // of the step that ended: refreshed step [s], max speed, save clock
    long long rec_count;
    int cur, skip, done, halted;
    int rec;                             // slot that receives this step's input depth (-1: none)
    int rec_last, rec_pending;
    int ended, accepted, refresh;        // a pending step ended, it was accepted, it refreshed the time step
};

// What every thread of a step's CTA shares: the step's scalars, constants and rain, and the
// CTA's reductions.
template <typename R, int NT> struct StepShared {
    StepScalars sc;      // as found (step_books brings them up to date)
    StepAcc acc;         // the pending step's sums
    StepPrep<R> p;       // this step's rain
    StepNow now;
    StepConsts<R> K;
    RainStep<R> rsn;     // the next step's rain
    double save_next;    // save clock of this step (the next launch ends it)
    int negn;            // an outlet cell would go below -1e-11 m after the next rain
    int last;            // ensemble item: this CTA finished its member and the step was accepted
    double stage;        // depth the stage overwrites of this CTA added [m]
    unsigned skipw;      // cells whose unchanged record this CTA did not rewrite
    unsigned skipr;      // of those, cells of skipped blocks (not read either)
    R red_s2[NT / 32];
    unsigned long long red_c[NT / 32];
    double red_d[3][NT / 32];
    int red_to[NT / 32];
    unsigned red_bad[NT / 32];
};

// words of a struct in global memory (written by other SMs in an earlier launch) into shared memory
template <int NT, typename T> __device__ __forceinline__ void copy_words(T& dst, const T* src, int tid) {
    static_assert(sizeof(T) % 4 == 0, "whole words");
    unsigned* d = reinterpret_cast<unsigned*>(&dst);
    const unsigned* s = reinterpret_cast<const unsigned*>(src);
#pragma unroll
    for (int w = 0; w < int(sizeof(T) / 4); w += NT)
        if (w + tid < int(sizeof(T) / 4)) d[w + tid] = __ldcg(s + w + tid);
}
template <typename T> __device__ __forceinline__ void store_words(T* dst, const T& src, int lane) {
    unsigned* d = reinterpret_cast<unsigned*>(dst);
    const unsigned* s = reinterpret_cast<const unsigned*>(&src);
#pragma unroll
    for (int w = 0; w < int(sizeof(T) / 4); w += 32)
        if (w + lane < int(sizeof(T) / 4)) d[w + lane] = s[w + lane];
}

// The verdict on a step: rejected when a row copy timed out, when more cells ended it non-finite
// or too negative than the run started with, or when the host's test hook names it.
__device__ __forceinline__ bool step_rejected(const StepScalars& sc, const StepAcc& acc) {
    return acc.timeout != 0u || acc.bad > sc.n_bad0 || (sc.fault_n > 0 && sc.k == sc.fault_k);
}

// The clock by one warp: ends the step `pending` (refreshing_timestep and the clock,
// HydroPol2D_Main_While.m:691-705, :779) from its scalars and sums, and forms the constants of the
// step that follows.  Only what that step's cells wait for is done here (the books are
// step_books'), in registers, with the independent FP64 divisions of a stage side by side in
// different lanes: one thread doing it all through memory took 8000 cycles, one warp with the
// books 3600.
// A rejected step commits nothing: the state stays in buffer cur and the clock and counters stay,
// and the launches halt until the host has prepared the retry (HydroPol2D_Main_While.m:926-993).
template <typename R>
__device__ __forceinline__ double save_clock(const FusedArgs<R>& a, double t) {
    return div_by((ceil(div_by(t * 60.0, a.tsc, a.inv_tsc)) - 1.0) * a.tsc, 60.0, 1.0 / 60.0);
}
template <typename R>
__device__ __forceinline__ void step_clock(const FusedArgs<R>& a, const StepScalars& sc, const StepAcc& acc,
                                           const StepPrep<R>& p, bool pending, StepNow& now, StepConsts<R>& K) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool accepted = pending && !step_rejected(sc, acc);
    const double t = sc.t_min, tp = sc.t_prev;
    const long long k = sc.k;
    double ts1 = sc.time_step, t1 = t;
    double tcr = 0.0, time_save = 0.0, vm = 0.0;
    bool refresh = false;
    int halted = sc.halted | ((pending && !accepted) ? 1 : 0);
    if (accepted) {
        // lane 0: max speed and the advective bound, lane 1: max celerity and the wave bound
        const unsigned long long cb = acc.cmax;
        const R arg = lane == 0 || !cb ? bits_to<R>(acc.vmax) : bits_to<R>(cb - 1ull);
        double m = double(sqrt(arg));
        if (lane != 0) m = !cb ? 0.0 : (a.adaptive == 1 ? fmax(m, double(R(1e-10))) : double(arg));
        const double q = (lane == 0 ? 1.0 * a.res : a.alfa_min * a.res) / (lane == 0 ? fmax(m, 1e-10) : m);
        time_save = p.key_b == t ? p.time_save : save_clock(a, t);
        refresh = (time_save - sc.tsp > 0 || k == 1) &&
                  (sc.refresh_every <= 1 || k == 1 || (k - 1) % sc.refresh_every == 0);
        vm = __shfl_sync(FULL, m, 0);
        const double nw = finalize_new(vm, __shfl_sync(FULL, m, 1), __shfl_sync(FULL, q, 0), __shfl_sync(FULL, q, 1),
                                       a.alfa_min, a.alfa_max, sc.max_dt, a.flag_timestep);
        tcr = refresh ? finalize_snap(div_by(nw, a.inc, a.inv_inc), a.min_dt, sc.max_dt, a.inc)
                      : ts1 * 60.0;   // refreshing_timestep.m:361-365
        ts1 = div_by(tcr, 60.0, 1.0 / 60.0);
        t1 = ts1 + t;
        if (refresh && tcr == a.min_dt && sc.dt_floor_stop) halted = 1;   // this step is kept; the next launches wait
    }
    // StepConsts::make, a constant per lane
    const double dts = ts1 * 60.0;
    const double q2 = (lane == 3 ? a.res : 1.0) / dts;
    const double v = lane == 0 ? dts : lane == 1 ? kG * dts : lane == 2 ? div_by(dts, a.res, a.inv_res) : q2;
    static_assert(sizeof(StepConsts<R>) == 9 * sizeof(R), "nine constants");
    if (lane < 9) reinterpret_cast<R*>(&K)[lane] = lane < 5 ? R(v) : a.k_const[lane < 5 ? 0 : lane - 5];
    if (lane == 0) {
        now.t_min = t1;
        now.time_step = ts1;
        now.dts = dts;
        // the next step's rain: update_spatial_BC over [t_previous, t]
        // (HydroPol2D_Main_While.m:721), then t_previous <- the clock increment on the first
        // step and t after it (:734-738), and the clock advances by the new step (:779)
        now.rain_a = accepted ? tp : sc.rain_a;
        now.rain_b = accepted ? t : sc.rain_b;
        now.t_prev = accepted ? (k == 1 ? ts1 : t) : tp;
        now.tcr = tcr;
        now.vm = vm;
        now.time_save = time_save;
        now.cur = sc.cur ^ (accepted ? 1 : 0);
        now.skip = accepted ? (acc.negn ? 1 : 0) : sc.skip_clamp;   // gathered by every CTA's outlets
        now.halted = halted;
        now.done = !(t1 <= a.t_end) || halted;
        now.ended = pending;
        now.accepted = accepted;
        now.refresh = refresh;
        now.rec = -1;
        if (a.rec.n_times > 0) {   // save_output_maps.m:25-27 with t_save = t + new dt (:740)
            long long count = sc.rec_count;
            int rp = sc.rec_pending, rl = sc.rec_last;
            if (accepted) {
                if (rp) { count += 1; rp = 0; }   // recorded by the step that ended
                const int idx = last_record_below(a.rec.times, a.rec.n_times, t + ts1);
                if (idx > rl && a.rec.n_slots > 0) rp = 1;
                if (idx > rl) rl = idx;
            }
            now.rec_count = count;
            now.rec_last = rl;
            now.rec_pending = rp;
            if (rp && a.rec.n_slots > 0) now.rec = int(count % a.rec.n_slots);
        }
    }
    __syncwarp();
}

// The books of the step that step_clock ended (one warp): sc, as found, becomes what the next
// launch or the host reads.
template <typename R, bool INFL>
__device__ __noinline__ void step_books(const FusedArgs<R>& a, StepScalars& __restrict__ sc, const StepAcc& __restrict__ acc,
                                         const StepNow& __restrict__ now) {
    if ((threadIdx.x & 31) == 0) {
        sc.pending = 0;
        if (now.ended) {
            if (acc.timeout) sc.status |= kStatusTimeout;
            if (acc.bad > sc.n_bad0) sc.status |= kStatusNumerical;
            if (sc.fault_n > 0 && sc.k == sc.fault_k) {   // the host's test hook
                sc.fault_n -= 1;
                sc.status |= kStatusNumerical;
            }
            sc.skipped_cells += acc.skipw;
            sc.skipped_read_cells += acc.skipr;
            sc.halted = now.halted;
        }
        if (now.accepted) {
            if (sc.skip_clamp) sc.neg_warn += 1;
            double rain_s = acc.rain;
            // uniform rain: the same depth on every cell with a finite depth
            if (a.rain.n_uniform) rain_s += sc.rain_cell * double(sc.n_finite);
            sc.tsp = now.time_save;
            sc.last_vbits = acc.vmax;
            sc.last_cbits = acc.cmax;
            sc.last_refreshed = now.refresh;
            sc.last_unstable = 0;
            if (now.refresh) {
                sc.vmax_last = now.vm;
                sc.last_unstable = now.tcr == a.min_dt;
                if (now.tcr == a.min_dt) {   // refreshing_timestep.m:357-359 (unstable)
                    sc.unstable += 1;
                    if (sc.dt_floor_stop) sc.status |= kStatusDtFloor;
                }
            }
            const double area = a.res * a.res;
            sc.rain_vol += rain_s * area;
            sc.inf_vol += acc.inf * area;
            sc.out_vol += acc.out * area;
            if constexpr (INFL) {
                if (a.inflow.n_gauges) {   // every cell of a gauge with a finite elevation got its depth
                    double v = 0.0;
                    for (int g = 0; g < a.inflow.n_gauges; ++g) v += double(a.inflow.depth[g]) * a.inflow.gauge_cells[g];
                    sc.inflow_vol += v * area;
                }
                if (a.inflow.n_stage) sc.stage_vol += acc.stage * area;
                if (a.strct.n) {   // the structures' extras this step applied
                    double v = 0.0;
                    for (int q = 0; q < a.strct.n_slots; ++q) v += double(a.strct.extra[q]) * area;
                    sc.struct_vol += v;
                }
            }
            if (a.rec.n_times > 0) {
                sc.rec_count = now.rec_count;
                sc.rec_pending = now.rec_pending;
                sc.rec_last = now.rec_last;
                if (now.rec >= 0) a.rec.snap_t[now.rec] = sc.t_min;
            }
            sc.rain_a = now.rain_a;
            sc.rain_b = now.rain_b;
            sc.t_prev = now.t_prev;
            sc.time_step = now.time_step;
            sc.t_min = now.t_min;
            sc.k += 1;
            sc.cur = now.cur;
            sc.skip_clamp = now.skip;
        }
    }
    __syncwarp();
}

// the next step's gauge depths and stages (one warp)
template <typename R> __device__ __forceinline__ void gauges_prepare(const FusedArgs<R>& a, const StepScalars& sc, int lane) {
    for (int g = lane; g < a.inflow.n_gauges; g += 32)
        a.inflow.depth[g] = R(inflow_integral(a.inflow, g, sc.rain_a, sc.rain_b) / 60000.0);
    for (int g = lane; g < a.inflow.n_stage; g += 32) a.inflow.stage_now[g] = R(stage_at(a.inflow, g, sc.t_min));
}

// The head of a step's CTA, by all its threads.  A solo grid's launch (SOLO) finds the step before
// pending and ends it here, in every CTA alike, from its scalars and sums: one round trip to L2,
// then warp 0's arithmetic while the other warps fetch their records (`early`, given the buffer that
// holds the state, which only needs the verdict).  This replaces a ticket and a tail in the last
// CTA, which the whole GPU waited for (release, ticket, reload and one thread's FP64 chain: 9000 of
// a small grid's 18000 cycles per step).  CTA 0 keeps the books for the next launch (step_publish).
// Items of an ensemble (not SOLO) find their member's scalars finished by step_finish's last CTA.
// The rain comes prepared from the step before (its table walk is off the critical path); thread 0
// makes what is missing on a call's first step.  ASYNC: the next step's rain is computed by warp 1
// after the last barrier here and is visible after the caller's next CTA barrier.
template <typename R, int NT>
__device__ __forceinline__ void step_next(const FusedArgs<R>& a, StepShared<R, NT>& sh, int lane) {
    RainStep<R>::make_warp(sh.rsn, a.rain, sh.now.t_prev, sh.now.t_min, lane);
    if (lane == 0) sh.save_next = save_clock(a, sh.now.t_min);
    __syncwarp();
}
template <typename R, int NT, bool ASYNC, bool SOLO, typename Early>
__device__ __forceinline__ void step_begin(const FusedArgs<R>& a, StepShared<R, NT>& sh, int phase, Early early) {
    const int tid = threadIdx.x, warp = tid >> 5;
    if (SOLO) {
        dependents_may_launch();
        wait_for_launches_before();
    }
    copy_words<NT>(sh.sc, a.sc + (SOLO ? (phase & 1) : 0), tid);
    copy_words<NT>(sh.p, a.prep + (SOLO ? (phase & 1) : 0), tid);
    if (SOLO) copy_words<NT>(sh.acc, a.acc + phase, tid);
    if (tid == 0) {
        sh.negn = 0;
        sh.stage = 0.0;
        sh.skipw = 0u;
        sh.skipr = 0u;
    }
    __syncthreads();
    const bool pending = SOLO && sh.sc.pending;
    early(sh.sc.cur ^ ((pending && !step_rejected(sh.sc, sh.acc)) ? 1 : 0));
    const int lane = tid & 31;
    if (warp == 0) {
        step_clock(a, sh.sc, sh.acc, sh.p, pending, sh.now, sh.K);
        if (!(sh.p.key_a == sh.now.rain_a && sh.p.key_b == sh.now.rain_b))
            RainStep<R>::make_warp(sh.p.rs, a.rain, sh.now.rain_a, sh.now.rain_b, lane);
        // the next step applies the rain of [t_previous, t] (HydroPol2D_Main_While.m:721)
        if (!ASYNC) step_next(a, sh, lane);
    }
    __syncthreads();
}

// step_begin and step_publish of the strip kernels, out of line: inlined, their registers would
// count against the row loop's
template <typename R, int NT, bool SOLO, bool INFL>
__device__ __noinline__ void step_begin_strips(const FusedArgs<R>& a, StepShared<R, NT>& sh, unsigned blk, int phase);

// CTA 0's warp 0, any time after step_begin (and step_next): the scalars, the
// next step's rain and a clear accumulator for the launches that follow.
template <typename R, int NT, bool INFL>
__device__ __forceinline__ void step_publish(const FusedArgs<R>& a, StepShared<R, NT>& sh, int phase) {
    const int lane = threadIdx.x & 31;
    step_books<R, INFL>(a, sh.sc, sh.acc, sh.now);
    if (lane == 0) {
        sh.sc.rain_cell = double(sh.p.rs.depth);
        sh.sc.pending = !sh.now.done;
        StepPrep<R>& np = a.prep[(phase + 1) & 1];
        np.key_a = sh.now.t_prev;
        np.key_b = sh.now.t_min;
        np.time_save = sh.save_next;
        np.rs = sh.rsn;
    }
    __syncwarp();
    store_words(a.sc + ((phase + 1) & 1), sh.sc, lane);
    unsigned* z = reinterpret_cast<unsigned*>(a.acc + ((phase + 2) & 3));
    for (int w = lane; w < int(sizeof(StepAcc) / 4); w += 32) z[w] = 0u;
}

template <typename R, int NT, bool SOLO, bool INFL>
__device__ __noinline__ void step_begin_strips(const FusedArgs<R>& a, StepShared<R, NT>& sh, unsigned blk, int phase) {
    step_begin<R, NT, false, SOLO>(a, sh, phase, [](int) {});
    if (SOLO && blk == 0 && threadIdx.x < 32) step_publish<R, NT, INFL>(a, sh, phase);
}

// warp maximum of ordered bits of non-negative numbers (or of the celerity code): one redux in FP32
template <typename R> __device__ __forceinline__ unsigned long long warp_max_code(unsigned long long v) {
    if constexpr (sizeof(R) == 4) return __reduce_max_sync(0xffffffffu, unsigned(v));
    else return warp_max_u(v);
}

// The end of a CTA's part of a step, called by all its threads: one warp reduction each of the
// sums the kernel can have, then the step's accumulators.  A solo grid is done with that: the next
// launch ends the step.  An ensemble item takes a ticket of its member, and the CTA that finishes
// the member last ends its step.  Returns false when one of the CTA's row copies timed out.
template <typename R, int NT, int INF, bool MAP, bool INFL, bool SOLO>
__device__ __forceinline__ bool step_finish(const FusedArgs<R>& a, StepShared<R, NT>& sh, double rain_acc,
                                            double inf_acc, double out_acc, R s2max, R cmaxv, unsigned nbad,
                                            bool timed_out, int phase, const typename Vec<R>::V4* sout,
                                            const typename Vec<R>::V2* gout) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int NWARP = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long scode = warp_max_code<R>(ord_bits(s2max));
    // 0: no non-stagnant cell; else the bits of the (non-negative, +0 for -0) maximum + 1
    unsigned long long cenc = warp_max_code<R>(cmaxv >= R(0) ? ord_bits(cmaxv + R(0)) + 1ull : 0ull);
    if (MAP) rain_acc = warp_sum(rain_acc);
    if (INF) inf_acc = warp_sum(inf_acc);
    if (__any_sync(FULL, out_acc != 0.0)) out_acc = warp_sum(out_acc);   // strips and tiles with outlets
    const int to_any = __any_sync(FULL, timed_out);
    nbad = __reduce_add_sync(FULL, nbad);
    if (lane == 0) {
        sh.red_bad[warp] = nbad;
        sh.red_s2[warp] = bits_to<R>(scode);
        sh.red_c[warp] = cenc;
        sh.red_d[0][warp] = rain_acc;
        sh.red_d[1][warp] = inf_acc;
        sh.red_d[2][warp] = out_acc;
        sh.red_to[warp] = to_any;
    }
    __syncthreads();
    bool cta_ok = true;
#pragma unroll
    for (int w = 0; w < NWARP; ++w) cta_ok = cta_ok && sh.red_to[w] == 0;
    if (warp == 0) {
        const int w = lane < NWARP ? lane : 0;
        scode = warp_max_code<R>(ord_bits(sh.red_s2[w]));
        cenc = warp_max_code<R>(sh.red_c[w]);
        const unsigned bad = __reduce_add_sync(FULL, lane < NWARP ? sh.red_bad[w] : 0u);
        double sum[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            if ((q == 0 && !MAP) || (q == 1 && !INF)) continue;
            const double v = lane < NWARP ? sh.red_d[q][w] : 0.0;
            if (__any_sync(FULL, v != 0.0)) sum[q] = warp_sum(v);
        }
        StepAcc* const acc = a.acc + (SOLO ? ((phase + 1) & 3) : 0);
        unsigned ticket = 0u;
        if (lane == 0) {
            if (!cta_ok) {   // a row copy did not arrive in time
                atomicOr(&acc->timeout, 1u);
                // an ensemble's CTA takes no more items after this: when all have given up, some of
                // the member's are left and no last ticket reports it
                if (!SOLO) atomicOr(&a.sc->status, kStatusTimeout);
            }
            if (bad) atomicAdd(&acc->bad, (unsigned long long)bad);
            if (scode) atomicMax(&acc->vmax, scode);
            if (cenc) atomicMax(&acc->cmax, cenc);
            if (sum[0] != 0.0) atomicAdd(&acc->rain, sum[0]);
            if (sum[1] != 0.0) atomicAdd(&acc->inf, sum[1]);
            if (sum[2] != 0.0) atomicAdd(&acc->out, sum[2]);
            if (sh.negn) atomicOr(&acc->negn, 1u);
            if (INFL && sh.stage != 0.0) atomicAdd(&acc->stage, sh.stage);
            if (sh.skipw) atomicAdd(&acc->skipw, (unsigned long long)sh.skipw);
            if (sh.skipr) atomicAdd(&acc->skipr, (unsigned long long)sh.skipr);
            // the accumulators above are released before the ticket, and acquired by the last CTA
            if (!SOLO)
                asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(ticket) : "l"(&a.sc->counter) : "memory");
        }
        if (!SOLO) {
            const bool last = __shfl_sync(FULL, ticket, 0) == a.n_ctas - 1;
            if (lane == 0) sh.last = 0;
            if (last) {
                copy_words<32>(sh.acc, a.acc, lane);
                __syncwarp();
                step_clock(a, sh.sc, sh.acc, sh.p, true, sh.now, sh.K);
                const bool accepted = sh.now.accepted;
                if (lane == 0) {
                    sh.sc.rain_cell = double(sh.p.rs.depth);   // of the step that ends
                    sh.sc.counter = 0u;
                    sh.last = accepted;
                    sh.p.key_a = sh.now.rain_a;
                    sh.p.key_b = sh.now.rain_b;
                    sh.p.rs = sh.rsn;
                }
                __syncwarp();
                step_books<R, INFL>(a, sh.sc, sh.acc, sh.now);
                store_words(a.sc, sh.sc, lane);
                if (accepted) store_words(a.prep, sh.p, lane);
                unsigned* z = reinterpret_cast<unsigned*>(a.acc);
                for (int q = lane; q < int(sizeof(StepAcc) / 4); q += 32) z[q] = 0u;
                if (INFL && accepted) gauges_prepare(a, sh.sc, lane);
            }
        }
    }
    if constexpr (INFL && !SOLO) {
        if (a.strct.n) {   // the next step's structure transfers, from its d_tot
            __syncthreads();
            if (sh.last) {
                __threadfence();   // records of other CTAs
                structure_prepare<R, INF, MAP, INFL>(a, sh.rsn, sh.sc.skip_clamp != 0, sh.K, sout, gout, tid, NT,
                                                     sh.sc.time_step);
            }
        }
    }
    return cta_ok;
}

// Ends the step that launch phase - 1 left pending (one CTA): after the last launch of a batch, for
// the host, and after every launch of a grid with gauges, stages or control structures, whose next
// step's depths, stages and transfers it prepares too.  Leaves the scalars in slot 0, nothing
// pending and every accumulator clear.
template <typename R, int INF, bool MAP>
__global__ void __launch_bounds__(128) k_step_flush(const __grid_constant__ FusedArgs<R> a, int phase) {
    __shared__ StepShared<R, 128> sh;
    const int tid = threadIdx.x, lane = tid & 31;
    copy_words<128>(sh.sc, a.sc + (phase & 1), tid);
    copy_words<128>(sh.acc, a.acc + phase, tid);
    copy_words<128>(sh.p, a.prep + (phase & 1), tid);
    __syncthreads();
    const bool pending = sh.sc.pending != 0;
    if (tid < 32) {
        step_clock(a, sh.sc, sh.acc, sh.p, pending, sh.now, sh.K);
        step_books<R, true>(a, sh.sc, sh.acc, sh.now);
        store_words(a.sc, sh.sc, lane);
        store_words(a.prep, sh.p, lane);
        if (sh.now.accepted) gauges_prepare(a, sh.sc, lane);
    }
    unsigned* z = reinterpret_cast<unsigned*>(a.acc);
    for (int w = tid; w < int(4 * sizeof(StepAcc) / 4); w += 128) z[w] = 0u;
    __syncthreads();
    if (a.strct.n && sh.now.accepted) {
        if (tid == 0) sh.rsn.make(a.rain, sh.sc.rain_a, sh.sc.rain_b);
        __syncthreads();
        structure_prepare<R, INF, MAP, true>(a, sh.rsn, sh.sc.skip_clamp != 0, sh.K, sh.sc.cur ? a.st1 : a.st0,
                                             sh.sc.cur ? a.gs1 : a.gs0, tid, 128, sh.sc.time_step);
    }
}

// the rain of a step at one cell, out of line (the few outlet cells of a grid with rain maps)
template <typename R> __device__ __noinline__ R rain_at_cell(const FusedArgs<R>& a, const RainStep<R>& rs, int i, int j) {
    return rs.at(a.rain, i, j, a.ny, a.nx);
}

template <typename R, int NT, int INF, bool MAP, int CPL, bool INFL, int SCH, bool SOLO>
__device__ __forceinline__ bool fused_item(const FusedArgs<R>& a, const unsigned blk, const int phase) {
    using V4 = typename Vec<R>::V4;
    using V2 = typename Vec<R>::V2;
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ StepShared<R, NT> sh;
    const int& s_rec = sh.now.rec;
    int& s_negn = sh.negn;
    double& s_stage = sh.stage;
    unsigned& s_skipw = sh.skipw;
    unsigned& s_skipr = sh.skipr;
    const RainStep<R>& s_rs = sh.p.rs;
    const RainStep<R>& s_rsn = sh.rsn;
    __shared__ R s_map[2][2][MAP ? NT * CPL : 1];   // rain maps in force: rows above / below, per cell of a lane
    __shared__ __align__(8) unsigned long long s_bar[NT / 32][kStages];
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    bool timed_out = false;

    const int tid = threadIdx.x;
    step_begin_strips<R, NT, SOLO, INFL>(a, sh, blk, phase);
    if (sh.now.done) return true;

    const StepConsts<R> K = sh.K;
    const int ny = a.ny, nx = a.nx;
    const int cur = sh.now.cur;
    const R clamp0 = sh.now.skip ? R(0) : R(1e-9);   // depths below are zero (Hydrological_Model.m:45-52)
    const RainStep<R> RS = s_rs;
    const V4* __restrict__ sin = cur ? a.st1 : a.st0;
    V4* __restrict__ sout = cur ? a.st0 : a.st1;
    const V2* __restrict__ gin = cur ? a.gs1 : a.gs0;
    V2* __restrict__ gout = cur ? a.gs0 : a.gs1;
    const V4* __restrict__ stat = a.stat;
    const R t_arr = R(sh.now.t_min * 60.0 + sh.now.dts);

    const int lane = tid & 31, warp = tid >> 5;
    const int wg = int(blk) * (NT / 32) + warp;

    double rain_acc = 0.0, inf_acc = 0.0, out_acc = 0.0;
    // per-lane partial sums of the volume ledger in the state precision, Kahan-compensated
    // (the warps' sums and everything after them are FP64)
    Kahan<R> rain_acc_r, inf_acc_r, out_acc_r;
    unsigned nbad = 0u;                       // own cells ending non-finite or below -tol
    unsigned dry = 0u;                        // bit i: row r-i dry across the strip
    unsigned marks = 0u;
    R s2max = R(0);
    R cmaxv = R(-1);   // largest celerity term of a non-stagnant cell (-1: none yet)

    if (wg < a.n_warps_total) {
        constexpr int SW = 32 * CPL;       // strip width: CPL cells per lane
        const int strip = wg % a.n_strips;
        const int rb = wg / a.n_strips;
        const int j_first = strip * (SW - 4) - 2;   // 2-column apron on each side
        int j[CPL];
        bool col_ok[CPL], own_lane[CPL];
#pragma unroll
        for (int h = 0; h < CPL; ++h) {
            j[h] = j_first + CPL * lane + h;
            col_ok[h] = j[h] >= 0 && j[h] < nx;
            own_lane[h] = lane >= 2 / CPL && lane < 32 - 2 / CPL && j[h] < nx;
        }
        const R rc_half = j[0] == 0 ? R(0.5) : R(1);   // refreshing_timestep.m's vel_left on the first column
        const int r0 = rb * a.rows_per_warp;
        const int r_end = min(r0 + a.rows_per_warp, ny);
        unsigned char* const dfl =
            a.dryflag ? a.dryflag + (size_t(cur ^ 1) * a.n_strips + strip) * size_t(a.dry_rows) : nullptr;
        unsigned own_n = 0;   // cells of the strip this warp stores
#pragma unroll
        for (int h = 0; h < CPL; ++h) own_n += __popc(__ballot_sync(FULL, own_lane[h]));
        // the flags of this warp's rows in the output buffer and in the input buffer, four per
        // lane (read once: each row's output flag changes only at that row, the input flags not
        // at all during the step)
        unsigned dfw = 0u, dfw_in = 0u;
        bool flagged = false;   // some row of the block is flagged in either buffer
        if (dfl && r0 + 4 * lane < r_end) {
            dfw = *reinterpret_cast<const unsigned*>(dfl + r0 + 4 * lane);
            dfw_in = *reinterpret_cast<const unsigned*>(a.dryflag + (size_t(cur) * a.n_strips + strip) * size_t(a.dry_rows) +
                                                        r0 + 4 * lane);
        }
        flagged = __any_sync(FULL, (dfw | dfw_in) != 0u);
        // The whole block of rows: when this step adds no rain and no infiltration and records
        // no map, and the flags show every input row r0-1..r_end+1 of this strip and of its
        // neighbours (the 2-column aprons) deep-dry and every output row already holding the
        // record the deep-dry path would write, the loop below would store nothing and
        // contribute nothing: skip it, copies included.  (A flag is only ever set on a row
        // whose 64 columns hold no outlet or boundary cell, so no inflow, stage or structure
        // water can reach the rows the flags cover, and the deep-dry path updates no velocity
        // or hazard maximum.)
        bool blk_skip = false;
        if constexpr (INF == 0 && !MAP) {
            if (dfl && s_rec < 0 && RS.depth == R(0) && K.thr > R(0)) {
                const int nrow = r_end - r0;
                const int nb = min(max(nrow - 4 * lane, 0), 4);
                const unsigned mask = nb == 4 ? 0xffffffffu : (1u << (8 * nb)) - 1u;
                const unsigned want = 0x01010101u & mask;
                bool ok = (dfw & mask) == want;
                const unsigned char* fin = a.dryflag + size_t(cur) * a.n_strips * size_t(a.dry_rows);
                for (int q = max(strip - 1, 0); q <= min(strip + 1, a.n_strips - 1); ++q) {
                    const unsigned char* fq = fin + size_t(q) * a.dry_rows;
                    if (nb > 0) ok = ok && (*reinterpret_cast<const unsigned*>(fq + r0 + 4 * lane) & mask) == want;
                    if (lane < 3) {
                        const int rr = lane == 0 ? r0 - 1 : r_end + lane - 1;
                        if (rr >= 0 && rr < ny) ok = ok && fq[rr] == 1;
                    }
                }
                blk_skip = __all_sync(FULL, ok);
            }
        }
        if (blk_skip) {
            if (lane == 0) {
                atomicAdd(&s_skipw, own_n * unsigned(r_end - r0));
                atomicAdd(&s_skipr, own_n * unsigned(r_end - r0));
            }
        } else {

        // rolling window (suffix = rows back), one entry per cell of the lane
        R hT1[CPL], hT2[CPL], qxu1[CPL], qyu1[CPL], hfx1[CPL], hfx2[CPL], hfy1[CPL], hfy2[CPL];
        R sc2[CPL], qxl2[CPL], qyl2[CPL], dm1[CPL], dm2[CPL];
        R qyp1[CPL];   // schemes 2/3: previous q_y of the row before
        // velocity of the face below row r-3, computed by the (F) of row r-3: after the shift it
        // is the face above row r-2 (qyl2 / hfy2 then hold the values it was computed from), so
        // the next (F) takes it instead of dividing again; vcar_ok (warp-uniform) says whether
        // the last row's (F) computed it
        R vcar[CPL];
        bool vcar_ok = false;
        bool lim2 = false;   // lim1 of the row before
        int map_iy = -1;   // row of the rain map whose interpolation s_map holds
        unsigned mt1[CPL], mt2[CPL];
#pragma unroll
        for (int h = 0; h < CPL; ++h) {
            qyp1[h] = R(0);
            vcar[h] = R(0);
            hT1[h] = hT2[h] = qxu1[h] = qyu1[h] = R(0);
            hfx1[h] = hfx2[h] = hfy1[h] = hfy2[h] = R(0);
            sc2[h] = R(1);
            qxl2[h] = qyl2[h] = dm1[h] = dm2[h] = R(0);
            mt1[h] = mt2[h] = 0u;
        }

        // TMA pipeline: the warp's two row records (static, state) of rows k+1..k+kStages-1
        // are in flight in a ring of kStages shared-memory stages while row k is
        // computed.  One 1-D bulk copy per record row (the strip's cells are contiguous),
        // the stage's mbarrier counts the bytes.
        const int seg_j0 = max(j_first, 0);
        const int seg_n = min(j_first + SW, nx) - seg_j0;
        const int seg_off = seg_j0 - j_first;
        const int last_k = (r_end + 1) - (r0 - 2);
        V4* ring = reinterpret_cast<V4*>(smem_dyn) + size_t(warp) * kStages * 2 * SW;
        const uint32_t bar0 = smem_addr(&s_bar[warp][0]);
        // lane 0 arms the stage's barrier (arrive + expected bytes) and copies the static
        // row, lane 1 copies the state row; a copy that lands before the arming only makes
        // the transaction count negative for a moment, and the phase cannot complete
        // before lane 0's arrival
        const uint32_t ring_base = smem_addr(ring + seg_off);
        const uint32_t bytes = uint32_t(seg_n) * uint32_t(sizeof(V4));
        const V4* src_base = lane == 0 ? stat : sin;
        const uint32_t dst_half = lane == 0 ? 0u : uint32_t(SW * sizeof(V4));
        auto issue = [&](int k) {
            const int s = k % kStages;
            const uint32_t bar = bar0 + 8u * s;
            const int rr = r0 - 2 + k;
            if (rr >= 0 && rr < ny && seg_n > 0) {
                if (lane == 0) mbar_expect_tx(bar, 2u * bytes);
                bulk_g2s(ring_base + uint32_t(s) * uint32_t(2 * SW * sizeof(V4)) + dst_half,
                         src_base + (size_t(rr) * nx + seg_j0), bytes, bar);
            } else if (lane == 0) {
                mbar_arrive(bar);
            }
        };
        if (lane == 0) {
            for (int s = 0; s < kStages; ++s) mbar_init(bar0 + 8u * s, 1u);
            mbar_fence_init();
        }
        // the ring's columns outside the grid, which no copy reaches: cells that stay dry whatever the
        // rain, their faces closed, that enter no maximum
        const R inf = R(__int_as_float(0x7f800000));
        const V4 pad_S{inf, inf, R(1), make_meta<R>(255u)}, pad_X{R(-3.0e38), R(0), R(0), inf};
#pragma unroll
        for (int h = 0; h < CPL; ++h)
            if (!col_ok[h])
                for (int s = 0; s < kStages; ++s) {
                    ring[s * 2 * SW + CPL * lane + h] = pad_S;
                    ring[s * 2 * SW + SW + CPL * lane + h] = pad_X;
                }
        __syncwarp();
        if (lane < 2) {
            fence_proxy_async_smem();   // reads of the ring by an earlier item come first
            for (int k = 0; k < kStages && k <= last_k; ++k) issue(k);
        }
#pragma unroll kRowUnroll
        for (int k = 0; k <= last_k; ++k) {
            const int r = r0 - 2 + k;
            const int s = k % kStages;
            // the dry flag of the output row r-2 in the buffer this step writes
            const bool frow_f = r - 2 >= r0 && r - 2 < r_end;
            unsigned flg = 0u, flg_in = 0u;
            if (flagged && frow_f) {
                const int fri = r - 2 - r0;
                flg = (__shfl_sync(FULL, dfw, fri >> 2) >> (8 * (fri & 3))) & 255u;
                flg_in = (__shfl_sync(FULL, dfw_in, fri >> 2) >> (8 * (fri & 3))) & 255u;
            }
            const bool landed = mbar_wait_bounded(bar0 + 8u * s, uint32_t((k / kStages) & 1), a.wait_polls);
            if (__any_sync(FULL, !landed)) {   // the whole warp leaves the loop together
                timed_out = true;
                // let every copy still in flight (rows k .. k+kStages-1, this one included) land
                // before the CTA leaves, with the long limit whatever a.wait_polls is
                for (int kk = k; kk < k + kStages && kk <= last_k; ++kk)
                    mbar_wait_bounded(bar0 + 8u * (kk % kStages), uint32_t((kk / kStages) & 1), 1u << 22);
                break;
            }
            V4 S[CPL], X[CPL];
#pragma unroll
            for (int h = 0; h < CPL; ++h) {
                S[h] = ring[s * 2 * SW + CPL * lane + h];
                X[h] = ring[s * 2 * SW + SW + CPL * lane + h];
            }
            __syncwarp();
            if (lane < 2 && k + kStages <= last_k) {
                fence_proxy_async_smem();
                issue(k + kStages);
            }
            const bool rok = r >= 0 && r < ny;
            const bool own_row = r >= r0 && r < r_end;
            if (!rok) {   // a row outside the grid, which no copy brings
#pragma unroll
                for (int h = 0; h < CPL; ++h) {
                    S[h] = pad_S;
                    X[h] = pad_X;
                }
            }
            R hT0[CPL];
            unsigned meta[CPL];
            bool all_dry = true, marked = false;
            // rain maps: the rows of the map around this row, and per lane their interpolation at its
            // columns, made anew only when those rows change (every ny / my rows) and kept in shared
            // memory (urban 2048^2 with 64 x 64 maps: four gathers and 30 instructions less per cell)
            R map_wy = R(0);
            if (MAP && rok) {
                const MapRow<R> mr = map_row<R>(r, a.rain.my, a.map_sy);
                map_wy = mr.wy;
                if (mr.iy0 != map_iy) {
                    map_iy = mr.iy0;
#pragma unroll 1
                    for (int q = 0; q < s_rs.nm; ++q)
#pragma unroll
                        for (int h = 0; h < CPL; ++h)
                            if (col_ok[h])
                                map_column<R>(a.rain.maps + size_t(s_rs.m[q]) * a.rain.my * a.rain.mx, mr, j[h],
                                              a.rain.mx, a.map_sx, s_map[q][0][h * NT + tid], s_map[q][1][h * NT + tid]);
                }
            }
            auto rain_row = [&](int h) -> R {   // RainStep::at of this row
                if (s_rs.nm == 0) return R(0);
                const R w1 = R(1) - map_wy;
                R v = s_rs.w[0] * (w1 * s_map[0][0][h * NT + tid] + map_wy * s_map[0][1][h * NT + tid]);
                if (s_rs.nm > 1) v = v + s_rs.w[1] * (w1 * s_map[1][0][h * NT + tid] + map_wy * s_map[1][1][h * NT + tid]);
                return v;
            };
#pragma unroll
            for (int h = 0; h < CPL; ++h) {
                // soil records: the row after next is brought to L1 (a register prefetch spilled)
                if (INF && col_ok[h] && r + 2 >= 0 && r + 2 < ny) prefetch_l1(gin + (size_t(r + 2) * nx + j[h]));
                meta[h] = meta_bits(S[h].w);
                marked = marked || (meta[h] >> 8) != 0u;
                // (A) hydrology of (r, j)
                hT0[h] = R(0);
                if constexpr (kFlatF<INF, MAP> && !INFL) {
                    const R hh = X[h].x + RS.depth;
                    hT0[h] = hh < clamp0 ? R(0) : hh;
                } else if (col_ok[h] && rok) {
                    const size_t c = size_t(r) * nx + j[h];
                    R hh = X[h].x;
                    const R rr = MAP ? rain_row(h) : RS.depth;
                    hh = hh + rr;
                    const bool own = own_lane[h] && own_row && r >= a.own_r0 && r < a.own_r1;
                    // uniform rain volume comes from the count of finite cells at the end
                    if (MAP && own && isfinite(hh)) rain_acc_r.add(rr);
                    if (INF) {
                        const unsigned sc = meta[h] & 255u;
                        const V2 Gs = gin[c];
                        V2 go = Gs;
                        if (sc != 255u) {
                            R Ic = Gs.x, Tc = Gs.y;
                            // Green-Ampt: {I, recovery timer}; van Genuchten: {I, water-table depth}
                            const R fd = INF == 1 ? green_ampt(hh, Ic, Tc, a.classes[sc], K)
                                                  : vg_infiltration(hh, Ic, Tc, a.classes_vg[sc], a.vg, K);
                            go.x = Ic;
                            go.y = Tc;
                            if (own && isfinite(fd)) inf_acc_r.add(fd);
                        }
                        if (own) gout[c] = go;
                    }
                    // inflow hydrographs after the infiltration (Hydrological_Model.m:27-28)
                    if (INFL) add_inflow(a.inflow, meta[h], hh);
                    hT0[h] = hh < clamp0 ? R(0) : hh;
                }
                all_dry = all_dry && hT0[h] == R(0);
            }
            // a pending map record keeps the depth this step starts from
            if (s_rec >= 0 && own_row) {
#pragma unroll
                for (int h = 0; h < CPL; ++h)
                    if (own_lane[h]) a.rec.snap[size_t(s_rec) * (size_t(ny) * nx) + size_t(r) * nx + j[h]] = X[h].x;
            }
            // bit i: row r-i has an outlet, inflow, stage or structure cell
            marks = (marks << 1) | (__any_sync(FULL, marked) ? 1u : 0u);
            // rows r-2..r dry across the whole strip: every face flux of row r and r-1 is
            // zero (Hf = 0), the donor scale of row r-1 is one and its limited faces are
            // zero, so (B)-(E) are skipped; the values below are what they would compute
            dry = (dry << 1) | (__all_sync(FULL, all_dry) ? 1u : 0u);
            // Deep-dry row: rows r-3..r dry across the strip and no outlet cell in row r-2.
            // Then (B)-(E) of this row and of the one before were skipped, so the window's
            // flux, face-depth and limited-flux registers hold +0 and the donor scale 1,
            // which is what this row's (B)-(E) and shift would store again; (F) for row r-2
            // gives depth hT2 + 0 = +0 (hT2 is a dry zero), fluxes +0 and the unchanged
            // maximum, with no arrival, outlet or CFL contribution.  Only the depth, maximum
            // and meta registers move.  (hfx2/hfy2 are left one row stale: they are read
            // only by a non-quiet (F), and the (F) after a deep-dry row is quiet.)  A depth
            // of +0 reaches the arrival threshold only when that is not positive.
            if ((dry & 15u) == 15u && K.thr > R(0)) {
                if (!(marks & 4u)) {
                    const int rm2 = r - 2;
                    if (frow_f && flg && flg_in) {
                        // this buffer already holds the row as this step would write it: the
                        // deep-dry record of two steps ago, and the step between wrote the
                        // deep-dry record into the other buffer (so the running maximum did not
                        // move; a row that got water in between and lost it again by the next
                        // step -- rain soaked up by the soil -- is written)
                        if (lane == 0) atomicAdd(&s_skipw, own_n);
                    } else if (frow_f) {
#pragma unroll
                        for (int h = 0; h < CPL; ++h)
                            if (own_lane[h]) {
                                V4 o4;
                                o4.x = R(0);
                                o4.y = R(0);
                                o4.z = R(0);
                                o4.w = R(0) > dm2[h] ? R(0) : dm2[h];
                                sout[size_t(rm2) * nx + j[h]] = o4;
                            }
                        if (dfl && lane == 0) dfl[rm2] = 1;
                    }
#pragma unroll
                    for (int h = 0; h < CPL; ++h) {
                        hT2[h] = hT1[h]; hT1[h] = hT0[h];
                        dm2[h] = dm1[h]; dm1[h] = X[h].w;
                        mt2[h] = mt1[h]; mt1[h] = meta[h];
                        if (SCH) qyp1[h] = X[h].z;
                    }
                    vcar_ok = false;
                    lim2 = false;
                    continue;
                }
            }
            R qxu0[CPL], hfx0[CPL], qyu0[CPL], hfy0[CPL], sc1[CPL], qxl1[CPL], qyl1[CPL];
#pragma unroll
            for (int h = 0; h < CPL; ++h) {
                qxu0[h] = hfx0[h] = qyu0[h] = hfy0[h] = qxl1[h] = qyl1[h] = R(0);
                sc1[h] = R(1);
            }
            bool lim1 = false;   // some cell of row r-1 has its faces limited (sc1 != 1)
            if ((dry & 7u) != 7u) {
                // (B) x face (r, j) between (r, j) and (r, j+1)
                R hR[CPL];
                right_of<R, CPL>(hT0, hR, lane);
                // schemes 2/3: previous q_x of the faces j-1 and j+1 (interior columns only);
                // lane 0's left neighbour lies outside the strip and is read from memory
                R qxa[CPL], qxb[CPL];
                if (SCH) {
                    R xq[CPL];
#pragma unroll
                    for (int h = 0; h < CPL; ++h) xq[h] = X[h].y;
                    left_of<R, CPL>(xq, qxa, lane);
                    right_of<R, CPL>(xq, qxb, lane);
                    if (lane == 0 && rok && j[0] >= 1) qxa[0] = sin[size_t(r) * nx + (j[0] - 1)].y;
#pragma unroll
                    for (int h = 0; h < CPL; ++h)
                        if (!(j[h] >= 1 && j[h] + 1 < nx)) qxa[h] = qxb[h] = R(0);
                }
                // (B) and (C) interleaved: the geometry of the 2 x CPL faces, then -- unless no
                // lane of the warp has a wet one -- their momentum updates without branches
                Two<R> Sl[CPL];
                R ya[CPL], yb[CPL];
                R hmax = R(0);
                bool edge = false;
#pragma unroll
                for (int h = 0; h < CPL; ++h) {
                    faces_open<R>(hT0[h], hR[h], hT1[h], S[h].x, S[h].y, hfx0[h], hfy0[h], Sl[h], K);
                    edge = edge || face_edge(fmax(fabs(S[h].x), fabs(S[h].y)));
                }
                if (__any_sync(FULL, edge)) {
#pragma unroll
                    for (int h = 0; h < CPL; ++h) {
                        if (face_edge(S[h].x)) hfx0[h] = R(0);
                        if (face_edge(S[h].y)) hfy0[h] = R(0);
                    }
                }
#pragma unroll
                for (int h = 0; h < CPL; ++h) {
                    hmax = fmax(hmax, fmax(hfx0[h], hfy0[h]));
                    ya[h] = yb[h] = R(0);
                    // schemes 2/3: the previous q_y of rows r-1 (kept from the row before) and r+1
                    if (SCH && col_ok[h] && r >= 1 && r + 1 < ny) {
                        ya[h] = qyp1[h];
                        yb[h] = sin[size_t(r + 1) * nx + j[h]].z;
                    }
                }
                if (__any_sync(FULL, hmax > R(0))) {
                    Two<R> p73[CPL];   // H^(7/3)
#pragma unroll
                    for (int h = 0; h < CPL; ++h) p73[h] = pow73_normal(hfx0[h], hfy0[h]);
                    if (sh.now.skip) {   // no clamp: depths of any size
#pragma unroll
                        for (int h = 0; h < CPL; ++h)
                            if ((hfx0[h] > R(0) && below_normal(hfx0[h])) || (hfy0[h] > R(0) && below_normal(hfy0[h])))
                                p73[h] = two(pow73_any(hfx0[h]), pow73_any(hfy0[h]));
                    }
#pragma unroll
                    for (int h = 0; h < CPL; ++h) {
                        qxu0[h] = X[h].y;
                        qyu0[h] = X[h].z;
                        faces_update<R, SCH>(hfx0[h], hfy0[h], p73[h], Sl[h], qxu0[h], qyu0[h], S[h].z, K, a.flag_critical,
                                             a.scheme, SCH ? qxa[h] : R(0), SCH ? qxb[h] : R(0), ya[h], yb[h]);
                    }
                }
                // (D) which cells of row r-1 have their faces limited
                R qxu1_left[CPL], out[CPL];
                left_of<R, CPL>(qxu1, qxu1_left, lane);
                const bool drow = r >= r0 && r - 1 >= 0 && r - 1 < ny;
                bool lim = false;
#pragma unroll
                for (int h = 0; h < CPL; ++h) {
                    out[h] = donor_out(qxu1[h], qxu1_left[h], qyu1[h], qyu0[h]);
                    lim = lim || out[h] > hT1[h] * K.dx_over_dt;
                }
                lim1 = drow && __any_sync(FULL, lim);
                if (lim1) {
#pragma unroll
                    for (int h = 0; h < CPL; ++h) {
                        const R avail = hT1[h] * K.dx_over_dt;
                        if (out[h] > avail) sc1[h] = avail / out[h];
                    }
                }
                // (E) limited faces of row r-1
                if (lim1 || lim2) {
                    R sc1_right[CPL];
                    right_of<R, CPL>(sc1, sc1_right, lane);
#pragma unroll
                    for (int h = 0; h < CPL; ++h) {
                        qxl1[h] = limit_by(qxu1[h], sc1[h], sc1_right[h]);
                        qyl1[h] = limit_by(qyu1[h], sc1[h], sc2[h]);
                    }
                } else {
#pragma unroll
                    for (int h = 0; h < CPL; ++h) {
                        qxl1[h] = qxu1[h];
                        qyl1[h] = qyu1[h];
                    }
                }
            }
            // (F) continuity, outlet, maxima and CFL of row r-2.  When rows r-3..r-1 are dry
            // across the strip every flux into row r-2 is +0 (and so are its face depths):
            // continuity gives hT2 + 0 and the cell adds nothing to the CFL reductions.
            const bool quiet = (dry & 14u) == 14u;
            R qxl2_left[CPL];
            if (quiet) {
#pragma unroll
                for (int h = 0; h < CPL; ++h) qxl2_left[h] = R(0);
            } else {
                left_of<R, CPL>(qxl2, qxl2_left, lane);
            }
            const int rm2 = r - 2;
            const bool frow = rm2 >= r0 && rm2 < r_end;
            const bool mine = rm2 >= a.own_r0 && rm2 < a.own_r1;   // enters the reductions
            if constexpr (kFlatF<INF, MAP>) {
                // The cells of the lane are computed without a per-lane branch (an apron lane's values
                // are computed and dropped: `act` masks every store and every reduction), so that the
                // compiler can interleave the CPL cells' arithmetic; frow is the same for the warp.
                if (frow) {
                    R hn[CPL], hf3[CPL];
                    const bool marked2 = (marks & 4u) != 0u;   // the rare cells of row r-2
#pragma unroll
                    for (int h = 0; h < CPL; ++h) {
                        R h_in = hT2[h];
                        if (INFL && marked2) {
                            // a control structure's transfers join the depth after the fluxes
                            // (Local_Inertial_Model_D4.m:318-344, :390)
                            if (own_lane[h] && (mt2[h] & kInflowBit)) {
                                const int ss = a.inflow.cell_struct[(mt2[h] >> 8) & 0x7FFFFFu];
                                if (ss >= 0) h_in = h_in + a.strct.extra[ss];
                            }
                        }
                        hn[h] = INFL && quiet ? h_in + R(0) : continuity(h_in, qxl2_left[h], qxl2[h], qyl2[h], qyl1[h], K);
                        hf3[h] = R(0);
                    }
                    if (marked2) {
#pragma unroll
                        for (int h = 0; h < CPL; ++h) {
                            const unsigned ord = INFL ? outlet_ord(mt2[h]) : mt2[h] >> 8;
                            if (own_lane[h] && ord) {
                                const int o = int(ord) - 1;
                                R ho;
                                const R qq = outlet_sink(hn[h], a.outlet_coef[o], a.outlet_type, K, ho);
                                hf3[h] = ho;
                                a.hf3[o] = ho;
                                a.qo[o] = qq;
                                if (mine) out_acc_r.add(qq * K.dt);
                                // the next step's clamp is skipped when an outlet cell (outside the
                                // infiltrating soils) stays negative after the next rain
                                // (Hydrological_Model.m:45-50); only outlet cells can end negative
                                if (mine && !(a.ga && (mt2[h] & 255u) != 255u) && hn[h] + s_rsn.depth < R(-1e-11))
                                    s_negn = 1;   // rare: kept in shared memory, not a register
                            }
                            // stage hydrograph: the cell's depth becomes the gauge's stage
                            // (update_spatial_BC.m:332-341, after the step's refreshing_timestep)
                            if (INFL && own_lane[h] && (mt2[h] & kInflowBit)) {
                                const int sg = a.inflow.cell_stage[(mt2[h] >> 8) & 0x7FFFFFu];
                                if (sg >= 0) {
                                    const R sv = a.inflow.stage_now[sg];
                                    atomicAdd(&s_stage, double(sv) - double(hn[h]));
                                    hn[h] = sv;
                                }
                            }
                        }
                    }
                    // arrival times, where a depth passes the threshold for the first time
                    bool arrived = false;
#pragma unroll
                    for (int h = 0; h < CPL; ++h) arrived = arrived || (dm2[h] < K.thr && hn[h] >= K.thr);
                    if (__any_sync(FULL, arrived)) {
#pragma unroll
                        for (int h = 0; h < CPL; ++h)
                            if (own_lane[h] && dm2[h] < K.thr && hn[h] >= K.thr) a.arrival[size_t(rm2) * nx + j[h]] = t_arr;
                    }
                    R vras[CPL];   // velocity raster: largest |face velocity| (refreshing_timestep.m:109-111)
#pragma unroll
                    for (int h = 0; h < CPL; ++h) vras[h] = R(0);
                    if (mine) {
                        // a non-finite depth (NaN walls included, counted against the run's start)
                        // or one below -depth_tolerance
#pragma unroll
                        for (int h = 0; h < CPL; ++h)
                            if (!(hn[h] >= -K.tol) && own_lane[h]) ++nbad;
                    }
                    // refreshing_timestep.m:61-89, :139-150, :181-238 for these cells; an apron lane's
                    // values are computed and dropped, so that the CPL cells interleave
                    if (mine && !quiet) {
                        R vr[CPL], vu[CPL], s2[CPL], dts[CPL];   // velocities with the other sign
                        if (vcar_ok) {
#pragma unroll
                            for (int h = 0; h < CPL; ++h) vu[h] = vcar[h];
                        } else {
#pragma unroll
                            for (int h = 0; h < CPL; ++h) vu[h] = -face_velocity(qyl2[h], hfy2[h], K);
                        }
#pragma unroll
                        for (int h = 0; h < CPL; ++h) {
                            R vb;
                            face_velocities_neg(qxl2[h], hfx2[h], qyl1[h], hfy1[h], K, vr[h], vb);
                            vcar[h] = vb;
                            if (INFL) vras[h] = fmax(fmax(fabs(vr[h]), fabs(vu[h])), fabs(vb));
                            const R rc = h == 0 ? vr[h] * rc_half : vr[h];
                            const R uc = R(0.5) * (vu[h] + vb);
                            s2[h] = rc * rc + uc * uc;
                            // the largest depth of a moving cell; its celerity is taken at the end (the
                            // product by g is monotone)
                            dts[h] = fmax(fmax(hfx2[h], hfy2[h]), hf3[h]);
                        }
                        if (a.adaptive != 1) {
#pragma unroll
                            for (int h = 0; h < CPL; ++h) {
                                const R wc = fmax(sqrt(K.g * fmax(dts[h], R(0))), R(1e-10));
                                dts[h] = fmax(fmax(fabs(vr[h]), fabs(vu[h])), fabs(vcar[h])) + wc;
                            }
                        }
#pragma unroll
                        for (int h = 0; h < CPL; ++h) {
                            if (own_lane[h]) s2max = fmax(s2max, s2[h]);
                            if (own_lane[h] && s2[h] >= a.stag_s2) cmaxv = fmax(cmaxv, dts[h]);
                        }
                    }
                    V4* const row = sout + size_t(rm2) * nx;
#pragma unroll
                    for (int h = 0; h < CPL; ++h) {
                        if (!own_lane[h]) continue;
                        V4 o4;
                        o4.x = hn[h];
                        o4.y = qxl2[h];
                        o4.z = qyl2[h];
                        o4.w = hn[h] > dm2[h] ? hn[h] : dm2[h];   // save_output_maps.m:598, max(d_t, dmax)
                        row[j[h]] = o4;
                    }
                    // running maxima of the velocity raster and of depth x velocity
                    // (save_output_maps.m:588-604, snisb_velocity_hazard_snapshot :832-848)
                    if (INFL && a.vmax) {
#pragma unroll
                        for (int h = 0; h < CPL; ++h) {
                            if (!own_lane[h]) continue;
                            const size_t c2 = size_t(rm2) * nx + j[h];
                            const R vo = a.vmax[c2];
                            a.vmax[c2] = vras[h] > vo ? vras[h] : vo;
                            const R hd = fmax(hn[h], R(0));
                            R hz = hd * vras[h];
                            if (hd < R(0.01) || !isfinite(hz)) hz = R(0);
                            const R ho = a.hzmax[c2];
                            a.hzmax[c2] = isnan(hn[h]) ? hn[h] : (hz > ho ? hz : ho);
                        }
                    }
                }
            } else {
            // the infiltration and rain-map instantiations keep the per-lane branch around the cell
            // body (fewer live registers: measured faster there)
    #pragma unroll
                for (int h = 0; h < CPL; ++h) {
                    if (own_lane[h] && frow) {
                        const size_t c2 = size_t(rm2) * nx + j[h];
                        // a control structure's transfers join the depth after the fluxes
                        // (Local_Inertial_Model_D4.m:318-344, :390)
                        R h_in = hT2[h];
                        if (INFL && (mt2[h] & kInflowBit)) {
                            const int ss = a.inflow.cell_struct[(mt2[h] >> 8) & 0x7FFFFFu];
                            if (ss >= 0) h_in = h_in + a.strct.extra[ss];
                        }
                        R hn = quiet ? h_in + R(0) : continuity(h_in, qxl2_left[h], qxl2[h], qyl2[h], qyl1[h], K);
                        const R negtol = -K.tol;
                        R hf3 = R(0);
                        const unsigned ord = INFL ? outlet_ord(mt2[h]) : mt2[h] >> 8;
                        if (ord) {
                            const int o = int(ord) - 1;
                            R ho;
                            const R qq = outlet_sink(hn, a.outlet_coef[o], a.outlet_type, K, ho);
                            hf3 = ho;
                            a.hf3[o] = ho;
                            a.qo[o] = qq;
                            if (mine) out_acc_r.add(qq * K.dt);
                            // the next step's clamp is skipped when an outlet cell (outside the
                            // infiltrating soils) stays negative after the next rain
                            // (Hydrological_Model.m:45-50); only outlet cells can end negative
                            if (mine && !(a.ga && (mt2[h] & 255u) != 255u) &&
                                hn + (MAP ? rain_at_cell(a, s_rsn, rm2, j[h]) : s_rsn.depth) < R(-1e-11))
                                s_negn = 1;   // rare: kept in shared memory, not a register
                        }
                        // stage hydrograph: the cell's depth becomes the gauge's stage
                        // (update_spatial_BC.m:332-341, after the step's refreshing_timestep)
                        if (INFL && (mt2[h] & kInflowBit)) {
                            const int sg = a.inflow.cell_stage[(mt2[h] >> 8) & 0x7FFFFFu];
                            if (sg >= 0) {
                                const R sv = a.inflow.stage_now[sg];
                                atomicAdd(&s_stage, double(sv) - double(hn));
                                hn = sv;
                            }
                        }
                        // a non-finite depth (NaN walls included, counted against the run's start)
                        // or one below -depth_tolerance
                        nbad += (hn >= negtol || !mine) ? 0u : 1u;
                        const R dm = dm2[h];
                        if (dm < K.thr && hn >= K.thr) a.arrival[c2] = t_arr;
                        // refreshing_timestep.m:61-89, :139-150, :181-238 for this cell
                        R vras = R(0);   // velocity raster: largest |face velocity| (refreshing_timestep.m:109-111)
                        if (!quiet && mine) {
                            const R vr = face_velocity(qxl2[h], hfx2[h], K);
                            R vu;
                            if (vcar_ok) vu = vcar[h];
                            else vu = face_velocity(qyl2[h], hfy2[h], K);
                            const R vb = face_velocity(qyl1[h], hfy1[h], K);
                            vcar[h] = vb;
                            if (INFL) vras = fmax(fmax(fabs(vr), fabs(vu)), fabs(vb));
                            const R rc = vr * (j[h] == 0 ? R(0.5) : R(1));
                            const R uc = R(0.5) * (vu + vb);
                            const R s2 = rc * rc + uc * uc;
                            s2max = fmax(s2max, s2);
                            if (s2 >= a.stag_s2) {
                                R dts = fmax(fmax(hfx2[h], hfy2[h]), hf3);
                                if (a.adaptive != 1) {
                                    const R wc = fmax(sqrt(K.g * fmax(dts, R(0))), R(1e-10));
                                    dts = fmax(fmax(fabs(vr), fabs(vu)), fabs(vb)) + wc;
                                }
                                cmaxv = fmax(cmaxv, dts);
                            }
                        }
                        V4 o4;
                        o4.x = hn;
                        o4.y = qxl2[h];
                        o4.z = qyl2[h];
                        o4.w = hn > dm ? hn : dm;   // save_output_maps.m:598, max(d_t, dmax)
                        sout[c2] = o4;
                        // running maxima of the velocity raster and of depth x velocity
                        // (save_output_maps.m:588-604, snisb_velocity_hazard_snapshot :832-848)
                        if (INFL && a.vmax) {
                            const R vo = a.vmax[c2];
                            a.vmax[c2] = vras > vo ? vras : vo;
                            const R hd = fmax(hn, R(0));
                            R hz = hd * vras;
                            if (hd < R(0.01) || !isfinite(hz)) hz = R(0);
                            const R ho = a.hzmax[c2];
                            a.hzmax[c2] = isnan(hn) ? hn : (hz > ho ? hz : ho);
                        }
                    }
                }
            }
            vcar_ok = !quiet && mine && frow;
            lim2 = lim1;
            if (flg && lane == 0) dfl[r - 2] = 0;   // rewritten: no longer known dry
            // (G) shift the window down one row
#pragma unroll
            for (int h = 0; h < CPL; ++h) {
                hT2[h] = hT1[h]; hT1[h] = hT0[h];
                qxu1[h] = qxu0[h]; qyu1[h] = qyu0[h];
                hfx2[h] = hfx1[h]; hfx1[h] = hfx0[h];
                hfy2[h] = hfy1[h]; hfy1[h] = hfy0[h];
                sc2[h] = sc1[h];
                qxl2[h] = qxl1[h]; qyl2[h] = qyl1[h];
                dm2[h] = dm1[h]; dm1[h] = X[h].w;
                mt2[h] = mt1[h]; mt1[h] = meta[h];
                if (SCH) qyp1[h] = X[h].z;
            }
        }
        // every phase of the ring's barriers has completed: retire them so that the next
        // item of a persistent CTA can initialise them again
        __syncwarp();
        if (lane == 0 && !timed_out)
            for (int s = 0; s < kStages; ++s) mbar_inval(bar0 + 8u * s);
        }  // !blk_skip
    }

    if (a.adaptive == 1 && cmaxv >= R(0)) cmaxv = K.g * cmaxv;
    if (MAP) rain_acc += rain_acc_r.value();
    if (INF) inf_acc += inf_acc_r.value();
    if (out_acc_r.any()) out_acc += out_acc_r.value();
    return step_finish<R, NT, INF, MAP, INFL, SOLO>(a, sh, rain_acc, inf_acc, out_acc, s2max, cmaxv, nbad, timed_out,
                                                    phase, sout, gout);
}

// Rain maps from gauges by inverse-distance weighting, one full-resolution map per record
// interval (Rainfall_Interpolator.m / idw_function.m with p = 2, the Euclidean norm and no
// radius): cell (i, j) sits at (x_ul + res (j+1), y_ul - res (i+1))
// (HydroPol2D_preprocessing.m:2420-2421); distance d = sqrt(dx^2 + dy^2), 0 -> eps, weight
// 1/d^2; gauges whose record is NaN are left out of that interval's map, and an interval
// without any gauge is dry.  Sums run over the gauges in order, in FP64.
static __global__ void k_idw_maps(int ny, int nx, double res, double x_ul, double y_ul, int ng, const double* xg,
                           const double* yg, int nt, const double* rate, float* maps) {
    const size_t n = size_t(ny) * nx;
    for (size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < n; c += size_t(gridDim.x) * blockDim.x) {
        const int i = int(c / nx), j = int(c % nx);
        const double X = x_ul + res * double(j + 1), Y = y_ul - res * double(i + 1);
        for (int m = 0; m < nt; ++m) {
            double num = 0.0, den = 0.0;
            for (int g = 0; g < ng; ++g) {
                const double r = rate[size_t(m) * ng + g];
                if (isnan(r)) continue;
                const double dx = fabs(X - xg[g]), dy = fabs(Y - yg[g]);
                double d = sqrt(dx * dx + dy * dy);
                if (d == 0.0) d = 2.220446049250313e-16;
                const double w = 1.0 / (d * d);
                num = num + w * r;
                den = den + w;
            }
            maps[size_t(m) * n + c] = den > 0.0 ? float(num / den) : 0.0f;
        }
    }
}

// ---------------- host boundary on the device: records built from the caller's arrays ----
// static record {dz_x, dz_y, n^2, meta} from the elevation and roughness in FP64 (dz formed in FP64 and rounded once; the closed domain edges +inf).  A cell
// of NaN elevation (idx_nan) gets n^2 = NaN: its own faces are closed by their NaN dz before
// n^2 is read, so the NaN only marks the cell as outside the domain (k_skip_flag reads it).
template <typename R>
__global__ void k_build_static(int ny, int nx, const double* z, const double* rough, const uint32_t* meta,
                               typename Vec<R>::V4* stat) {
    const size_t n = size_t(ny) * nx;
    const double edge = __longlong_as_double(0x7ff0000000000000ll);   // +inf
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x) {
        const int i = int(k / nx), j = int(k % nx);
        const R a = R((j + 1 < nx) ? z[k + 1] - z[k] : edge);
        const R b = R((i >= 1) ? z[k - nx] - z[k] : edge);
        const R c = isnan(z[k]) ? R(__longlong_as_double(0x7ff8000000000000ll)) : R(rough[k] * rough[k]);
        stat[k] = typename Vec<R>::V4{a, b, c, make_meta<R>(meta[k])};
    }
}
// state record {h, q_x, q_y, dmax = -inf} from depths.d_t [mm] and outflow_bates pages 1-2
// [mm/h] (NULL: zero fluxes)
template <typename R>
__global__ void k_build_state(size_t n, const double* d, const double* outflow, double res,
                              typename Vec<R>::V4* st) {
    const R ninf = R(__longlong_as_double(0xfff0000000000000ll));
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x) {
        typename Vec<R>::V4 x;
        x.x = R(d[k] / 1000.0);
        // outflow_bates [mm/h] -> q [m^2/s]: mm/h / 1000 / 3600 * dx (LIM_D4.m:198)
        x.y = outflow ? R(outflow[k] / 3.6e6 * res) : R(0);
        x.z = outflow ? R(outflow[n + k] / 3.6e6 * res) : R(0);
        x.w = ninf;
        st[k] = x;
    }
}
template <typename R> __global__ void k_fill(size_t n, R* p, R v) {
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x)
        p[k] = v;
}
// one component of the state records (0..3 = h, q_x, q_y, dmax), for read-back
template <typename R>
__global__ void k_state_component(size_t n, const typename Vec<R>::V4* st, int comp, R* out) {
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x) {
        const auto v = st[k];
        out[k] = comp == 0 ? v.x : comp == 1 ? v.y : comp == 2 ? v.z : v.w;
    }
}

// read-back into FP64: one component of the state records (0..3 = h, q_x, q_y, dmax) or a plain
// array, times `scale` (the conversion to the caller's units happens on the device)
template <typename R>
__global__ void k_state_component_f64(size_t n, const typename Vec<R>::V4* st, int comp, double scale, double* out) {
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x) {
        const auto v = st[k];
        const R x = comp == 0 ? v.x : comp == 1 ? v.y : comp == 2 ? v.z : v.w;
        out[k] = double(x) * scale;
    }
}
template <typename R> __global__ void k_scaled_f64(size_t n, const R* src, double scale, double* out) {
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x)
        out[k] = double(src[k]) * scale;
}
template <typename R> __global__ void k_divided_f64(size_t n, const R* src, double div, double* out) {
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x)
        out[k] = double(src[k]) / div;
}
// the soil storage I of the soil records, times `scale`
template <typename R>
__global__ void k_soil_component_f64(size_t n, const typename Vec<R>::V2* gs, double scale, double* out) {
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x)
        out[k] = double(gs[k].x) * scale;
}
// qout_left (-q_x of the cell to the left, -0 on the first column) or qout_down (-q_y of the
// cell below, -0 on the last row) [mm/h] (Local_Inertial_Model_D4.m:347-350)
template <typename R>
__global__ void k_shifted_flux_f64(int ny, int nx, const typename Vec<R>::V4* st, int down, double scale, double* out) {
    const size_t n = size_t(ny) * nx;
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x) {
        const int i = int(k / nx), j = int(k % nx);
        if (down) out[k] = i + 1 == ny ? -0.0 : -double(st[k + nx].z) * scale;
        else out[k] = j == 0 ? -0.0 : -double(st[k - 1].y) * scale;
    }
}
// CA_States.I_tot_end_cell [m^3] (Local_Inertial_Model_D4.m:512-514): |right + up + outlet flux|
// [mm/h] x dt over the cell area, from the state records and each outlet cell's sink rate
template <typename R>
__global__ void k_itot_f64(size_t n, const typename Vec<R>::V4* st, const typename Vec<R>::V4* stat, const R* qo,
                           double to_mmh, double dts, double res, double* out) {
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x) {
        const auto v = st[k];
        const unsigned ord = outlet_ord(meta_bits(stat[k].w));
        const double of = ord ? double(qo[ord - 1]) * 3.6e6 : 0.0;
        out[k] = fabs(double(v.y) * to_mmh + double(v.z) * to_mmh + of) * dts / 1000.0 / 3600.0 * res * res;
    }
}

// a map record taken by the host when no step follows the one that triggered it
template <typename R> __global__ void k_record_depth(size_t n, const typename Vec<R>::V4* st, R* dst) {
    for (size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < n; c += size_t(gridDim.x) * blockDim.x)
        dst[c] = st[c].x;
}

// gauge depths of the current rain interval (after a host change of the inflow or clock)
template <typename R> __global__ void k_inflow_depth(InflowDesc<R> d, const StepScalars* sc) {
    const double ra = sc->rain_a, rb = sc->rain_b, t = sc->t_min;
    for (int g = threadIdx.x; g < d.n_gauges; g += blockDim.x)
        d.depth[g] = R(inflow_integral(d, g, ra, rb) / 60000.0);
    for (int g = threadIdx.x; g < d.n_stage; g += blockDim.x) d.stage_now[g] = R(stage_at(d, g, t));
}

// Retry of a rejected step (HydroPol2D_Main_While.m:928-951): the reference's new step needs
// the wave celerity sqrt(g max(max(d_tot), max(d_p))) of the attempt.  Over the state the
// attempt started from (buffer cur, untouched by it) this restates phase (A) per cell -- rain,
// infiltration, inflow and clamps give d_tot -- and reduces max(d_p, d_tot) (NaN skipped, as
// MATLAB's max) into sc->retry_dmax.  It also takes back the arrival times the attempt wrote:
// a cell whose arrival equals the attempt's t_arr and whose start-of-step maximum is below the
// threshold was marked by it (a block of temporal blocking marks with the times of its
// sub-steps, the range [t_arr_lo, t_arr_hi]).  inf: 0 none, 1 Green-Ampt, 2 van Genuchten.
template <typename R>
__global__ void k_retry_scan(const FusedArgs<R> a, int inf, R t_arr_lo, R t_arr_hi) {
    StepScalars* sc = a.sc;
    RainStep<R> RS;
    RS.make(a.rain, sc->rain_a, sc->rain_b);
    StepConsts<R> K;
    K.make(sc->time_step * 60.0, a.res, a.tol_mm, a.thr_mm);
    const bool skip = sc->skip_clamp != 0;
    const typename Vec<R>::V4* st = sc->cur ? a.st1 : a.st0;
    const typename Vec<R>::V2* gs = sc->cur ? a.gs1 : a.gs0;
    const size_t n = size_t(a.ny) * a.nx;
    R m = R(0);
    for (size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < n; c += size_t(gridDim.x) * blockDim.x) {
        const int r = int(c / a.nx), j = int(c % a.nx);
        const auto rec = st[c];
        R hh = rec.x;
        m = fmax(m, hh);
        hh = hh + RS.at(a.rain, r, j, a.ny, a.nx);
        const unsigned meta = meta_bits(a.stat[c].w);
        if (inf && (meta & 255u) != 255u) {
            R Ic = gs[c].x, Tc = gs[c].y;
            if (inf == 1) green_ampt(hh, Ic, Tc, a.classes[meta & 255u], K);
            else vg_infiltration(hh, Ic, Tc, a.classes_vg[meta & 255u], a.vg, K);
        }
        if (a.inflow.n_gauges) add_inflow(a.inflow, meta, hh);
        if (!skip && hh < R(1e-9)) hh = R(0);
        if (hh < R(0)) hh = R(0);
        m = fmax(m, hh);
        const R ar = a.arrival[c];
        if (ar >= t_arr_lo && ar <= t_arr_hi && rec.w < K.thr) a.arrival[c] = R(__int_as_float(0x7f800000));
    }
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0 && m > R(0)) atomicMax(&sc->retry_dmax, ord_bits(m));
}

// the structure transfers of the first fused step of a call (one block)
template <typename R, int INF, bool MAP>
__global__ void k_struct_prime(const FusedArgs<R> a) {
    __shared__ RainStep<R> s_r;
    __shared__ StepConsts<R> s_k;
    __shared__ int s_skip, s_cur;
    __shared__ double s_ts;
    if (threadIdx.x == 0) {
        const StepScalars* sc = a.sc;
        s_r.make(a.rain, sc->rain_a, sc->rain_b);
        s_ts = sc->time_step;
        s_k.make(s_ts * 60.0, a.res, a.tol_mm, a.thr_mm);
        s_skip = sc->skip_clamp;
        s_cur = sc->cur;
    }
    __syncthreads();
    structure_prepare<R, INF, MAP, true>(a, s_r, s_skip != 0, s_k, s_cur ? a.st1 : a.st0, s_cur ? a.gs1 : a.gs0,
                                         threadIdx.x, blockDim.x, s_ts);
}

template <typename R, int NT, int INF, bool MAP, int CPL = 1, bool INFL = false, int SCH = 0>
__global__ void __launch_bounds__(NT, FusedOcc<R, CPL>::minb) k_fused_step(const __grid_constant__ FusedArgs<R> a, int phase) {
    fused_item<R, NT, INF, MAP, CPL, INFL, SCH, true>(a, blockIdx.x, phase);
}

// a step's launch, allowed to begin before the launch before it has ended (step_begin waits)
template <typename K, typename... A>
inline void launch_step(K kernel, unsigned grid, unsigned block, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

// ---- batched ensemble ----------------------------------------------------------------
// Members are independent grids, each with its own FusedArgs (clock, dt, buffers).  Each
// step, k_ens_plan lists the CTA-sized items of the members still running (exclusive
// prefix over members) and k_ens_step -- a persistent grid sized to the resident CTA
// slots -- pulls items from a queue head.  Items of one launch never wait on each other;
// the CTA that completes a member's last item refreshes that member's dt and clock.
struct EnsQueue {
    unsigned head;       // next item to hand out
    unsigned total;      // items of this step
    unsigned n_active;   // members running this step
    unsigned stalled;    // members stopped by a failed row copy
};

template <typename R>
__global__ void k_ens_plan(const FusedArgs<R>* __restrict__ members, int n_members, unsigned* prefix, EnsQueue* q) {
    // one CTA of 1024 threads; members are scanned in chunks of 1024
    __shared__ unsigned s_run[1024];
    __shared__ unsigned s_base, s_act, s_stall;
    const int tid = threadIdx.x;
    if (tid == 0) { s_base = 0; s_act = 0; s_stall = 0; }
    __syncthreads();
    for (int m0 = 0; m0 < n_members; m0 += 1024) {
        const int m = m0 + tid;
        unsigned items = 0;
        if (m < n_members) {
            const FusedArgs<R>& a = members[m];
            const StepScalars* sc = a.sc;
            const bool stalled = (sc->status & kStatusTimeout) != 0u;
            const bool running = sc->t_min <= a.t_end && !stalled && !sc->halted;
            items = running ? a.n_ctas : 0u;
            if (running) atomicAdd(&s_act, 1u);
            if (stalled) atomicAdd(&s_stall, 1u);
        }
        s_run[tid] = items;
        __syncthreads();
        // Hillis-Steele inclusive scan over the chunk
        for (int o = 1; o < 1024; o <<= 1) {
            const unsigned v = tid >= o ? s_run[tid - o] : 0u;
            __syncthreads();
            s_run[tid] += v;
            __syncthreads();
        }
        if (m < n_members) prefix[m] = s_base + s_run[tid] - items;
        __syncthreads();
        if (tid == 0) s_base += s_run[1023];
        __syncthreads();
    }
    if (tid == 0) {
        prefix[n_members] = s_base;
        q->head = 0;
        q->total = s_base;
        q->n_active = s_act;
        q->stalled = s_stall;
    }
}

template <typename R, int NT, int INF, bool MAP, int CPL = 1, bool INFL = false, int SCH = 0>
__global__ void __launch_bounds__(NT, FusedOcc<R, CPL>::minb)
k_ens_step(const FusedArgs<R>* __restrict__ members, int n_members, const unsigned* __restrict__ prefix,
           EnsQueue* q) {
    __shared__ FusedArgs<R> s_a;
    __shared__ unsigned s_item, s_local;
    __shared__ int s_m;
    const int tid = threadIdx.x;
    const unsigned total = q->total;   // written by k_ens_plan before this launch
    for (;;) {
        __syncthreads();   // the previous item is finished with s_a and the ring
        if (tid == 0) {
            const unsigned it = atomicAdd(&q->head, 1u);
            s_item = it;
            if (it < total) {
                // member m with prefix[m] <= it < prefix[m+1] (members without items have
                // prefix[m] == prefix[m+1] and are passed over)
                int lo = 0, hi = n_members - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (prefix[mid] <= it) lo = mid; else hi = mid - 1;
                }
                s_m = lo;
                s_local = it - prefix[lo];
            }
        }
        __syncthreads();
        if (s_item >= total) return;
        {
            const unsigned* src = reinterpret_cast<const unsigned*>(members + s_m);
            unsigned* dst = reinterpret_cast<unsigned*>(&s_a);
            for (int w = tid; w < int(sizeof(FusedArgs<R>) / 4); w += NT) dst[w] = src[w];
        }
        __syncthreads();
        if (!fused_item<R, NT, INF, MAP, CPL, INFL, SCH, false>(s_a, s_local, 0)) return;   // ring unusable after a timeout
    }
}

// Clamp-skip flag for the first fused step of a call, over every cell (the state may
// have been set from the host).  sc->skip_clamp must be zero on entry.  Also counts the cells
// with a finite depth (n_finite) and with a non-finite one (n_bad0, the count a healthy step
// keeps), and flags a non-finite depth in a cell of finite elevation (bad_domain).
template <typename R>
__global__ void k_skip_flag(const typename Vec<R>::V4* st, const typename Vec<R>::V4* stat, int ny, int nx,
                            RainDesc rain, int ga, double res, double tol_mm, double thr_mm, StepScalars* sc,
                            int own_r0, int own_r1) {
    const size_t n = size_t(ny) * nx;
    RainStep<R> RS;
    RS.make(rain, sc->rain_a, sc->rain_b);
    int neg = 0;
    unsigned long long fin = 0;
    for (size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < n; c += size_t(gridDim.x) * blockDim.x) {
        const R hc = st[c].x;
        const auto sr = stat[c];
        const int ci = int(c / nx);
        if (ci < own_r0 || ci >= own_r1) continue;   // a row slab counts its own rows only
        if (isfinite(hc)) ++fin;
        else {
            atomicAdd(&sc->n_bad0, 1ull);
            if (!isnan(sr.z)) atomicOr(&sc->bad_domain, 1);
        }
        if (ga && (meta_bits(sr.w) & 255u) != 255u) continue;
        const int i = int(c / nx), j = int(c % nx);
        if (hc + RS.at(rain, i, j, ny, nx) < R(-1e-11)) neg = 1;
    }
    for (int o = 16; o > 0; o >>= 1) fin += __shfl_xor_sync(0xffffffffu, fin, o);
    if ((threadIdx.x & 31) == 0 && fin) atomicAdd(&sc->n_finite, fin);
    if (__syncthreads_or(neg) && threadIdx.x == 0) atomicOr(&sc->skip_clamp, 1);
}

}  // namespace hp2d
