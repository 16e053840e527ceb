// Unfused kernels: one reference function per C-ABI call (hp2d_hydrology_step, hp2d_li_step,
// hp2d_cfl_dt, hp2d_track_maxima).  They exist so that a MATLAB caller that keeps calling
// Local_Inertial_Model_D4 / Infiltration_Module / refreshing_timestep separately gets the same
// numbers as the fused step; they share every formula with it (hp2d_device.cuh).  The routing step is
// the tile kernel without its clock (hp2d_tile.cuh, k_tile_li).
//
// The calls work on the state records themselves, one pass each: hydrology and routing from the
// current buffer into the other one, the time step and the maxima on the current one.  Columns run
// over the threads and rows over the blocks, so no cell needs a division for its place.  1024^2 FP64:
// hydrology 41 us, routing 73 (its FP64 quotients), time step 42, maxima 16.
#pragma once

#include "hp2d_device.cuh"
#include "hp2d_fused.cuh"

namespace hp2d {

constexpr int kRowsPerBlock = 8;   // rows a thread of the row kernels walks
inline dim3 rows_grid(int ny, int nx) {
    return dim3(unsigned((nx + 127) / 128), unsigned(std::min((ny + kRowsPerBlock - 1) / kRowsPerBlock, 65535)));
}

// block sum of v into *to (one atomic per block that has any)
__device__ __forceinline__ void block_add(double v, double* to, double* part) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < 4; ++w) s += part[w];
        if (s != 0.0) atomicAdd(to, s);
    }
    __syncthreads();
}

// Rain, infiltration, inflow and the depth clamp (Hydrological_Model.m:14-55) from buffer cur into
// the other one.  The clamp is skipped when some depth ends below -1e-8 mm (acc_neg): pass 0 clamps
// and reports, pass 1 runs only if it did and does it again without the clamp.  INF: 0 none, 1
// Green-Ampt, 2 van Genuchten.
template <typename R, int INF, bool MAP>
__global__ void __launch_bounds__(128) k_hydrology(const __grid_constant__ FusedArgs<R> a, int cur, double rain_a, double rain_b,
                                                   const StepConsts<R> K, int pass) {
    using V4 = typename Vec<R>::V4;
    using V2 = typename Vec<R>::V2;
    __shared__ RainStep<R> s_rs;
    __shared__ double s_part[4];
    if (pass == 1 && __ldcg(&a.sc->acc_neg) == 0) return;
    if (threadIdx.x < 32) RainStep<R>::make_warp(s_rs, a.rain, rain_a, rain_b, threadIdx.x);
    __syncthreads();
    const V4* __restrict__ sin = cur ? a.st1 : a.st0;
    V4* __restrict__ sout = cur ? a.st0 : a.st1;
    const V2* __restrict__ gin = cur ? a.gs1 : a.gs0;
    V2* __restrict__ gout = cur ? a.gs0 : a.gs1;
    const int j = blockIdx.x * 128 + threadIdx.x;
    double racc = 0.0, iacc = 0.0;
    int neg = 0;
    if (j < a.nx)
        for (int q = blockIdx.y; q * kRowsPerBlock < a.ny; q += gridDim.y) {
            const int r1 = min((q + 1) * kRowsPerBlock, a.ny);
#pragma unroll 2
            for (int r = q * kRowsPerBlock; r < r1; ++r) {
                const size_t c = size_t(r) * a.nx + j;
                V4 x = sin[c];
                R rr = s_rs.depth;
                if constexpr (MAP) {
                    rr = R(0);
                    const MapRow<R> mr = map_row<R>(r, a.rain.my, a.map_sy);
                    for (int m = 0; m < s_rs.nm; ++m) {
                        R top, bot;
                        map_column<R>(a.rain.maps + size_t(s_rs.m[m]) * a.rain.my * a.rain.mx, mr, j, a.rain.mx, a.map_sx,
                                      top, bot);
                        const R v = s_rs.w[m] * ((R(1) - mr.wy) * top + mr.wy * bot);
                        rr = m == 0 ? v : rr + v;
                    }
                }
                R hh = x.x + rr;
                if (isfinite(hh)) racc += double(rr);
                unsigned meta = 0u;
                if (INF || a.inflow.n_gauges) meta = meta_bits(a.stat[c].w);
                if (INF) {
                    V2 gs = gin[c];
                    const unsigned scl = meta & 255u;
                    if (scl != 255u) {
                        R Ic = gs.x, Tc = gs.y;
                        const R fd = INF == 1 ? green_ampt(hh, Ic, Tc, a.classes[scl], K)
                                              : vg_infiltration(hh, Ic, Tc, a.classes_vg[scl], a.vg, K);
                        gs.x = Ic;
                        gs.y = Tc;
                        if (isfinite(fd)) iacc += double(fd);
                    }
                    gout[c] = gs;
                }
                if (a.inflow.n_gauges) add_inflow(a.inflow, meta, hh);   // Hydrological_Model.m:27-28
                if (hh < R(-1e-11)) neg = 1;
                if (pass == 0 && hh < R(1e-9)) hh = R(0);
                if (hh < R(0)) hh = R(0);
                x.x = hh;
                sout[c] = x;
            }
        }
    if (pass == 0) {
        block_add(racc, &a.sc->acc_rain, s_part);
        if (INF) block_add(iacc, &a.sc->acc_inf, s_part);
        if (__syncthreads_or(neg) && threadIdx.x == 0) atomicOr(&a.sc->acc_neg, 1);
    }
}

// control-structure transfers of an unfused step (Local_Inertial_Model_D4.m:318-344), one
// thread: from the d_tot the fluxes use; the extras join the depth in the continuity update
template <typename R>
__global__ void k_struct_unfused(StructDesc<R> s, const typename Vec<R>::V4* st, double time_step, double area, StepScalars* sc) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    for (int i = 0; i < s.n; ++i) s.hres[i] = st[s.slot_cell[s.slot[3 * i]]].x;
    sc->struct_vol += structure_transfers(s, time_step, area);
}

// CFL reductions (refreshing_timestep.m:61-238) over the current records and the last routing step's
// face depths; accumulates into sc->acc_vmax/acc_cmax
template <typename R>
__global__ void __launch_bounds__(128) k_cfl(const __grid_constant__ FusedArgs<R> a, int cur, const StepConsts<R> K,
                                             const R* __restrict__ hfx, const R* __restrict__ hfy,
                                             const uint32_t* outlet_bits, int bit_words) {
    const typename Vec<R>::V4* __restrict__ st = cur ? a.st1 : a.st0;
    __shared__ R s_v[4], s_c[4];
    const int j = blockIdx.x * 128 + threadIdx.x;
    R vmax = R(0), cmax = R(0);
    if (j < a.nx)
        for (int q = blockIdx.y; q * kRowsPerBlock < a.ny; q += gridDim.y) {
            const int r1 = min((q + 1) * kRowsPerBlock, a.ny);
            size_t c = size_t(q) * kRowsPerBlock * a.nx + j;
            auto x = st[c];
            R hy = hfy[c];
            for (int r = q * kRowsPerBlock; r < r1; ++r, c += a.nx) {
                const bool last = r + 1 >= a.ny;
                auto xb = x;
                R hb = R(0), qyb = R(0);
                if (!last) {
                    xb = st[c + a.nx];
                    hb = hfy[c + a.nx];
                    qyb = xb.z;
                }
                R h3 = R(0);
                if (a.n_outlets && ((outlet_bits[size_t(r) * bit_words + (j >> 5)] >> (j & 31)) & 1u)) {
                    const int o = find_outlet(a.outlet_cells, a.n_outlets, int(c));
                    if (o >= 0) h3 = a.hf3[o];
                }
                R sp, ce;
                cfl_cell(x.y, x.z, qyb, hfx[c], hy, hb, h3, j == 0, a.adaptive, K, sp, ce);
                vmax = fmax(vmax, sp);
                cmax = fmax(cmax, ce);
                x = xb;
                hy = hb;
            }
        }
    vmax = warp_max(vmax);
    cmax = warp_max(cmax);
    if ((threadIdx.x & 31) == 0) {
        s_v[threadIdx.x >> 5] = vmax;
        s_c[threadIdx.x >> 5] = cmax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 4; ++w) {
            vmax = fmax(vmax, s_v[w]);
            cmax = fmax(cmax, s_c[w]);
        }
        if (vmax > R(0)) atomicMax(&a.sc->acc_vmax, ord_bits(vmax));
        if (cmax > R(0)) atomicMax(&a.sc->acc_cmax, ord_bits(cmax));
    }
}

// running maximum depth and arrival time (save_output_maps.m:588-600) in the current records
template <typename R>
__global__ void k_track(size_t n, typename Vec<R>::V4* st, R* arrival, R thr, R t_end) {
    for (size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < n; c += size_t(gridDim.x) * blockDim.x) {
        const auto v = st[c];
        if (v.w < thr && v.x >= thr) arrival[c] = t_end;
        if (v.x > v.w) st[c].w = v.x;
    }
}

// The end of an unfused call on the device, so that the host reads the scalars once: the call's sums
// into the cumulative volumes, and the buffer that now holds the state.
enum UnfusedCall { CALL_HYDROLOGY, CALL_ROUTING, CALL_TIME_STEP };
template <typename R>
__global__ void k_unfused_end(const __grid_constant__ FusedArgs<R> a, int call, double max_dt) {
    if (threadIdx.x != 0) return;
    StepScalars* sc = a.sc;
    const double area = a.res * a.res;
    if (call == CALL_TIME_STEP) {   // refreshing_timestep's refresh branch
        const double vm = from_ord(sc->acc_vmax, sizeof(R) == 8), cm = from_ord(sc->acc_cmax, sizeof(R) == 8);
        const double tcr = finalize_dt(vm, cm, a.res, a.alfa_min, a.alfa_max, a.min_dt, max_dt, a.inc, a.flag_timestep);
        sc->vmax_last = vm;
        sc->refreshed_s = tcr;
        if (tcr == a.min_dt) sc->unstable += 1;
        sc->acc_vmax = sc->acc_cmax = 0ull;
        return;
    }
    if (call == CALL_HYDROLOGY) {
        if (sc->acc_neg) sc->neg_warn += 1;
        for (int g = 0; g < a.inflow.n_gauges; ++g) sc->inflow_vol += double(a.inflow.depth[g]) * a.inflow.gauge_cells[g] * area;
    }
    sc->rain_vol += sc->acc_rain * area;
    sc->inf_vol += sc->acc_inf * area;
    sc->out_vol += sc->acc_out * area;
    sc->acc_rain = sc->acc_inf = sc->acc_out = 0.0;
    sc->acc_vmax = sc->acc_cmax = 0ull;
    sc->acc_neg = 0;
    sc->cur ^= 1;
}

}  // namespace hp2d
