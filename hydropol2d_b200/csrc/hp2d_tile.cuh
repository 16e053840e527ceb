// Fused surface-flow step on tiles: the step of hp2d_fused.cuh with a cell per thread (times RPT
// rows) instead of a warp walking down a strip, for grids whose strips cannot fill the GPU.
//
// A CTA holds rows of 32 columns, lane L the column L: warp 0 the first row, each other warp RPT
// consecutive ones.  All but two rows and two columns on each side are the tile's output (the
// draining limiter makes a cell depend on cells two away).  Neighbours in x come from other lanes
// by shuffles, neighbours in y from the thread's own rows or, across warps, through one shared
// row per warp and phase; four CTA barriers separate the phases
//   (A) rain, infiltration, clamp      (B, C) unlimited faces      (D) donor scales
//   (E) limited faces, face velocities (F) continuity, outlets, maxima, CFL terms.
// Every cell runs the operations of the strip kernel on the same values, so the results are the
// same bit for bit.
//
// Why: a strip's warp takes about 2.4 us per row (one warp's dependent chain of ~1000
// instructions), so a small grid of strips is bound by rows per warp, not by work: us per step,
// strips / tiles, 200 x 200 FP64 155 / 7.7, 512 x 512 FP32 46 / 10, 1000 x 1000 wet FP32 43 / 29.
//
// Dry tiles: a flag per tile and state buffer records that the tile's whole output was written as
// dry records there.  A tile whose depths are all zero after (A), two-cell apron included, and
// that holds no outlet or boundary cell writes zero depth and fluxes and the unchanged maximum --
// or nothing when both buffers' flags say that the record is there already; and a step without
// rain, infiltration and map record does not even read a tile when its eight neighbours are
// flagged too (the neighbours' outputs are its apron).
#pragma once

#include <mutex>

#include "hp2d_fused.cuh"

namespace hp2d {

// A CTA's warps and the rows per thread.  Warp 0 holds the first apron row only, the others RPT
// consecutive rows each.
template <typename R, int RPT> struct TileShape {
    static constexpr int NW = RPT == 1 && sizeof(R) == 4 ? 16 : 12;
    static constexpr int NT = 32 * NW;
    static constexpr int OR = 1 + (NW - 1) * RPT - 4;   // output rows
    static constexpr int OC = 28;                       // output columns
    static constexpr int MINB = 2;   // CTAs per SM
};

// named barriers over NTH threads
template <int ID, int NTH> __device__ __forceinline__ void bar_sync() {
    asm volatile("barrier.sync %0, %1;" ::"n"(ID), "n"(NTH) : "memory");
}
template <int ID, int NTH> __device__ __forceinline__ bool bar_or(bool p) {
    int any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.red.or.pred q, %2, %3, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
                 : "=r"(any) : "r"(int(p)), "n"(ID), "n"(NTH) : "memory");
    return any != 0;
}
template <int ID, int NTH> __device__ __forceinline__ void bar_arrive() {
    asm volatile("barrier.arrive %0, %1;" ::"n"(ID), "n"(NTH) : "memory");
}

// The routing step alone (Local_Inertial_Model_D4 as a call of its own, hp2d_li_step), LI: no rain,
// clock, maxima or CFL terms, the face depths kept; buffer `phase` to the other one, with the
// constants kc of the caller's time step.
template <typename R> struct LiArgs {
    StepConsts<R> kc;
    R* hfx; R* hfy;
};

template <typename R, int RPT, int INF, bool MAP, bool INFL, int SCH, bool LI>
__device__ __forceinline__ void tile_body(const FusedArgs<R>& a, int phase, const LiArgs<R>& li) {
    using V4 = typename Vec<R>::V4;
    using V2 = typename Vec<R>::V2;
    using Sh = TileShape<R, RPT>;
    constexpr int NW = Sh::NW, NT = Sh::NT, OR = Sh::OR, OC = Sh::OC;
    constexpr unsigned FULL = 0xffffffffu;
    __shared__ StepShared<R, NT> sh;
    __shared__ R x_h[NW][32], x_q[NW][32], x_s[NW][32], x_l[NW][32], x_v[NW][32];
    // dry flags of this tile and of the next: bit 0 output buffer, 1 input buffer, 2 both and all neighbours
    __shared__ unsigned s_flags[2];
    // the records of the tile that comes next, each thread's own: static, state
    extern __shared__ __align__(16) unsigned char smem_tile[];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ny = a.ny, nx = a.nx;
    const unsigned n_tiles = a.n_ctas;
    V4* const next_S = reinterpret_cast<V4*>(smem_tile) + tid;
    V4* const next_X = next_S + NT * RPT;
    // this thread's cells of tile t: column, first row
    int tx, ty, j, rw;
    bool col_ok;
    auto place = [&](unsigned t) {
        ty = int(t / unsigned(a.tile_nx));
        tx = int(t) - ty * a.tile_nx;
        j = tx * OC - 2 + lane;
        rw = ty * OR - 2 + (warp == 0 ? 0 : 1 + (warp - 1) * RPT);
        col_ok = j >= 0 && j < nx;
    };
    auto fetch = [&](V4* dst, const V4* src, V4 outside) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = rw + i;
            if (col_ok && r >= 0 && r < ny && (i == 0 || warp != 0)) copy_async(dst + i * NT, src + (size_t(r) * nx + j));
            else dst[i * NT] = outside;
        }
    };
    // infiltration: the next tile's soil records to L1, for the hydrology (with the map rows kept from row
    // to row: urban 2048^2 FP32 14.3 to 13.8 ms a pass, 1000^2 FP64 3.94 to 3.77)
    auto prefetch_soil = [&](const V2* src) {
#pragma unroll
        for (int i = 0; i < RPT; ++i)
            if (col_ok && rw + i >= 0 && rw + i < ny && (i == 0 || warp != 0)) prefetch_l1(src + (size_t(rw + i) * nx + j));
    };
    // warp 1: the dry flags of tile (tx, ty): lanes 0..8 the input flags of the 3 x 3 tiles around it,
    // lane 9 its output flag (c: the buffer that holds the state)
    auto flags = [&](unsigned t, int c) -> unsigned {
        const unsigned char* fl = a.dryflag + size_t(c) * n_tiles;
        const int ty_n = int(n_tiles) / a.tile_nx;
        bool f = lane > 9;
        if (lane < 9) {
            const int qx = tx + lane % 3 - 1, qy = ty + lane / 3 - 1;
            f = !(qx >= 0 && qx < a.tile_nx && qy >= 0 && qy < ty_n) || fl[qy * a.tile_nx + qx] != 0;
        } else if (lane == 9) {
            f = a.dryflag[size_t(c ^ 1) * n_tiles + t] != 0;
        }
        const unsigned b = __ballot_sync(FULL, f);
        return ((b >> 9) & 1u) | ((b >> 4) & 1u) << 1 | (b == FULL ? 4u : 0u);
    };
    const R inf = R(__int_as_float(0x7f800000));
    const V4 out_S{inf, inf, R(1), make_meta<R>(255u)}, out_X{R(0), R(0), R(0), R(0)};   // closed faces

    // the static records do not depend on the step's scalars; the state records and the dry flags are
    // fetched while warp 0 ends the step before
    place(blockIdx.x);
    fetch(next_S, a.stat, out_S);
    bool publish = !LI && blockIdx.x == 0 && warp == 0, next_made = LI;
    if constexpr (LI) {
        fetch(next_X, phase ? a.st1 : a.st0, out_X);
    } else {
        step_begin<R, NT, true, true>(a, sh, phase, [&](int c) {
            fetch(next_X, c ? a.st1 : a.st0, out_X);
            if (INF) prefetch_soil(c ? a.gs1 : a.gs0);
            if (a.dryflag && warp == 1) {
                const unsigned f = flags(blockIdx.x, c);
                if (lane == 0) s_flags[0] = f;
            }
        });
        if (sh.now.done) {
            copy_wait_all();
            if (publish) {
                step_next(a, sh, lane);
                step_publish<R, NT, INFL>(a, sh, phase);
            }
            return;
        }
    }

    const StepConsts<R>& K = LI ? li.kc : sh.K;
    const int cur = LI ? phase : sh.now.cur;
    const R clamp0 = LI ? R(0) : sh.now.skip ? R(0) : R(1e-9);   // depths below are zero (Hydrological_Model.m:45-52)
    const V4* __restrict__ sin = cur ? a.st1 : a.st0;
    V4* __restrict__ sout = cur ? a.st0 : a.st1;
    const V2* __restrict__ gin = cur ? a.gs1 : a.gs0;
    V2* __restrict__ gout = cur ? a.gs0 : a.gs1;

    double rain_acc = 0.0, inf_acc = 0.0, out_acc = 0.0;
    Kahan<R> rain_acc_r, inf_acc_r, out_acc_r;
    unsigned nbad = 0u;
    R s2max = R(0), cmaxv = R(-1);
    for (unsigned tile = blockIdx.x, it = 0; tile < n_tiles; tile += gridDim.x, ++it) {
    V4 S[RPT], X[RPT];
    copy_wait_all();   // this thread's own copies: no barrier needed
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        S[i] = next_S[i * NT];
        X[i] = next_X[i * NT];
    }
    const int r0 = ty * OR, r_end = min(r0 + OR, ny);
    const int j = tx * OC - 2 + lane, rw = r0 - 2 + (warp == 0 ? 0 : 1 + (warp - 1) * RPT);
    const bool col_ok = j >= 0 && j < nx;
    const bool own_lane = lane >= 2 && lane < 30 && j < nx;
    const R first_col = j == 0 ? R(0.5) : R(1);   // refreshing_timestep.m's vel_left on the first column
    const int tile_cells = (r_end - r0) * (min(tx * OC + OC, nx) - tx * OC);
    const unsigned fbits = !LI && a.dryflag ? s_flags[it & 1u] : 0u;
    unsigned char* const fl_out = !LI && a.dryflag ? a.dryflag + size_t(cur ^ 1) * n_tiles + tile : nullptr;
    const bool fo = (fbits & 1u) != 0u, fi = (fbits & 2u) != 0u;
    bool tile_skip = false;
    if constexpr (INF == 0 && !MAP && !LI)
        tile_skip = (fbits & 4u) && sh.now.rec < 0 && sh.p.rs.depth == R(0) && K.thr > R(0);
    const unsigned next = tile + gridDim.x;
    const bool more = next < n_tiles;
    if (more) {   // the next tile's records and flags arrive while this one is computed
        place(next);
        fetch(next_S, a.stat, out_S);
        fetch(next_X, sin, out_X);
        if (INF) prefetch_soil(gin);
        if (!LI && a.dryflag && warp == 1) {
            const unsigned f = flags(next, cur);
            if (lane == 0) s_flags[(it + 1u) & 1u] = f;
        }
    }
    if (tile_skip) {
        if (tid == 0) { sh.skipw += unsigned(tile_cells); sh.skipr += unsigned(tile_cells); }
    } else {
        // (A) hydrology
        R hT[RPT];
        bool wet = false;
        R map_top[2] = {R(0), R(0)}, map_bot[2] = {R(0), R(0)};   // rain maps: the two rows around r at column j
        int map_iy = -1;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = rw + i;
            hT[i] = R(0);
            if (col_ok && r >= 0 && r < ny && (i == 0 || warp != 0)) {
                const size_t c = size_t(r) * nx + j;
                const unsigned meta = meta_bits(S[i].w);
                R hh = X[i].x;
                if constexpr (LI) {   // the depth as it is; the fluxes see its positive part
                    hT[i] = fmax(hh, R(0));
                    wet = wet || hh != R(0) || (meta >> 8) != 0u;
                    continue;
                }
                const bool own_cell = own_lane && warp != 0 && r >= r0 && r < r_end;
                // a pending map record keeps the depth this step starts from
                if (sh.now.rec >= 0 && own_cell) a.rec.snap[size_t(sh.now.rec) * (size_t(ny) * nx) + c] = hh;
                R rr;
                if constexpr (MAP) {   // RainStep::at
                    rr = R(0);
                    const MapRow<R> mr = map_row<R>(r, a.rain.my, a.map_sy);
                    if (mr.iy0 != map_iy) {   // a thread's rows mostly lie between the same two of the map
                        map_iy = mr.iy0;
#pragma unroll
                        for (int q = 0; q < 2; ++q)
                            if (q < sh.p.rs.nm)
                                map_column<R>(a.rain.maps + size_t(sh.p.rs.m[q]) * a.rain.my * a.rain.mx, mr, j, a.rain.mx,
                                              a.map_sx, map_top[q], map_bot[q]);
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        if (q >= sh.p.rs.nm) continue;
                        const R v = sh.p.rs.w[q] * ((R(1) - mr.wy) * map_top[q] + mr.wy * map_bot[q]);
                        rr = q == 0 ? v : rr + v;
                    }
                } else {
                    rr = sh.p.rs.depth;
                }
                hh = hh + rr;
                const bool own = own_cell && r >= a.own_r0 && r < a.own_r1;
                if (MAP && own && isfinite(hh)) rain_acc_r.add(rr);
                if (INF) {
                    const V2 Gs = gin[c];
                    const unsigned scl = meta & 255u;
                    V2 go = Gs;
                    if (scl != 255u) {
                        R Ic = Gs.x, Tc = Gs.y;
                        const R fd = INF == 1 ? green_ampt(hh, Ic, Tc, a.classes[scl], K)
                                              : vg_infiltration(hh, Ic, Tc, a.classes_vg[scl], a.vg, K);
                        go.x = Ic;
                        go.y = Tc;
                        if (own && isfinite(fd)) inf_acc_r.add(fd);
                    }
                    if (own) gout[c] = go;
                }
                if (INFL) add_inflow(a.inflow, meta, hh);
                hT[i] = hh < clamp0 ? R(0) : hh;
                hh = hT[i];
                wet = wet || hh != R(0) || (own_cell && (meta >> 8) != 0u);
            }
        }
        x_h[warp][lane] = warp == 0 ? hT[0] : hT[RPT - 1];
        const bool busy = __syncthreads_or(wet || (!LI && !(K.thr > R(0)))) != 0;
        if (!busy) {
            // dry through: what (B)-(F) would store
            if (fo && fi) {
                if (tid == 0) sh.skipw += unsigned(tile_cells);
            } else {
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const int r = rw + i;
                    if (own_lane && warp != 0 && r >= r0 && r < r_end) {
                        const size_t c = size_t(r) * nx + j;
                        sout[c] = V4{R(0), R(0), R(0), !LI && R(0) > X[i].w ? R(0) : X[i].w};
                        if (LI) li.hfx[c] = li.hfy[c] = R(0);
                    }
                }
                if (fl_out && tid == 0) *fl_out = 1;
            }
        } else {
            if (fo && tid == 0) *fl_out = 0;
            if (warp == 0) {
                // an apron row: nothing below needs its fluxes.  The warp makes the next step's rain,
                // which (F) of the others waits for, and CTA 0's keeps the books meanwhile.
                if (!next_made) step_next(a, sh, lane);
                next_made = true;
                bar_arrive<2, NT>();
                if (publish) step_publish<R, NT, INFL>(a, sh, phase);
                publish = false;
            } else {
            // (B, C) unlimited faces
            R hfx[RPT], hfy[RPT], qxu[RPT], qyu[RPT];
            Two<R> Sl[RPT];
            R hmax = R(0);
            bool edge = false;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const R hR = __shfl_down_sync(FULL, hT[i], 1);
                const R hU = i > 0 ? hT[i > 0 ? i - 1 : 0] : x_h[warp - 1][lane];
                faces_open<R>(hT[i], hR, hU, S[i].x, S[i].y, hfx[i], hfy[i], Sl[i], K);
                edge = edge || face_edge(fmax(fabs(S[i].x), fabs(S[i].y)));
                qxu[i] = qyu[i] = R(0);
            }
            if (__any_sync(FULL, edge)) {   // the grid's edges, cells outside it
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    if (face_edge(S[i].x)) hfx[i] = R(0);
                    if (face_edge(S[i].y)) hfy[i] = R(0);
                }
            }
#pragma unroll
            for (int i = 0; i < RPT; ++i) hmax = fmax(hmax, fmax(hfx[i], hfy[i]));
            if (__any_sync(FULL, hmax > R(0))) {
                Two<R> p73[RPT];   // H^(7/3)
#pragma unroll
                for (int i = 0; i < RPT; ++i) p73[i] = pow73_normal(hfx[i], hfy[i]);
                if (LI || sh.now.skip) {   // no clamp: depths of any size
#pragma unroll
                    for (int i = 0; i < RPT; ++i)
                        if ((hfx[i] > R(0) && below_normal(hfx[i])) || (hfy[i] > R(0) && below_normal(hfy[i])))
                            p73[i] = two(pow73_any(hfx[i]), pow73_any(hfy[i]));
                }
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const int r = rw + i;
                    R xa = R(0), xb = R(0), ya = R(0), yb = R(0);
                    if (SCH) {   // previous fluxes of the neighbouring faces (interior columns / rows only)
                        const size_t c = size_t(r) * nx + j;
                        if (hfx[i] > R(0) && j >= 1 && j + 1 < nx) {
                            xa = sin[c - 1].y;
                            xb = sin[c + 1].y;
                        }
                        if (hfy[i] > R(0) && r >= 1 && r + 1 < ny) {
                            ya = sin[c - nx].z;
                            yb = sin[c + nx].z;
                        }
                    }
                    qxu[i] = X[i].y;
                    qyu[i] = X[i].z;
                    faces_update<R, SCH>(hfx[i], hfy[i], p73[i], Sl[i], qxu[i], qyu[i], S[i].z, K, a.flag_critical, a.scheme,
                                         xa, xb, ya, yb);
                }
            }
            x_q[warp][lane] = qyu[0];
            bar_sync<1, NT - 32>();
            // (D) which cells' faces are limited: none in most tiles away from wet / dry fronts
            R out[RPT];
            bool lim = false;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int r = rw + i;
                const R qL = __shfl_up_sync(FULL, qxu[i], 1);
                const R qD = i + 1 < RPT ? qyu[i + 1 < RPT ? i + 1 : i]
                                         : (warp + 1 < NW ? x_q[warp + 1 < NW ? warp + 1 : 0][lane] : R(0));
                out[i] = donor_out(qxu[i], qL, qyu[i], qD);
                // (the rows outside the grid have no flux; the apron's outer columns are not looked at)
                lim = lim || (out[i] > hT[i] * K.dx_over_dt && lane > 0 && r >= r0 - 1);
            }
            R qxl[RPT], qyl[RPT], vu[RPT], vr[RPT];
            if (bar_or<1, NT - 32>(lim)) {
                R sc[RPT];
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const R avail = hT[i] * K.dx_over_dt;
                    sc[i] = out[i] > avail ? avail / out[i] : R(1);
                }
                x_s[warp][lane] = sc[RPT - 1];
                bar_sync<1, NT - 32>();
                // (E) limited faces
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const R scR = __shfl_down_sync(FULL, sc[i], 1);
                    const R scU = i > 0 ? sc[i > 0 ? i - 1 : 0] : (warp > 1 ? x_s[warp - 1][lane] : R(1));
                    qxl[i] = limit_by(qxu[i], sc[i], scR);
                    qyl[i] = limit_by(qyu[i], sc[i], scU);
                }
            } else {
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    qxl[i] = qxu[i];
                    qyl[i] = qyu[i];
                }
            }
#pragma unroll
            for (int i = 0; i < RPT; ++i) {   // of the upper and the right face, with the other sign
                vu[i] = vr[i] = R(0);
                if (!LI) face_velocities_neg(qyl[i], hfy[i], qxl[i], hfx[i], K, vu[i], vr[i]);
            }
            x_l[warp][lane] = qyl[0];
            x_v[warp][lane] = vu[0];
            bar_sync<2, NT>();
            // (F) continuity, outlets, maxima, CFL terms
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int r = rw + i;
                const R qxl_left = __shfl_up_sync(FULL, qxl[i], 1);
                if (!(own_lane && r >= r0 && r < r_end)) continue;
                const R qyd = i + 1 < RPT ? qyl[i + 1 < RPT ? i + 1 : i] : x_l[warp + 1 < NW ? warp + 1 : 0][lane];
                const R vb = i + 1 < RPT ? vu[i + 1 < RPT ? i + 1 : i] : x_v[warp + 1 < NW ? warp + 1 : 0][lane];
                const size_t c = size_t(r) * nx + j;
                const unsigned meta = meta_bits(S[i].w);
                const bool mine = r >= a.own_r0 && r < a.own_r1;
                // a control structure's transfers join the depth after the fluxes
                R h_in = LI ? X[i].x : hT[i];
                if (INFL && (meta & kInflowBit)) {
                    const int ss = a.inflow.cell_struct[(meta >> 8) & 0x7FFFFFu];
                    if (ss >= 0) h_in = h_in + a.strct.extra[ss];
                }
                R hn = continuity(h_in, qxl_left, qxl[i], qyl[i], qyd, K);
                R dts = fmax(hfx[i], hfy[i]);
                // LI's instantiation says nothing of gauge and stage cells: it takes any meta word
                const unsigned ord = INFL || LI ? outlet_ord(meta) : meta >> 8;
                if (ord) {
                    const int o = int(ord) - 1;
                    R ho;
                    const R qq = outlet_sink(hn, a.outlet_coef[o], a.outlet_type, K, ho);
                    dts = fmax(dts, ho);
                    a.hf3[o] = ho;
                    a.qo[o] = qq;
                    if (mine) out_acc_r.add(qq * K.dt);
                    if (!LI && mine && !(a.ga && (meta & 255u) != 255u) &&
                        hn + (MAP ? rain_at_cell(a, sh.rsn, r, j) : sh.rsn.depth) < R(-1e-11))
                        sh.negn = 1;
                }
                if (!LI && INFL && (meta & kInflowBit)) {   // stage hydrograph
                    const int sg = a.inflow.cell_stage[(meta >> 8) & 0x7FFFFFu];
                    if (sg >= 0) {
                        const R sv = a.inflow.stage_now[sg];
                        atomicAdd(&sh.stage, double(sv) - double(hn));
                        hn = sv;
                    }
                }
                if constexpr (LI) {
                    sout[c] = V4{hn, qxl[i], qyl[i], X[i].w};
                    li.hfx[c] = hfx[i];
                    li.hfy[c] = hfy[i];
                    continue;
                }
                const R negtol = -K.tol;
                nbad += (hn >= negtol || !mine) ? 0u : 1u;
                const R dm = X[i].w;
                if (dm < K.thr && hn >= K.thr) a.arrival[c] = R(sh.now.t_min * 60.0 + sh.now.dts);
                R vras = R(0);   // velocity raster: largest |face velocity|
                if (mine) {
                    if (INFL) vras = fmax(fmax(fabs(vr[i]), fabs(vu[i])), fabs(vb));
                    const R rc = vr[i] * first_col;
                    const R uc = R(0.5) * (vu[i] + vb);
                    const R s2 = rc * rc + uc * uc;
                    s2max = fmax(s2max, s2);
                    // the largest depth of a moving cell; its celerity is taken at the end (the product
                    // by g is monotone)
                    if (s2 >= a.stag_s2) {
                        if (a.adaptive != 1)
                            dts = fmax(fmax(fabs(vr[i]), fabs(vu[i])), fabs(vb)) + fmax(sqrt(K.g * fmax(dts, R(0))), R(1e-10));
                        cmaxv = fmax(cmaxv, dts);
                    }
                }
                V4 o4;
                o4.x = hn;
                o4.y = qxl[i];
                o4.z = qyl[i];
                o4.w = hn > dm ? hn : dm;
                sout[c] = o4;
                if (INFL && a.vmax) {   // running maxima of the velocity raster and of depth x velocity
                    const R vo = a.vmax[c];
                    a.vmax[c] = vras > vo ? vras : vo;
                    const R hd = fmax(hn, R(0));
                    R hz = hd * vras;
                    if (hd < R(0.01) || !isfinite(hz)) hz = R(0);
                    const R ho = a.hzmax[c];
                    a.hzmax[c] = isnan(hn) ? hn : (hz > ho ? hz : ho);
                }
            }
            }
        }
    }
    if (more) __syncthreads();   // the next tile's flags; warp 0 must not run ahead into its rows
    }
    if (publish) {   // no busy tile in CTA 0
        if (!next_made) step_next(a, sh, lane);
        step_publish<R, NT, INFL>(a, sh, phase);
    }
    if (a.adaptive == 1 && cmaxv >= R(0)) cmaxv = K.g * cmaxv;
    if (MAP) rain_acc += rain_acc_r.value();
    if (INF) inf_acc += inf_acc_r.value();
    if (out_acc_r.any()) out_acc += out_acc_r.value();
    if constexpr (LI) {
        if (__any_sync(FULL, out_acc != 0.0)) {
            out_acc = warp_sum(out_acc);
            if (lane == 0) atomicAdd(&a.sc->acc_out, out_acc);
        }
    } else {
        step_finish<R, NT, INF, MAP, INFL, true>(a, sh, rain_acc, inf_acc, out_acc, s2max, cmaxv, nbad, false, phase, sout,
                                                 gout);
    }
}

template <typename R, int RPT, int INF, bool MAP, bool INFL, int SCH>
__global__ void __launch_bounds__(TileShape<R, RPT>::NT, TileShape<R, RPT>::MINB)
k_tile_step(const __grid_constant__ FusedArgs<R> a, int phase) {
    const LiArgs<R> none{};
    tile_body<R, RPT, INF, MAP, INFL, SCH, false>(a, phase, none);
}
template <typename R, int RPT, bool INFL, int SCH>
__global__ void __launch_bounds__(TileShape<R, RPT>::NT, TileShape<R, RPT>::MINB)
k_tile_li(const __grid_constant__ FusedArgs<R> a, int cur, const __grid_constant__ LiArgs<R> li) {
    tile_body<R, RPT, 0, false, INFL, SCH, true>(a, cur, li);
}

// the tile step of a grid: infiltration model, rain from maps, boundary-cell variant, faces of
// schemes 2/3 (defined in hp2d_tile_f32.cu and hp2d_tile_f64.cu)
template <typename R> void launch_tile_step(const FusedArgs<R>& a, int inf, bool map, bool infl, bool sch, int phase, cudaStream_t st);
// the routing step alone, from buffer `cur` to the other one (infl: control structures)
template <typename R> void launch_tile_li(const FusedArgs<R>& a, const LiArgs<R>& li, bool infl, bool sch, int cur, cudaStream_t st);

#ifdef HP2D_TILE_INSTANTIATE
// kernels whose shared memory exceeds the default opt in, once per device; one TileOptIn per group of
// kernels
struct TileOptIn {
    std::mutex mu;
    unsigned long long done[4] = {};
};
template <typename K> static void tile_opt_in(K kernel, size_t smem, int v, TileOptIn* o) {
    if (smem + 20 * 1024 <= 48 * 1024) return;   // with the static part
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(o->mu);
    if (dev > 63 || !((o->done[v] >> dev) & 1ull)) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (dev <= 63) o->done[v] |= 1ull << dev;
    }
}
template <typename R, int RPT, int INF, bool MAP>
static void launch_tile_v(const FusedArgs<R>& a, bool infl, bool sch, int phase, cudaStream_t st) {
    constexpr int NT = TileShape<R, RPT>::NT;
    constexpr size_t smem = 2 * sizeof(typename Vec<R>::V4) * NT * RPT;
    const unsigned grid = a.n_ctas < a.tile_grid ? a.n_ctas : a.tile_grid;
    auto* const kernel = sch ? k_tile_step<R, RPT, INF, MAP, true, 1>
                         : infl ? k_tile_step<R, RPT, INF, MAP, true, 0> : k_tile_step<R, RPT, INF, MAP, false, 0>;
    static TileOptIn opt;
    tile_opt_in(kernel, smem, sch ? 2 : infl ? 1 : 0, &opt);
    launch_step(kernel, grid, NT, smem, st, a, phase);
}
template <typename R, int RPT>
static void launch_tile_r(const FusedArgs<R>& a, int inf, bool map, bool infl, bool sch, int phase, cudaStream_t st) {
    if (inf == 1) {
        if (map) launch_tile_v<R, RPT, 1, true>(a, infl, sch, phase, st);
        else launch_tile_v<R, RPT, 1, false>(a, infl, sch, phase, st);
    } else if (inf == 2) {
        if (map) launch_tile_v<R, RPT, 2, true>(a, infl, sch, phase, st);
        else launch_tile_v<R, RPT, 2, false>(a, infl, sch, phase, st);
    } else {
        if (map) launch_tile_v<R, RPT, 0, true>(a, infl, sch, phase, st);
        else launch_tile_v<R, RPT, 0, false>(a, infl, sch, phase, st);
    }
}
template <typename R, int RPT>
static void launch_li_r(const FusedArgs<R>& a, const LiArgs<R>& li, bool infl, bool sch, int cur, cudaStream_t st) {
    constexpr int NT = TileShape<R, RPT>::NT;
    constexpr size_t smem = 2 * sizeof(typename Vec<R>::V4) * NT * RPT;
    const unsigned grid = a.n_ctas < a.tile_grid ? a.n_ctas : a.tile_grid;
    auto* const kernel = sch ? (infl ? k_tile_li<R, RPT, true, 1> : k_tile_li<R, RPT, false, 1>)
                             : (infl ? k_tile_li<R, RPT, true, 0> : k_tile_li<R, RPT, false, 0>);
    static TileOptIn opt;
    tile_opt_in(kernel, smem, (sch ? 2 : 0) + (infl ? 1 : 0), &opt);
    kernel<<<grid, NT, smem, st>>>(a, cur, li);
}
template <typename R> void launch_tile_li(const FusedArgs<R>& a, const LiArgs<R>& li, bool infl, bool sch, int cur, cudaStream_t st) {
    if (a.tile_rpt == 2) launch_li_r<R, 2>(a, li, infl, sch, cur, st);
    else launch_li_r<R, 1>(a, li, infl, sch, cur, st);
}
template <typename R> void launch_tile_step(const FusedArgs<R>& a, int inf, bool map, bool infl, bool sch, int phase, cudaStream_t st) {
    if (a.tile_rpt == 2) launch_tile_r<R, 2>(a, inf, map, infl, sch, phase, st);
    else launch_tile_r<R, 1>(a, inf, map, infl, sch, phase, st);
}
#endif

}  // namespace hp2d
