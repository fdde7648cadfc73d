/*
 * One RKHEVI step on device mirrors (src/time_stepping/manage_rkhevi.c:20-100),
 * templated on the horizontal precision R.  Included by step_f64.cu (R =
 * double, compiled without FMA contraction, every operation in the
 * reference's order) and step_mixed.cu (R = float).
 */
#pragma once

#include "context.h"
#include "diff.h"
#include "kernels.cuh"
#include "solvers.cuh"
#include "solvers_df.cuh"

namespace game {

inline unsigned nblocks(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

template <typename R>
HGrid<R> &hgrid(Context *c);
template <>
inline HGrid<double> &hgrid<double>(Context *c) { return c->hg64; }
template <>
inline HGrid<float> &hgrid<float>(Context *c) { return c->hg32; }
template <typename R>
Work<R> &work(Context *c);
template <>
inline Work<double> &work<double>(Context *c) { return c->w64; }
template <>
inline Work<float> &work<float>(Context *c) { return c->w32; }

/* capacities of the local-memory sweeps for other layer counts */
constexpr int SWEEP_SMALL = 64, SWEEP_LARGE = 256;
/* the mixed path solves a batch of fewer systems than this with the warp
 * cyclic reduction: one thread per system leaves most of the 152 SMs idle
 * there, while above it the per-thread sweeps, with log2(n) times less FP64
 * work, are faster (cloud-free, mixed: 3210 tracer systems of 256 layers 0.55
 * ms a step against 0.79 by the sweeps, 12810 of 128 layers 0.72 against 0.39;
 * 2562 wave systems of 128 layers 0.19 against 0.40, 10242 0.60 against 0.50).
 * The count is of all systems, those of absent constituents too.  The FP64 path keeps the reference's elimination order at any
 * depth. */
constexpr long long PCR_SYSTEMS_BELOW = 6144;

enum { COLUMN_REGISTERS, COLUMN_LOCAL, COLUMN_PCR };
/* the solver for a batch of n_systems columns (game_gpu_set_column_solver:
 * 0 chosen by layer count, batch size and precision, 1 per-thread Thomas
 * sweeps, 2 warp cyclic reduction) */
inline int column_mode(const Context *c, bool exact, long long n_systems)
{
    if (c->column_solver == 2) return COLUMN_PCR;
    if (c->nl == NL_FIXED) return COLUMN_REGISTERS;
    if (c->column_solver == 0 && !exact && n_systems < PCR_SYSTEMS_BELOW) return COLUMN_PCR;
    return COLUMN_LOCAL;
}

inline WavesWork waves_work(Context *c)
{
    WavesWork w;
    const long long ns = c->ns, ni = (long long)(c->nl - 1) * c->nc;
    double *a = c->wv_layer, *b = c->wv_rows;
    w.rho_expl = a; w.rt_expl = a + ns; w.alpha = a + 2 * ns; w.beta = a + 3 * ns; w.gam = a + 4 * ns;
    w.tp_expl = a + 5 * ns; w.ep_expl = a + 6 * ns; w.thl = a + 7 * ns;
    w.c = b; w.d = b + ni; w.e = b + 2 * ni; w.r = b + 3 * ni; w.th_int = b + 4 * ni; w.rho_io = b + 5 * ni;
    w.r_rho_io = b + 6 * ni;
    w.inv_vol = c->inv_vol;
    w.inv_area_v = c->inv_area_v;
    w.damp_den = c->damp_den;
    w.damp_inv = c->damp_inv;
    w.geo = c->wv_geo;
    return w;
}

/* read view of state_new in precision R and the FP32 shadow (mixed path) */
template <typename R>
struct Views {
    SView<R> sv;
    Shadow sh;
};
template <typename R>
Views<R> views(Context *c, StateMirror *sn);
template <>
inline Views<double> views<double>(Context *c, StateMirror *sn)
{
    Views<double> v{};
    v.sv = {sn->ds.rho, sn->ds.rhotheta_v, sn->ds.theta_v_pert, sn->ds.exner_pert, sn->ds.w, sn->ds.u};
    v.sh = Shadow{};
    return v;
}
template <>
inline Views<float> views<float>(Context *c, StateMirror *sn)
{
    Views<float> v{};
    const long long ns = c->ns;
    float *b = c->shadow;
    v.sh.rho = b;
    v.sh.rhotheta_v = b + (long long)c->n_const * ns;
    v.sh.theta_v_pert = v.sh.rhotheta_v + ns;
    v.sh.exner_pert = v.sh.theta_v_pert + ns;
    v.sh.w = v.sh.exner_pert + ns;
    v.sh.u = v.sh.w + (long long)(c->nl + 1) * c->nc;
    v.sh.present = c->present;
    v.sv = {v.sh.rho, v.sh.rhotheta_v, v.sh.theta_v_pert, v.sh.exner_pert, v.sh.w, v.sh.u};
    return v;
}

/* the FP64 path's scalar tendencies; theta: rho theta_v / rho_gas */
inline void launch_scalar_tend64(Context *c, const StepParams &p, const SView<double> &sv, const double *rho_prev,
                                 double *st_rho, double *st_rt, const double *theta, const double *cp_ice,
                                 const double *cp_water, const double *pt_rates, const double *pt_heat,
                                 const double *sed_heat, int rk, const IrrTerms &irr)
{
    const HGrid<double> &g = c->hg64;
    const long long nu = (long long)c->nl * c->ne, nw = (long long)(c->nl + 1) * c->nc;
    double *fm = c->edge_flux64, *ft = fm + nu, *cr = c->level_corr64;
    cudaStream_t s = c->stream;
    k_edge_flux<<<layer_grid(c->nl, c->ne, 256), 256, 0, s>>>(g, sv.rho + (long long)c->n_cond * c->ns, theta, sv.u, fm,
                                                             ft);
    c->kernel_launches += 2;
    if (c->n_tilt) {
        const dim3 nb = layer_grid(c->n_oro, c->nc, 256);
        if (p.n_const > 1)
            k_level_corr<true><<<nb, 256, 0, s>>>(g, fm, ft, sv.u, cr, cr + nw, cr + 2 * nw);
        else
            k_level_corr<false><<<nb, 256, 0, s>>>(g, fm, ft, sv.u, cr, cr + nw, cr + 2 * nw);
        c->kernel_launches++;
    }
    const dim3 nb = layer_grid(c->nl, c->nc, 128);
    if (p.irr)
        k_scalar_tend64<true><<<nb, 128, 0, s>>>(g, p, sv, rho_prev, st_rho, st_rt, fm, ft, cr, theta, cp_ice, cp_water,
                                                 pt_rates, pt_heat, sed_heat, rk, irr);
    else
        k_scalar_tend64<false><<<nb, 128, 0, s>>>(g, p, sv, rho_prev, st_rho, st_rt, fm, ft, cr, theta, cp_ice, cp_water,
                                                  pt_rates, pt_heat, sed_heat, rk, irr);
}

template <typename R>
PgCells<R> pg_cells(Context *c);
template <>
inline PgCells<float> pg_cells<float>(Context *c)
{
    return {c->pg_cell};
}
template <>
inline PgCells<double> pg_cells<double>(Context *c)
{
    return {c->pg_cell64, c->grad_pi_v, c->w64.v2g_v, c->level_q64, c->level_q64 + (long long)(c->nl + 1) * c->nc,
            c->gas_share64};
}

template <typename R, bool ADV, bool PG>
static void launch_momentum_v(Context *c, const StepParams &p, const Views<R> &v, StateMirror *st, double new_w,
                              double old_w, cudaStream_t stream)
{
    HGrid<R> &g = hgrid<R>(c);
    Work<R> &w = work<R>(c);
    ProfScope ps(c, "k_momentum_v");
    const double *fric_w = p.irr ? c->dbuf->fric : nullptr;
    k_momentum_v<R, ADV, PG><<<layer_grid(c->nl + 1, c->nc, 256), 256, 0, stream>>>(
        g, p, v.sv, st->ds.w, w.P_v, w.pvt_v, w.v2g_v, w.flux_h, w.zh, w.v2, new_w, old_w, fric_w,
        pg_cells<R>(c));
    c->kernel_launches++;
}

template <typename R, bool ADV, bool PG>
static void launch_momentum_h(Context *c, const StepParams &p, const Views<R> &v, StateMirror *so, StateMirror *sn,
                              StateMirror *st, double new_w, double old_w)
{
    HGrid<R> &g = hgrid<R>(c);
    Work<R> &w = work<R>(c);
    ProfScope ps(c, "k_momentum_h");
    const double *fric_u = p.irr ? c->dbuf->fric + (long long)(c->nl + 1) * c->nc : nullptr;
    k_momentum_h<R, ADV, PG><<<layer_grid(c->nl, c->ne, 256), 256, 0, c->stream>>>(
        g, p, v.sv, sn->ds.u, v.sh.u, so->ds.u, st->ds.u, w.P_h, w.pg_old_h, w.pvt_h, w.v2g_h, w.flux_h, w.flux_v,
        w.zh, w.zv, w.v2, new_w, old_w, fric_u, pg_cells<R>(c));
    c->kernel_launches++;
}

template <typename R, bool ADV, bool PG>
static void launch_momentum(Context *c, const StepParams &p, const Views<R> &v, StateMirror *so, StateMirror *sn,
                            StateMirror *st, double new_w, double old_w, cudaStream_t v_stream)
{
    launch_momentum_v<R, ADV, PG>(c, p, v, st, new_w, old_w, v_stream);
    launch_momentum_h<R, ADV, PG>(c, p, v, so, sn, st, new_w, old_w);
}

/* implicit vertical sound waves (column_solvers.c:19-383) */
template <bool EXACT>
void launch_waves(Context *c, const StepParams &p, StateMirror *so, StateMirror *sn, StateMirror *st, int rk,
                  const Shadow &sh, const double *theta = nullptr)
{
    const long long ns = c->ns;
    WavesWork ww = waves_work(c);
    if constexpr (!EXACT) {
        if (p.dfloat && column_mode(c, EXACT, c->nc) == COLUMN_REGISTERS) {
            {
                ProfScope ps(c, "k_waves_layer");
                k_waves_layer_df<<<nblocks(ns, 256), 256, 0, c->stream>>>(c->vg, p, so->ds, sn->ds, st->ds, ww,
                                                                          c->dfg, rk);
            }
            {
                ProfScope ps(c, "k_waves_rows");
                k_waves_rows_df<<<layer_grid(c->nl - 1, c->nc, 256), 256, 0, c->stream>>>(
                    c->vg, p, so->ds, st->ds, ww, c->dfg);
            }
            {
                ProfScope ps(c, "k_waves_thomas");
                /* two lanes per column (twisted elimination) */
                k_waves_thomas_df<NL_FIXED><<<nblocks(2 * (long long)c->nc, WAVES_BLOCK), WAVES_BLOCK, 0,
                                              c->stream>>>(c->nc, ww, c->dfg);
            }
            {
                ProfScope ps(c, "k_waves_apply");
                k_waves_apply_df<<<nblocks(ns, 256), 256, 0, c->stream>>>(c->vg, p, so->ds, sn->ds, ww, c->dfg, sh,
                                                                          rk == 0 ? c->theta32 : nullptr);
            }
            c->kernel_launches += 4;
            return;
        }
    }
    {
        ProfScope ps(c, "k_waves_layer");
        k_waves_layer<EXACT><<<nblocks(ns, 256), 256, 0, c->stream>>>(c->vg, p, so->ds, sn->ds, st->ds, ww, rk, theta);
    }
    {
        ProfScope ps(c, "k_waves_rows");
        const dim3 nb = layer_grid(c->nl - 1, c->nc, 256);
        if (EXACT)
            k_waves_rows<<<nb, 256, 0, c->stream>>>(c->vg, p, so->ds, st->ds, ww);
        else
            k_waves_rows_mixed<<<nb, 256, 0, c->stream>>>(c->vg, p, so->ds, st->ds, ww);
    }
    {
        ProfScope ps(c, "k_waves_thomas");
        const int mode = column_mode(c, EXACT, c->nc);
        if (mode == COLUMN_REGISTERS)
            k_waves_thomas<NL_FIXED, EXACT><<<nblocks(c->nc, 64), 64, 0, c->stream>>>(c->nc, ww);
        else if (mode == COLUMN_LOCAL && c->nl - 1 <= SWEEP_SMALL)
            k_waves_thomas_any<SWEEP_SMALL, EXACT><<<nblocks(c->nc, 64), 64, 0, c->stream>>>(c->nc, c->nl, ww);
        else if (mode == COLUMN_LOCAL)
            k_waves_thomas_any<SWEEP_LARGE, EXACT><<<nblocks(c->nc, 64), 64, 0, c->stream>>>(c->nc, c->nl, ww);
        else
            k_waves_pcr<EXACT><<<nblocks(c->nc, PCR_WARPS), 32 * PCR_WARPS,
                                 (size_t)PCR_WARPS * 6 * (c->nl - 1) * sizeof(double), c->stream>>>(c->nc, c->nl, ww);
    }
    {
        ProfScope ps(c, "k_waves_apply");
        k_waves_apply<EXACT><<<nblocks(ns, 256), 256, 0, c->stream>>>(c->vg, p, so->ds, sn->ds, ww, sh);
    }
    c->kernel_launches += 4;
}

/* implicit vertical advection and sedimentation of the non-main constituents
 * (column_solvers.c:385-639); temperature and its c_p tables as of the start
 * of the step, sedimentation heat written at rk 0 */
template <bool EXACT>
void launch_tracers(Context *c, const StepParams &p, StateMirror *so, StateMirror *sn, StateMirror *st, int rk,
                    const Shadow &sh, const double *temperature, const double *cp_ice, const double *cp_water,
                    double *sed_heat, cudaStream_t strm = nullptr)
{
    if (c->n_const <= 1) return;
    if (!strm) strm = c->stream;
    const long long ns = c->ns;
    TracerWork tw{cp_ice, cp_water, c->inv_vol};
    const long long nsys = (long long)(c->n_const - 1) * c->nc;
    const int mode = column_mode(c, EXACT, nsys);
    if (rk == 0) {
        ProfScope ps(c, "k_tracers_sedheat");
        if (!EXACT && p.dfloat)
            k_tracers_sedheat_df<<<nblocks(ns, 128), 128, 0, strm>>>(c->vg, p, so->ds, sn->ds, temperature, tw,
                                                                     c->dfg, sed_heat);
        else if (EXACT)
            k_tracers_sedheat64<<<layer_grid(c->nl, c->nc, 128), 128, 0, strm>>>(c->vg, p, so->ds, sn->ds, temperature,
                                                                                 tw, sed_heat);
        else
            k_tracers_sedheat<<<nblocks(c->nc, 128), 128, 0, strm>>>(c->vg, p, so->ds, sn->ds, temperature, tw,
                                                                     sed_heat);
        c->kernel_launches++;
    }
    ProfScope ps(c, "k_tracers_solve");
    if constexpr (!EXACT) {
        if (p.dfloat && mode == COLUMN_REGISTERS) {
            k_tracers_solve_df<NL_FIXED><<<nblocks(nsys, TRACER_BLOCK), TRACER_BLOCK, 0, strm>>>(
                c->vg, p, so->ds, sn->ds, st->ds, c->dfg, sh.rho, sh.present);
            c->kernel_launches++;
            return;
        }
    }
    if (mode == COLUMN_REGISTERS)
        k_tracers_solve<NL_FIXED, NL_FIXED, EXACT><<<nblocks(nsys, 64), 64, 0, strm>>>(c->vg, p, so->ds, sn->ds,
                                                                                        st->ds, tw, sh.rho, sh.present);
    /* sweeps in local memory: blocks of one warp, since a small grid's systems
     * (80 layers, RES_ID 4: 80 warps of vapour) then lie on as many SMs (125 ->
     * 121 us; the same at RES_ID 6) */
    else if (mode == COLUMN_LOCAL && c->nl <= SWEEP_SMALL)
        k_tracers_solve<0, SWEEP_SMALL, EXACT><<<nblocks(nsys, 32), 32, 0, strm>>>(c->vg, p, so->ds, sn->ds, st->ds,
                                                                                    tw, sh.rho, sh.present);
    else if (mode == COLUMN_LOCAL)
        k_tracers_solve<0, SWEEP_LARGE, EXACT><<<nblocks(nsys, 32), 32, 0, strm>>>(c->vg, p, so->ds, sn->ds, st->ds,
                                                                                    tw, sh.rho, sh.present);
    else
        k_tracers_pcr<EXACT><<<nblocks(nsys, PCR_WARPS), 32 * PCR_WARPS,
                               (size_t)PCR_WARPS * 6 * c->nl * sizeof(double), strm>>>(c->vg, p, so->ds, sn->ds,
                                                                                       st->ds, tw, sh.rho, sh.present);
    c->kernel_launches++;
}

/* the second stream's work starts after what c->stream holds so far; c->stream
 * goes on after what the second stream holds */
inline void fork_second(Context *c)
{
    cudaEventRecord(c->ev_fork, c->stream);
    cudaStreamWaitEvent(c->stream2, c->ev_fork, 0);
}
inline void join_second(Context *c)
{
    cudaEventRecord(c->ev_join, c->stream2);
    cudaStreamWaitEvent(c->stream, c->ev_join, 0);
}

/* the kernel sequence of one step on c->stream (and c->stream2 for the tracer branch) */
template <typename R>
void launch_step(Context *c, const StepParams &p, StateMirror *so, StateMirror *sn, StateMirror *st)
{
    constexpr bool EXACT = sizeof(R) == sizeof(double);
    HGrid<R> &g = hgrid<R>(c);
    Work<R> &w = work<R>(c);
    const int bs = 256;
    const long long ns = c->ns;
    const Views<R> v = views<R>(c, sn);
    R *theta = EXACT ? (R *)c->theta : (R *)c->theta32;
    const R *cpi = EXACT ? (const R *)c->cp_ice : (const R *)c->cp32_ice;
    const R *cpw = EXACT ? (const R *)c->cp_water : (const R *)c->cp32_water;
    const bool parallel = !c->profiling;
    /* Kernels that share no output run side by side on the second stream (a
     * parallel branch of the captured graph): the thermodynamics of state_old
     * (FP64-bound; first read by the diffusion branch and the scalar
     * tendencies) beside the conversion to the shadow and the pressure-gradient
     * factors, the kinetic energy beside the vorticities, and the vertical
     * beside the horizontal momentum.  On a small grid each saves a launch's
     * latency, on a large one the idle end of a kernel.  Serial while
     * profiling.  RES_ID 3 dry, mixed, 2 steps: 337 -> 314 us; RES_ID 6 moist,
     * mixed, 8 steps: 9.82 -> 9.73 ms, FP64, 2 steps: 8.52 -> 8.44 ms. */
    if (parallel) fork_second(c);
    {
        cudaStream_t side = parallel ? c->stream2 : c->stream;
        ProfScope ps(c, "k_cell_prepare");
        if (EXACT)
            k_cell_prepare<<<nblocks(ns, bs), bs, 0, side>>>(c->vg, p, so->ds, c->temperature, c->pt_rates, c->pt_heat,
                                                             c->cp_ice, c->cp_water);
        else
            k_cell_prepare_f32<<<nblocks(ns, bs), bs, 0, side>>>(c->vg, p, so->ds, c->temperature, c->pt_rates,
                                                                 c->pt_heat, c->cp_ice, c->cp_water, c->cp32_ice,
                                                                 c->cp32_water);
        c->kernel_launches++;
    }
    if (!EXACT) {
        ProfScope ps(c, "k_make_shadow");
        const long long n_rho = (long long)c->n_const * ns, nw = (long long)(c->nl + 1) * c->nc,
                        nu = (long long)c->nl * c->ne;
        const long long pairs = (std::max(std::max(n_rho, nw), nu) + 1) / 2;
        if (c->n_const > 1)
            cudaMemsetAsync(c->present.by_layer, 0, ((size_t)c->nl + 8 * c->n_const) * sizeof(int), c->stream);
        k_make_shadow<<<nblocks(pairs, bs), bs, 0, c->stream>>>(n_rho, ns, nw, nu, sn->ds, v.sh);
        c->kernel_launches++;
    }
    {
        /* the first substage's pressure-gradient factors per cell (the
         * diffusion branch, which runs before it, changes none of its inputs) */
        ProfScope ps(c, "k_pg_cells");
        if constexpr (EXACT)
            k_pg_cells64<<<layer_grid(c->nl, c->nc, bs), bs, 0, c->stream>>>(g, p, v.sv, c->pg_cell64, c->grad_pi_v,
                                                                                 c->theta);
        else
            k_pg_cells<<<layer_grid(c->nl, c->nc, bs), bs, 0, c->stream>>>(c->hg32, p, v.sv, c->pg_cell, c->theta32,
                                                                             c->present);
        c->kernel_launches++;
    }
    const R *rho_gas = v.sv.rho + (long long)c->n_cond * ns;
    /* Substage 0's tracer solve (FP64-bound) and substage 1's advection and
     * horizontal momentum (FP32, memory-bound) read and write disjoint
     * fields: the tracer solve runs on a second stream (a parallel branch of
     * the captured graph) and joins before substage 1's vertical momentum,
     * whose condensate term reads the tracer densities.  Serial while
     * profiling. */
    const bool fork = c->n_const > 1 && parallel;
    bool join_pending = false;
    for (int rk = 0; rk < 2; ++rk) {
        const bool adv = rk == 1 || p.first_step;
        const double new_w = rk == 1 ? 0.5 : 1.0, old_w = 1.0 - new_w;
        /* the second stream is free beside this substage's momentum */
        const bool beside = parallel && !join_pending;
        cudaStream_t side = beside ? c->stream2 : c->stream;
        if (adv) {
            if (beside) fork_second(c);
            {
                ProfScope ps(c, "k_tri_vort");
                k_tri_vort<R><<<layer_grid(c->nl, c->nt, bs), bs, 0, c->stream>>>(g, v.sv.u, w.tri_vort);
            }
            {
                ProfScope ps(c, "k_edge_vort");
                k_edge_vort<R><<<layer_grid(c->nl + 1, c->ne, bs), bs, 0, c->stream>>>(
                    g, v.sv.u, v.sv.w, rho_gas, w.tri_vort, w.zh, w.zv, w.flux_h);
            }
            {
                ProfScope ps(c, "k_cell_kinetic");
                k_cell_kinetic<R><<<layer_grid(c->nl, c->nc, bs), bs, 0, side>>>(g, v.sv.u, v.sv.w, rho_gas, w.v2, w.flux_v);
            }
            if constexpr (EXACT) {
                ProfScope ps(c, "k_level_terms");
                k_level_terms<<<layer_grid(c->nl + 1, c->nc, bs), bs, 0, side>>>(
                    g, w.v2, w.flux_v, w.v2g_v, c->level_q64, c->level_q64 + (long long)(c->nl + 1) * c->nc);
                c->kernel_launches++;
            }
            if (beside) join_second(c);
            c->kernel_launches += 3;
        }
        /* diffusion branch: momentum part on state_new before the wind update */
        if (rk == 0 && p.diff) {
            if (parallel) join_second(c); /* reads the temperature */
            launch_diffusion_momentum(c, p, v.sv);
        }
        if (beside) fork_second(c);
        if (rk == 0) {
            if (adv)
                launch_momentum<R, true, true>(c, p, v, so, sn, st, new_w, old_w, side);
            else
                launch_momentum<R, false, true>(c, p, v, so, sn, st, new_w, old_w, side);
        } else {
            launch_momentum_h<R, true, false>(c, p, v, so, sn, st, new_w, old_w);
            if (join_pending) join_second(c);
            if constexpr (EXACT) {
                ProfScope ps(c, "k_theta");
                k_theta_share<<<nblocks(ns, bs), bs, 0, side>>>(ns, c->n_cond, c->n_const, v.sv, c->theta, c->gas_share64);
                c->kernel_launches++;
            }
            launch_momentum_v<R, true, false>(c, p, v, st, new_w, old_w, side);
        }
        if (beside) join_second(c);
        join_pending = false;
        /* diffusion branch: temperature and mass diffusion */
        if (rk == 0 && (p.diff & DIFF_RAD_HS)) launch_held_suarez_radiation(c, so->ds);
        if (rk == 0 && p.diff) launch_diffusion_scalar(c, p, v.sv);
        /* theta_v: at rk 0 from k_pg_cells, at rk 1 from k_waves_apply_df or,
         * without the double-float solve, here */
        if constexpr (!EXACT)
            if (rk == 1 && !(p.dfloat && column_mode(c, EXACT, c->nc) == COLUMN_REGISTERS)) {
                ProfScope ps(c, "k_theta");
                k_theta<R><<<nblocks(ns, bs), bs, 0, c->stream>>>(c->nl, c->nc, c->n_cond, v.sv, theta);
                c->kernel_launches++;
            }
        {
            ProfScope ps(c, "k_scalar_tend");
            IrrTerms irr{};
            if (p.irr) irr = {c->dbuf->hdiss, c->dbuf->tdh, c->dbuf->rad, c->dbuf->mdt};
            if constexpr (EXACT) {
                launch_scalar_tend64(c, p, v.sv, st->ds.rho, st->ds.rho, st->ds.rhotheta_v, theta, cpi, cpw, c->pt_rates,
                                     c->pt_heat, c->sed_heat, rk, irr);
            } else {
                const int tilt_blocks = (int)nblocks(c->n_tilt, 128);
                auto tend = [&](auto kernel) {
                    kernel<<<dim3(tilt_blocks + nblocks(c->nc, 128), (unsigned)c->nl), 128, 0, c->stream>>>(
                        g, p, v.sv, st->ds, theta, cpi, cpw, c->pt_rates, c->pt_heat, c->sed_heat, c->inv_vol, c->present,
                        rk, irr, c->tilt_cells, c->n_tilt, tilt_blocks);
                };
                if (c->n_tilt)
                    p.irr ? tend(k_scalar_tend32<true, true>) : tend(k_scalar_tend32<false, true>);
                else
                    p.irr ? tend(k_scalar_tend32<true, false>) : tend(k_scalar_tend32<false, false>);
            }
        }
        c->kernel_launches += EXACT ? 0 : 1; /* launch_scalar_tend64 counts its own */
        /* the tendency is final from here on: a host-in/host-out call copies
         * it out while the solvers run */
        if (rk == 1) {
            /* inside a graph capture: an external event node, which streams
             * outside the graph can wait on */
            cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
            cudaStreamIsCapturing(c->stream, &cs);
            if (cs == cudaStreamCaptureStatusActive)
                cudaEventRecordWithFlags(c->ev_tend, c->stream, cudaEventRecordExternal);
            else
                cudaEventRecord(c->ev_tend, c->stream);
        }
        launch_waves<EXACT>(c, p, so, sn, st, rk, v.sh, EXACT ? c->theta : nullptr);
        if (rk == 0 && fork) {
            fork_second(c);
            launch_tracers<EXACT>(c, p, so, sn, st, rk, v.sh, c->temperature, c->cp_ice, c->cp_water, c->sed_heat,
                                  c->stream2);
            join_pending = true;
        } else {
            launch_tracers<EXACT>(c, p, so, sn, st, rk, v.sh, c->temperature, c->cp_ice, c->cp_water, c->sed_heat);
        }
    }
}

}  // namespace game
