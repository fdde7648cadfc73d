/*
 * Vertical implicit solvers of the RKHEVI step (src/time_stepping/column_solvers.c),
 * FP64, restructured for the GPU:
 *
 * sound waves (column_solvers.c:19-383) in four kernels
 *   k_waves_layer   per (layer, column): explicit predictors and the
 *                   partial derivatives alpha, beta, gamma (:102-139)
 *   k_waves_rows    per (interface, column): the tridiagonal rows c, d, e, r
 *                   (:142-189) and the Klemp damping denominator (:285-298);
 *                   k_waves_rows_mixed is its mixed-path rearrangement
 *   k_waves_thomas  per column: the elimination, with the sweep held in
 *                   registers (layer count a compile-time constant)
 *   k_waves_apply   per (layer, column): back-substitution into rho, rho*theta_v,
 *                   w, theta_v', Pi' (:305-370)
 * tracers (column_solvers.c:385-639)
 *   k_tracers_solve per (constituent, column): rows built on the fly, Thomas
 *                   sweep in registers, clipping
 *   k_tracers_sedheat64 per (layer, column), k_tracers_sedheat (mixed path
 *                   with FP64 eliminations) per column: sedimentation enthalpy
 *                   flux divergence, accumulated over the condensates in the
 *                   reference's order
 *
 * EXACT = true keeps the reference's operation order (FP64 parity path), its
 * quotients by reciprocals at hand where one serves several (div_rcp,
 * div_sweep: IEEE's results); EXACT = false (mixed path) multiplies by precomputed
 * reciprocals of the grid metrics and of repeated denominators, which moves
 * results by a few ulps but removes most FP64 divisions.
 */
#pragma once

#include "kernels.cuh"

namespace game {
namespace {

struct WavesWork {
    /* per layer [L][Nc] */
    double *rho_expl, *rt_expl, *alpha, *beta, *gam, *tp_expl, *ep_expl, *thl;
    /* per inner interface [L-1][Nc] */
    double *c, *d, *e, *r, *th_int, *rho_io, *r_rho_io;
    /* mixed path: reciprocal grid metrics */
    const double *inv_vol;    /* [L][Nc] */
    const double *inv_area_v; /* [L+1][Nc] */
    /* 1 + dt * Klemp damping coefficient of the inner interfaces [L-1][Nc]
     * for the current dt, and its reciprocal */
    const double *damp_den, *damp_inv;
    /* mixed path: grid terms of the rows of inner interface j [6][L-1][Nc]:
     * dz = z(j) - z(j+1), H = (Pi_bg(j) - Pi_bg(j+1)) / 2, G1 = 2 / A_v,
     * G2 = (1/V(j+1) - 1/V(j)) / 2, Cz = dz / V(j), Ez = dz / V(j+1)
     * (layers j, j+1 above and below the interface) */
    const double *geo;
};

/* 1 + dt times the Klemp (2008) damping coefficient at inner interface j + 1 of every column
 * (column_solvers.c:285-298).  It depends on the grid and the two damping
 * parameters only, so it is tabulated once per parameter pair instead of
 * once per substage. */
__global__ void k_damping_table(VGrid vg, double start_height, double coeff_max, double dt, double *den, double *inv_den,
                                float2 *inv_den_df)
{
    const long long n = (long long)(vg.nl - 1) * vg.nc, q = gtid();
    if (q >= n) return;
    const long long wi = q + vg.nc;
    const double zad = vg.z_v[wi] - start_height;
    double r = 0.0;
    if (zad >= 0.0) {
        const double s = sin(0.5 * M_PI * zad / (vg.z_v[0] - start_height));
        r = coeff_max * (s * s);
    }
    den[q] = 1.0 + dt * r;
    const double inv = 1.0 / den[q];
    inv_den[q] = inv;
    const float hi = (float)inv;
    inv_den_df[q] = make_float2(hi, (float)(inv - (double)hi));
}

/* alpha, beta, gamma of a cell over its volume (column_solvers.c:102-139),
 * FP64 path: every quotient correctly rounded as the reference's, the
 * divisions by rho, rho^2 and the volume through one reciprocal each
 * (div_rcp) */
struct WaveCoeffs {
    double alpha, beta, gam;
};
__device__ __forceinline__ WaveCoeffs wave_coeffs(int rk, double ro, double rto, double ebg, double epo, double rn,
                                                  double rtn, double irn, double epn, double vol, double rv)
{
    const double pdw = 0.5, iro = 1.0 / ro;
    const double ao = div_rcp(-rto, ro * ro, iro * iro);
    auto gamma = [&](double rt, double e) { return R_D / (C_D_V * rt) * (ebg + e); };
    const double go = gamma(rto, epo);
    if (rk == 0) return {div_rcp(ao, vol, rv), div_rcp(iro, vol, rv), div_rcp(go, vol, rv)};
    const double an = div_rcp(-rtn, rn * rn, irn * irn);
    const double gn = gamma(rtn, epn);
    return {div_rcp((1.0 - pdw) * ao + pdw * an, vol, rv), div_rcp((1.0 - pdw) * iro + pdw * irn, vol, rv),
            div_rcp((1.0 - pdw) * go + pdw * gn, vol, rv)};
}

template <bool EXACT>
__global__ void k_waves_layer(VGrid vg, StepParams p, DState so, DState sn, DState st, WavesWork ww, int rk,
                              const double *theta)
{
    const long long ns = (long long)vg.nl * vg.nc, b = gtid();
    if (b >= ns) return;
    const long long gp = p.n_cond * ns;
    const double dt = p.dt;
    const double vol = vg.volume[b];
    const double ro = so.rho[gp + b], rto = so.rhotheta_v[b];
    if (EXACT) {
        const double rv = vg.r_volume[b];
        const double rn = sn.rho[gp + b], rtn = sn.rhotheta_v[b];
        const double irn = rk != 0 || !theta ? 1.0 / rn : 0.0;
        const WaveCoeffs w = wave_coeffs(rk, ro, rto, vg.exner_bg[b], so.exner_pert[b], rn, rtn, irn,
                                         rk == 0 ? 0.0 : sn.exner_pert[b], vol, rv);
        const double str = st.rho[gp + b], strt = st.rhotheta_v[b], dtv = dt * vol;
        ww.alpha[b] = w.alpha;
        ww.beta[b] = w.beta;
        ww.gam[b] = w.gam;
        ww.rho_expl[b] = ro + dt * str;
        ww.rt_expl[b] = rto + dt * strt;
        ww.tp_expl[b] = so.theta_v_pert[b] + dtv * (w.alpha * str + w.beta * strt);
        ww.ep_expl[b] = so.exner_pert[b] + dtv * w.gam * strt;
        ww.thl[b] = theta ? theta[b] : div_rcp(rtn, rn, irn);
    } else {
        double alpha, beta, gam;
        const double iv = ww.inv_vol[b], iro = rcp_nr<1>(ro);
        const double rn = sn.rho[gp + b], rtn = sn.rhotheta_v[b], irn = rk == 0 ? 0.0 : rcp_nr<1>(rn);
        const double go = (R_D / C_D_V) * (vg.exner_bg[b] + so.exner_pert[b]) * rcp_nr<1>(rto);
        if (rk == 0) {
            alpha = -rto * iro * iro * iv;
            beta = iro * iv;
            gam = go * iv;
        } else {
            const double gn = (R_D / C_D_V) * (vg.exner_bg[b] + sn.exner_pert[b]) * rcp_nr<1>(rtn);
            alpha = 0.5 * (-rto * iro * iro - rtn * irn * irn) * iv;
            beta = 0.5 * (iro + irn) * iv;
            gam = 0.5 * (go + gn) * iv;
        }
        const double str = st.rho[gp + b], strt = st.rhotheta_v[b];
        ww.alpha[b] = alpha;
        ww.beta[b] = beta;
        ww.gam[b] = gam;
        ww.rho_expl[b] = ro + dt * str;
        ww.rt_expl[b] = rto + dt * strt;
        ww.tp_expl[b] = so.theta_v_pert[b] + dt * vol * (alpha * str + beta * strt);
        ww.ep_expl[b] = so.exner_pert[b] + dt * vol * gam * strt;
        ww.thl[b] = rtn * (rk == 0 ? rcp_nr<1>(rn) : irn);
    }
}

/* FP64 path: the rows in the reference's operation order.  Thread (interface
 * j, column) forms d_j, r_j, the super-diagonal e_j of row j and the
 * sub-diagonal c_{j-1} of row j - 1, whose theta_v, rho, w and heights are
 * those of interface j: the two share their quotients.  FP64 issue bounds
 * the kernel; one division per interface (1 / rho), the others by div_rcp:
 * 96 -> 56 us at RES_ID 5, 360 -> 193 us at RES_ID 6. */
__global__ void k_waves_rows(VGrid vg, StepParams p, DState so, DState st, WavesWork ww)
{
    const int nc = vg.nc, nl = vg.nl;
    const LayerPoint pt_ = layer_point(nc);
    if (!pt_.in) return;
    const long long q = pt_.i;
    const int j = pt_.l;
    const long long ns = (long long)nl * nc, gp = p.n_cond * ns;
    const long long b = q, lo = q + nc, wi = q + nc;
    const double dt = p.dt;
    const double rho_io = 0.5 * (so.rho[gp + b] + so.rho[gp + lo]), r_rio = rcp_nr<2>(rho_io);
    const double rho_ie = 0.5 * (ww.rho_expl[b] + ww.rho_expl[lo]);
    const double tl_b = ww.thl[b], tl_lo = ww.thl[lo];
    const double th = 0.5 * (tl_b + tl_lo);
    const double dz = vg.z_scalar[b] - vg.z_scalar[lo], dpi = vg.exner_bg[b] - vg.exner_bg[lo];
    const double half_dpi = 0.5 * dpi;
    const double wo = so.w[wi], rv_b = vg.r_volume[b], rv_lo = vg.r_volume[lo];
    const double a0 = ww.alpha[b], a1 = ww.alpha[lo], b0 = ww.beta[b], b1 = ww.beta[lo];
    const double g0 = ww.gam[b], g1 = ww.gam[lo];
    const double dz_a = div_rcp(dz, p.rows_a, p.r_rows_a);
    ww.d[q] = -(th * th) * (g0 + g1) + half_dpi * (a1 - a0 + th * (b1 - b0))
              - div_rcp(dz, p.rows_a * rho_io, p.r_rows_a * r_rio)
                    * (2.0 * vg.r_area_v[wi] + dt * wo * 0.5 * (-rv_b + rv_lo));
    ww.r[q] = div_rcp(-(wo + dt * st.w[wi]) * dz, p.rows_a, p.r_rows_a)
              + div_rcp(th * (ww.ep_expl[b] - ww.ep_expl[lo]), dt, p.inv_dt)
              + p.half_inv_dt * (ww.tp_expl[b] + ww.tp_expl[lo]) * dpi - div_rcp(dz_a * wo * rho_ie, rho_io, r_rio);
    ww.th_int[q] = th;
    ww.rho_io[q] = rho_io;
    ww.r_rho_io[q] = r_rio;
    /* the terms of c and e with the old w, before the layer's volume */
    const double wt = div_rcp(dz, p.rows_b, p.r_rows_b) * 0.5 * wo;
    if (j < nl - 2) {
        const double th1 = 0.5 * (tl_lo + ww.thl[lo + nc]);
        ww.e[q] = th * g1 * th1 - half_dpi * (a1 + b1 * th1) + div_rcp(wt, vg.volume[lo] * rho_io, rv_lo * r_rio);
    }
    if (j > 0) {
        const double th0 = 0.5 * (ww.thl[b - nc] + tl_b);
        ww.c[q - nc] = th * g0 * th0 + half_dpi * (a0 + b0 * th0) - div_rcp(wt, vg.volume[b] * rho_io, rv_b * r_rio);
    }
}

/* Mixed path: the rows of column_solvers.c:142-189 rearranged so that every
 * inner interface needs one reciprocal.  Thread (interface j, column) forms
 * d_j, r_j, the super-diagonal e_j of row j and the sub-diagonal c_{j-1} of
 * row j-1: c_{j-1} depends on the quantities of interface j (theta_v, rho,
 * w, heights) and on layer j, so the thread of interface j owns it.  Grid
 * terms come from the geo tables; 1/rho at the interface is kept in rho_io
 * for k_waves_apply. */
__global__ void k_waves_rows_mixed(VGrid vg, StepParams p, DState so, DState st, WavesWork ww)
{
    const int nc = vg.nc, nl = vg.nl;
    const long long n = (long long)(nl - 1) * nc;
    const LayerPoint pt_ = layer_point(nc);
    if (!pt_.in) return;
    const long long q = pt_.i;
    const int j = pt_.l;
    const long long ns = (long long)nl * nc, gp = p.n_cond * ns;
    const long long b = q, lo = q + nc, wi = q + nc;
    const double dt = p.dt;
    const double *geo = ww.geo;
    const double dz = geo[q], H = geo[n + q], G1 = geo[2 * n + q], G2 = geo[3 * n + q];
    const double rho_io = 0.5 * (so.rho[gp + b] + so.rho[gp + lo]);
    const double irio = rcp_nr<1>(rho_io);
    const double rho_ie = 0.5 * (ww.rho_expl[b] + ww.rho_expl[lo]);
    const double tl_b = ww.thl[b], tl_lo = ww.thl[lo];
    const double th = 0.5 * (tl_b + tl_lo);
    const double wo = so.w[wi];
    const double a0 = ww.alpha[b], a1 = ww.alpha[lo], b0 = ww.beta[b], b1 = ww.beta[lo];
    const double g0 = ww.gam[b], g1 = ww.gam[lo];
    const double k1 = dz * p.k_rows;
    ww.d[q] = -(th * th) * (g0 + g1) + H * (a1 - a0 + th * (b1 - b0)) - k1 * irio * (G1 + dt * wo * G2);
    ww.r[q] = -(wo + dt * st.w[wi]) * k1 + th * (ww.ep_expl[b] - ww.ep_expl[lo]) * p.inv_dt
              + p.inv_dt * (ww.tp_expl[b] + ww.tp_expl[lo]) * H - k1 * wo * rho_ie * irio;
    ww.th_int[q] = th;
    ww.rho_io[q] = irio;
    const double sw = p.k_rows2 * wo * irio;
    if (j < nl - 2) {
        const double th_next = 0.5 * (tl_lo + ww.thl[lo + nc]);
        ww.e[q] = th * g1 * th_next - H * (a1 + b1 * th_next) + geo[5 * n + q] * sw;
    }
    if (j > 0) {
        const double th_prev = 0.5 * (ww.thl[b - nc] + tl_b);
        ww.c[q - nc] = th * g0 * th_prev + H * (a0 + b0 * th_prev) - geo[4 * n + q] * sw;
    }
}

/* tridiagonal elimination of one column (column_solvers.c:641-669), forward
 * sweep kept in registers; solution divided by the damping denominator and
 * written over r */
template <int NL, bool EXACT>
__global__ void k_waves_thomas(int nc, WavesWork ww)
{
    const int i = (int)gtid();
    if (i >= nc) return;
    constexpr int n = NL - 1;
    double ep[n], rp[n];
#pragma unroll
    for (int j = 0; j < n; ++j) {
        const long long q = (long long)j * nc + i;
        const double dj = ww.d[q], rj = ww.r[q];
        if (j == 0) {
            if (EXACT) {
                const double inv = rcp_sweep(dj);
                ep[0] = div_sweep(ww.e[q], dj, inv);
                rp[0] = div_sweep(rj, dj, inv);
            } else {
                const double inv = rcp_nr<2>(dj);
                ep[0] = ww.e[q] * inv;
                rp[0] = rj * inv;
            }
        } else {
            const double cm = ww.c[q - nc];
            const double den = dj - ep[j - 1] * cm;
            if (EXACT) {
                const double inv = rcp_sweep(den);
                if (j < n - 1) ep[j] = div_sweep(ww.e[q], den, inv);
                rp[j] = div_sweep(rj - rp[j - 1] * cm, den, inv);
            } else {
                const double inv = rcp_nr<2>(den);
                if (j < n - 1) ep[j] = ww.e[q] * inv;
                rp[j] = (rj - rp[j - 1] * cm) * inv;
            }
        }
    }
    /* damping: divide by 1 + dt * coefficient (mixed path: multiply by the
     * tabulated reciprocal) */
    auto damp = [&](double x, long long q) {
        return EXACT ? div_sweep(x, ww.damp_den[q], ww.damp_inv[q]) : x * ww.damp_inv[q];
    };
    double x = rp[n - 1];
    ww.r[(long long)(n - 1) * nc + i] = damp(x, (long long)(n - 1) * nc + i);
#pragma unroll
    for (int j = n - 2; j >= 0; --j) {
        x = rp[j] - ep[j] * x;
        ww.r[(long long)j * nc + i] = damp(x, (long long)j * nc + i);
    }
}

/* generic layer count (nl - 1 <= CAP): the sweep in local memory, FP64
 * divisions on both paths */
template <int CAP, bool EXACT>
__global__ void k_waves_thomas_any(int nc, int nl, WavesWork ww)
{
    const int i = (int)gtid();
    if (i >= nc) return;
    const int n = nl - 1;
    double ep[CAP], rp[CAP];
    for (int j = 0; j < n; ++j) {
        const long long q = (long long)j * nc + i;
        const double dj = ww.d[q], rj = ww.r[q];
        if (j == 0) {
            ep[0] = ww.e[q] / dj;
            rp[0] = rj / dj;
        } else {
            const double cm = ww.c[q - nc];
            const double den = dj - ep[j - 1] * cm;
            if (j < n - 1) ep[j] = ww.e[q] / den;
            rp[j] = (rj - rp[j - 1] * cm) / den;
        }
    }
    auto damp = [&](double x, long long q) {
        return EXACT ? div_rcp(x, ww.damp_den[q], ww.damp_inv[q]) : x * ww.damp_inv[q];
    };
    double x = rp[n - 1];
    ww.r[(long long)(n - 1) * nc + i] = damp(x, (long long)(n - 1) * nc + i);
    for (int j = n - 2; j >= 0; --j) {
        x = rp[j] - ep[j] * x;
        ww.r[(long long)j * nc + i] = damp(x, (long long)j * nc + i);
    }
}

template <bool EXACT>
__global__ void k_waves_apply(VGrid vg, StepParams p, DState so, DState sn, WavesWork ww, Shadow sh)
{
    const int nc = vg.nc, nl = vg.nl;
    const long long ns = (long long)nl * nc;
    const long long b = gtid();
    if (b >= ns) return;
    const int j = row_of(b, nc);
    const long long gp = p.n_cond * ns;
    const double dt = p.dt;
    const double *sol = ww.r;
    auto rho_new = [&](int jj, long long bb) {
        const double ve = EXACT ? vg.volume[bb] : 0.0;
        const double iv = EXACT ? 0.0 : ww.inv_vol[bb];
        double num;
        if (jj == 0) num = sol[bb];
        else if (jj == nl - 1) num = -sol[bb - nc];
        else num = -sol[bb - nc] + sol[bb];
        return EXACT ? ww.rho_expl[bb] + div_rcp(dt * num, ve, vg.r_volume[bb]) : ww.rho_expl[bb] + dt * num * iv;
    };
    const double r_new = rho_new(j, b);
    double num;
    if (j == 0) num = ww.th_int[b] * sol[b];
    else if (j == nl - 1) num = -ww.th_int[b - nc] * sol[b - nc];
    else num = -ww.th_int[b - nc] * sol[b - nc] + ww.th_int[b] * sol[b];
    const double rt_new = EXACT ? ww.rt_expl[b] + div_rcp(dt * num, vg.volume[b], vg.r_volume[b])
                                : ww.rt_expl[b] + dt * num * ww.inv_vol[b];
    const double tp_new =
        (EXACT ? div_rcp(rt_new, r_new, rcp_nr<2>(r_new)) : rt_new * rcp_nr<1>(r_new)) - vg.theta_v_bg[b];
    const double ep_new = so.exner_pert[b] + vg.volume[b] * ww.gam[b] * (rt_new - so.rhotheta_v[b]);
    sn.rho[gp + b] = r_new;
    sn.rhotheta_v[b] = rt_new;
    sn.theta_v_pert[b] = tp_new;
    sn.exner_pert[b] = ep_new;
    if (sh.rho) {
        sh.rho[gp + b] = to_float(r_new);
        sh.rhotheta_v[b] = to_float(rt_new);
        sh.theta_v_pert[b] = to_float(tp_new);
        sh.exner_pert[b] = to_float(ep_new);
    }
    if (j < nl - 1) {
        const long long wi = b + nc;
        const double r_below = rho_new(j + 1, b + nc);
        const double dint = 0.5 * (r_new + r_below);
        double wn;
        if (EXACT)
            wn = div_rcp(div_rcp(2.0 * sol[b], vg.area_v[wi], vg.r_area_v[wi]) - dint * so.w[wi], ww.rho_io[b],
                         ww.r_rho_io[b]);
        else /* rho_io holds 1 / rho at the interface on the mixed path */
            wn = (2.0 * sol[b] * ww.inv_area_v[wi] - dint * so.w[wi]) * ww.rho_io[b];
        sn.w[wi] = wn;
        if (sh.w) sh.w[wi] = to_float(wn);
    }
}

/* ------------------------------------------------------------- tracers */
/* layers (bits of held) that received a density, into one word of
 * Present::by_const: one atomic at most per warp and word, from the threads of
 * the warp that are here (a store per layer and warp cost k_tracers_solve_df
 * 486 -> 884 us at RES_ID 7 with tracers everywhere) */
__device__ __forceinline__ void mark_layers(unsigned *words, int word, unsigned held)
{
    const unsigned same = __match_any_sync(__activemask(), word);
    held = __reduce_or_sync(same, held);
    if ((threadIdx.x & 31) == __ffs(same) - 1 && (held & ~*(volatile unsigned *)(words + word)))
        atomicOr(words + word, held);
}

struct TracerWork {
    const double *cp_ice, *cp_water; /* c_p of ice / liquid water at the cell temperature [L][Nc] */
    const double *inv_vol;           /* mixed path */
};

__device__ __forceinline__ double sink_velocity(const StepParams &p, int k, bool &has)
{
    const int cond = p.n_cond;
    has = true;
    if (k < cond / 4) return p.snow_velocity;
    if (k < cond / 2) return p.rain_velocity;
    if (k < cond) return p.cloud_velocity;
    has = false;
    return 0.0;
}

/* layers tested for a density at a time */
constexpr int EMPTY_BATCH = 13;
/* whether a constituent's old density and tendency are 0 in every layer of
 * column i: the lowest layer first, which tells most of the others, then
 * batches of loads in flight */
__device__ __forceinline__ bool absent_from_column(const double *ro, const double *tr, int nl, int nc, int i)
{
    const long long low = (long long)(nl - 1) * nc + i;
    bool empty = is_zero(ro[low]) && is_zero(tr[low]);
#pragma unroll 1
    for (int j0 = 0; j0 < nl && empty; j0 += EMPTY_BATCH) {
        unsigned long long any = 0;
#pragma unroll
        for (int d = 0; d < EMPTY_BATCH; ++d) {
            if (j0 + d >= nl) continue;
            const long long b = (long long)(j0 + d) * nc + i;
            any |= (unsigned long long)(__double_as_longlong(ro[b]) | __double_as_longlong(tr[b]));
        }
        empty = (any << 1) == 0ULL;
    }
    return empty;
}

/* vertical advection + sedimentation of constituent k in one column
 * (column_solvers.c:398-635); thread = (k-slot, column).  NL > 0: the layer
 * count is a compile-time constant and the sweep stays in registers; NL = 0:
 * the layer count is vg.nl (at most CAP) and the sweep lives in local memory */
template <int NL, int CAP, bool EXACT>
__global__ void k_tracers_solve(VGrid vg, StepParams p, DState so, DState sn, DState st, TracerWork tw, float *sh_rho,
                                Present present)
{
    const int nc = vg.nc;
    const int nl = NL > 0 ? NL : vg.nl;
    const long long ns = (long long)nl * nc;
    const long long q = gtid();
    const int n_tr = p.n_const - 1;
    if (q >= (long long)n_tr * nc) return;
    /* the last slot (the vapour, in every column of a moist run) first, the
     * columns without condensates fill in behind its solves */
    const int row = (int)(q / nc), slot = n_tr - 1 - row, i = (int)(q - (long long)row * nc);
    const int k = slot < p.n_cond ? slot : slot + 1; /* skip the main gas */
    bool has_sink;
    const double vsink = sink_velocity(p, k, has_sink);
    const double dt = p.dt, iw = 0.5, ew = 1.0 - iw, half_dt = 0.5 * dt;
    const double *ro = so.rho + k * ns;
    const double *tr = st.rho + k * ns;
    const long long bot = i + ns - nc;
    /* a constituent absent from the column, old density and tendency 0 in
     * every layer: so is the solution.  FP64, with the volumes' reciprocals
     * and one division per row: RES_ID 6, cloud-free, 1088 -> 103 us;
     * RES_ID 5 with clouds everywhere 221 -> 120 us.  Mixed, 80 layers,
     * RES_ID 4, cloud-free, with the rows' inputs loaded a row ahead and blocks
     * of one warp: 189 -> 121 us */
    if (absent_from_column(ro, tr, nl, nc, i)) {
        double *rn = sn.rho + k * ns;
        float *rs = sh_rho ? sh_rho + k * ns : nullptr;
#pragma unroll 1
        for (int j = 0; j < nl; ++j) {
            rn[i + (long long)j * nc] = 0.0;
            if (rs) rs[i + (long long)j * nc] = 0.f;
        }
        return;
    }
    const double a_sfc = vg.area_v[(long long)nl * nc + i];
    double ep[NL > 0 ? NL : CAP], rp[NL > 0 ? NL : CAP];
    /* FP64 path: iw dt / V of the layer, shared by its flux terms */
    double gq = EXACT ? div_sweep(iw * dt, vg.volume[i], vg.r_volume[i]) : 0.0;
    double fi_prev = 0.0, fr_prev = 0.0, c_prev = 0.0;
    /* what row j reads; where the layer count is a run-time one, a row ahead of
     * its use (with a compile-time one the compiler places the loads) */
    struct Row {
        double ro, ro_lo, tr, wo, wn, ar, iv;
    };
    auto load = [&](int j) {
        const long long b = i + (long long)j * nc;
        return Row{ro[b], j < nl - 1 ? ro[b + nc] : 0.0, tr[b], so.w[b + nc], sn.w[b + nc], vg.area_v[b + nc],
                   EXACT ? 0.0 : tw.inv_vol[b]};
    };
    Row next = load(0);
#pragma unroll
    for (int j = 0; j < nl; ++j) {
        const Row in = NL > 0 ? load(j) : next;
        if (NL == 0 && j < nl - 1) next = load(j + 1);
        const long long b = i + (long long)j * nc;
        const double vol = EXACT ? vg.volume[b] : 0.0, rvol = EXACT ? vg.r_volume[b] : 0.0;
        double gq_next = 0.0;
        if (EXACT && j < nl - 1) gq_next = div_sweep(iw * dt, vg.volume[b + nc], vg.r_volume[b + nc]);
        /* mixed path: implicit and explicit weights are both 1/2, so every
         * flux term of row j carries the factor g = dt / (2 V_j) */
        const double g = EXACT ? 0.0 : half_dt * in.iv;
        /* flux at interface j (below layer j) */
        double fi = 0.0, fr = 0.0, cj = 0.0, ej = 0.0;
        if (j < nl - 1) {
            double a_ = in.wo, b_ = in.wn;
            if (has_sink) {
                a_ -= vsink;
                b_ -= vsink;
            }
            a_ = in.ar * a_;
            b_ = in.ar * b_;
            const double dio = nonneg<EXACT>(b_) ? in.ro_lo : in.ro;
            fi = a_;
            fr = dio * b_;
            if (EXACT) {
                if (nonneg<EXACT>(fi)) ej = -gq * fi;
                else cj = gq_next * fi;
            } else if (nonneg<EXACT>(fi)) {
                ej = -g * fi;
            }
        }
        if (!EXACT) /* sub-diagonal of row j - 1, formed with row j's factor */
            c_prev = nonneg<EXACT>(fi_prev) ? 0.0 : g * fi_prev;
        double dj, rj = in.ro + dt * in.tr;
        if (EXACT) {
            if (j == 0) {
                dj = fi >= 0.0 ? 1.0 : 1.0 - gq * fi;
                rj += div_sweep(ew * dt * fr, vol, rvol);
            } else if (j == nl - 1) {
                dj = fi_prev >= 0.0 ? 1.0 + gq * fi_prev : 1.0;
                if (has_sink) dj += div_sweep(iw * vsink * dt * a_sfc, vol, rvol);
                rj += div_sweep(-ew * dt * fr_prev, vol, rvol);
                if (has_sink) rj += div_sweep(-ew * vsink * dt * ro[bot] * a_sfc, vol, rvol);
            } else {
                dj = 1.0;
                if (fi_prev >= 0.0) dj += gq * fi_prev;
                if (fi < 0.0) dj -= gq * fi;
                rj += div_sweep(ew * dt * (-fr_prev + fr), vol, rvol);
            }
        } else {
            if (j == 0) {
                dj = nonneg<EXACT>(fi) ? 1.0 : 1.0 - g * fi;
                rj += g * fr;
            } else if (j == nl - 1) {
                dj = nonneg<EXACT>(fi_prev) ? 1.0 + g * fi_prev : 1.0;
                rj -= g * fr_prev;
                if (has_sink) {
                    const double gs = g * vsink * a_sfc;
                    dj += gs;
                    rj -= gs * ro[bot];
                }
            } else {
                dj = 1.0 + (nonneg<EXACT>(fi_prev) ? g * fi_prev : 0.0) - (nonneg<EXACT>(fi) ? 0.0 : g * fi);
                rj += g * (fr - fr_prev);
            }
        }
        /* forward elimination */
        if (j == 0) {
            if (EXACT) {
                const double inv = rcp_sweep(dj);
                ep[0] = div_sweep(ej, dj, inv);
                rp[0] = div_sweep(rj, dj, inv);
            } else {
                const double inv = rcp_nr<2>(dj);
                ep[0] = ej * inv;
                rp[0] = rj * inv;
            }
        } else {
            const double den = dj - ep[j - 1] * c_prev;
            if (EXACT) {
                const double inv = rcp_sweep(den);
                if (j < nl - 1) ep[j] = div_sweep(ej, den, inv);
                rp[j] = div_sweep(rj - rp[j - 1] * c_prev, den, inv);
            } else {
                const double inv = rcp_nr<2>(den);
                if (j < nl - 1) ep[j] = ej * inv;
                rp[j] = (rj - rp[j - 1] * c_prev) * inv;
            }
        }
        fi_prev = fi;
        fr_prev = fr;
        if (EXACT) {
            c_prev = cj;
            gq = gq_next;
        }
    }
    double *rn = sn.rho + k * ns;
    float *rs = sh_rho ? sh_rho + k * ns : nullptr;
    double x = rp[nl - 1];
    unsigned held = 0; /* layers of a 32-layer group that receive a density */
    {
        const double v = EXACT ? (x < 0.0 ? 0.0 : x) : (nonneg<false>(x) ? x : 0.0);
        rn[(long long)(nl - 1) * nc + i] = v;
        if (rs) {
            rs[(long long)(nl - 1) * nc + i] = to_float(v);
            held = (is_zero(v) ? 0u : 1u) << ((nl - 1) & 31);
        }
    }
#pragma unroll
    for (int j = nl - 2; j >= 0; --j) {
        x = rp[j] - ep[j] * x;
        const double v = EXACT ? (x < 0.0 ? 0.0 : x) : (nonneg<false>(x) ? x : 0.0);
        rn[(long long)j * nc + i] = v;
        if (rs) {
            rs[(long long)j * nc + i] = to_float(v);
            if ((j & 31) == 31) {
                mark_layers(present.by_const, 8 * k + (j >> 5) + 1, held);
                held = 0;
            }
            held |= (is_zero(v) ? 0u : 1u) << (j & 31);
        }
    }
    if (rs) mark_layers(present.by_const, 8 * k, held);
}

/* sedimentation heating (rk 0 only), mixed path with FP64 eliminations:
 * thread = column, walking down the
 * layers so that each interface's enthalpy fluxes are formed once and reused
 * by the layer below; the condensates' contributions are added in the
 * reference's constituent order, with the same operations as the per-layer
 * form (column_solvers.c:455-462, 551-623) */
constexpr int SEDHEAT_MAX_COND = 4;
__global__ void k_tracers_sedheat(VGrid vg, StepParams p, DState so, DState sn, const double *temperature,
                                  TracerWork tw, double *sed_heat)
{
    const int nc = vg.nc, nl = vg.nl;
    const long long ns = (long long)nl * nc;
    const long long ii = gtid();
    if (ii >= nc) return;
    const int i = (int)ii, n_cond = p.n_cond;
    const long long bot = i + ns - nc;
    const double a_sfc = vg.area_v[(long long)nl * nc + i];
    /* enthalpy flux of constituent k at interface jj (below layer jj) */
    auto fe = [&](int k, int jj, double vsink, bool has) {
        const long long bb = i + (long long)jj * nc, wi = bb + nc;
        double b_ = sn.w[wi];
        if (has) b_ -= vsink;
        b_ = vg.area_v[wi] * b_;
        const long long up = nonneg<false>(b_) ? bb + nc : bb;
        const double dio = so.rho[k * ns + up], tio = temperature[up];
        const double fr = dio * b_;
        const double cp = (k % 2 == 0) ? tw.cp_ice[up] : tw.cp_water[up];
        return cp * tio * fr;
    };
    double h_up[SEDHEAT_MAX_COND];
    for (int j = 0; j < nl; ++j) {
        const long long b = i + (long long)j * nc;
        const double ivol = tw.inv_vol[b];
        auto per_vol = [&](double x) { return x * ivol; };
        double sh = 0.0;
#pragma unroll
        for (int k = 0; k < SEDHEAT_MAX_COND; ++k) {
            if (k >= n_cond) break;
            bool has;
            const double vs = sink_velocity(p, k, has);
            if (j == 0) {
                h_up[k] = fe(k, j, vs, has);
                sh += per_vol(h_up[k]);
            } else if (j == nl - 1) {
                sh += per_vol(-h_up[k]);
                const double tb = temperature[bot];
                const double cp = (k % 2 == 0) ? tw.cp_ice[bot] : tw.cp_water[bot];
                sh += per_vol(-vs * tb * cp * so.rho[k * ns + bot] * a_sfc);
            } else {
                const double h = fe(k, j, vs, has);
                sh += per_vol(-h_up[k] + h);
                h_up[k] = h;
            }
        }
        sed_heat[b] = sh;
    }
}

/* the same on the FP64 path, thread = (layer, column): each forms the
 * enthalpy fluxes of both its interfaces, twice the products of the walk down
 * a column but a layer count more threads (a walk of RES_ID 4's 2562 columns
 * fills 20 blocks); an absent condensate's flux is a zero and left out.
 * RES_ID 6, cloud-free: 328 -> 16 us. */
__global__ void k_tracers_sedheat64(VGrid vg, StepParams p, DState so, DState sn, const double *temperature,
                                    TracerWork tw, double *sed_heat)
{
    const LayerPoint pt = layer_point(vg.nc);
    if (!pt.in) return;
    const int nc = vg.nc, nl = vg.nl, j = pt.l, i = pt.x;
    const long long ns = (long long)nl * nc, b = pt.i;
    const int n_cond = p.n_cond < SEDHEAT_MAX_COND ? p.n_cond : SEDHEAT_MAX_COND;
    /* enthalpy flux of constituent k at the interface below box bb */
    auto fe = [&](int k, long long bb, double vsink, bool has) {
        const double r_hi = so.rho[k * ns + bb], r_lo = so.rho[k * ns + bb + nc];
        if (is_zero(r_hi) && is_zero(r_lo)) return 0.0;
        const long long wi = bb + nc;
        double b_ = sn.w[wi];
        if (has) b_ -= vsink;
        b_ = vg.area_v[wi] * b_;
        const bool from_below = nonneg<true>(b_);
        const long long up = from_below ? bb + nc : bb;
        const double fr = (from_below ? r_lo : r_hi) * b_;
        const double cp = (k % 2 == 0) ? tw.cp_ice[up] : tw.cp_water[up];
        return cp * temperature[up] * fr;
    };
    /* no condensate here or in the layers around: no arithmetic at all (the
     * tests inside fe alone are run ahead of) */
    unsigned long long any = 0;
    for (int k = 0; k < n_cond; ++k) {
        const double *r = so.rho + k * ns + b;
        any |= (unsigned long long)(__double_as_longlong(r[0]) | (j > 0 ? __double_as_longlong(r[-nc]) : 0LL)
                                    | (j < nl - 1 ? __double_as_longlong(r[nc]) : 0LL));
    }
    if ((any << 1) == 0ULL) {
        sed_heat[b] = 0.0;
        return;
    }
    const double vol = vg.volume[b], rvol = vg.r_volume[b];
    double sh = 0.0;
#pragma unroll 1
    for (int k = 0; k < n_cond; ++k) {
        bool has;
        const double vs = sink_velocity(p, k, has);
        if (j == 0) {
            sh += div_rcp(fe(k, b, vs, has), vol, rvol);
        } else if (j == nl - 1) {
            sh += div_rcp(-fe(k, b - nc, vs, has), vol, rvol);
            const double r = so.rho[k * ns + b];
            if (!is_zero(r)) {
                const double cp = (k % 2 == 0) ? tw.cp_ice[b] : tw.cp_water[b];
                sh += div_rcp(-vs * temperature[b] * cp * r * vg.area_v[(long long)nl * nc + i], vol, rvol);
            }
        } else {
            sh += div_rcp(-fe(k, b - nc, vs, has) + fe(k, b, vs, has), vol, rvol);
        }
    }
    sed_heat[b] = sh;
}

/* ------------------------------------------------ deep columns: warp PCR
 * One warp solves one tridiagonal system a_j x_{j-1} + b_j x_j + c_j x_{j+1}
 * = d_j (j < n, a_0 = c_{n-1} = 0) by parallel cyclic reduction (Hockney and
 * Jesshope): in step s = 1, 2, 4, ... every row eliminates its couplings at
 * distance s with the rows j - s and j + s, so after ceil(log2 n) steps row j
 * reads x_j = d_j.  Rows are kept normalised to b_j = 1, one reciprocal per
 * row and step (an FP64 division on the FP64 path, a Newton-refined
 * reciprocal on the mixed path).
 * A block holds PCR_WARPS systems of neighbouring columns.  Its threads load
 * and store the rows cooperatively, PCR_WARPS consecutive columns of one row
 * per group of threads, so that the [layer][cell] accesses fill whole
 * sectors; warp w then reduces system w in shared memory, double-buffered
 * (one __syncwarp per step), lane l handling rows l, l + 32, ....
 * Shared memory: 6 n doubles per system, 48 KB per block at n = 256. */
constexpr int PCR_MAX_ROWS = 256;
constexpr int PCR_WARPS = 4; /* systems (warps) per block */
static_assert(PCR_WARPS * 6 * PCR_MAX_ROWS * sizeof(double) <= 48 * 1024, "PCR block exceeds 48 KB");

template <bool EXACT>
__device__ __forceinline__ double pcr_inv(double b)
{
    return EXACT ? 1.0 / b : rcp_nr<2>(b);
}

/* reduction steps for n rows: ceil(log2 n) */
__device__ __forceinline__ int pcr_steps(int n)
{
    int s = 0;
    for (int st = 1; st < n; st <<= 1) ++s;
    return s;
}

/* s: [a | c | d] of n normalised rows followed by the second buffer; the
 * solution ends in d of buffer pcr_steps(n) & 1 */
template <bool EXACT>
__device__ __forceinline__ void pcr_warp(double *s, int n)
{
    const int lane = threadIdx.x & 31;
    double *cur = s, *nxt = s + 3 * n;
    for (int st = 1; st < n; st <<= 1) {
        const double *a = cur, *c = cur + n, *d = cur + 2 * n;
        for (int j = lane; j < n; j += 32) {
            double an = 0.0, cn = 0.0, bn = 1.0, dn = d[j];
            if (j - st >= 0) {
                const double k = a[j];
                an = -k * a[j - st];
                bn -= k * c[j - st];
                dn -= k * d[j - st];
            }
            if (j + st < n) {
                const double k = c[j];
                cn = -k * c[j + st];
                bn -= k * a[j + st];
                dn -= k * d[j + st];
            }
            const double r = pcr_inv<EXACT>(bn);
            nxt[j] = an * r;
            nxt[n + j] = cn * r;
            nxt[2 * n + j] = dn * r;
        }
        __syncwarp();
        double *tmp = cur;
        cur = nxt;
        nxt = tmp;
    }
}

__device__ __forceinline__ const double *pcr_solution(const double *s, int n)
{
    return s + (pcr_steps(n) & 1) * 3 * n + 2 * n;
}

/* sound waves: the rows of k_waves_rows(_mixed) of PCR_WARPS neighbouring
 * columns, solution divided by the damping denominator into r */
template <bool EXACT>
__global__ void __launch_bounds__(32 * PCR_WARPS) k_waves_pcr(int nc, int nl, WavesWork ww)
{
    extern __shared__ double smem[];
    const int n = nl - 1;
    const int t = threadIdx.x, warp = t >> 5, sys = t % PCR_WARPS, row0 = t / PCR_WARPS;
    const int i0 = blockIdx.x * PCR_WARPS, i = i0 + sys;
    double *s = smem + (size_t)sys * 6 * n;
    if (i < nc)
        for (int j = row0; j < n; j += 32) {
            const long long q = (long long)j * nc + i;
            const double r = pcr_inv<EXACT>(ww.d[q]);
            s[j] = j > 0 ? ww.c[q - nc] * r : 0.0;
            s[n + j] = j < n - 1 ? ww.e[q] * r : 0.0;
            s[2 * n + j] = ww.r[q] * r;
        }
    __syncthreads();
    if (i0 + warp < nc) pcr_warp<EXACT>(smem + (size_t)warp * 6 * n, n);
    __syncthreads();
    if (i < nc) {
        const double *x = pcr_solution(s, n);
        for (int j = row0; j < n; j += 32) {
            const long long q = (long long)j * nc + i;
            ww.r[q] = EXACT ? div_rcp(x[j], ww.damp_den[q], ww.damp_inv[q]) : x[j] * ww.damp_inv[q];
        }
    }
}

/* tracers: vertical advection and sedimentation of constituent k (the rows of
 * k_tracers_solve, column_solvers.c:398-635) for PCR_WARPS consecutive
 * (k-slot, column) systems, clipped at 0; the sedimentation heat comes from
 * k_tracers_sedheat.  The interface fluxes are staged in the second buffer,
 * which the reduction overwrites only after the rows are built. */
template <bool EXACT>
__global__ void __launch_bounds__(32 * PCR_WARPS)
    k_tracers_pcr(VGrid vg, StepParams p, DState so, DState sn, DState st, TracerWork tw, float *sh_rho,
                                Present present)
{
    extern __shared__ double smem[];
    const int nc = vg.nc, nl = vg.nl, n = nl;
    const int t = threadIdx.x, warp = t >> 5, sys = t % PCR_WARPS, row0 = t / PCR_WARPS;
    const int n_tr = p.n_const - 1;
    const long long nsys = (long long)n_tr * nc, q0 = (long long)blockIdx.x * PCR_WARPS, q = q0 + sys;
    const bool valid = q < nsys;
    const int slot = valid ? (int)(q / nc) : 0, i = valid ? (int)(q - (long long)slot * nc) : 0;
    const int k = slot < p.n_cond ? slot : slot + 1;
    const long long ns = (long long)nl * nc;
    bool has_sink;
    const double vsink = sink_velocity(p, k, has_sink);
    const double dt = p.dt, iw = 0.5, ew = 1.0 - iw, half_dt = 0.5 * dt;
    const double *ro = so.rho + k * ns, *tr = st.rho + k * ns;
    double *s = smem + (size_t)sys * 6 * n;
    double *fi = s + 3 * n, *fr = s + 4 * n;
    /* interface fluxes (below layer j) */
    if (valid)
        for (int j = row0; j < n; j += 32) {
            double a_ = 0.0, f_ = 0.0;
            if (j < nl - 1) {
                const long long b = i + (long long)j * nc, wi = b + nc;
                double wo = so.w[wi], wn = sn.w[wi];
                if (has_sink) {
                    wo -= vsink;
                    wn -= vsink;
                }
                const double ar = vg.area_v[wi];
                a_ = ar * wo;
                const double b_ = ar * wn;
                f_ = (nonneg<EXACT>(b_) ? ro[b + nc] : ro[b]) * b_;
            }
            fi[j] = a_;
            fr[j] = f_;
        }
    __syncthreads();
    if (valid) {
        const long long bot = i + ns - nc;
        const double a_sfc = vg.area_v[(long long)nl * nc + i];
        for (int j = row0; j < n; j += 32) {
            const long long b = i + (long long)j * nc;
            const double fij = j < nl - 1 ? fi[j] : 0.0, fip = j > 0 ? fi[j - 1] : 0.0;
            const double frj = j < nl - 1 ? fr[j] : 0.0, frp = j > 0 ? fr[j - 1] : 0.0;
            double aj = 0.0, cj = 0.0, dj, rj = ro[b] + dt * tr[b];
            if (EXACT) {
                const double vol = vg.volume[b];
                if (j > 0 && fip < 0.0) aj = iw * dt / vol * fip;
                if (j < nl - 1 && fij >= 0.0) cj = -iw * dt / vol * fij;
                if (j == 0) {
                    dj = fij >= 0.0 ? 1.0 : 1.0 - iw * dt / vol * fij;
                    rj += ew * dt * frj / vol;
                } else if (j == nl - 1) {
                    dj = fip >= 0.0 ? 1.0 + iw * dt / vol * fip : 1.0;
                    if (has_sink) dj += iw * vsink * dt * a_sfc / vol;
                    rj += -ew * dt * frp / vol;
                    if (has_sink) rj += -ew * vsink * dt * ro[bot] * a_sfc / vol;
                } else {
                    dj = 1.0;
                    if (fip >= 0.0) dj += iw * dt / vol * fip;
                    if (fij < 0.0) dj -= iw * dt / vol * fij;
                    rj += ew * dt * (-frp + frj) / vol;
                }
            } else {
                const double g = half_dt * tw.inv_vol[b];
                if (j > 0 && !nonneg<false>(fip)) aj = g * fip;
                if (j < nl - 1 && nonneg<false>(fij)) cj = -g * fij;
                if (j == 0) {
                    dj = nonneg<false>(fij) ? 1.0 : 1.0 - g * fij;
                    rj += g * frj;
                } else if (j == nl - 1) {
                    dj = nonneg<false>(fip) ? 1.0 + g * fip : 1.0;
                    rj -= g * frp;
                    if (has_sink) {
                        const double gs = g * vsink * a_sfc;
                        dj += gs;
                        rj -= gs * ro[bot];
                    }
                } else {
                    dj = 1.0 + (nonneg<false>(fip) ? g * fip : 0.0) - (nonneg<false>(fij) ? 0.0 : g * fij);
                    rj += g * (frj - frp);
                }
            }
            const double r = pcr_inv<EXACT>(dj);
            s[j] = aj * r;
            s[n + j] = cj * r;
            s[2 * n + j] = rj * r;
        }
    }
    __syncthreads();
    if (q0 + warp < nsys) pcr_warp<EXACT>(smem + (size_t)warp * 6 * n, n);
    __syncthreads();
    if (valid) {
        const double *x = pcr_solution(s, n);
        double *rn = sn.rho + k * ns;
        float *rs = sh_rho ? sh_rho + k * ns : nullptr;
        for (int j = row0; j < n; j += 32) {
            const double v = EXACT ? (x[j] < 0.0 ? 0.0 : x[j]) : (nonneg<false>(x[j]) ? x[j] : 0.0);
            rn[i + (long long)j * nc] = v;
            if (rs) {
                rs[i + (long long)j * nc] = to_float(v);
                if (!is_zero(v)) mark_layers(present.by_const, 8 * k + (j >> 5), 1u << (j & 31));
            }
        }
    }
}

}  // namespace
}  // namespace game
