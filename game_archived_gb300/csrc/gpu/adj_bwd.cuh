/*
 * Hand-written adjoint kernels of the dry RKHEVI step (the reverse mode of
 * adj_fwd.cuh).  Each kernel takes the bar (adjoint) of one forward
 * kernel's outputs, recomputes the forward point values it needs from the
 * tape, and accumulates the bars of that kernel's inputs: x_bar += (dy/dx)^T
 * y_bar.  Gathers of the forward become scatters here; they use FP64
 * atomicAdd, so the summation order of a bar varies between runs by rounding
 * (about 1e-16 relative), which the dot-product test tolerates by orders of
 * magnitude.  Pointwise inputs are accumulated without atomics.
 */
#pragma once

#include "adj_fwd.cuh"

namespace game {
namespace {

__device__ __forceinline__ void acc(double *p, double v) { atomicAdd(p, v); }

/* ---------------------------------------------------- operator adjoints */
__device__ __forceinline__ void b_gv(const HGrid<double> &g, double *fb, int k, int c, double gb)
{
    const double q = gb / g.nd_v[(long long)k * g.nc + c];
    acc(&fb[(long long)(k - 1) * g.nc + c], q);
    acc(&fb[(long long)k * g.nc + c], -q);
}

__device__ __forceinline__ void b_grad_h(const HGrid<double> &g, double *fb, int l, int e, double ob)
{
    const int fr = g.from[e], to = g.to[e];
    const long long le = (long long)l * g.ne + e;
    const double q = ob / g.nd_h[le];
    acc(&fb[(long long)l * g.nc + to], q);
    acc(&fb[(long long)l * g.nc + fr], -q);
    if (l >= g.nl - g.n_oro) {
        const double cb = 0.5 * (-g.slope_h[le] * ob);
        b_gv(g, fb, l, fr, ipw_d(g, 6, l, fr) * cb);
        b_gv(g, fb, l, to, ipw_d(g, 6, l, to) * cb);
        if (l < g.nl - 1) {
            b_gv(g, fb, l + 1, fr, ipw_d(g, 7, l, fr) * cb);
            b_gv(g, fb, l + 1, to, ipw_d(g, 7, l, to) * cb);
        }
    }
}

__device__ __forceinline__ void b_hor_cov(const HGrid<double> &g, double *ub, double *wb, int l, int e, double rb)
{
    const long long le = (long long)l * g.ne + e;
    acc(&ub[le], rb);
    if (l >= g.nl - g.n_oro) {
        const int fr = g.from[e], to = g.to[e];
        const double cb = 0.5 * (g.slope_h[le] * rb);
        acc(&wb[(long long)l * g.nc + fr], ipw_d(g, 6, l, fr) * cb);
        acc(&wb[(long long)l * g.nc + to], ipw_d(g, 6, l, to) * cb);
        if (l < g.nl - 1) {
            acc(&wb[(long long)(l + 1) * g.nc + fr], ipw_d(g, 7, l, fr) * cb);
            acc(&wb[(long long)(l + 1) * g.nc + to], ipw_d(g, 7, l, to) * cb);
        }
    }
}

__device__ __forceinline__ void b_rel_tan(const HGrid<double> &g, double *ub, double *wb, int k, int e, double rb)
{
    const int nl = g.nl;
    if (k == 0) k = 1;
    const double ia = 1.0 / g.dual_area_h[(long long)k * g.ne + e];
    if (k == nl) {
        b_hor_cov(g, ub, wb, k - 1, e, ia * g.nd_h[(long long)(k - 1) * g.ne + e] * rb);
        return;
    }
    const int fr = g.from[e], to = g.to[e];
    const double s = ia * rb;
    b_hor_cov(g, ub, wb, k, e, -g.nd_h[(long long)k * g.ne + e] * s);
    acc(&wb[(long long)k * g.nc + fr], g.nd_v[(long long)k * g.nc + fr] * s);
    b_hor_cov(g, ub, wb, k - 1, e, g.nd_h[(long long)(k - 1) * g.ne + e] * s);
    acc(&wb[(long long)k * g.nc + to], -g.nd_v[(long long)k * g.nc + to] * s);
}

__device__ __forceinline__ void b_dens_tan(const HGrid<double> &g, double *rb, int k, int e, double db)
{
    const int nl = g.nl, nc = g.nc, ne = g.ne, fr = g.from[e], to = g.to[e];
    if (k == 0) {
        const double f = g.pvz[e] / g.pvz[ne + e];
        const double tb = 0.5 * (db * (1.0 + f)), bb = 0.5 * (-db * f);
        acc(&rb[fr], tb);
        acc(&rb[to], tb);
        acc(&rb[nc + fr], bb);
        acc(&rb[nc + to], bb);
        return;
    }
    if (k == nl) {
        const long long a = (long long)(nl - 1) * nc, b = (long long)(nl - 2) * nc;
        const double f = g.pvz[2 * (long long)ne + e] / g.pvz[3 * (long long)ne + e];
        const double lb = 0.5 * (db * (1.0 - f)), ab = 0.5 * (db * f);
        acc(&rb[a + fr], lb);
        acc(&rb[a + to], lb);
        acc(&rb[b + fr], ab);
        acc(&rb[b + to], ab);
        return;
    }
    const long long uf = (long long)(k - 1) * nc + fr, ut = (long long)(k - 1) * nc + to;
    const double q = 0.25 * db;
    acc(&rb[uf], q);
    acc(&rb[ut], q);
    acc(&rb[uf + nc], q);
    acc(&rb[ut + nc], q);
}

/* theta_v' = rho theta_v / rho - theta_bg: the bar of theta_v' moves to
 * rho theta_v and rho and is consumed */
__global__ void ba_rediag(long long ns, const double *rho, const double *rt, double *tp_b, double *rho_b, double *rt_b)
{
    const long long i = gtid();
    if (i >= ns) return;
    const double tb = tp_b[i], r = rho[i];
    rt_b[i] += tb / r;
    rho_b[i] -= tb * (rt[i] / r) / r;
    tp_b[i] = 0.0;
}

/* theta = rho theta_v / rho */
__global__ void ba_theta(long long ns, const double *rho, const double *rt, const double *theta_b, double *rho_b,
                         double *rt_b)
{
    const long long i = gtid();
    if (i >= ns) return;
    const double tb = theta_b[i], r = rho[i];
    rt_b[i] += tb / r;
    rho_b[i] -= tb * (rt[i] / r) / r;
}

__global__ void ba_pgrad(HGrid<double> g, AParams ap, AState<double> s, const double *P_b, double *tp_b,
                         double *ep_b, double *rho_all_b = nullptr)
{
    const long long nw = (long long)(g.nl + 1) * g.nc, n = nw + (long long)g.nl * g.ne;
    const long long ns = (long long)g.nl * g.nc;
    const long long i = gtid();
    if (i >= n) return;
    const double cdp = C_D_P;
    double pb = P_b[i];
    if (pb == 0.0) return;
    const bool moist = ap.n_const > 1 && rho_all_b;
    /* moist: P = dec (nl + l), dec = 0.5 (d_a + d_b), d = rho_gas / rho_total */
    auto decel = [&](long long a, long long b, double nl_plus_l) {
        double d = 0.0;
        for (const long long cell : {a, b}) {
            double tot = 0.0;
            for (int q = 0; q < ap.n_const; ++q) tot += s.rho_all[q * ns + cell];
            const double rg = s.rho[cell];
            d += 0.5 * (rg / tot);
            const double hb = 0.5 * nl_plus_l * pb;
            for (int q = 0; q < ap.n_const; ++q) {
                const double dq = ((q == ap.n_cond ? tot : 0.0) - rg) / (tot * tot);
                acc(&rho_all_b[q * ns + cell], dq * hb);
            }
        }
        return d;
    };
    if (i < nw) {
        const int k = row_of(i, g.nc), c = (int)(i - (long long)k * g.nc);
        if (k == 0 || k == g.nl) return;
        const long long up = (long long)(k - 1) * g.nc + c, lo = (long long)k * g.nc + c;
        const double G = a_gv(g, s.ep, k, c);
        const double S = 0.5 * (cdp * (g.theta_v_bg[up] + s.tp[up]) + cdp * (g.theta_v_bg[lo] + s.tp[lo]));
        if (moist) {
            const double lt = (0.5 * (cdp * s.tp[up] + cdp * s.tp[lo])) * g.exner_bg_grad_v[(long long)k * g.nc + c];
            pb = pb * decel(up, lo, S * G + lt);
        }
        const double tb = 0.5 * cdp * (G * pb) + 0.5 * cdp * g.exner_bg_grad_v[(long long)k * g.nc + c] * pb;
        acc(&tp_b[up], tb);
        acc(&tp_b[lo], tb);
        b_gv(g, ep_b, k, c, S * pb);
    } else {
        const long long j = i - nw;
        const int l = row_of(j, g.ne), e = (int)(j - (long long)l * g.ne);
        const int fr = g.from[e], to = g.to[e];
        const long long cf = (long long)l * g.nc + fr, ct = (long long)l * g.nc + to;
        const double G = a_grad_h(g, s.ep, l, e);
        const double S = 0.5 * (cdp * (g.theta_v_bg[ct] + s.tp[ct]) + cdp * (g.theta_v_bg[cf] + s.tp[cf]));
        if (moist) {
            const double lt = (0.5 * (cdp * s.tp[ct] + cdp * s.tp[cf])) * g.exner_bg_grad_h[(long long)l * g.ne + e];
            pb = pb * decel(ct, cf, S * G + lt);
        }
        const double tb = 0.5 * cdp * (G * pb) + 0.5 * cdp * g.exner_bg_grad_h[(long long)l * g.ne + e] * pb;
        acc(&tp_b[ct], tb);
        acc(&tp_b[cf], tb);
        b_grad_h(g, ep_b, l, e, S * pb);
    }
}

__global__ void ba_tri(HGrid<double> g, const double *tri_b, double *u_b)
{
    const long long n = (long long)g.nl * g.nt;
    const long long i = gtid();
    if (i >= n) return;
    const double tb = tri_b[i] / g.dual_area_t[i];
    if (tb == 0.0) return;
    const int l = row_of(i, g.nt), t = (int)(i - (long long)l * g.nt);
    for (int j = 0; j < 3; ++j) {
        const int e = g.vort_i[j * g.nt + t];
        const long long le = (long long)l * g.ne + e;
        double rescale = 1.0, dz = 0.0;
        long long lo_e = le;
        if (l >= g.nl - g.n_oro) {
            const double zt = g.dual_z_t[i];
            rescale = (g.radius + zt) / (g.radius + g.z_h[le]);
            dz = zt - g.z_h[le];
            int lo;
            if (dz > 0.0) lo = l - 1;
            else if (l == g.nl - 1) lo = l - 1;
            else lo = l + 1;
            lo_e = (long long)lo * g.ne + e;
        }
        const double vb = rescale * g.nd_h[le] * double(g.vort_s[j * g.nt + t]) * tb;
        acc(&u_b[le], vb);
        if (l >= g.nl - g.n_oro) {
            const double q = dz * vb / (g.z_h[le] - g.z_h[lo_e]);
            acc(&u_b[le], q);
            acc(&u_b[lo_e], -q);
        }
    }
}

__global__ void ba_edge(HGrid<double> g, const double *u, const double *rho, const double *zh, const double *zv,
                        const double *zh_b, const double *zv_b, const double *fh_b, double *u_b, double *w_b,
                        double *rho_b, double *tri_b)
{
    const long long n = (long long)(g.nl + 1) * g.ne;
    const long long i = gtid();
    if (i >= n) return;
    const int k = row_of(i, g.ne), e = (int)(i - (long long)k * g.ne);
    const int nl = g.nl, nc = g.nc, ne = g.ne;
    {
        const double zb = zh_b[i];
        if (zb != 0.0) {
            const double dens = a_dens_tan(g, rho, k, e);
            b_rel_tan(g, u_b, w_b, k, e, zb / dens);
            b_dens_tan(g, rho_b, k, e, -zb * zh[i] / dens);
        }
    }
    if (k < nl) {
        const long long le = (long long)k * ne + e;
        const double vb = zv_b[le];
        if (vb != 0.0) {
            double dens = 0.0;
            for (int j = 0; j < 4; ++j)
                dens += g.rhombi_w[j * (long long)ne + e] * rho[(long long)k * nc + g.rhombi_i[j * (long long)ne + e]];
            const double pb = vb / dens, db = -vb * zv[le] / dens;
            for (int j = 0; j < 4; ++j)
                acc(&rho_b[(long long)k * nc + g.rhombi_i[j * (long long)ne + e]], g.rhombi_w[j * (long long)ne + e] * db);
            const int tf = g.dual_from[e], tt = g.dual_to[e];
            const long long kt = (long long)k * g.nt;
            const double af = g.dual_area_t[kt + tf], at = g.dual_area_t[kt + tt];
            acc(&tri_b[kt + tf], af / (af + at) * pb);
            acc(&tri_b[kt + tt], at / (af + at) * pb);
        }
        const double fb = fh_b[le];
        if (fb != 0.0) {
            const long long ct = (long long)k * nc + g.to[e], cf = (long long)k * nc + g.from[e];
            acc(&u_b[le], 0.5 * (rho[ct] + rho[cf]) * fb);
            const double q = 0.5 * u[le] * fb;
            acc(&rho_b[ct], q);
            acc(&rho_b[cf], q);
        }
    }
}

__global__ void ba_kin(HGrid<double> g, const double *u, const double *w, const double *rho, const double *v2_b,
                       const double *fv_b, double *u_b, double *w_b, double *rho_b)
{
    const long long ns = (long long)g.nl * g.nc;
    const long long i = gtid();
    if (i >= ns) return;
    const int l = row_of(i, g.nc), c = (int)(i - (long long)l * g.nc);
    const int n_edges = c < N_PENT ? 5 : 6;
    const double vb = v2_b[i];
    if (vb != 0.0) {
        for (int j = 0; j < n_edges; ++j) {
            const long long le = (long long)l * g.ne + g.adj[j * g.nc + c];
            acc(&u_b[le], 2.0 * ipw_d(g, j, l, c) * u[le] * vb);
        }
        acc(&w_b[i], 2.0 * ipw_d(g, 6, l, c) * w[i] * vb);
        acc(&w_b[i + g.nc], 2.0 * ipw_d(g, 7, l, c) * w[i + g.nc] * vb);
    }
    if (l >= 1) {
        const double fb = fv_b[i];
        if (fb != 0.0) {
            acc(&w_b[i], 0.5 * (rho[i - g.nc] + rho[i]) * fb);
            const double q = 0.5 * w[i] * fb;
            acc(&rho_b[i - g.nc], q);
            acc(&rho_b[i], q);
        }
    }
}

__device__ __forceinline__ void b_vflux_h(const HGrid<double> &g, const double *flux_h, const double *flux_v,
                                          const double *zh, const double *zv, double *fh_b, double *fv_b,
                                          double *zh_b, double *zv_b, int l, int e, double ob)
{
    const long long ne = g.ne, nc = g.nc;
    const double *mf = flux_h + (long long)l * ne, *pv = zv + (long long)l * ne;
    double *mfb = fh_b + (long long)l * ne, *pvb = zv_b + (long long)l * ne;
    const int fr = g.from[e], to = g.to[e];
    auto term = [&](int j, bool half) {
        const double w = g.trsk_w[j * ne + e];
        const int ti = g.trsk_i[j * ne + e], tm = g.trsk_m[j * ne + e];
        if (half) {
            acc(&mfb[ti], w * 0.5 * (pv[tm] + pv[e]) * ob);
            const double q = w * mf[ti] * 0.5 * ob;
            acc(&pvb[tm], q);
            acc(&pvb[e], q);
        } else {
            acc(&mfb[ti], w * pv[tm] * ob);
            acc(&pvb[tm], w * mf[ti] * ob);
        }
    };
    if (fr < N_PENT)
        for (int j = 0; j < 4; ++j) term(j, false);
    else
        for (int j = 0; j < 5; ++j) term(j, j == 2);
    if (to < N_PENT)
        for (int j = 5; j < 9; ++j) term(j, false);
    else
        for (int j = 5; j < 10; ++j) term(j, j == 7);
    const double zt = zh[(long long)l * ne + e], zb = zh[(long long)(l + 1) * ne + e];
    const double i6f = 0.5 * ipw_d(g, 6, l, fr), i6t = 0.5 * ipw_d(g, 6, l, to);
    const double i7f = 0.5 * ipw_d(g, 7, l, fr), i7t = 0.5 * ipw_d(g, 7, l, to);
    acc(&fv_b[l * nc + fr], -i6f * zt * ob);
    acc(&fv_b[l * nc + to], -i6t * zt * ob);
    acc(&fv_b[(l + 1) * nc + fr], -i7f * zb * ob);
    acc(&fv_b[(l + 1) * nc + to], -i7t * zb * ob);
    acc(&zh_b[(long long)l * ne + e], -(i6f * flux_v[l * nc + fr] + i6t * flux_v[l * nc + to]) * ob);
    acc(&zh_b[(long long)(l + 1) * ne + e],
        -(i7f * flux_v[(l + 1) * nc + fr] + i7t * flux_v[(l + 1) * nc + to]) * ob);
}

/* horizontal momentum: t_b holds the bar of this substage's tendency from its
 * later uses, u_new_b the bar of the new wind; pvt_b / v2g_b may already hold
 * bars from the next step (they are lagged into it) */
__global__ void ba_mom_h(HGrid<double> g, AParams ap, int adv, double new_w, double old_w, const double *flux_h,
                         const double *flux_v, const double *zh, const double *zv, const double *t_b,
                         const double *u_new_b, double *u_old_b, double *tend_in_b, double *P_b, double *pgo_b,
                         double *pvt_b, double *v2g_b, double *fh_b, double *fv_b, double *zh_b, double *zv_b,
                         double *v2_b)
{
    const long long n = (long long)g.nl * g.ne;
    const long long i = gtid();
    if (i >= n) return;
    const long long nw = (long long)(g.nl + 1) * g.nc, vi = nw + i;
    const int l = row_of(i, g.ne), e = (int)(i - (long long)l * g.ne);
    const double ub = u_new_b[i];
    u_old_b[i] += ub;
    const double tb = t_b[vi] + ap.dt * ub;
    double yb;
    if (new_w == 1.0) {
        yb = tb;
    } else {
        tend_in_b[vi] += old_w * tb;
        yb = new_w * tb;
    }
    const double cur_hor = 0.5 + ap.impl_thermo_weight, old_hor = 1.0 - (0.5 + ap.impl_thermo_weight);
    pgo_b[vi] += old_hor * yb;
    P_b[vi] += -cur_hor * yb;
    const double pb = pvt_b[vi] + yb, gb = v2g_b[vi] - 0.5 * yb;
    pvt_b[vi] = pb;
    v2g_b[vi] = gb;
    if (adv) {
        if (pb != 0.0) b_vflux_h(g, flux_h, flux_v, zh, zv, fh_b, fv_b, zh_b, zv_b, l, e, pb);
        if (gb != 0.0) b_grad_h(g, v2_b, l, e, gb);
    }
}

__global__ void ba_mom_v(HGrid<double> g, AParams ap, int adv, double new_w, double old_w, const double *flux_h,
                         const double *zh, const double *t_b, double *tend_in_b, double *P_b, double *pvt_b,
                         double *v2g_b, double *fh_b, double *zh_b, double *v2_b, const double *rho_all = nullptr,
                         double *rho_all_b = nullptr)
{
    const long long n = (long long)(g.nl + 1) * g.nc;
    const long long i = gtid();
    if (i >= n) return;
    const int k = row_of(i, g.nc), c = (int)(i - (long long)k * g.nc);
    const int nl = g.nl;
    double pb = pvt_b[i];
    if (k != 0 && k != nl) {
        const double tb = t_b[i];
        double yb;
        if (new_w == 1.0) {
            yb = tb;
        } else {
            tend_in_b[i] += old_w * tb;
            yb = new_w * tb;
        }
        const double cur_ver = 1.0 - ap.impl_thermo_weight;
        P_b[i] += -cur_ver * yb;
        pb += yb;
        if (rho_all && yb != 0.0) {
            /* condensate term 0.5 (d_up + d_lo) g_m, d = rho_gas / rho_total - 1 */
            const long long ns = (long long)nl * g.nc, gp = (long long)ap.n_cond * ns;
            const double hb = 0.5 * g.gravity_m_v[i] * yb;
            for (const long long cell : {(long long)(k - 1) * g.nc + c, (long long)k * g.nc + c}) {
                double tot = 0.0;
                for (int q = 0; q < ap.n_const; ++q) tot += rho_all[q * ns + cell];
                const double rg = rho_all[gp + cell];
                /* d(rg / tot) / d rho_q = (delta_q,gas tot - rg) / tot^2 */
                for (int q = 0; q < ap.n_const; ++q) {
                    const double dq = ((q == ap.n_cond ? tot : 0.0) - rg) / (tot * tot);
                    acc(&rho_all_b[q * ns + cell], dq * hb);
                }
            }
        }
        const double gb = v2g_b[i] - 0.5 * yb;
        v2g_b[i] = gb;
        if (adv && gb != 0.0) b_gv(g, v2_b, k, c, gb);
    }
    pvt_b[i] = pb;
    if (adv && pb != 0.0) {
        const int n_edges = c < N_PENT ? 5 : 6;
        const double vw = (k == 0 || k == nl) ? 1.0 : 0.5;
        const double *z = zh + (long long)k * g.ne;
        double *zb = zh_b + (long long)k * g.ne;
        if (k >= 1)
            for (int j = 0; j < n_edges; ++j) {
                const int a = g.adj[j * g.nc + c];
                const double wv = vw * ipw_d(g, j, k - 1, c);
                acc(&fh_b[(long long)(k - 1) * g.ne + a], wv * z[a] * pb);
                acc(&zb[a], wv * flux_h[(long long)(k - 1) * g.ne + a] * pb);
            }
        if (k <= nl - 1)
            for (int j = 0; j < n_edges; ++j) {
                const int a = g.adj[j * g.nc + c];
                const double wv = vw * ipw_d(g, j, k, c);
                acc(&fh_b[(long long)k * g.ne + a], wv * z[a] * pb);
                acc(&zb[a], wv * flux_h[(long long)k * g.ne + a] * pb);
            }
    }
}

/* mass and rho theta_v tendencies (fa_scalar) */
__global__ void ba_scalar(HGrid<double> g, const double *rho, const double *theta, const double *u,
                          const double *st_rho_b, const double *st_rt_b, double *rho_b, double *theta_b, double *u_b)
{
    const long long ns = (long long)g.nl * g.nc;
    const long long i = gtid();
    if (i >= ns) return;
    const double yb = st_rho_b[i], ytb = st_rt_b[i];
    if (yb == 0.0 && ytb == 0.0) return;
    const int nl = g.nl, n_oro = g.n_oro;
    const int l = row_of(i, g.nc), c = (int)(i - (long long)l * g.nc);
    const long long nc = g.nc, ne = g.ne;
    const int n_edges = c < N_PENT ? 5 : 6;
    const bool oro = l >= nl - n_oro - 1;
    const bool up_corr = oro && l >= nl - n_oro;
    const bool lo_corr = oro && l < nl - 1;
    const bool up_has_prev = up_corr && l > nl - n_oro;
    const bool lo_has_curr = lo_corr && l + 1 > nl - n_oro;
    const double inv_vol = 1.0 / g.volume[i];
    const double area_up = g.area_v[(long long)l * nc + c], area_lo = g.area_v[(long long)(l + 1) * nc + c];
    const double hb = -inv_vol * yb, htb = -inv_vol * ytb;
    double umb = 0.0, lmb = 0.0, utb = 0.0, ltb = 0.0;
    if (oro) {
        if (l == nl - n_oro - 1) {
            lmb = -area_lo * hb;
            ltb = -area_lo * htb;
        } else if (l == nl - 1) {
            umb = area_up * hb;
            utb = area_up * htb;
        } else {
            umb = area_up * hb;
            utb = area_up * htb;
            lmb = -area_lo * hb;
            ltb = -area_lo * htb;
        }
    }
    auto layer_pass = [&](int ll, bool to_h, bool to_up, bool to_lo) {
        const long long o = (long long)ll * nc;
        const double fs = rho[o + c], ts = theta[o + c];
        for (int j = 0; j < n_edges; ++j) {
            const int nb = g.adj_nbr[j * nc + c], ed = g.adj[j * nc + c];
            const long long le = (long long)ll * ne + ed;
            double fmb = 0.0, ftb = 0.0;
            if (to_h) {
                const double ar = g.area_h[le];
                const double sg = g.adj_sign[j * nc + c] > 0 ? 1.0 : -1.0;
                fmb += sg * ar * hb;
                ftb += sg * ar * htb;
            }
            if (to_up || to_lo) {
                const double wc = -0.5 * ipw_d(g, j, ll, c) * g.slope_h[le];
                if (to_up) {
                    fmb += wc * umb;
                    ftb += wc * utb;
                }
                if (to_lo) {
                    fmb += wc * lmb;
                    ftb += wc * ltb;
                }
            }
            const double uv = u[le];
            const double fm = (0.5 * (fs + rho[o + nb])) * uv;
            /* ft = 0.5 (theta_c + theta_nb) fm */
            fmb += 0.5 * (ts + theta[o + nb]) * ftb;
            const double qt = 0.5 * fm * ftb;
            acc(&theta_b[o + c], qt);
            acc(&theta_b[o + nb], qt);
            /* fm = 0.5 (rho_c + rho_nb) u */
            const double qr = 0.5 * uv * fmb;
            acc(&rho_b[o + c], qr);
            acc(&rho_b[o + nb], qr);
            acc(&u_b[le], 0.5 * (fs + rho[o + nb]) * fmb);
        }
    };
    if (up_has_prev) layer_pass(l - 1, false, true, false);
    layer_pass(l, true, up_corr, lo_has_curr);
    if (lo_corr) layer_pass(l + 1, false, false, true);
}

/* ------------------------------------------------- sound-wave solver adjoints */

/* The wave solver's adjoint writes every bar from the thread that owns it (no
 * atomics, nothing to zero): quantities shared by the two layers of an
 * interface are kept per interface and gathered by the layers.  Quotients by
 * rho, the volumes and the run constants go through one reciprocal each.
 * RES_ID 5: 632 -> 207 us per substage. */

/* apply, phase 1 (per layer and the interface below it): theta_v', Pi', w and
 * the TOA / surface copies of w; the bar of the interface's mean density
 * stays in db for phase 2 */
__global__ void ba_apply_state(VGrid vg, AState<double> so, const double *wl, const double *wr, AState<double> out,
                               AState<double> out_b, double *rn_b, double *rtn_b, double *db, AState<double> so_b,
                               double *wl_b, double *wr_b)
{
    const LayerPoint pt = layer_point(vg.nc);
    if (!pt.in) return;
    const int nc = vg.nc, nl = vg.nl, j = pt.l;
    const long long ns = (long long)nl * nc, m = ns - nc, b = pt.i;
    const double vg_b = vg.volume[b] * wl[WL_G * ns + b];
    const double rn = out.rho[b], rtn = out.rt[b], irn = 1.0 / rn;
    const double tpb = out_b.tp[b], epb = out_b.ep[b], t = div_rcp(tpb, rn, irn), v = epb * vg_b;
    rtn_b[b] = out_b.rt[b] + t + v;
    rn_b[b] = out_b.rho[b] - t * div_rcp(rtn, rn, irn);
    so_b.ep[b] += epb;
    so_b.rt[b] -= v;
    wl_b[WL_G * ns + b] = epb * vg.volume[b] * (rtn - so.rt[b]);
    if (j == 0) so_b.w[b] += out_b.w[b];
    if (j == nl - 1) {
        so_b.w[b + nc] += out_b.w[b + nc];
        return;
    }
    const long long wi = b + nc;
    const double wb = out_b.w[wi], q = div_rcp(wb, wr[WR_RIO * m + b], wr[WR_RRIO * m + b]);
    const double dint = 0.5 * (rn + out.rho[wi]);
    wr_b[WR_SOL * m + b] = 2.0 * div_rcp(q, vg.area_v[wi], vg.r_area_v[wi]);
    db[b] = -q * so.w[wi];
    so_b.w[wi] -= q * dint;
    wr_b[WR_RIO * m + b] = -q * out.w[wi];
}

/* apply, phase 2 (per layer and the interface below it): rho and rho theta_v
 * from the solution */
__global__ void ba_apply_rho(VGrid vg, double dt, const double *wr, const double *rn_b, const double *rtn_b,
                             const double *db, double *wl_b, double *wr_b)
{
    const LayerPoint pt = layer_point(vg.nc);
    if (!pt.in) return;
    const int nc = vg.nc, nl = vg.nl, j = pt.l;
    const long long ns = (long long)nl * nc, m = ns - nc, b = pt.i;
    const double here = j < nl - 1 ? db[b] : 0.0;
    const double rb = rn_b[b] + 0.5 * ((j > 0 ? db[b - nc] : 0.0) + here), rtb = rtn_b[b];
    wl_b[WL_REXP * ns + b] = rb;
    wl_b[WL_RTEXP * ns + b] = rtb;
    if (j == nl - 1) return;
    const long long lo = b + nc;
    const double rb1 = rn_b[lo] + 0.5 * (here + (j < nl - 2 ? db[lo] : 0.0));
    const double f0 = div_rcp(dt, vg.volume[b], vg.r_volume[b]), f1 = div_rcp(dt, vg.volume[lo], vg.r_volume[lo]);
    const double nb = rb * f0 - rb1 * f1, ntb = rtb * f0 - rtn_b[lo] * f1;
    wr_b[WR_SOL * m + b] += nb + wr[WR_TH * m + b] * ntb;
    wr_b[WR_TH * m + b] = wr[WR_SOL * m + b] * ntb;
}

/* transposed tridiagonal solve per column: lambda = A^-T xbar with xbar the
 * bar of the undamped solution; then rbar = lambda and the coefficient bars
 * -lambda x^T on the three diagonals.  NL > 0: the layer count is a
 * compile-time constant and the sweep stays in registers, so that the rows'
 * loads run ahead of the elimination (135 -> 43 us at RES_ID 5). */
template <int NL, int CAP>
__global__ void ba_thomas(int nc, int nl_arg, const double *dden, const double *r_dden, const double *wr, double *wr_b)
{
    const int i = (int)gtid();
    if (i >= nc) return;
    const int n = (NL > 0 ? NL : nl_arg) - 1;
    const long long m = (long long)n * nc;
    const double *cc = wr + WR_C * m, *dd = wr + WR_D * m, *ee = wr + WR_E * m, *x = wr + WR_X * m;
    double ep[NL > 0 ? NL : CAP], rp[NL > 0 ? NL : CAP];
#pragma unroll
    for (int j = 0; j < n; ++j) {
        const long long q = (long long)j * nc + i;
        const double xb = div_sweep(wr_b[WR_SOL * m + q], dden[q], r_dden[q]);
        const double sub = j > 0 ? ee[q - nc] : 0.0; /* (A^T)_{j,j-1} = e_{j-1} */
        const double den = j > 0 ? dd[q] - ep[j - 1] * sub : dd[q], inv = rcp_sweep(den);
        if (j < n - 1) ep[j] = div_sweep(cc[q], den, inv); /* (A^T)_{j,j+1} = c_j */
        rp[j] = div_sweep(j > 0 ? xb - rp[j - 1] * sub : xb, den, inv);
    }
    double lam_next = 0.0, x_next = 0.0;
#pragma unroll
    for (int j = n - 1; j >= 0; --j) {
        const long long q = (long long)j * nc + i;
        const double lam = (j == n - 1) ? rp[j] : rp[j] - ep[j] * lam_next, xj = x[q];
        wr_b[WR_R * m + q] = lam;
        wr_b[WR_D * m + q] = -lam * xj;
        if (j < n - 1) {
            wr_b[WR_E * m + q] = -lam * x_next;
            wr_b[WR_C * m + q] = -lam_next * xj;
        }
        lam_next = lam;
        x_next = xj;
    }
}

/* bars of the rows, per inner interface (BR_N arrays [L-1][Nc]): alpha, beta,
 * gamma of the layers above (0) and below (1), theta_v and rho at the
 * interface, the mean explicit density and the explicit Pi' and theta_v' */
enum { BR_A0, BR_A1, BR_B0, BR_B1, BR_G0, BR_G1, BR_TH, BR_RIE, BR_EP, BR_TP, BR_RIO, BR_N };

/* the rows (fa_waves_rows) per inner interface.  c_{j-1} and e_{j-1} read this
 * interface's theta_v and rho too: their share is formed here. */
__global__ void ba_waves_rows(VGrid vg, StepParams p, AState<double> so, const double *wl, const double *wr,
                              const double *wr_b, double *br, AState<double> so_b, double *st_w_b)
{
    const LayerPoint pt = layer_point(vg.nc);
    if (!pt.in) return;
    const int nc = vg.nc, nl = vg.nl, j = pt.l;
    const long long ns = (long long)nl * nc, n = ns - nc, q = pt.i;
    const long long b = q, lo = q + nc, wi = q + nc;
    const double dt = p.dt;
    const double *be = wl + WL_B * ns, *ga = wl + WL_G * ns, *rexp = wl + WL_REXP * ns;
    const double *epx = wl + WL_EPEXP * ns;
    const double r_rio = wr[WR_RRIO * n + q], th = wr[WR_TH * n + q];
    const double rho_ie = 0.5 * (rexp[b] + rexp[lo]);
    const double dz = vg.z_scalar[b] - vg.z_scalar[lo], ebg_b = vg.exner_bg[b], ebg_lo = vg.exner_bg[lo];
    const double dpi = ebg_b - ebg_lo, hdpi = 0.5 * dpi;
    const double wo = so.w[wi], rv_b = vg.r_volume[b], rv_lo = vg.r_volume[lo];
    const double b0 = be[b], b1 = be[lo], g0 = ga[b], g1 = ga[lo];
    const double db = wr_b[WR_D * n + q], rb = wr_b[WR_R * n + q];
    /* dz / K1 and dz / (K1 rho), K1 = w dt^2 c_p; dz / (2 K2), K2 = w dt c_p */
    const double dz_a = div_rcp(dz, p.rows_a, p.r_rows_a), dz_ar = dz_a * r_rio;
    const double dz_b = 0.5 * div_rcp(dz, p.rows_b, p.r_rows_b);
    double thb = wr_b[WR_TH * n + q], riob = wr_b[WR_RIO * n + q];
    /* d */
    const double dv = dt * 0.5 * (rv_lo - rv_b), geo = 2.0 * vg.r_area_v[wi] + wo * dv;
    const double hd = db * hdpi, dth2 = db * (th * th);
    thb += db * (hdpi * (b1 - b0) - 2.0 * th * (g0 + g1));
    double g1b = -dth2, a1b = hd, b1b = hd * th, g0b = -dth2, a0b = -hd, b0b = -b1b;
    riob += db * dz_ar * geo * r_rio;
    double wob = -db * dz_ar * dv;
    /* r */
    const double rie_r = rho_ie * r_rio, rz = rb * dz_ar * wo;
    wob -= rb * (dz_a + dz_a * rie_r);
    st_w_b[wi] -= rb * (dt * dz_a);
    thb += div_rcp(rb * (epx[b] - epx[lo]), dt, p.inv_dt);
    riob += rz * rie_r;
    if (j < nl - 2) {
        /* row j's c = th1 g1 th + H1 (a1 + b1 th) - ..., e = th g1 th1 - hdpi (a1 + b1 th1) + ... */
        const double th1 = wr[WR_TH * n + q + nc], H1 = 0.5 * (ebg_lo - vg.exner_bg[lo + nc]);
        const double cb = wr_b[WR_C * n + q], eb = wr_b[WR_E * n + q], r2 = rv_lo * r_rio;
        const double cH = cb * H1, eh = eb * hdpi, s = eb * dz_b * r2;
        thb += cb * (th1 * g1 + H1 * b1) + eb * g1 * th1;
        g1b += (cb + eb) * (th1 * th);
        a1b += cH - eh;
        b1b += cH * th - eh * th1;
        wob += s;
        riob -= s * wo * r_rio;
    }
    if (j > 0) {
        /* row j-1's c = th g0 th0 + hdpi (a0 + b0 th0) - wt / (V_b rho), and
         * its e = th0 g0 th - hdpi0 (a0 + b0 th) + ... */
        const double th0 = wr[WR_TH * n + q - nc], hdpi0 = 0.5 * (vg.exner_bg[b - nc] - ebg_b);
        const double cb = wr_b[WR_C * n + q - nc], eb = wr_b[WR_E * n + q - nc], s = cb * dz_b * (rv_b * r_rio);
        thb += (cb + eb) * (g0 * th0) - eb * (hdpi0 * b0);
        wob -= s;
        riob += s * wo * r_rio;
    }
    br[BR_A0 * n + q] = a0b;
    br[BR_A1 * n + q] = a1b;
    br[BR_B0 * n + q] = b0b;
    br[BR_B1 * n + q] = b1b;
    br[BR_G0 * n + q] = g0b;
    br[BR_G1 * n + q] = g1b;
    br[BR_TH * n + q] = thb;
    br[BR_RIE * n + q] = -rz;
    br[BR_EP * n + q] = div_rcp(rb * th, dt, p.inv_dt);
    br[BR_TP * n + q] = rb * p.half_inv_dt * dpi;
    br[BR_RIO * n + q] = riob;
    so_b.w[wi] += wob;
}

/* the per-layer predictors (fa_waves_layer), their bars gathered from the
 * interfaces above and below; at rk 0 sn is so and sn_b is so_b */
__global__ void ba_waves_layer(VGrid vg, double dt, int rk, AState<double> so, AState<double> sn, const double *st_rho,
                               const double *st_rt, const double *wl, const double *wl_b, const double *br,
                               AState<double> so_b, AState<double> sn_b, double *st_rho_b, double *st_rt_b)
{
    const LayerPoint pt = layer_point(vg.nc);
    if (!pt.in) return;
    const int nc = vg.nc, nl = vg.nl, j = pt.l;
    const long long ns = (long long)nl * nc, n = ns - nc, b = pt.i, u = b - nc;
    double ab = 0.0, bb = 0.0, gb = wl_b[WL_G * ns + b], thlb = 0.0, rexpb = 0.0, epxb = 0.0, tpxb = 0.0, ro_b = 0.0;
    if (j > 0) {
        ab = br[BR_A1 * n + u];
        bb = br[BR_B1 * n + u];
        gb += br[BR_G1 * n + u];
        thlb = br[BR_TH * n + u];
        rexpb = br[BR_RIE * n + u];
        epxb = -br[BR_EP * n + u];
        tpxb = br[BR_TP * n + u];
        ro_b = br[BR_RIO * n + u];
    }
    if (j < nl - 1) {
        ab += br[BR_A0 * n + b];
        bb += br[BR_B0 * n + b];
        gb += br[BR_G0 * n + b];
        thlb += br[BR_TH * n + b];
        rexpb += br[BR_RIE * n + b];
        epxb += br[BR_EP * n + b];
        tpxb += br[BR_TP * n + b];
        ro_b += br[BR_RIO * n + b];
    }
    thlb *= 0.5;
    ro_b *= 0.5;
    rexpb = 0.5 * rexpb + wl_b[WL_REXP * ns + b];
    const double rtxb = wl_b[WL_RTEXP * ns + b];
    const double vol = vg.volume[b], rv = vg.r_volume[b], dtv = dt * vol;
    const double alpha = wl[WL_A * ns + b], beta = wl[WL_B * ns + b], gam = wl[WL_G * ns + b];
    const double sr = st_rho[b], srt = st_rt[b], tv = tpxb * dtv, ev = epxb * dtv;
    /* tp_expl, ep_expl, rho_expl, rt_expl */
    so_b.tp[b] += tpxb;
    ab += tv * sr;
    bb += tv * srt;
    gb += ev * srt;
    const double sr_b = tv * alpha + dt * rexpb, srt_b = tv * beta + ev * gam + dt * rtxb;
    ro_b += rexpb;
    double rto_b = rtxb, epo_b = epxb, rn_b = 0.0, rtn_b = 0.0, epn_b = 0.0;
    const double ro = so.rho[b], rto = so.rt[b], pe = vg.exner_bg[b] + so.ep[b];
    const double iro = 1.0 / ro, irto = 1.0 / rto;
    const double rn = sn.rho[b], rtn = sn.rt[b], irn = rk == 0 ? iro : 1.0 / rn;
    /* thl = rt_n / rho_n */
    const double tq = thlb * irn;
    rtn_b += tq;
    rn_b -= tq * div_rcp(rtn, rn, irn);
    /* alpha, beta, gamma: over the volume, at rk 1 the mean of old and new */
    const double kg = R_D / C_D_V;
    const double w = rk == 0 ? 1.0 : 0.5;
    const double hab = div_rcp(w * ab, vol, rv), hbb = div_rcp(w * bb, vol, rv), hgb = div_rcp(w * gb, vol, rv);
    auto part = [&](double r, double ir, double rt, double irt, double pi, double &r_b, double &rt_b, double &e_b) {
        const double x = ir * ir, y = hgb * kg * irt;
        r_b += (2.0 * hab * (rt * ir) - hbb) * x;
        rt_b -= hab * x + y * pi * irt;
        e_b += y;
    };
    part(ro, iro, rto, irto, pe, ro_b, rto_b, epo_b);
    if (rk != 0) part(rn, irn, rtn, 1.0 / rtn, vg.exner_bg[b] + sn.ep[b], rn_b, rtn_b, epn_b);
    so_b.rho[b] += ro_b;
    so_b.rt[b] += rto_b;
    so_b.ep[b] += epo_b;
    sn_b.rho[b] += rn_b;
    sn_b.rt[b] += rtn_b;
    sn_b.ep[b] += epn_b;
    st_rho_b[b] += sr_b;
    st_rt_b[b] += srt_b;
}

}  // namespace
}  // namespace game
