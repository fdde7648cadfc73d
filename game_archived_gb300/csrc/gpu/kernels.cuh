/*
 * RKHEVI step kernels.
 *
 * Every device function restates one reference operator at one point and
 * keeps the reference's order of floating-point operations, so that the FP64
 * instantiation (compiled with --fmad=false) rounds like the reference C.
 * Horizontal operators are templated on R: double on the FP64 path, float on
 * the mixed path, where the prognostic state, the vertical solves and the
 * density/mass-flux divergence accumulation stay in double.
 *
 * Kernels of one RK substage (src/time_stepping/manage_rkhevi.c:48-97):
 *   k_cell_prepare      T, theta_v, moist phase-transition rates (once per step)
 *   k_tri_vort          vertical relative vorticity on triangles        (rk 1)
 *   k_edge_vort         rhombus / tangential potential vorticity, mass flux (rk 1)
 *   k_cell_kinetic      kinetic energy, vertical mass flux               (rk 1)
 *   k_momentum_h        pressure gradient + vorticity flux + KE gradient
 *                       -> horizontal tendency and wind update
 *   k_momentum_v        the same for w at the interfaces
 *   k_scalar_tend       mass / rho*theta_v flux divergences -> tendencies
 * The implicit vertical column solves (sound waves, tracer advection and
 * sedimentation) are in solvers.cuh.
 */
#pragma once

#include <cuda_runtime.h>

#include "devgrid.cuh"
#include "dfloat.cuh"
#include "numeric.cuh"

namespace game {
/* internal linkage: the FP64 and the mixed translation unit each compile
 * their own copy with their own contraction flags */
namespace {

template <typename R>
__device__ __forceinline__ R ipw_at(const HGrid<R> &g, int j, int l, int c)
{
    return g.ipw[((long long)j * g.nl + l) * g.nc + c];
}

/* vertical covariant gradient of a cell field at an inner interface k
 * (src/spatial_operators/gradient_operators.c:35-54) */
template <typename R, typename F>
__device__ __forceinline__ R grad_v(const HGrid<R> &g, const F *f, int k, int c)
{
    const long long i = (long long)k * g.nc + c;
    return div_tab(R(f[i - g.nc]) - R(f[i]), g.nd_v, g.r_nd_v, i);
}

/* Slopes and height differences are exactly 0 away from orography, and what
 * they multiply is left out there (tests on integers: no FP64 comparison): a
 * zero for finite values; a field that is infinite or NaN in a neighbouring
 * layer does not become a NaN through it.  ALL: nothing is left out (the
 * single operators, whose NaN are the reference's for any field). */
__device__ __forceinline__ bool zero_slope(double s) { return is_zero(s); }
__device__ __forceinline__ bool zero_slope(float s) { return s == 0.0f; }

/* horizontal gradient at edge e of layer l from the field and its vertical
 * gradients gv at the inner interfaces: grad_h's operations in its order */
__device__ __forceinline__ double grad_h_pre(const HGrid<double> &g, double f_to, double f_fr, const double *gv, int l,
                                             int e, int fr, int to)
{
    const long long le = (long long)l * g.ne + e;
    double out = div_tab(f_to - f_fr, g.nd_h, g.r_nd_h, le);
    if (l < g.nl - g.n_oro) return out;
    const double slope = g.slope_h[le];
    if (zero_slope(slope)) return out;
    const double *gl = gv + (long long)l * g.nc;
    double c = ipw_at(g, 6, l, fr) * gl[fr];
    c += ipw_at(g, 6, l, to) * gl[to];
    if (l < g.nl - 1) {
        c += ipw_at(g, 7, l, fr) * gl[g.nc + fr];
        c += ipw_at(g, 7, l, to) * gl[g.nc + to];
    }
    c = 0.5 * c;
    out += -slope * c;
    return out;
}

/* horizontal gradient at edge e of layer l, with the terrain-following
 * covariant -> contravariant correction in the orography layers
 * (gradient_operators.c:14-33, averaging.c:14-39 and :113-133) */
template <bool ALL = false, typename R, typename F>
__device__ __forceinline__ R grad_h(const HGrid<R> &g, const F *f, int l, int e)
{
    const int fr = g.from[e], to = g.to[e];
    const long long le = (long long)l * g.ne + e;
    R out = div_tab(R(f[(long long)l * g.nc + to]) - R(f[(long long)l * g.nc + fr]), g.nd_h, g.r_nd_h, le);
    if (l >= g.nl - g.n_oro) {
        /* a zero slope adds a zero */
        if (!ALL && zero_slope(g.slope_h[le])) return out;
        R c = ipw_at(g, 6, l, fr) * grad_v(g, f, l, fr);
        c += ipw_at(g, 6, l, to) * grad_v(g, f, l, to);
        if (l < g.nl - 1) {
            c += ipw_at(g, 7, l, fr) * grad_v(g, f, l + 1, fr);
            c += ipw_at(g, 7, l, to) * grad_v(g, f, l + 1, to);
        }
        c = R(0.5) * c;
        out += -g.slope_h[le] * c;
    }
    return out;
}

/* horizontal covariant wind component (averaging.c:97-111) */
template <bool ALL = false, typename R, typename F>
__device__ __forceinline__ R hor_covariant(const HGrid<R> &g, const F *u, const F *w, int l, int e)
{
    const long long le = (long long)l * g.ne + e;
    R r = R(u[le]);
    if (l >= g.nl - g.n_oro) {
        const R slope = g.slope_h[le];
        /* a zero slope adds a zero */
        if (!ALL && zero_slope(slope)) return r;
        const int fr = g.from[e], to = g.to[e];
        R c = ipw_at(g, 6, l, fr) * R(w[(long long)l * g.nc + fr]);
        c += ipw_at(g, 6, l, to) * R(w[(long long)l * g.nc + to]);
        if (l < g.nl - 1) {
            c += ipw_at(g, 7, l, fr) * R(w[(long long)(l + 1) * g.nc + fr]);
            c += ipw_at(g, 7, l, to) * R(w[(long long)(l + 1) * g.nc + to]);
        }
        c = R(0.5) * c;
        r += slope * c;
    }
    return r;
}

/* sum of all constituent densities (src/constituents/derived_quantities.c:83-95) */
__device__ __forceinline__ double density_total(const double *rho, int n_const, long long ns, long long i)
{
    double r = 0.0;
    for (int k = 0; k < n_const; ++k) r += rho[k * ns + i];
    return r;
}

/* ------------------------------------------------------ thermodynamics
 * src/constituents/dictionary.c (FP64 on both paths) */
/* t^3 and t^4 with the products' rounding errors carried along (TwoProd):
 * correctly rounded (tested), the reference's pow(t, n) to its last bit, at five
 * or six FP64 instructions instead of some 150 */
__device__ __forceinline__ double cube(double t)
{
    const double s = t * t, se = __fma_rn(t, t, -s), p = s * t;
    return p + __fma_rn(se, t, __fma_rn(s, t, -p));
}
__device__ __forceinline__ double fourth(double t)
{
    const double s = t * t, se = __fma_rn(t, t, -s), p = s * s;
    return p + __fma_rn(2.0 * s, se, __fma_rn(s, s, -p));
}

__device__ __forceinline__ double c_p_ice(double t)
{
    if (t > T_0) t = T_0;
    if (t < 20.0) t = 20.0;
    double q = div_rcp(t, 125.1, 1.0 / 125.1);
    double r = -2.0572 + 0.14644 * t + 0.06163 * t * exp(-(q * q));
    return div_rcp(r, M_V, 1.0 / M_V);
}

__device__ __forceinline__ double c_p_water(double t)
{
    double tc = t - T_0, r;
    if (tc >= 0.0) {
        if (tc > 35.0) tc = 35.0;
        double a = tc - 35.0;
        r = 0.9979 + 3.1e-6 * (a * a) + 3.8e-9 * fourth(a);
    } else {
        if (tc < -37.0) tc = -37.0;
        r = 1.000938 - 2.7052e-3 * tc - 2.3235e-5 * (tc * tc) + 4.3778e-6 * cube(tc) + 2.7136e-7 * fourth(tc);
    }
    return 4186.8 * r;
}

__device__ __forceinline__ double c_p_cond(int id, double t) { return (id % 2 == 0) ? c_p_ice(t) : c_p_water(t); }

__device__ __forceinline__ double enthalpy_evaporation(double t)
{
    double r;
    if (t < T_0) {
        if (t < 30.0) t = 30.0;
        r = 56579.0 - 42.212 * t + exp(0.1149 * (281.6 - t));
        r = div_rcp(r, M_V, 1.0 / M_V);
    } else {
        if (t > T_0 + 100.0) t = T_0 + 100.0;
        r = 3151378.0 - 2386.0 * t;
    }
    return r;
}

__device__ __forceinline__ double enthalpy_sublimation(double t)
{
    if (t < 30.0) t = 30.0;
    if (t > T_0) t = T_0;
    double q = div_rcp(t, 123.75, 1.0 / 123.75);
    double r = 46782.5 + 35.8925 * t - 0.07414 * (t * t) + 541.5 * exp(-(q * q));
    return div_rcp(r, M_V, 1.0 / M_V);
}

__device__ __forceinline__ double sat_pressure_water(double t)
{
    double tc = t - T_0, r;
    if (tc > 100.0) tc = 100.0;
    if (tc > 0.0) {
        r = exp(34.494 - 4924.99 / (tc + 237.1)) / pow(tc + 105.0, 1.57);
    } else {
        if (tc < -50.0) tc = -50.0;
        r = 6.107799961 + 4.436518521e-1 * tc + 1.428945805e-2 * (tc * tc) + 2.650648471e-4 * pow(tc, 3.0)
            + 3.031240396e-6 * pow(tc, 4.0) + 2.034080948e-8 * pow(tc, 5.0) + 6.136820929e-11 * pow(tc, 6.0);
        r = 100.0 * r;
    }
    return r;
}

__device__ __forceinline__ double sat_pressure_ice(double t)
{
    double tc = t - T_0;
    if (tc < -80.0) tc = -80.0;
    if (tc > 0.0) tc = 0.0;
    double a = tc + 868.0;
    return exp(43.494 - 6545.8 / (tc + 278.0)) / (a * a);
}

/* mass-weighted c_v (derived_quantities.c:97-115); cp_ice / cp_water are
 * c_p_cond of the even (ice) and odd (liquid) condensates at the cell's
 * temperature, evaluated once per step */
__device__ __forceinline__ double c_v_mass_weighted(const double *rho, int n_cond, int moist, long long ns,
                                                    long long i, double cp_ice, double cp_water)
{
    double r = 0.0;
    for (int k = 0; k < n_cond; ++k) r += rho[k * ns + i] * ((k % 2 == 0) ? cp_ice : cp_water);
    r += rho[n_cond * ns + i] * C_D_V;
    if (moist) r += rho[(n_cond + 1) * ns + i] * C_V_V;
    return r;
}

/* --------------------------------------------------- k_cell_prepare
 * temperature (derived_quantities.c:15-40) from state_old and, for the moist
 * build, phase-transition rates and heating (phase_trans.c:16-311).  Bound by
 * FP64 issue: the five exponentials are left; powers by products (cube,
 * fourth), quotients by shared reciprocals: 1292 -> 633 us at RES_ID 6 */
__global__ void k_cell_prepare(VGrid vg, StepParams p, DState so, double *temperature, double *pt_rates,
                               double *pt_heat, double *cp_ice_out, double *cp_water_out)
{
    const long long ns = (long long)vg.nl * vg.nc;
    const long long i = gtid();
    if (i >= ns) return;
    const int cond = p.n_cond;
    double T;
    if (!p.moist) {
        T = (vg.theta_v_bg[i] + so.theta_v_pert[i]) * (vg.exner_bg[i] + so.exner_pert[i]);
        temperature[i] = T;
        return;
    }
    const double *rho = so.rho;
    const double rg = rho[cond * ns + i], rv = rho[(cond + 1) * ns + i];
    T = (vg.theta_v_bg[i] + so.theta_v_pert[i]) * (vg.exner_bg[i] + so.exner_pert[i]);
    /* without vapour the divisor is 1 */
    if (!is_zero(rv)) T = T / (1.0 + rv / rg * (M_D / M_V - 1.0));
    temperature[i] = T;
    const double cpi = c_p_ice(T), cpw = c_p_water(T);
    cp_ice_out[i] = cpi;
    cp_water_out[i] = cpw;
    const double dt = p.dt, inv_dt = p.inv_dt;
    const double max_cloud_water = 0.2e-3;
    /* saturation pressure and the bracket of its derivative; each
     * transcendental and each reciprocal evaluated once, the quotients by
     * div_rcp: reused values are the numbers the reference recomputes */
    const bool warm = T >= T_0;
    double tc = T - T_0, sat0, bracket;
    if (warm) {
        if (tc > 100.0) tc = 100.0;
        const double x = tc + 237.1, rx = 1.0 / x;
        if (tc > 0.0) sat0 = exp(34.494 - div_rcp(4924.99, x, rx)) / pow(tc + 105.0, 1.57);
        else sat0 = sat_pressure_water(T);
        bracket = div_rcp(4924.99, x * x, rx * rx) - 1.57 / (tc + 105.0);
    } else {
        if (tc < -80.0) tc = -80.0;
        const double x = tc + 278.0, rx = 1.0 / x, a = tc + 868.0, ra = 1.0 / a;
        sat0 = div_rcp(exp(43.494 - div_rcp(6545.8, x, rx)), a * a, ra * ra);
        bracket = div_rcp(6545.8, x * x, rx * rx) - 2.0 * ra;
    }
    double wvp = rv * R_V * T;
    double dry = (rg - rv) * R_D * T;
    double air = dry + wvp;
    double ef = warm ? 1.00071 * exp(0.000000045 * air) : 0.99882 * exp(0.00000008 * air);
    double sat = ef * sat0;
    const double dsat = sat0 * bracket;
    const double h_evap = enthalpy_evaporation(T), h_subl = enthalpy_sublimation(T);
    const double h_melt = h_subl - h_evap;
    const double cw_ice = rho[2 * ns + i], cw_liq = rho[3 * ns + i];
    const double cv = c_v_mass_weighted(rho, cond, 1, ns, i, cpi, cpw), r_cv = 1.0 / cv;
    const double pth = warm ? h_evap : h_subl;
    const double a = div_rcp(-R_V * pth, cv, r_cv), r_a = 1.0 / a;
    const double b = R_V * T - div_rcp(R_V * rv * pth, cv, r_cv) + div_rcp(ef * dsat * pth, cv, r_cv);
    const double cc = wvp - sat;
    const double pp = div_rcp(b, a, r_a);
    const double q = div_rcp(cc, a, r_a);
    const double diff = -0.5 * pp - sqrt(0.25 * (pp * pp) - q);
    auto per_dt = [&](double x) { return div_rcp(x, dt, inv_dt); };
    double r0, r1, r2, r3, r4, heat;
    /* warm: ice melts, liquid water evaporates or vapour condenses to it;
     * cold: the other way round */
    const double ptd = sat >= wvp ? fmin(warm ? cw_liq : cw_ice, diff) : diff;
    r4 = per_dt(ptd);
    if (warm) {
        r2 = per_dt(-cw_ice);
        r3 = per_dt(cw_ice) - r4;
        heat = r2 * h_melt - per_dt(ptd * h_evap);
    } else {
        r3 = per_dt(-cw_liq);
        r2 = per_dt(cw_liq) - r4;
        heat = -r3 * h_melt - per_dt(ptd * h_subl);
    }
    r0 = 0.0;
    r1 = 0.0;
    if (T < T_0) {
        r0 = div_rcp(fmax(cw_ice - max_cloud_water * rho[4 * ns + i], 0.0), 1000.0, 1.0 / 1000.0);
        r2 -= r0;
    } else if (T >= T_0) {
        r1 = div_rcp(fmax(cw_liq - max_cloud_water * rho[4 * ns + i], 0.0), 1000.0, 1.0 / 1000.0);
        r3 -= r1;
    }
    if (T >= T_0 && rho[i] > 0.0) {
        r0 = per_dt(-rho[i]);
        r1 -= r0;
        heat += r0 * h_melt;
    }
    if (T < T_0 && rho[ns + i] > 0.0) {
        r1 = per_dt(-rho[ns + i]);
        r0 -= r1;
        heat += -r1 * h_melt;
    }
    pt_rates[i] = r0;
    pt_rates[ns + i] = r1;
    pt_rates[2 * ns + i] = r2;
    pt_rates[3 * ns + i] = r3;
    pt_rates[4 * ns + i] = r4;
    pt_heat[i] = heat;
}

/* ------------------------------------------------ k_cell_prepare_f32
 * the same diagnostics and phase-transition rates in FP32 (mixed path).  The
 * condensation quadratic's root -p/2 - sqrt(p^2/4 - q) is evaluated as
 * q / (-p/2 + sqrt(p^2/4 - q)) when p < 0, the algebraically identical form
 * without cancellation, which FP32 needs. */
__device__ __forceinline__ float c_p_ice_f(float t)
{
    if (t > float(T_0)) t = float(T_0);
    if (t < 20.f) t = 20.f;
    const float q = t / 125.1f;
    return (-2.0572f + 0.14644f * t + 0.06163f * t * expf(-(q * q))) / float(M_V);
}
__device__ __forceinline__ float c_p_water_f(float t)
{
    float tc = t - float(T_0), r;
    if (tc >= 0.f) {
        if (tc > 35.f) tc = 35.f;
        const float a = tc - 35.f, a2 = a * a;
        r = 0.9979f + 3.1e-6f * a2 + 3.8e-9f * (a2 * a2);
    } else {
        if (tc < -37.f) tc = -37.f;
        const float t2 = tc * tc;
        r = 1.000938f - 2.7052e-3f * tc - 2.3235e-5f * t2 + 4.3778e-6f * (t2 * tc) + 2.7136e-7f * (t2 * t2);
    }
    return 4186.8f * r;
}
__device__ __forceinline__ float enthalpy_evaporation_f(float t)
{
    if (t < float(T_0)) {
        if (t < 30.f) t = 30.f;
        return (56579.0f - 42.212f * t + expf(0.1149f * (281.6f - t))) / float(M_V);
    }
    if (t > float(T_0) + 100.f) t = float(T_0) + 100.f;
    return 3151378.0f - 2386.0f * t;
}
__device__ __forceinline__ float enthalpy_sublimation_f(float t)
{
    if (t < 30.f) t = 30.f;
    if (t > float(T_0)) t = float(T_0);
    const float q = t / 123.75f;
    return (46782.5f + 35.8925f * t - 0.07414f * (t * t) + 541.5f * expf(-(q * q))) / float(M_V);
}

__global__ void k_cell_prepare_f32(VGrid vg, StepParams p, DState so, double *temperature, double *pt_rates,
                                   double *pt_heat, double *cp_ice_out, double *cp_water_out, float *cp32_ice,
                                   float *cp32_water)
{
    const long long ns = (long long)vg.nl * vg.nc;
    const long long i = gtid();
    if (i >= ns) return;
    const int cond = p.n_cond;
    const double *rho = so.rho;
    const float th = to_float(vg.theta_v_bg[i] + so.theta_v_pert[i]), pi = to_float(vg.exner_bg[i] + so.exner_pert[i]);
    if (!p.moist) {
        temperature[i] = to_double(th) * to_double(pi);
        return;
    }
    float r[6];
    for (int k = 0; k < 6; ++k) r[k] = to_float(rho[k * ns + i]);
    const float rv = r[cond + 1], rg = r[cond];
    const float T = th * pi / (1.f + rv / rg * float(M_D / M_V - 1.0));
    temperature[i] = to_double(T);
    const float cpi = c_p_ice_f(T), cpw = c_p_water_f(T);
    cp_ice_out[i] = to_double(cpi);
    cp_water_out[i] = to_double(cpw);
    cp32_ice[i] = cpi;
    cp32_water[i] = cpw;
    const float dt = float(p.dt), T0 = float(T_0);
    const bool warm = T >= T0;
    float tc = T - T0, sat0, dsat_fac;
    if (warm) {
        float tw = tc > 100.f ? 100.f : tc;
        if (tw > 0.f) {
            sat0 = expf(34.494f - 4924.99f / (tw + 237.1f)) / powf(tw + 105.0f, 1.57f);
        } else {
            const float t2 = tw * tw;
            sat0 = 100.f * (6.107799961f + 4.436518521e-1f * tw + 1.428945805e-2f * t2 + 2.650648471e-4f * t2 * tw
                            + 3.031240396e-6f * t2 * t2 + 2.034080948e-8f * t2 * t2 * tw
                            + 6.136820929e-11f * t2 * t2 * t2);
        }
        float td = tc > 100.f ? 100.f : (tc < 0.f ? 0.f : tc);
        const float q0 = td + 237.1f;
        dsat_fac = 4924.99f / (q0 * q0) - 1.57f / (td + 105.0f);
    } else {
        float ti = tc < -80.f ? -80.f : (tc > 0.f ? 0.f : tc);
        const float a = ti + 868.0f;
        sat0 = expf(43.494f - 6545.8f / (ti + 278.0f)) / (a * a);
        const float q0 = ti + 278.0f;
        dsat_fac = 6545.8f / (q0 * q0) - 2.0f / (ti + 868.0f);
    }
    const float wvp = rv * float(R_V) * T;
    const float air = (rg - rv) * float(R_D) * T + wvp;
    const float ef = warm ? 1.00071f * expf(0.000000045f * air) : 0.99882f * expf(0.00000008f * air);
    const float sat = ef * sat0;
    const float h_evap = enthalpy_evaporation_f(T), h_subl = enthalpy_sublimation_f(T), h_melt = h_subl - h_evap;
    float cv = 0.f;
    for (int k = 0; k < cond; ++k) cv += r[k] * ((k % 2 == 0) ? cpi : cpw);
    cv += rg * float(C_D_V) + rv * float(C_V_V);
    const float pth = warm ? h_evap : h_subl;
    const float a = -float(R_V) * pth / cv;
    const float b = float(R_V) * T - float(R_V) * rv * pth / cv + ef * (sat0 * dsat_fac) * pth / cv;
    const float pp = b / a, q = (wvp - sat) / a;
    const float sq = sqrtf(0.25f * (pp * pp) - q);
    const float diff = pp < 0.f ? q / (-0.5f * pp + sq) : -0.5f * pp - sq;
    float r0, r1, r2, r3, r4, heat;
    if (sat >= wvp) {
        if (warm) {
            r2 = -r[2] / dt;
            const float ptd = fminf(r[3], diff);
            r4 = ptd / dt;
            r3 = r[2] / dt - ptd / dt;
            heat = r2 * h_melt - ptd * h_evap / dt;
        } else {
            r3 = -r[3] / dt;
            const float ptd = fminf(r[2], diff);
            r4 = ptd / dt;
            r2 = r[3] / dt - ptd / dt;
            heat = -r3 * h_melt - ptd * h_subl / dt;
        }
    } else {
        if (warm) {
            r2 = -r[2] / dt;
            r4 = diff / dt;
            r3 = r[2] / dt - diff / dt;
            heat = r2 * h_melt - diff * h_evap / dt;
        } else {
            r3 = -r[3] / dt;
            r4 = diff / dt;
            r2 = r[3] / dt - diff / dt;
            heat = -r3 * h_melt - diff * h_subl / dt;
        }
    }
    r0 = 0.f;
    r1 = 0.f;
    const float max_cloud_water = 0.2e-3f;
    if (!warm) {
        r0 = fmaxf(r[2] - max_cloud_water * r[4], 0.f) / 1000.f;
        r2 -= r0;
    } else {
        r1 = fmaxf(r[3] - max_cloud_water * r[4], 0.f) / 1000.f;
        r3 -= r1;
    }
    if (warm && r[0] > 0.f) {
        r0 = -r[0] / dt;
        r1 -= r0;
        heat += r0 * h_melt;
    }
    if (!warm && r[1] > 0.f) {
        r1 = -r[1] / dt;
        r0 -= r1;
        heat += -r1 * h_melt;
    }
    /* widened by integer operations (to_double): the FP64 pipe was this
     * kernel's bound */
    pt_rates[i] = to_double(r0);
    pt_rates[ns + i] = to_double(r1);
    pt_rates[2 * ns + i] = to_double(r2);
    pt_rates[3 * ns + i] = to_double(r3);
    pt_rates[4 * ns + i] = to_double(r4);
    pt_heat[i] = to_double(heat);
}

/* FP32 shadow of the state at the start of a mixed step.  Each thread
 * converts the pairs 2i, 2i + 1 of every field with one 16-byte load and one
 * 8-byte store (every field length is even: 10 * 4^RES_ID + 2 cells, 30 *
 * 4^RES_ID edges, so every field of the mirror and of the shadow starts on
 * an even element), rounding with to_float (the conversion instruction's
 * bits, on the integer pipe instead of the FP64 pipe). */
__device__ __forceinline__ void shadow_pair(const double *src, float *dst, long long j)
{
    const double2 v = reinterpret_cast<const double2 *>(src)[j];
    reinterpret_cast<float2 *>(dst)[j] = make_float2(to_float(v.x), to_float(v.y));
}
__global__ void k_make_shadow(long long n_rho, long long ns, long long nw, long long nu, DState s, Shadow sh)
{
    const long long j = gtid();
    if (2 * j < n_rho) shadow_pair(s.rho, sh.rho, j);
    if (2 * j < ns) {
        shadow_pair(s.rhotheta_v, sh.rhotheta_v, j);
        shadow_pair(s.theta_v_pert, sh.theta_v_pert, j);
        shadow_pair(s.exner_pert, sh.exner_pert, j);
    }
    if (2 * j < nw) shadow_pair(s.w, sh.w, j);
    if (2 * j < nu) shadow_pair(s.u, sh.u, j);
}

/* ------------------------------------------------------- k_tri_vort
 * vertical relative vorticity on triangles (vorticities.c:167-222) */
template <typename R, bool ALL = false>
__global__ void __launch_bounds__(256, sizeof(R) == sizeof(float) ? 8 : 1) k_tri_vort(HGrid<R> g, const R *u, R *tri_vort)
{
    const LayerPoint pt_ = layer_point(g.nt);
    if (!pt_.in) return;
    const long long n = (long long)g.nl * g.nt, i = pt_.i;
    const int l = pt_.l, t = pt_.x;
    R acc = R(0);
    if constexpr (sizeof(R) == sizeof(double)) {
        /* FP64 issue bounds this kernel: the circulation weights come from a
         * table and the vertical shear's denominator from its reciprocal, a
         * third of the FP64 instructions (three divisions and two products
         * less per edge) for three more streamed words: 96 -> 41 us at
         * RES_ID 5 with the mountain, 345 -> 100 us at RES_ID 6 flat */
        for (int j = 0; j < 3; ++j) {
            const int e = g.vort_i[j * g.nt + t];
            const long long le = (long long)l * g.ne + e;
            double vel = u[le];
            if (l >= g.nl - g.n_oro) {
                const double zh = g.z_h[le], dz = g.dual_z_t[i] - zh;
                if (ALL || !is_zero(dz)) {
                    const bool above = __double_as_longlong(dz) > 0 || l == g.nl - 1;
                    const long long lo_e = above ? le - g.ne : le + g.ne;
                    const double r = above ? -g.r_dz_h[le] : g.r_dz_h[le + g.ne];
                    vel += dz * div_rcp(vel - u[lo_e], zh - g.z_h[lo_e], r);
                }
            }
            acc += g.tri_circ[j * n + i] * vel;
        }
        tri_vort[i] = div_tab(acc, g.dual_area_t, g.r_dual_area_t, i);
        return;
    }
    for (int j = 0; j < 3; ++j) {
        const int e = g.vort_i[j * g.nt + t];
        const long long le = (long long)l * g.ne + e;
        R vel = u[le];
        R rescale = R(1);
        if (l >= g.nl - g.n_oro) {
            const R zt = g.dual_z_t[i];
            rescale = (g.radius + zt) / (g.radius + g.z_h[le]);
            R dz = zt - g.z_h[le];
            int lo;
            if (dz > R(0)) lo = l - 1;
            else if (l == g.nl - 1) lo = l - 1;
            else lo = l + 1;
            const long long lo_e = (long long)lo * g.ne + e;
            R vgrad = (u[le] - u[lo_e]) / (g.z_h[le] - g.z_h[lo_e]);
            vel += dz * vgrad;
        }
        acc += rescale * g.nd_h[le] * R(g.vort_s[j * g.nt + t]) * vel;
    }
    tri_vort[i] = acc / g.dual_area_t[i];
}

/* tangential relative vorticity at level k, edge e (vorticities.c:104-165) */
template <bool ALL = false, typename R>
__device__ __forceinline__ R rel_vort_tangential(const HGrid<R> &g, const R *u, const R *w, int k, int e)
{
    const int nl = g.nl;
    if (k == 0) k = 1; /* no vertical shear of the tangential vorticity at the TOA */
    const long long ke = (long long)k * g.ne + e;
    R inv_area;
    if constexpr (sizeof(R) == sizeof(double)) inv_area = g.r_dual_area_h[ke];
    else inv_area = R(1) / g.dual_area_h[ke];
    if (k == nl) {
        R c2 = hor_covariant<ALL>(g, u, w, k - 1, e);
        return inv_area * g.nd_h[(long long)(k - 1) * g.ne + e] * c2;
    }
    const int fr = g.from[e], to = g.to[e];
    R c0 = hor_covariant<ALL>(g, u, w, k, e);
    R c2 = hor_covariant<ALL>(g, u, w, k - 1, e);
    return inv_area * (-g.nd_h[(long long)k * g.ne + e] * c0
                       + g.nd_v[(long long)k * g.nc + fr] * w[(long long)k * g.nc + fr]
                       + g.nd_h[(long long)(k - 1) * g.ne + e] * c2
                       - g.nd_v[(long long)k * g.nc + to] * w[(long long)k * g.nc + to]);
}

/* --------------------------------------------------------- k_edge_vort
 * potential vorticity (vorticities.c:18-85) and the horizontal mass flux
 * density (multiplications.c:45-66), one thread per (edge, level 0..L) */
template <typename R>
__global__ void __launch_bounds__(256, sizeof(R) == sizeof(float) ? 8 : 1) k_edge_vort(HGrid<R> g, const R *u, const R *w, const R *rho_gas, const R *tri_vort, R *zh, R *zv,
                            R *flux_h)
{
    const LayerPoint pt_ = layer_point(g.ne);
    if (!pt_.in) return;
    const long long i = pt_.i;
    const int k = pt_.l, e = pt_.x;
    const int nl = g.nl, nc = g.nc, ne = g.ne;
    const int fr = g.from[e], to = g.to[e];
    /* tangential component at level k */
    {
        R rel = rel_vort_tangential(g, u, w, k, e);
        R pv = rel + g.f_vec[e];
        R dens;
        if (k == 0) {
            R top = R(0.5) * (rho_gas[fr] + rho_gas[to]);
            R below = R(0.5) * (rho_gas[nc + fr] + rho_gas[nc + to]);
            dens = top + (top - below) / g.pvz[ne + e] * g.pvz[e];
        } else if (k == nl) {
            long long a = (long long)(nl - 1) * nc, b = (long long)(nl - 2) * nc;
            R low = R(0.5) * (rho_gas[a + fr] + rho_gas[a + to]);
            R above = R(0.5) * (rho_gas[b + fr] + rho_gas[b + to]);
            dens = low + (above - low) / g.pvz[3 * (long long)ne + e] * g.pvz[2 * (long long)ne + e];
        } else {
            long long uf = (long long)(k - 1) * nc + fr, ut = (long long)(k - 1) * nc + to;
            dens = R(0.25) * (rho_gas[uf] + rho_gas[ut] + rho_gas[uf + nc] + rho_gas[ut + nc]);
        }
        zh[i] = pv / dens;
    }
    if (k < nl) {
        const long long le = (long long)k * ne + e;
        /* rhombus: area-weighted mean of the two triangles */
        const int tf = g.dual_from[e], tt = g.dual_to[e];
        const long long kt = (long long)k * g.nt;
        R af = g.dual_area_t[kt + tf], at = g.dual_area_t[kt + tt];
        R rel = af * tri_vort[kt + tf] + at * tri_vort[kt + tt];
        if constexpr (sizeof(R) == sizeof(double)) rel = div_tab(rel, g.rhombus_area, g.r_rhombus_area, le);
        else rel = rel / (af + at);
        R pv = rel + g.f_vec[ne + e];
        R dens = R(0);
        for (int j = 0; j < 4; ++j)
            dens += g.rhombi_w[j * (long long)ne + e] * rho_gas[(long long)k * nc + g.rhombi_i[j * (long long)ne + e]];
        zv[le] = pv / dens;
        /* mass flux density */
        R sv = R(0.5) * (rho_gas[(long long)k * nc + to] + rho_gas[(long long)k * nc + fr]);
        flux_h[le] = sv * u[le];
    }
}

/* ------------------------------------------------------ k_cell_kinetic
 * kinetic energy v^2 (inner_product.c:13-43) at (cell, layer) and the vertical
 * mass flux density (multiplications.c:98-117) at the inner interfaces */
template <typename R>
__global__ void k_cell_kinetic(HGrid<R> g, const R *u, const R *w, const R *rho_gas, R *v2, R *flux_v)
{
    const long long ns = (long long)g.nl * g.nc;
    const LayerPoint pt_ = layer_point(g.nc);
    if (!pt_.in) return;
    const long long i = pt_.i;
    const int l = pt_.l, c = pt_.x;
    const int n_edges = c < N_PENT ? 5 : 6;
    R acc = R(0);
    for (int j = 0; j < n_edges; ++j) {
        R ue = u[(long long)l * g.ne + g.adj[j * g.nc + c]];
        acc += ipw_at(g, j, l, c) * ue * ue;
    }
    R wu = w[i], wl = w[i + g.nc];
    acc += ipw_at(g, 6, l, c) * wu * wu;
    acc += ipw_at(g, 7, l, c) * wl * wl;
    v2[i] = acc;
    if (l >= 1) {
        R sv = R(0.5) * (rho_gas[i - g.nc] + rho_gas[i]);
        flux_v[i] = sv * wu;
    }
}

/* x / 2; on the FP64 path without an FP64 instruction (exact, so where a
 * product takes the factor does not change it) */
__device__ __forceinline__ float halved(float x) { return 0.5f * x; }
__device__ __forceinline__ double halved(double x) { return half_of(x); }

/* modified TRSK sum of the vorticity flux at edge e of layer l
 * (vorticity_flux.c:35-113) */
template <typename R>
__device__ __forceinline__ R trsk_sum(const HGrid<R> &g, const R *flux_h, const R *zv, int l, int e)
{
    const long long ne = g.ne;
    const R *mf = flux_h + (long long)l * ne;
    const R *pv = zv + (long long)l * ne;
    const int fr = g.from[e], to = g.to[e];
    R out = R(0);
    /* the middle edge of each side counts with the mean of two vorticities */
    auto mean_term = [&](int j) {
        if constexpr (sizeof(R) == sizeof(double))
            return half_of(g.trsk_w[j * ne + e]) * mf[g.trsk_i[j * ne + e]] * (pv[g.trsk_m[j * ne + e]] + pv[e]);
        else
            return g.trsk_w[j * ne + e] * mf[g.trsk_i[j * ne + e]] * R(0.5) * (pv[g.trsk_m[j * ne + e]] + pv[e]);
    };
    if (fr < N_PENT) {
        for (int j = 0; j < 4; ++j)
            out += g.trsk_w[j * ne + e] * mf[g.trsk_i[j * ne + e]] * pv[g.trsk_m[j * ne + e]];
    } else {
        for (int j = 0; j < 5; ++j) {
            if (j == 2) out += mean_term(j);
            else out += g.trsk_w[j * ne + e] * mf[g.trsk_i[j * ne + e]] * pv[g.trsk_m[j * ne + e]];
        }
    }
    if (to < N_PENT) {
        for (int j = 5; j < 9; ++j)
            out += g.trsk_w[j * ne + e] * mf[g.trsk_i[j * ne + e]] * pv[g.trsk_m[j * ne + e]];
    } else {
        for (int j = 5; j < 10; ++j) {
            if (j == 7) out += mean_term(j);
            else out += g.trsk_w[j * ne + e] * mf[g.trsk_i[j * ne + e]] * pv[g.trsk_m[j * ne + e]];
        }
    }
    return out;
}

/* modified TRSK vorticity flux at edge e of layer l (vorticity_flux.c:35-137) */
template <typename R>
__device__ __forceinline__ R vorticity_flux_h(const HGrid<R> &g, const R *flux_h, const R *flux_v, const R *zh,
                                              const R *zv, int l, int e)
{
    const long long ne = g.ne;
    const int fr = g.from[e], to = g.to[e];
    R out = trsk_sum(g, flux_h, zv, l, e);
    const R zt = zh[(long long)l * ne + e], zb = zh[(long long)(l + 1) * ne + e];
    const long long nc = g.nc;
    out -= halved(ipw_at(g, 6, l, fr)) * flux_v[l * nc + fr] * zt;
    out -= halved(ipw_at(g, 6, l, to)) * flux_v[l * nc + to] * zt;
    out -= halved(ipw_at(g, 7, l, fr)) * flux_v[(l + 1) * nc + fr] * zb;
    out -= halved(ipw_at(g, 7, l, to)) * flux_v[(l + 1) * nc + to] * zb;
    return out;
}

/* What an edge's horizontal momentum reads of its two cells' levels, formed
 * once per level instead of by each of the cell's six edges (FP64 path): the
 * vertical gradient of v^2 at the inner interfaces, and the vertical mass
 * flux times half the inner-product weight of the layer below (hi) and above
 * (lo) the level, the factors of vorticity_flux.c:115-137. */
__global__ void k_level_terms(HGrid<double> g, const double *v2, const double *flux_v, double *grad_v2, double *q_hi,
                              double *q_lo)
{
    const LayerPoint p = layer_point(g.nc);
    if (!p.in) return;
    const int k = p.l, c = p.x;
    const double f = flux_v[p.i];
    if (k > 0 && k < g.nl) grad_v2[p.i] = grad_v(g, v2, k, c);
    if (k < g.nl) q_hi[p.i] = half_of(ipw_at(g, 6, k, c)) * f;
    if (k > 0) q_lo[p.i] = half_of(ipw_at(g, 7, k - 1, c)) * f;
}

/* vorticity_flux_h from them */
__device__ __forceinline__ double vorticity_flux_levels(const HGrid<double> &g, const double *flux_h, const double *q_hi,
                                                        const double *q_lo, const double *zh, const double *zv, int l,
                                                        int e)
{
    const int fr = g.from[e], to = g.to[e];
    const long long nc = g.nc, lc = l * nc;
    double out = trsk_sum(g, flux_h, zv, l, e);
    const double zt = zh[(long long)l * g.ne + e], zb = zh[(long long)(l + 1) * g.ne + e];
    out -= q_hi[lc + fr] * zt;
    out -= q_hi[lc + to] * zt;
    out -= q_lo[lc + nc + fr] * zb;
    out -= q_lo[lc + nc + to] * zb;
    return out;
}

/* sum of all constituent densities in R (derived_quantities.c:83-95) */
template <typename R>
__device__ __forceinline__ R density_total_r(const R *rho, int n_const, long long ns, long long i)
{
    R r = R(0);
    for (int k = 0; k < n_const; ++k) r += rho[k * ns + i];
    return r;
}

/* decelerated pressure-gradient sum nl + l at edge e, layer l
 * (manage_pressure_gradient.c:17-72) */
template <typename R>
__device__ __forceinline__ void pgrad_h_parts(const HGrid<R> &g, const StepParams &p, const SView<R> &s, int l, int e,
                                              R &nl, R &l_term)
{
    const long long ns = (long long)g.nl * g.nc;
    const int fr = g.from[e], to = g.to[e];
    const long long cf = (long long)l * g.nc + fr, ct = (long long)l * g.nc + to;
    const R cdp = R(C_D_P);
    nl = grad_h<true>(g, s.exner_pert, l, e);
    R s_to = cdp * (g.theta_v_bg[ct] + s.theta_v_pert[ct]), s_fr = cdp * (g.theta_v_bg[cf] + s.theta_v_pert[cf]);
    nl = (R(0.5) * (s_to + s_fr)) * nl;
    l_term = (R(0.5) * (cdp * s.theta_v_pert[ct] + cdp * s.theta_v_pert[cf])) * g.exner_bg_grad_h[(long long)l * g.ne + e];
    R d_to = s.rho[p.n_cond * ns + ct] / density_total_r(s.rho, p.n_const, ns, ct);
    R d_fr = s.rho[p.n_cond * ns + cf] / density_total_r(s.rho, p.n_const, ns, cf);
    R dec = R(0.5) * (d_to + d_fr);
    nl = dec * nl;
    l_term = dec * l_term;
}

/* the same at the inner interface k of cell c */
template <typename R>
__device__ __forceinline__ void pgrad_v_parts(const HGrid<R> &g, const StepParams &p, const SView<R> &s, int k, int c,
                                              R &nl, R &l_term)
{
    const long long ns = (long long)g.nl * g.nc;
    const long long up = (long long)(k - 1) * g.nc + c, lo = (long long)k * g.nc + c;
    const R cdp = R(C_D_P);
    nl = grad_v(g, s.exner_pert, k, c);
    R s_up = cdp * (g.theta_v_bg[up] + s.theta_v_pert[up]), s_lo = cdp * (g.theta_v_bg[lo] + s.theta_v_pert[lo]);
    nl = (R(0.5) * (s_up + s_lo)) * nl;
    l_term = (R(0.5) * (cdp * s.theta_v_pert[up] + cdp * s.theta_v_pert[lo])) * g.exner_bg_grad_v[(long long)k * g.nc + c];
    R d_up = s.rho[p.n_cond * ns + up] / density_total_r(s.rho, p.n_const, ns, up);
    R d_lo = s.rho[p.n_cond * ns + lo] / density_total_r(s.rho, p.n_const, ns, lo);
    R dec = R(0.5) * (d_up + d_lo);
    nl = dec * nl;
    l_term = dec * l_term;
}

/* Mixed path: the cell factors of the pressure gradient at the step start,
 * one float4 per (layer, cell): x = Pi', y = c_p (theta_v_bg + theta_v'),
 * z = c_p theta_v', w = rho_gas / (sum of all densities) -- the float
 * expressions of pgrad_h_parts / pgrad_v_parts, so that the first
 * substage's gradients gather two float4 per edge (or interface) instead of
 * some twenty scalars.  Read from the FP32 shadow of state_new, which the
 * first substage's pressure gradient reads.  Also the first substage's
 * theta_v (k_theta) and the flags of the constituents each layer holds. */
__global__ void k_pg_cells(HGrid<float> g, StepParams p, SView<float> s, float4 *pc, float *theta,
                           Present present)
{
    const LayerPoint pt = layer_point(g.nc);
    const long long ns = (long long)g.nl * g.nc, i = pt.i;
    int held = 0; /* constituents with a density here */
    if (pt.in) {
        const float cdp = float(C_D_P);
        const float tp = s.theta_v_pert[i];
        pc[i] = make_float4(s.exner_pert[i], cdp * (g.theta_v_bg[i] + tp), cdp * tp,
                            s.rho[p.n_cond * ns + i] / density_total_r(s.rho, p.n_const, ns, i));
        theta[i] = s.rhotheta_v[i] / s.rho[p.n_cond * ns + i];
        for (int k = 0; k < p.n_const; ++k) held |= (s.rho[k * ns + i] != 0.f) << k;
    }
    if (p.n_const == 1) return;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) held |= __shfl_xor_sync(0xffffffffu, held, d);
    __shared__ int any;
    if (threadIdx.x == 0) any = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && held) atomicOr(&any, held);
    __syncthreads();
    if (threadIdx.x == 0) {
        int *row = present.by_layer + pt.l;
        if (any & ~*(volatile int *)row) atomicOr(row, any);
    }
}

/* FP64 path: the same cell factors in double with the operations of
 * pgrad_h_parts / pgrad_v_parts (the dry build's density ratio is rho / rho =
 * 1 and is left out), the vertical gradient of Pi' at the interface above
 * the cell, and theta_v.  Formed once per cell instead of once per edge and
 * interface that reads it (up to eight times). */
__global__ void k_pg_cells64(HGrid<double> g, StepParams p, SView<double> s, Quad *pc, double *grad_pi, double *theta)
{
    const LayerPoint pt = layer_point(g.nc);
    if (!pt.in) return;
    const long long ns = (long long)g.nl * g.nc, i = pt.i;
    const double cdp = C_D_P, tp = s.theta_v_pert[i];
    pc[i] = Quad{s.exner_pert[i], cdp * (g.theta_v_bg[i] + tp), cdp * tp,
                 p.n_const > 1 ? s.rho[p.n_cond * ns + i] / density_total_r(s.rho, p.n_const, ns, i) : 1.0};
    if (pt.l > 0) grad_pi[i] = grad_v(g, s.exner_pert, pt.l, pt.x);
    theta[i] = s.rhotheta_v[i] / s.rho[p.n_cond * ns + i];
}

__device__ __forceinline__ double pgrad_h_cells(const HGrid<double> &g, const Quad *pc, const double *grad_pi, int l,
                                                int e, bool dry)
{
    const int fr = g.from[e], to = g.to[e];
    const Quad a = pc[(long long)l * g.nc + fr], b = pc[(long long)l * g.nc + to];
    double nl = grad_h_pre(g, b.x, a.x, grad_pi, l, e, fr, to);
    nl = (0.5 * (b.y + a.y)) * nl;
    double l_term = (0.5 * (b.z + a.z)) * g.exner_bg_grad_h[(long long)l * g.ne + e];
    if (!dry) {
        const double dec = 0.5 * (b.w + a.w);
        nl = dec * nl;
        l_term = dec * l_term;
    }
    return nl + l_term;
}

/* u, d: the factors of the cells above and below the interface i */
__device__ __forceinline__ double pgrad_v_cells(const HGrid<double> &g, const Quad &u, const Quad &d,
                                                const double *grad_pi, long long i, bool dry)
{
    double nl = grad_pi[i];
    nl = (0.5 * (u.y + d.y)) * nl;
    double l_term = (0.5 * (u.z + d.z)) * g.exner_bg_grad_v[i];
    if (!dry) {
        const double dec = 0.5 * (u.w + d.w);
        nl = dec * nl;
        l_term = dec * l_term;
    }
    return nl + l_term;
}

/* pgrad_h from the cell factors (mixed path, first substage) */
__device__ __forceinline__ float pgrad_h_packed(const HGrid<float> &g, const float4 *pc, const SView<float> &s, int l,
                                                int e)
{
    const int fr = g.from[e], to = g.to[e];
    const long long le = (long long)l * g.ne + e;
    const float4 a = pc[(long long)l * g.nc + fr], b = pc[(long long)l * g.nc + to];
    float nl = (b.x - a.x) / g.nd_h[le];
    const float slope = l >= g.nl - g.n_oro ? g.slope_h[le] : 0.0f;
    if (slope != 0.0f) { /* a zero slope adds -0 */
        float c = ipw_at(g, 6, l, fr) * grad_v(g, s.exner_pert, l, fr);
        c += ipw_at(g, 6, l, to) * grad_v(g, s.exner_pert, l, to);
        if (l < g.nl - 1) {
            c += ipw_at(g, 7, l, fr) * grad_v(g, s.exner_pert, l + 1, fr);
            c += ipw_at(g, 7, l, to) * grad_v(g, s.exner_pert, l + 1, to);
        }
        c = 0.5f * c;
        nl += -slope * c;
    }
    nl = (0.5f * (b.y + a.y)) * nl;
    float l_term = (0.5f * (b.z + a.z)) * g.exner_bg_grad_h[le];
    const float dec = 0.5f * (b.w + a.w);
    nl = dec * nl;
    l_term = dec * l_term;
    return nl + l_term;
}

/* pgrad_v from the cell factors of the interface's two cells */
__device__ __forceinline__ float pgrad_v_packed(const HGrid<float> &g, float4 u, float4 d, int k, int c)
{
    float nl = (u.x - d.x) / g.nd_v[(long long)k * g.nc + c];
    nl = (0.5f * (u.y + d.y)) * nl;
    float l_term = (0.5f * (u.z + d.z)) * g.exner_bg_grad_v[(long long)k * g.nc + c];
    const float dec = 0.5f * (u.w + d.w);
    nl = dec * nl;
    l_term = dec * l_term;
    return nl + l_term;
}

/* what the momentum kernels read of the first substage's pressure gradient
 * (mixed path: k_pg_cells; FP64 path: k_pg_cells64) and, FP64 path, of the
 * levels' terms (k_level_terms) and, at rk 1, rho_gas / rho_total */
template <typename R>
struct PgCells;
template <>
struct PgCells<float> {
    const float4 *cell;
};
template <>
struct PgCells<double> {
    const Quad *cell;
    const double *grad_pi, *grad_v2, *q_hi, *q_lo, *gas_share;
};

/* ------------------------------------------------------- k_momentum_h
 * horizontal momentum: explicit tendency (vector_tendencies_expl.c:74-131) and
 * the wind update (manage_rkhevi.c:67-75).  ADV: the advection terms are
 * recomputed in this substage; PG: the pressure gradient is recomputed from
 * the cell factors.  FP64 issue bounds the FP64 instantiation: with the
 * vertical gradients and cell factors formed once, the zero slopes skipped
 * and div_rcp for the distances it went from 182 to 101 us at RES_ID 5
 * with the mountain (789 to 378 us at RES_ID 6, flat, moist), with the levels'
 * terms formed once and the halves taken off the exponent to 89 (320).  The wind update
 * is FP64; u_shadow (mixed path) receives its FP32 copy. */
template <typename R, bool ADV, bool PG>
__global__ void __launch_bounds__(256, sizeof(R) == sizeof(float) ? 8 : 1) k_momentum_h(HGrid<R> g, StepParams p, SView<R> sv, double *u_new, float *u_shadow, const double *u_old,
                             double *tend_u, R *P_h, R *pg_old_h, R *pvt_h, R *v2g_h, const R *flux_h,
                             const R *flux_v, const R *zh, const R *zv, const R *v2, double new_w, double old_w,
                             const double *fric_u, PgCells<R> pg)
{
    const LayerPoint pt_ = layer_point(g.ne);
    if (!pt_.in) return;
    const long long i = pt_.i;
    const int l = pt_.l, e = pt_.x;
    R P, pgo;
    if (PG) {
        if constexpr (sizeof(R) == sizeof(float))
            P = pgrad_h_packed(g, pg.cell, sv, l, e);
        else
            P = pgrad_h_cells(g, pg.cell, pg.grad_pi, l, e, p.n_const == 1);
        pgo = p.first_step ? -P : -P_h[i];
        P_h[i] = P;
        pg_old_h[i] = pgo;
    } else {
        P = P_h[i];
        pgo = pg_old_h[i];
    }
    R pvt, v2g;
    if (ADV) {
        if constexpr (sizeof(R) == sizeof(float)) {
            pvt = vorticity_flux_h(g, flux_h, flux_v, zh, zv, l, e);
            v2g = grad_h(g, v2, l, e);
        } else {
            pvt = vorticity_flux_levels(g, flux_h, pg.q_hi, pg.q_lo, zh, zv, l, e);
            const int fr = g.from[e], to = g.to[e];
            v2g = grad_h_pre(g, v2[(long long)l * g.nc + to], v2[(long long)l * g.nc + fr], pg.grad_v2, l, e, fr, to);
        }
        pvt_h[i] = pvt;
        v2g_h[i] = v2g;
    } else {
        pvt = pvt_h[i];
        v2g = v2g_h[i];
    }
    constexpr bool F = sizeof(R) == sizeof(float);
    const R cur_hor = F ? R(p.cur_hor_f) : R(p.cur_hor), old_hor = F ? R(p.old_hor_f) : R(p.old_hor);
    R y = old_hor * pgo - cur_hor * P + pvt - halved(v2g);
    /* friction acceleration of the diffusion branch, when it is active */
    if (fric_u) y = y + as<R>(fric_u[i]);
    /* the pressure gradient is recomputed in substage 0 only, where the new
     * weight is 1 */
    double t;
    if (PG) t = wide(y);
    else if (F) t = old_w * tend_u[i] + new_w * wide(y);
    else t = half_of(tend_u[i] + wide(y)); /* both weights 1/2 */
    tend_u[i] = t;
    const double un = u_old[i] + p.dt * t;
    u_new[i] = un;
    if (u_shadow) u_shadow[i] = to_float(un);
}

/* ------------------------------------------------------- k_momentum_v
 * vertical momentum at interface k of cell c: tendency including the
 * condensate term (manage_pressure_gradient.c:74-87) */
template <typename R, bool ADV, bool PG>
__global__ void __launch_bounds__(256, sizeof(R) == sizeof(float) ? 8 : 1) k_momentum_v(HGrid<R> g, StepParams p, SView<R> sv, double *tend_w, R *P_v, R *pvt_v, R *v2g_v,
                             const R *flux_h, const R *zh, const R *v2, double new_w, double old_w,
                             const double *fric_w, PgCells<R> pg)
{
    const LayerPoint pt_ = layer_point(g.nc);
    if (!pt_.in) return;
    const long long i = pt_.i;
    const int k = pt_.l, c = pt_.x;
    const int nl = g.nl;
    R pvt = R(0);
    if (ADV) {
        /* vertical part of the vorticity flux (vorticity_flux.c:143-183), all levels */
        const int n_edges = c < N_PENT ? 5 : 6;
        /* the weight 1/2 of the inner levels goes to every term (mixed path)
         * or, exact in either place, to their sum */
        const R vw = (k == 0 || k == nl || sizeof(R) == sizeof(double)) ? R(1) : R(0.5);
        auto weight = [&](int j, int ll) {
            if constexpr (sizeof(R) == sizeof(double)) return ipw_at(g, j, ll, c);
            else return vw * ipw_at(g, j, ll, c);
        };
        const R *z = zh + (long long)k * g.ne;
        if (k >= 1)
            for (int j = 0; j < n_edges; ++j) {
                const int a = g.adj[j * g.nc + c];
                pvt += weight(j, k - 1) * flux_h[(long long)(k - 1) * g.ne + a] * z[a];
            }
        if (k <= nl - 1)
            for (int j = 0; j < n_edges; ++j) {
                const int a = g.adj[j * g.nc + c];
                pvt += weight(j, k) * flux_h[(long long)k * g.ne + a] * z[a];
            }
        if (sizeof(R) == sizeof(double) && k > 0 && k < nl) pvt = halved(pvt);
        pvt_v[i] = pvt;
    }
    if (k == 0 || k == nl) {
        tend_w[i] = 0.0;
        return;
    }
    /* the first substage takes the pressure gradient and the condensate
     * factors from the cell factors of k_pg_cells / k_pg_cells64 */
    constexpr bool F = sizeof(R) == sizeof(float);
    const bool dry = !F && p.n_const == 1;
    R P, v2g, d_up = R(0), d_lo = R(0);
    if constexpr (PG) {
        const auto fu = pg.cell[i - g.nc], fd = pg.cell[i];
        if constexpr (F) P = pgrad_v_packed(g, fu, fd, k, c);
        else P = pgrad_v_cells(g, fu, fd, pg.grad_pi, i, dry);
        d_up = fu.w - R(1);
        d_lo = fd.w - R(1);
        P_v[i] = P;
    } else {
        P = P_v[i];
    }
    if (!ADV) pvt = pvt_v[i];
    if constexpr (ADV && F) {
        v2g = grad_v(g, v2, k, c);
        v2g_v[i] = v2g;
    } else {
        v2g = v2g_v[i]; /* FP64 path: written by k_level_terms */
    }
    if constexpr (!PG && !F) {
        if (!dry) {
            d_up = pg.gas_share[i - g.nc] - R(1);
            d_lo = pg.gas_share[i] - R(1);
        }
    } else if (!PG) {
        const long long ns = (long long)nl * g.nc;
        const long long up = (long long)(k - 1) * g.nc + c, lo = (long long)k * g.nc + c;
        d_up = sv.rho[p.n_cond * ns + up] / density_total_r(sv.rho, p.n_const, ns, up) - R(1);
        d_lo = sv.rho[p.n_cond * ns + lo] / density_total_r(sv.rho, p.n_const, ns, lo) - R(1);
    }
    R pgc = (R(0.5) * (d_up + d_lo)) * g.gravity_m_v[i];
    const R cur_ver = sizeof(R) == sizeof(float) ? R(p.cur_ver_f) : R(p.cur_ver);
    R y = -cur_ver * P + pvt - halved(v2g);
    if (fric_w) y = y + as<R>(fric_w[i]);
    y = y + pgc;
    double t;
    if (PG) t = wide(y);
    else if (F) t = old_w * tend_w[i] + new_w * wide(y);
    else t = half_of(tend_w[i] + wide(y)); /* both weights 1/2 */
    tend_w[i] = t;
}

/* ------------------------------------------------------ k_scalar_tend32
 * explicit mass and rho*theta_v tendencies (scalar_tendencies_expl.c:90-178)
 * at (cell, layer) */

/* vertical_contravariant_corr (averaging.c:41-95) of an edge field given
 * by the functor flux(l, j) at level k of cell c */
template <typename R, typename FX>
__device__ __forceinline__ R contra_corr(const HGrid<R> &g, int k, int c, int n_edges, FX flux)
{
    R r = R(0);
    if (k >= g.nl - g.n_oro) {
        if (k > g.nl - g.n_oro)
            for (int j = 0; j < n_edges; ++j) {
                const int a = g.adj[j * g.nc + c];
                r += R(-0.5) * ipw_at(g, j, k - 1, c) * g.slope_h[(long long)(k - 1) * g.ne + a] * flux(k - 1, j);
            }
        for (int j = 0; j < n_edges; ++j) {
            const int a = g.adj[j * g.nc + c];
            r += R(-0.5) * ipw_at(g, j, k, c) * g.slope_h[(long long)k * g.ne + a] * flux(k, j);
        }
    }
    return r;
}

template <typename R>
__global__ void k_theta(int nl, int nc, int n_cond, SView<R> sv, R *theta)
{
    const long long ns = (long long)nl * nc;
    const long long i = gtid();
    if (i >= ns) return;
    theta[i] = sv.rhotheta_v[i] / sv.rho[n_cond * ns + i];
}

/* FP64 path, rk 1: theta_v and rho_gas / rho_total of every cell, which two
 * interfaces' condensate terms read */
__global__ void k_theta_share(long long ns, int n_cond, int n_const, SView<double> sv, double *theta, double *share)
{
    const long long i = gtid();
    if (i >= ns) return;
    const double rg = sv.rho[n_cond * ns + i];
    theta[i] = sv.rhotheta_v[i] / rg;
    if (n_const > 1) share[i] = rg / density_total_r(sv.rho, n_const, ns, i);
}

/* Sum of edge fluxes of one cell.  R = double: plain double accumulation
 * (the reference's).  R = float: Knuth's TwoSum keeps the exact rounding
 * error of every FP32 addition in a second FP32 word, so the pair (hi, lo)
 * carries the sum to ~2^-48 relative before being rounded once to double --
 * FP64-class accumulation of the mass fluxes at FP32 instruction cost. */
template <typename R>
struct FluxSum {
    double s = 0.0;
    __device__ __forceinline__ void add(R x) { s += double(x); }
    __device__ __forceinline__ double value() const { return s; }
};
template <>
struct FluxSum<float> {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float x)
    {
        const float t = hi + x;
        const float bp = t - hi;
        const float err = (hi - (t - bp)) + (x - bp);
        hi = t;
        lo += err;
    }
    __device__ __forceinline__ bool zero() const { return hi == 0.f && lo == 0.f; }
    __device__ __forceinline__ double value() const { return to_double(hi) + to_double(lo); }
};

/* irreversible terms of the tendencies (scalar_tendencies_expl.c:125-176):
 * dissipative and diffusive heating, radiation, mass diffusion [C][L][Nc] */
struct IrrTerms {
    const double *heating_diss, *temp_diff_heating, *radiation, *mass_diff;
};

/* The mixed path's tendencies at (cell, layer) where the terrain corrections
 * vanish: in the columns without a sloping edge (all of them on a flat grid)
 * and above the terrain-following layers.
 * Edge fluxes are FP32 products, their divergences double-word FP32 sums
 * (FluxSum), the tendencies FP64.  The cell's edges, neighbours, orientation,
 * wind and face areas are loaded once for all constituents.
 *
 * Bounds: load latency of the gathers, then FP64 issue (one warp instruction
 * per 16 cycles).  Hence: a constituent absent from the layer (present: set
 * by k_pg_cells and the tracer solve) is neither gathered nor
 * summed; a zero flux and a zero rate leave the tendency without FP64
 * arithmetic; sums with exact zeros are left out, the rk 1 mean takes one
 * addition.  RES_ID 6 moist, cloud-free: 141 -> 85 us per launch. */
template <bool IRR>
__device__ __forceinline__ void scalar_tend_flat(const HGrid<float> &g, const StepParams &p, const SView<float> &sv,
                                                 const DState &st, const float *theta, const float *cp_ice,
                                                 const float *cp_water, const double *pt_rates, const double *pt_heat,
                                                 const double *sed_heat, const double *inv_vol_tab,
                                                 const Present &present, int rk, const IrrTerms &irr, int l, int c)
{
    const long long ns = (long long)g.nl * g.nc;
    const long long i = (long long)l * g.nc + c;
    const long long nc = g.nc, ne = g.ne;
    const int n_edges = c < N_PENT ? 5 : 6;
    const int cond = p.n_cond;
    const double inv_vol = inv_vol_tab[i];
    int ej[6], nbj[6];
    bool sfj[6];
    float uj[6], arj[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const bool on = j < n_edges;
        ej[j] = on ? g.adj[j * nc + c] : 0;
        nbj[j] = on ? g.adj_nbr[j * nc + c] : c;
        sfj[j] = on && g.adj_sign[j * nc + c] > 0;
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const bool on = j < n_edges;
        uj[j] = on ? sv.u[(long long)l * ne + ej[j]] : 0.f;
        arj[j] = on ? g.area_h[(long long)l * ne + ej[j]] : 0.f;
    }
    /* the main gas: centred mass flux and, from it, the rho*theta_v flux
     * (new weight 1 in both substages) */
    {
        const float *f = sv.rho + cond * ns;
        FluxSum<float> hm, ht;
        const long long o = (long long)l * nc;
        const float fs = f[o + c], ts = theta[o + c];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            if (j >= n_edges) continue;
            const float fm = (0.5f * (fs + f[o + nbj[j]])) * uj[j];
            const float ft = (0.5f * (ts + theta[o + nbj[j]])) * fm;
            const float am = fm * arj[j], at = ft * arj[j];
            hm.add(sfj[j] ? am : -am);
            ht.add(sfj[j] ? at : -at);
        }
        const double dm = hm.value(), dt_ = ht.value();
        const double div = inv_vol * dm;
        double y = -div;
        if (IRR) y = y + irr.mass_diff[cond * ns + i];
        if (p.moist) y = y + pt_rates[cond * ns + i];
        st.rho[cond * ns + i] = y;
        const double div_t = inv_vol * dt_;
        double yt = -div_t;
        if (p.moist || IRR) {
            /* diabatic heating: c_v-weighted, divided by c_p * Pi */
            float cv = 0.f;
            for (int kk = 0; kk < cond; ++kk) cv += sv.rho[kk * ns + i] * ((kk % 2 == 0) ? cp_ice[i] : cp_water[i]);
            cv += sv.rho[cond * ns + i] * float(C_D_V);
            if (p.moist) cv += sv.rho[(cond + 1) * ns + i] * float(C_V_V);
            double heat = pt_heat[i] + sed_heat[i], rate = pt_rates[cond * ns + i];
            if (IRR) {
                heat = irr.heating_diss[i] + irr.temp_diff_heating[i] + irr.radiation[i] + pt_heat[i] + sed_heat[i];
                rate = pt_rates[cond * ns + i] + irr.mass_diff[cond * ns + i];
            }
            const float fac = float(C_D_V) * sv.rho[cond * ns + i] / cv / (float(C_D_P) * (g.exner_bg[i] + sv.exner_pert[i]));
            yt = yt + wide(fac) * heat + rate * wide(theta[i]);
        }
        st.rhotheta_v[i] = yt;
    }
    if (p.n_const == 1) return;
    /* the other constituents: upstream flux */
    const long long o = (long long)l * nc;
#pragma unroll 1
    for (int k = 0; k < p.n_const; ++k) {
        if (k == cond) continue;
        const float *f = sv.rho + k * ns;
        double sum = 0.0;
        if (present.holds(k, l)) {
            FluxSum<float> h;
            const float fs = f[o + c];
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                if (j >= n_edges) continue;
                const float ue = uj[j];
                const float fv = ((ue >= 0.f) == sfj[j] ? fs : f[o + nbj[j]]) * ue;
                const float a = fv * arj[j];
                h.add(sfj[j] ? a : -a);
            }
            if (!h.zero()) sum = guarded_add(to_double(h.hi), to_double(h.lo));
        }
        double rate = 0.0;
        if (p.moist) rate = pt_rates[(k == cond + 1 ? k - 1 : k) * ns + i];
        double y = 0.0;
        if (IRR || !is_zero(sum) || !is_zero(rate)) {
            if (IRR) {
                y = guarded_fma(-inv_vol, sum, irr.mass_diff[k * ns + i]);
                if (p.moist) y = guarded_add(y, rate);
            } else {
                y = guarded_mul(-inv_vol, sum);
                if (p.moist) y = guarded_add(y, rate);
            }
        }
        if (rk != 0) {
            const double old = st.rho[k * ns + i];
            if (!is_zero(old) || !is_zero(y)) y = half_of(guarded_add(old, y));
        }
        st.rho[k * ns + i] = y;
    }
}

/* the same in the terrain-following layers of the columns with a sloping edge,
 * with the terrain corrections: the cell's edges are streamed one layer at a
 * time, every accumulator in the reference's order (layer l-1 before l, edges
 * j = 0..5) */
template <bool IRR>
__device__ __forceinline__ void scalar_tend_tilt(const HGrid<float> &g, const StepParams &p, const SView<float> &sv,
                                                 const DState &st, const float *theta, const float *cp_ice,
                                                 const float *cp_water, const double *pt_rates, const double *pt_heat,
                                                 const double *sed_heat, const double *inv_vol_tab, int rk,
                                                 const IrrTerms &irr, int l, int c)
{
    const long long ns = (long long)g.nl * g.nc;
    const int nl = g.nl, n_oro = g.n_oro;
    const long long i = (long long)l * g.nc + c;
    const long long nc = g.nc, ne = g.ne;
    const int n_edges = c < N_PENT ? 5 : 6;
    const int cond = p.n_cond;
    /* terrain-following corrections: in the orography layers */
    const bool oro = l >= nl - n_oro - 1;
    const bool up_corr = oro && l >= nl - n_oro;            /* contra_corr at level l needed   */
    const bool lo_corr = oro && l < nl - 1;                 /* contra_corr at level l+1 needed */
    const bool up_has_prev = up_corr && l > nl - n_oro;     /* level l sums layer l-1, then l  */
    const bool lo_has_curr = lo_corr && l + 1 > nl - n_oro; /* level l+1 sums layer l, then l+1 */
    const double inv_vol = inv_vol_tab[i];
    const float area_up = g.area_v[(long long)l * nc + c], area_lo = g.area_v[(long long)(l + 1) * nc + c];
    auto edge = [&](int j) { return g.adj[j * nc + c]; };
    auto wcorr = [&](int ll, int j) {
        return float(-0.5) * ipw_at(g, j, ll, c) * g.slope_h[(long long)ll * ne + edge(j)];
    };
    auto uval = [&](int ll, int j) { return sv.u[(long long)ll * ne + edge(j)]; };
    auto comp_v = [&](float up, float lo) -> double {
        if (!oro) return 0.0;
        if (l == nl - n_oro - 1) return wide(-lo * area_lo);
        if (l == nl - 1) return wide(up * area_up);
        return wide(up * area_up - lo * area_lo);
    };
    /* terrain correction of the wind at levels l and l+1 (shared by the tracers) */
    float w_up = float(0), w_lo = float(0);
    if (oro) {
        if (up_has_prev)
            for (int j = 0; j < n_edges; ++j) w_up += wcorr(l - 1, j) * uval(l - 1, j);
        for (int j = 0; j < n_edges; ++j) {
            const float t = wcorr(l, j) * uval(l, j);
            if (up_corr) w_up += t;
            if (lo_has_curr) w_lo += t;
        }
        if (lo_corr)
            for (int j = 0; j < n_edges; ++j) w_lo += wcorr(l + 1, j) * uval(l + 1, j);
    }
    /* the main gas: centred mass flux and, from it, the rho*theta_v flux
     * (new weight 1 in both substages) */
    {
        const float *f = sv.rho + cond * ns;
        FluxSum<float> hm, ht;
        float um = float(0), ut = float(0), lm = float(0), lt = float(0);
        auto layer_pass = [&](int ll, bool to_h, bool to_up, bool to_lo) {
            const long long o = (long long)ll * nc;
            const float fs = f[o + c], ts = theta[o + c];
            for (int j = 0; j < n_edges; ++j) {
                const int nb = g.adj_nbr[j * nc + c];
                const float fm = (float(0.5) * (fs + f[o + nb])) * uval(ll, j);
                const float ft = (float(0.5) * (ts + theta[o + nb])) * fm;
                if (to_h) {
                    const float ar = g.area_h[(long long)ll * ne + edge(j)];
                    const bool self_from = g.adj_sign[j * nc + c] > 0;
                    const float am = fm * ar, at = ft * ar;
                    hm.add(self_from ? am : -am);
                    ht.add(self_from ? at : -at);
                }
                if (to_up || to_lo) {
                    const float wc = wcorr(ll, j);
                    if (to_up) {
                        um += wc * fm;
                        ut += wc * ft;
                    }
                    if (to_lo) {
                        lm += wc * fm;
                        lt += wc * ft;
                    }
                }
            }
        };
        if (up_has_prev) layer_pass(l - 1, false, true, false);
        layer_pass(l, true, up_corr, lo_has_curr);
        if (lo_corr) layer_pass(l + 1, false, false, true);
        const double div = inv_vol * (hm.value() + comp_v(um, lm));
        double y = -div;
        if (IRR) y = y + irr.mass_diff[cond * ns + i];
        if (p.moist) y = y + pt_rates[cond * ns + i];
        st.rho[cond * ns + i] = y;
        const double div_t = inv_vol * (ht.value() + comp_v(ut, lt));
        double yt = -div_t;
        if (p.moist || IRR) {
            /* diabatic heating: c_v-weighted, divided by c_p * Pi */
            float cv = float(0);
            for (int kk = 0; kk < cond; ++kk) cv += sv.rho[kk * ns + i] * ((kk % 2 == 0) ? cp_ice[i] : cp_water[i]);
            cv += sv.rho[cond * ns + i] * float(C_D_V);
            if (p.moist) cv += sv.rho[(cond + 1) * ns + i] * float(C_V_V);
            double heat = pt_heat[i] + sed_heat[i], rate = pt_rates[cond * ns + i];
            if (IRR) {
                heat = irr.heating_diss[i] + irr.temp_diff_heating[i] + irr.radiation[i] + pt_heat[i] + sed_heat[i];
                rate = pt_rates[cond * ns + i] + irr.mass_diff[cond * ns + i];
            }
            const float fac = float(C_D_V) * sv.rho[cond * ns + i] / cv / (float(C_D_P) * (g.exner_bg[i] + sv.exner_pert[i]));
            yt = yt + wide(fac) * heat + rate * wide(theta[i]);
        }
        st.rhotheta_v[i] = yt;
    }
    if (p.n_const == 1) return;
    /* the other constituents: upstream flux.  The cell's edges, neighbours,
     * orientation and layer-l wind and face areas are loaded once for all
     * of them. */
    int ej[6], nbj[6];
    bool sfj[6];
    float uj[6], arj[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const bool on = j < n_edges;
        ej[j] = on ? g.adj[j * nc + c] : 0;
        nbj[j] = on ? g.adj_nbr[j * nc + c] : c;
        sfj[j] = on && g.adj_sign[j * nc + c] > 0;
        uj[j] = on ? sv.u[(long long)l * ne + ej[j]] : float(0);
        arj[j] = on ? g.area_h[(long long)l * ne + ej[j]] : float(0);
    }
    const long long o = (long long)l * nc;
    for (int k = 0; k < p.n_const; ++k) {
        if (k == cond) continue;
        const float *f = sv.rho + k * ns;
        FluxSum<float> h;
        const float fs = f[o + c];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            if (j >= n_edges) continue;
            const float ue = uj[j];
            const float fv = ((ue >= float(0)) == sfj[j] ? fs : f[o + nbj[j]]) * ue;
            const float a = fv * arj[j];
            h.add(sfj[j] ? a : -a);
        }
        double cv = 0.0;
        if (oro) {
            const float d_here = f[i];
            if (l == nl - n_oro - 1) {
                const float d_lo = w_lo <= float(0) ? d_here : f[i + nc];
                cv = wide(-d_lo * w_lo * area_lo);
            } else if (l == nl - 1) {
                const float d_up = w_up <= float(0) ? f[i - nc] : d_here;
                cv = wide(d_up * w_up * area_up);
            } else {
                const float d_up = w_up <= float(0) ? f[i - nc] : d_here;
                const float d_lo = w_lo <= float(0) ? d_here : f[i + nc];
                cv = wide(d_up * w_up * area_up - d_lo * w_lo * area_lo);
            }
        }
        const double div = inv_vol * (h.value() + cv);
        double y = -div;
        if (IRR) y = y + irr.mass_diff[k * ns + i];
        if (p.moist) {
            long long pt = k * ns;
            if (k == cond + 1) pt -= ns;
            y = y + pt_rates[pt + i];
        }
        st.rho[k * ns + i] = rk == 0 ? y : half_of(st.rho[k * ns + i] + y);
    }
}

/* One launch for both: the first tilt_blocks blocks of a layer take the columns
 * of tilt_cells, the others every cell and leave those out; the tilted columns
 * take the shorter way above the terrain-following layers.  Against one kernel
 * that decides per cell, with the mountain and all constituents: RES_ID 6 202 ->
 * 172 us, RES_ID 3 and 4, where both wait for the latency of their gathers, 21 ->
 * 24 and 24 -> 28 us (two launches one after the other 38).  64 registers (eight
 * blocks per SM; 72 without the bound, which spills 48 bytes of the tilted form:
 * 657 against 628 us at RES_ID 7) and no corrections compiled in for a flat grid
 * (TILT = false; RES_ID 6, cloud-free: 96 -> 85 us). */
template <bool IRR, bool TILT>
__global__ void __launch_bounds__(128, 8) k_scalar_tend32(HGrid<float> g, StepParams p, SView<float> sv, DState st,
                                                       const float *theta, const float *cp_ice, const float *cp_water,
                                                       const double *pt_rates, const double *pt_heat,
                                                       const double *sed_heat, const double *inv_vol_tab,
                                                       Present present, int rk, IrrTerms irr, const int *tilt_cells,
                                                       int n_tilt, int tilt_blocks)
{
    const int l = (int)blockIdx.y, b = (int)blockIdx.x, top = g.nl - g.n_oro - 1;
    if (TILT && b < tilt_blocks) {
        const int x = b * (int)blockDim.x + (int)threadIdx.x;
        if (l < top || x >= n_tilt) return;
        scalar_tend_tilt<IRR>(g, p, sv, st, theta, cp_ice, cp_water, pt_rates, pt_heat, sed_heat, inv_vol_tab, rk, irr, l,
                              tilt_cells[x]);
    } else {
        const int c = (b - (TILT ? tilt_blocks : 0)) * (int)blockDim.x + (int)threadIdx.x;
        if (c >= g.nc || (TILT && l >= top && g.tilt[c])) return;
        scalar_tend_flat<IRR>(g, p, sv, st, theta, cp_ice, cp_water, pt_rates, pt_heat, sed_heat, inv_vol_tab, present, rk,
                              irr, l, c);
    }
}

/* ---- the same tendencies on the FP64 path (k_scalar_tend64), in three kernels.  FP64 issue
 * bounds them, so nothing is formed twice: the fluxes of an edge once
 * (k_edge_flux) instead of by both its cells in up to three layer passes, the
 * terrain corrections of a level once (k_level_corr) instead of by the cells
 * above and below it, with tabulated weights, and only in columns with a
 * sloping edge; constituents absent around an edge and zero heating are
 * skipped (they add zeros).  Every accumulator receives the reference's terms
 * in its order (layer k-1 before k, edges j = 0..5).
 * RES_ID 5 with the mountain: 180 -> 72 us per substage; RES_ID 6 moist,
 * flat: 1175 -> 228 us. */

/* horizontal mass flux of the main gas and rho theta_v flux of every edge */
__global__ void k_edge_flux(HGrid<double> g, const double *rho_gas, const double *theta, const double *u, double *flux_m,
                            double *flux_t)
{
    const LayerPoint p = layer_point(g.ne);
    if (!p.in) return;
    const long long o = (long long)p.l * g.nc;
    const int fr = g.from[p.x], to = g.to[p.x];
    const double fm = (0.5 * (rho_gas[o + fr] + rho_gas[o + to])) * u[p.i];
    flux_m[p.i] = fm;
    flux_t[p.i] = (0.5 * (theta[o + fr] + theta[o + to])) * fm;
}

/* terrain corrections at level k (from layers k-1 and k, averaging.c:41-95)
 * of the mass and rho theta_v fluxes, times the interface's area, and of the
 * wind (WIND: for the tracers).  Grid: levels nl - n_oro .. nl - 1. */
template <bool WIND>
__global__ void k_level_corr(HGrid<double> g, const double *flux_m, const double *flux_t, const double *u,
                             double *corr_m, double *corr_t, double *corr_w)
{
    const LayerPoint p = layer_point(g.nc);
    if (!p.in || !g.tilt[p.x]) return;
    const int c = p.x, k = p.l + g.nl - g.n_oro, n_edges = c < N_PENT ? 5 : 6;
    const long long ns = (long long)g.nl * g.nc, kc = (long long)k * g.nc + c;
    int e[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) e[j] = j < n_edges ? g.adj[j * g.nc + c] : 0;
    double m = 0.0, t = 0.0, w = 0.0;
    for (int ll = p.l > 0 ? k - 1 : k; ll <= k; ++ll) {
        const double *cw = g.corr_w + (long long)ll * g.nc + c;
        const long long lo = (long long)ll * g.ne;
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            if (j >= n_edges) continue;
            const double wc = cw[j * ns];
            m += wc * flux_m[lo + e[j]];
            t += wc * flux_t[lo + e[j]];
            if (WIND) w += wc * u[lo + e[j]];
        }
    }
    const double area = g.area_v[kc];
    corr_m[kc] = m * area;
    corr_t[kc] = t * area;
    if (WIND) corr_w[kc] = w;
}

/* the tendencies of a cell from them; rho_prev: the tendencies of the
 * previous substage (old weight 1/2 at rk 1, non-main constituents) */
template <bool IRR>
__global__ void __launch_bounds__(128)
    k_scalar_tend64(HGrid<double> g, StepParams p, SView<double> sv, const double *rho_prev, double *st_rho,
                    double *st_rt, const double *flux_m, const double *flux_t, const double *corr, const double *theta,
                    const double *cp_ice, const double *cp_water, const double *pt_rates, const double *pt_heat,
                    const double *sed_heat, int rk, IrrTerms irr)
{
    const LayerPoint pt_ = layer_point(g.nc);
    if (!pt_.in) return;
    const long long i = pt_.i, nc = g.nc, ne = g.ne, ns = (long long)g.nl * nc, nw = ns + nc;
    const int l = pt_.l, c = pt_.x, nl = g.nl, n_oro = g.n_oro, cond = p.n_cond;
    const int n_edges = c < N_PENT ? 5 : 6;
    /* corrections at the level above (up) and below (lo) the layer */
    const bool oro = l >= nl - n_oro - 1 && g.tilt[c];
    const bool up = oro && l >= nl - n_oro, lo = oro && l < nl - 1;
    const double inv_vol = g.r_volume[i];
    int ej[6];
    bool sfj[6];
    double arj[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const bool on = j < n_edges;
        ej[j] = on ? g.adj[j * nc + c] : 0;
        sfj[j] = on && g.adj_sign[j * nc + c] > 0;
        arj[j] = on ? g.area_h[(long long)l * ne + ej[j]] : 0.0;
    }
    auto comp_v = [&](const double *cr) {
        const double a = up ? cr[i] : 0.0, b = lo ? cr[i + nc] : 0.0;
        return up ? (lo ? a - b : a) : -b;
    };
    const long long lo_e = (long long)l * ne;
    {
        double hm = 0.0, ht = 0.0;
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            if (j >= n_edges) continue;
            const double am = flux_m[lo_e + ej[j]] * arj[j], at = flux_t[lo_e + ej[j]] * arj[j];
            hm += sfj[j] ? am : -am;
            ht += sfj[j] ? at : -at;
        }
        double y = -(inv_vol * (oro ? hm + comp_v(corr) : hm));
        double yt = -(inv_vol * (oro ? ht + comp_v(corr + nw) : ht));
        double rate = p.moist ? pt_rates[cond * ns + i] : 0.0;
        if (IRR) y = y + irr.mass_diff[cond * ns + i];
        if (p.moist) y = y + rate;
        st_rho[cond * ns + i] = y;
        if (p.moist || IRR) {
            /* diabatic heating: c_v-weighted, divided by c_p * Pi */
            double heat = pt_heat[i] + sed_heat[i];
            if (IRR) {
                heat = irr.heating_diss[i] + irr.temp_diff_heating[i] + irr.radiation[i] + pt_heat[i] + sed_heat[i];
                rate = pt_rates[cond * ns + i] + irr.mass_diff[cond * ns + i];
            }
            if (!is_zero(heat)) {
                const double rg = sv.rho[cond * ns + i];
                double cv = 0.0;
                for (int kk = 0; kk < cond; ++kk) {
                    const double r = sv.rho[kk * ns + i];
                    if (!is_zero(r)) cv = guarded_add(cv, guarded_mul(r, (kk % 2 == 0) ? cp_ice[i] : cp_water[i]));
                }
                cv += rg * C_D_V;
                if (p.moist) cv += sv.rho[(cond + 1) * ns + i] * C_V_V;
                yt = yt + C_D_V * rg / cv * heat / (C_D_P * (g.exner_bg[i] + sv.exner_pert[i]));
            }
            yt = yt + rate * theta[i];
        }
        st_rt[i] = yt;
    }
    if (p.n_const == 1) return;
    /* the other constituents: upstream flux */
    int nbj[6];
    double uj[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const bool on = j < n_edges;
        uj[j] = on ? sv.u[lo_e + ej[j]] : 0.0;
        /* the upstream cell: the cell itself where the wind leaves it (u =
         * -0 picks the other one, whose product is a zero as well) */
        nbj[j] = on && nonneg<false>(uj[j]) != sfj[j] ? g.adj_nbr[j * nc + c] : c;
    }
    const double w_up = up ? corr[2 * nw + i] : 0.0, w_lo = lo ? corr[2 * nw + i + nc] : 0.0;
    const double area_up = oro ? g.area_v[i] : 0.0, area_lo = oro ? g.area_v[i + nc] : 0.0;
    const double *fl = sv.rho + (long long)l * nc;
#pragma unroll 1
    for (int k = 0; k < p.n_const; ++k, fl += ns) {
        if (k == cond) continue;
        double h = 0.0, d[6];
        unsigned long long any = 0;
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            d[j] = j < n_edges ? fl[nbj[j]] : 0.0;
            any |= (unsigned long long)__double_as_longlong(d[j]);
        }
        if (any << 1)
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                if (j >= n_edges) continue;
                const double a = d[j] * uj[j] * arj[j];
                h += sfj[j] ? a : -a;
            }
        if (oro) {
            const double d_up = up ? (w_up <= 0.0 ? fl[c - nc] : fl[c]) : 0.0;
            const double d_lo = lo ? (w_lo <= 0.0 ? fl[c] : fl[c + nc]) : 0.0;
            double cv;
            if (!up) cv = -d_lo * w_lo * area_lo;
            else if (!lo) cv = d_up * w_up * area_up;
            else cv = d_up * w_up * area_up - d_lo * w_lo * area_lo;
            h = h + cv;
        }
        double y = is_zero(h) ? 0.0 : guarded_mul(-inv_vol, h);
        if (IRR) y = y + irr.mass_diff[k * ns + i];
        if (p.moist) {
            const double rate = pt_rates[(k == cond + 1 ? k - 1 : k) * ns + i];
            if (!is_zero(rate)) y = guarded_add(y, rate);
        }
        if (rk != 0) { /* 0.5 old + 0.5 y */
            const double old = rho_prev[k * ns + i];
            if (!is_zero(old) || !is_zero(y)) y = half_of(guarded_add(old, y));
        }
        st_rho[k * ns + i] = y;
    }
}

/* per-thread column sweeps of the adjoint hold at most this many layers */
constexpr int MAX_L = 64;
/* the layer count the register-resident column sweeps are compiled for
 * (NO_OF_LAYERS of every GAME configuration) */
constexpr int NL_FIXED = 26;

}  // namespace
}  // namespace game

