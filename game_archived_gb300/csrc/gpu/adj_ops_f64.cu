/*
 * Adjoints of the single operators (the reverse mode of grad, divv_h,
 * divv_h_tracer, scalar_times_vector, inner_product, calc_pot_vort,
 * vorticity_flux and the tracer column solver on device-layout fields),
 * compiled with --fmad=false.  They use the scatter
 * helpers of the step adjoint (adj_bwd.cuh): bars of a forward's inputs are
 * accumulated, x_bar += (dy/dx)^T y_bar.
 */
#include "adj_bwd.cuh"
#include "adj_ops.h"

namespace game {
namespace {

inline unsigned nb(long long n, int bs = 256) { return (unsigned)((n + bs - 1) / bs); }

/* grad (gradient_operators.c:66-74): vector bar [w | u] -> scalar bar; the
 * TOA and surface entries of the output are not written by grad and carry
 * no dependence on the input */
__global__ void kop_grad_adj(HGrid<double> g, const double *out_b, double *in_b)
{
    const long long nw = (long long)(g.nl + 1) * g.nc, n = nw + (long long)g.nl * g.ne;
    const long long i = gtid();
    if (i >= n) return;
    const double ob = out_b[i];
    if (ob == 0.0) return;
    if (i < nw) {
        const int k = row_of(i, g.nc), c = (int)(i - (long long)k * g.nc);
        if (k == 0 || k == g.nl) return;
        b_gv(g, in_b, k, c, ob);
    } else {
        const long long j = i - nw;
        const int l = row_of(j, g.ne), e = (int)(j - (long long)l * g.ne);
        b_grad_h(g, in_b, l, e, ob);
    }
}

/* divv_h (divergences.c:14-64): scalar bar -> bar of the horizontal part of
 * the vector field, through the edge sum and the terrain correction */
__global__ void kop_divv_adj(HGrid<double> g, const double *out_b, double *in_b_u)
{
    const long long ns = (long long)g.nl * g.nc;
    const long long i = gtid();
    if (i >= ns) return;
    const double yb = out_b[i];
    if (yb == 0.0) return;
    const int nl = g.nl, n_oro = g.n_oro;
    const int l = row_of(i, g.nc), c = (int)(i - (long long)l * g.nc);
    const long long nc = g.nc, ne = g.ne;
    const int n_edges = c < N_PENT ? 5 : 6;
    const bool oro = l >= nl - n_oro - 1;
    const bool up_corr = oro && l >= nl - n_oro;
    const bool lo_corr = oro && l < nl - 1;
    const bool up_has_prev = up_corr && l > nl - n_oro;
    const bool lo_has_curr = lo_corr && l + 1 > nl - n_oro;
    const double hb = yb / g.volume[i];
    const double area_up = g.area_v[(long long)l * nc + c], area_lo = g.area_v[(long long)(l + 1) * nc + c];
    double upb = 0.0, lob = 0.0;
    if (oro) {
        if (l == nl - n_oro - 1) lob = -area_lo * hb;
        else if (l == nl - 1) upb = area_up * hb;
        else {
            upb = area_up * hb;
            lob = -area_lo * hb;
        }
    }
    auto pass = [&](int ll, bool to_h, bool to_up, bool to_lo) {
        for (int j = 0; j < n_edges; ++j) {
            const int ed = g.adj[j * nc + c];
            const long long le = (long long)ll * ne + ed;
            double fb = 0.0;
            if (to_h) fb += double(g.adj_sign[j * nc + c]) * g.area_h[le] * hb;
            if (to_up || to_lo) {
                const double wc = -0.5 * ipw_d(g, j, ll, c) * g.slope_h[le];
                if (to_up) fb += wc * upb;
                if (to_lo) fb += wc * lob;
            }
            if (fb != 0.0) acc(&in_b_u[le], fb);
        }
    };
    if (up_has_prev) pass(l - 1, false, true, false);
    pass(l, true, up_corr, lo_has_curr);
    if (lo_corr) pass(l + 1, false, false, true);
}

/* scalar_times_vector (multiplications.c:35-117): edge average (all edges)
 * and interface average (inner interfaces) times the vector */
__global__ void kop_stv_adj(HGrid<double> g, const double *s, const double *v, const double *out_b, double *s_b,
                            double *v_b)
{
    const long long nw = (long long)(g.nl + 1) * g.nc, n = nw + (long long)g.nl * g.ne;
    const long long i = gtid();
    if (i >= n) return;
    const double ob = out_b[i];
    if (ob == 0.0) return;
    if (i < nw) {
        const int k = row_of(i, g.nc), c = (int)(i - (long long)k * g.nc);
        if (k == 0 || k == g.nl) return;
        const long long up = (long long)(k - 1) * g.nc + c, lo = (long long)k * g.nc + c;
        acc(&v_b[i], 0.5 * (s[up] + s[lo]) * ob);
        const double q = 0.5 * v[i] * ob;
        acc(&s_b[up], q);
        acc(&s_b[lo], q);
    } else {
        const long long j = i - nw;
        const int l = row_of(j, g.ne), e = (int)(j - (long long)l * g.ne);
        const long long ct = (long long)l * g.nc + g.to[e], cf = (long long)l * g.nc + g.from[e];
        acc(&v_b[i], 0.5 * (s[ct] + s[cf]) * ob);
        const double q = 0.5 * v[i] * ob;
        acc(&s_b[ct], q);
        acc(&s_b[cf], q);
    }
}

/* inner_product (inner_product.c:13-43) of vectors a, b (device layout) */
__global__ void kop_inner_adj(HGrid<double> g, const double *a, const double *b, const double *out_b, double *a_b,
                              double *b_b)
{
    const long long ns = (long long)g.nl * g.nc;
    const long long i = gtid();
    if (i >= ns) return;
    const double ob = out_b[i];
    if (ob == 0.0) return;
    const int l = row_of(i, g.nc), c = (int)(i - (long long)l * g.nc);
    const int n_edges = c < N_PENT ? 5 : 6;
    const long long nw = (long long)(g.nl + 1) * g.nc;
    for (int j = 0; j < n_edges; ++j) {
        const long long vi = nw + (long long)l * g.ne + g.adj[j * g.nc + c];
        const double wgt = ipw_d(g, j, l, c);
        acc(&a_b[vi], wgt * b[vi] * ob);
        acc(&b_b[vi], wgt * a[vi] * ob);
    }
    const long long top = i, bot = i + g.nc;
    acc(&a_b[top], ipw_d(g, 6, l, c) * b[top] * ob);
    acc(&b_b[top], ipw_d(g, 6, l, c) * a[top] * ob);
    acc(&a_b[bot], ipw_d(g, 7, l, c) * b[bot] * ob);
    acc(&b_b[bot], ipw_d(g, 7, l, c) * a[bot] * ob);
}

/* vorticity_flux (vorticity_flux.c:16-187): horizontal part per edge */
__global__ void kop_vflux_h_adj(HGrid<double> g, const double *flux_v, const double *flux_h, const double *zh,
                                const double *zv, const double *out_b_u, double *fv_b, double *fh_b, double *zh_b,
                                double *zv_b)
{
    const long long n = (long long)g.nl * g.ne;
    const long long i = gtid();
    if (i >= n) return;
    const double ob = out_b_u[i];
    if (ob == 0.0) return;
    const int l = row_of(i, g.ne), e = (int)(i - (long long)l * g.ne);
    b_vflux_h(g, flux_h, flux_v, zh, zv, fh_b, fv_b, zh_b, zv_b, l, e, ob);
}

/* vertical part per interface (all levels) */
__global__ void kop_vflux_v_adj(HGrid<double> g, const double *flux_h, const double *zh, const double *out_b_w,
                                double *fh_b, double *zh_b)
{
    const long long n = (long long)(g.nl + 1) * g.nc;
    const long long i = gtid();
    if (i >= n) return;
    const double pb = out_b_w[i];
    if (pb == 0.0) return;
    const int k = row_of(i, g.nc), c = (int)(i - (long long)k * g.nc);
    const int nl = g.nl, n_edges = c < N_PENT ? 5 : 6;
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


/* divv_h_tracer (divergences.c:66-148): the horizontal part is linear in the
 * flux field; the terrain vertical term is rho_up * corr(wind) * area_v with
 * rho_up the density upstream of the contravariant correction corr (the
 * pick is held fixed: the derivative of the piecewise form) */
__global__ void kop_divv_tracer_adj(HGrid<double> g, const double *density, const double *wind_u,
                                    const double *out_b, double *in_b_u, double *dens_b, double *wind_b_u)
{
    const long long ns = (long long)g.nl * g.nc;
    const long long i = gtid();
    if (i >= ns) return;
    const double yb = out_b[i];
    if (yb == 0.0) return;
    const int nl = g.nl, n_oro = g.n_oro;
    const int l = row_of(i, g.nc), c = (int)(i - (long long)l * g.nc);
    const long long nc = g.nc, ne = g.ne;
    const int n_edges = c < N_PENT ? 5 : 6;
    const double hb = yb / g.volume[i];
    for (int j = 0; j < n_edges; ++j) {
        const long long vi = (long long)l * ne + g.adj[j * nc + c];
        acc(&in_b_u[vi], double(g.adj_sign[j * nc + c]) * g.area_h[vi] * hb);
    }
    auto fw = [&](int ll, int j) { return wind_u[(long long)ll * ne + g.adj[j * nc + c]]; };
    /* bar of contra_corr(g, k, c, ...) into the edge winds it reads */
    auto corr_b = [&](int k, double cb) {
        if (k < nl - n_oro || cb == 0.0) return;
        for (int kk = (k > nl - n_oro ? k - 1 : k); kk <= k; ++kk)
            for (int j = 0; j < n_edges; ++j) {
                const long long le = (long long)kk * ne + g.adj[j * nc + c];
                acc(&wind_b_u[le], -0.5 * ipw_at(g, j, kk, c) * g.slope_h[le] * cb);
            }
    };
    if (l == nl - n_oro - 1 || (l > nl - n_oro - 1 && l < nl - 1)) { /* lower interface term, - rho * corr * A */
        const double lo = contra_corr(g, l + 1, c, n_edges, fw);
        const long long id = lo <= 0.0 ? i : i + nc;
        const double a = g.area_v[(long long)(l + 1) * nc + c];
        acc(&dens_b[id], -lo * a * hb);
        corr_b(l + 1, -density[id] * a * hb);
    }
    if (l > nl - n_oro - 1) { /* upper interface term, + rho * corr * A */
        const double up = contra_corr(g, l, c, n_edges, fw);
        const long long id = up <= 0.0 ? i - nc : i;
        const double a = g.area_v[(long long)l * nc + c];
        acc(&dens_b[id], up * a * hb);
        corr_b(l, density[id] * a * hb);
    }
}

/* d/dT of c_p(T) * T for the condensate kinds of c_p_cond (dictionary.c:111-190),
 * from the same fits: Murphy and Koop (2005) Eq. (4) for ice, Pruppacher and
 * Klett (2010) Eqs. (3-15), (3-16) for water; zero where the fits clip */
__device__ double d_cpT(int id, double t)
{
    double dcp = 0.0;
    if (id % 2 == 0) {
        if (t <= T_0 && t >= 20.0) {
            const double q = t / 125.1;
            dcp = (0.14644 + 0.06163 * exp(-(q * q)) * (1.0 - 2.0 * q * q)) / M_V;
        }
    } else {
        const double tc = t - T_0;
        if (tc >= 0.0) {
            if (tc <= 35.0) {
                const double a = tc - 35.0;
                dcp = 4186.8 * (2.0 * 3.1e-6 * a + 4.0 * 3.8e-9 * a * a * a);
            }
        } else if (tc >= -37.0) {
            dcp = 4186.8 * (-2.7052e-3 - 2.0 * 2.3235e-5 * tc + 3.0 * 4.3778e-6 * tc * tc
                            + 4.0 * 2.7136e-7 * tc * tc * tc);
        }
    }
    return dcp * t + c_p_cond(id, t);
}

/* three_band_solver_gen_densities (column_solvers.c:385-639) in reverse mode,
 * in three kernels over its (tracer, column) systems: the rows per (tracer,
 * layer, column), the two tridiagonal solves per (tracer, column) -- the
 * unclipped solution x and the bar y of the right-hand side, the transposed
 * system's -- and the bars of the inputs per (tracer, layer, column) again:
 * the old density and tendency of the tracer, the old and new vertical wind
 * and, at rk 0, the temperature through the sedimentation heat.  One kernel
 * with a column per thread did all of it in local memory with 200 blocks of
 * work at RES_ID 4: 551 -> 152 us.  Upwind picks and flux-sign branches are
 * held fixed; clipped outputs carry no derivative.  The bar of the new
 * density is taken and left zero (the forward overwrites that field without
 * reading it).
 * work: 4 arrays [C-1][L][Nc]: c, d (x after the solve), e, r (y after it). */
struct TracerRows {
    double *c, *d, *e, *r;
};
struct TracerSlot {
    int k;       /* constituent */
    bool sink;   /* sediments */
    double vs;   /* its velocity */
};
__device__ __forceinline__ TracerSlot tracer_slot(const StepParams &p, int slot)
{
    const int cond = p.n_cond, k = slot < cond ? slot : slot + 1;
    const bool sink = k < cond;
    return {k, sink,
            k < cond / 4 ? p.snow_velocity : k < cond / 2 ? p.rain_velocity : sink ? p.cloud_velocity : 0.0};
}

/* grid: x cells, y layers, z tracer slots */
__global__ void ka_gen_rows(VGrid vg, StepParams p, DState so, DState sn, DState st, TracerRows w)
{
    const LayerPoint pt = layer_point(vg.nc);
    if (!pt.in) return;
    const int nc = vg.nc, nl = vg.nl, j = pt.l;
    const long long ns = (long long)nl * nc, b = pt.i, o = (long long)blockIdx.z * ns + b;
    const TracerSlot s = tracer_slot(p, blockIdx.z);
    const double *ro = so.rho + s.k * ns;
    const double dt = p.dt, h = 0.5 * dt, v = vg.volume[b], rv = vg.r_volume[b];
    const double g = div_rcp(h, v, rv);
    double c = 0.0, d = 1.0, e = 0.0, r = ro[b] + dt * st.rho[s.k * ns + b];
    if (j < nl - 1) {
        const long long wi = b + nc;
        const double ar = vg.area_v[wi], f = ar * (so.w[wi] - s.vs), bw = ar * (sn.w[wi] - s.vs);
        const double fr = (nonneg<true>(bw) ? ro[wi] : ro[b]) * bw;
        if (nonneg<true>(f)) {
            e = -g * f;
        } else {
            c = div_rcp(h, vg.volume[wi], vg.r_volume[wi]) * f;
            d -= g * f;
        }
        r += div_rcp(h * fr, v, rv);
    }
    if (j > 0) {
        const double ar = vg.area_v[b], f = ar * (so.w[b] - s.vs), bw = ar * (sn.w[b] - s.vs);
        const double fr = (nonneg<true>(bw) ? ro[b] : ro[b - nc]) * bw;
        if (nonneg<true>(f)) d += g * f;
        r -= div_rcp(h * fr, v, rv);
    }
    if (j == nl - 1 && s.sink) {
        const double a = h * s.vs * vg.area_v[b + nc];
        d += div_rcp(a, v, rv);
        r -= div_rcp(a * ro[b], v, rv);
    }
    w.c[o] = c;
    w.d[o] = d;
    w.e[o] = e;
    w.r[o] = r;
}

/* x over d, y over r.  NL > 0: the layer count is a compile-time constant and
 * the sweeps stay in registers; else the layer count is nl (at most CAP) */
template <int NL, int CAP>
__global__ void ka_gen_solve(int nc, int nl_arg, int n_tr, int n_cond, TracerRows w, DState sn_b)
{
    const long long q = gtid();
    if (q >= (long long)n_tr * nc) return;
    const int nl = NL > 0 ? NL : nl_arg;
    const int slot = row_of(q, nc), i = (int)(q - (long long)slot * nc);
    const long long ns = (long long)nl * nc;
    const double *cc = w.c + slot * ns + i, *ee = w.e + slot * ns + i;
    double *dx = w.d + slot * ns + i, *ry = w.r + slot * ns + i;
    double *rn_b = sn_b.rho + (slot < n_cond ? slot : slot + 1) * ns + i;
    double ep[NL > 0 ? NL : CAP], rp[NL > 0 ? NL : CAP], dd[NL > 0 ? NL : CAP];
#pragma unroll
    for (int j = 0; j < nl; ++j) {
        const long long o = (long long)j * nc;
        dd[j] = dx[o];
        const double cm = j > 0 ? cc[o - nc] : 0.0, r = ry[o];
        const double den = j > 0 ? dd[j] - ep[j - 1] * cm : dd[j], inv = rcp_sweep(den);
        ep[j] = j < nl - 1 ? div_sweep(ee[o], den, inv) : 0.0;
        rp[j] = div_sweep(j > 0 ? r - rp[j - 1] * cm : r, den, inv);
    }
    double x = 0.0;
#pragma unroll
    for (int j = nl - 1; j >= 0; --j) {
        x = j < nl - 1 ? rp[j] - ep[j] * x : rp[j];
        dx[(long long)j * nc] = x;
        rp[j] = x; /* its sign clips the bar below */
    }
    /* transposed system A^T y = xbar (sub-diagonal e, super-diagonal c) */
#pragma unroll
    for (int j = 0; j < nl; ++j) {
        const long long o = (long long)j * nc;
        const double g = rp[j] < 0.0 ? 0.0 : rn_b[o];
        rn_b[o] = 0.0;
        const double sub = j > 0 ? ee[o - nc] : 0.0;
        const double den = j > 0 ? dd[j] - ep[j - 1] * sub : dd[j], inv = rcp_sweep(den);
        ep[j] = j < nl - 1 ? div_sweep(cc[o], den, inv) : 0.0;
        rp[j] = div_sweep(j > 0 ? g - rp[j - 1] * sub : g, den, inv);
    }
    double y = 0.0;
#pragma unroll
    for (int j = nl - 1; j >= 0; --j) {
        y = j < nl - 1 ? rp[j] - ep[j] * y : rp[j];
        ry[(long long)j * nc] = y;
    }
}

/* grid: x cells, y layers, z tracer slots; a layer's thread takes the interface
 * below it too.  The wind and the temperature are shared by the tracers, the
 * upstream density by a layer's two interfaces: atomic. */
__global__ void ka_gen_bars(VGrid vg, StepParams p, DState so, DState sn, const double *temperature, int rk,
                            const double *sed_b, TracerRows w, DState so_b, DState sn_b, DState st_b, double *t_b)
{
    const LayerPoint pt = layer_point(vg.nc);
    if (!pt.in) return;
    const int nc = vg.nc, nl = vg.nl, j = pt.l;
    const long long ns = (long long)nl * nc, b = pt.i, o = (long long)blockIdx.z * ns + b;
    const TracerSlot s = tracer_slot(p, blockIdx.z);
    const bool heat = rk == 0 && s.sink;
    const double *ro = so.rho + s.k * ns;
    double *ro_b = so_b.rho + s.k * ns;
    const double dt = p.dt, h = 0.5 * dt, y = w.r[o], rv = vg.r_volume[b], yv = div_rcp(y, vg.volume[b], rv);
    st_b.rho[s.k * ns + b] += dt * y;
    double own = y; /* bar of this layer's old density */
    if (j == nl - 1) {
        if (s.sink) {
            const double a_sfc = vg.area_v[b + nc];
            own -= h * s.vs * a_sfc * yv;
            if (heat) {
                const double hb = div_rcp(sed_b[b], vg.volume[b], rv) * a_sfc, tb = temperature[b];
                own -= s.vs * c_p_cond(s.k, tb) * tb * hb;
                acc(&t_b[b], -s.vs * d_cpT(s.k, tb) * ro[b] * hb);
            }
        }
        acc(&ro_b[b], own);
        return;
    }
    const long long wi = b + nc;
    const double ar = vg.area_v[wi], f = ar * (so.w[wi] - s.vs), bw = ar * (sn.w[wi] - s.vs);
    const bool below = nonneg<true>(bw);
    const long long id = below ? wi : b;
    const double rv1 = vg.r_volume[wi], v1 = vg.volume[wi], y1v = div_rcp(w.r[o + nc], v1, rv1), dio = ro[id];
    double frb = h * (yv - y1v);
    if (heat) {
        const double hb = div_rcp(sed_b[b], vg.volume[b], rv) - div_rcp(sed_b[wi], v1, rv1), t = temperature[id];
        frb += c_p_cond(s.k, t) * t * hb;
        acc(&t_b[id], d_cpT(s.k, t) * dio * bw * hb);
    }
    if (below) acc(&ro_b[wi], bw * frb);
    else own += bw * frb;
    acc(&ro_b[b], own);
    acc(&sn_b.w[wi], ar * dio * frb);
    /* rows j (e, d) and j + 1 (c, d) */
    const double xs = nonneg<true>(f) ? w.d[o + nc] : w.d[o];
    acc(&so_b.w[wi], ar * (h * (yv - y1v) * xs));
}

}  // namespace

void op_grad_adj(Context *c, const double *out_b, double *in_b)
{
    kop_grad_adj<<<nb(c->nv), 256, 0, c->stream>>>(c->hg64, out_b, in_b);
    c->kernel_launches++;
}

void op_divv_adj(Context *c, const double *out_b, double *in_b)
{
    kop_divv_adj<<<nb(c->ns), 256, 0, c->stream>>>(c->hg64, out_b, in_b + (long long)(c->nl + 1) * c->nc);
    c->kernel_launches++;
}

void op_stv_adj(Context *c, const double *s, const double *v, const double *out_b, double *s_b, double *v_b)
{
    kop_stv_adj<<<nb(c->nv), 256, 0, c->stream>>>(c->hg64, s, v, out_b, s_b, v_b);
    c->kernel_launches++;
}

void op_inner_adj(Context *c, const double *a, const double *b, const double *out_b, double *a_b, double *b_b)
{
    kop_inner_adj<<<nb(c->ns), 256, 0, c->stream>>>(c->hg64, a, b, out_b, a_b, b_b);
    c->kernel_launches++;
}

void op_vflux_adj(Context *c, const double *flux, const double *pv, const double *out_b, double *flux_b, double *pv_b)
{
    const long long nw = (long long)(c->nl + 1) * c->nc, nzh = (long long)(c->nl + 1) * c->ne;
    kop_vflux_h_adj<<<nb((long long)c->nl * c->ne), 256, 0, c->stream>>>(c->hg64, flux, flux + nw, pv, pv + nzh,
                                                                          out_b + nw, flux_b, flux_b + nw, pv_b,
                                                                          pv_b + nzh);
    kop_vflux_v_adj<<<nb(nw), 256, 0, c->stream>>>(c->hg64, flux + nw, pv, out_b, flux_b + nw, pv_b);
    c->kernel_launches += 2;
}

void op_pot_vort_adj(Context *c, const double *wind, const double *rho, const double *pv, const double *pv_b,
                     const double *zero_u, double *wind_b, double *rho_b, double *tri_b)
{
    const long long nw = (long long)(c->nl + 1) * c->nc, nzh = (long long)(c->nl + 1) * c->ne;
    ba_edge<<<nb(nzh), 256, 0, c->stream>>>(c->hg64, wind + nw, rho, pv, pv + nzh, pv_b, pv_b + nzh, zero_u,
                                            wind_b + nw, wind_b, rho_b, tri_b);
    ba_tri<<<nb((long long)c->nl * c->nt), 256, 0, c->stream>>>(c->hg64, tri_b, wind_b + nw);
    c->kernel_launches += 2;
}

void op_divv_tracer_adj(Context *c, const double *density, const double *wind, const double *out_b, double *in_b,
                        double *dens_b, double *wind_b)
{
    const long long nw = (long long)(c->nl + 1) * c->nc;
    kop_divv_tracer_adj<<<nb(c->ns), 256, 0, c->stream>>>(c->hg64, density, wind + nw, out_b, in_b + nw, dens_b,
                                                          wind_b + nw);
    c->kernel_launches++;
}

int adj_gen_densities(Context *c, const StepParams &p, StateMirror *so, StateMirror *sn, StateMirror *st,
                      const double *temperature, int rk, double *sed_b, StateMirror *so_b, StateMirror *sn_b,
                      StateMirror *st_b, double *t_b)
{
    if (c->n_const <= 1) return 0;
    if (c->nl > 256) return fail("three_band_solver_gen_densities_adj: more than 256 layers");
    const int n_tr = c->n_const - 1;
    const long long nsys = (long long)n_tr * c->nc, len = (long long)n_tr * c->ns;
    double *work = tracer_adj_work(c);
    if (!work) return -1;
    const TracerRows w{work, work + len, work + 2 * len, work + 3 * len};
    const dim3 boxes(nb(c->nc, 128), (unsigned)c->nl, (unsigned)n_tr);
    ka_gen_rows<<<boxes, 128, 0, c->stream>>>(c->vg, p, so->ds, sn->ds, st->ds, w);
    const unsigned cols = nb(nsys, 64);
    if (c->nl == NL_FIXED)
        ka_gen_solve<NL_FIXED, NL_FIXED><<<cols, 64, 0, c->stream>>>(c->nc, c->nl, n_tr, c->n_cond, w, sn_b->ds);
    else if (c->nl <= 64)
        ka_gen_solve<0, 64><<<cols, 64, 0, c->stream>>>(c->nc, c->nl, n_tr, c->n_cond, w, sn_b->ds);
    else
        ka_gen_solve<0, 256><<<cols, 64, 0, c->stream>>>(c->nc, c->nl, n_tr, c->n_cond, w, sn_b->ds);
    ka_gen_bars<<<boxes, 128, 0, c->stream>>>(c->vg, p, so->ds, sn->ds, temperature, rk, sed_b, w, so_b->ds, sn_b->ds,
                                              st_b->ds, t_b);
    c->kernel_launches += 3;
    /* the forward overwrites the sedimentation heat at rk 0 */
    if (rk == 0) CK(cudaMemsetAsync(sed_b, 0, (size_t)c->ns * sizeof(double), c->stream));
    CK(cudaGetLastError());
    return 0;
}

}  // namespace game
