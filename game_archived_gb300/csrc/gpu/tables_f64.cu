/*
 * The FP64 path's tables of reciprocals and products of grid quantities
 * (HGrid<double>), formed on the device from the grid tables already there:
 * IEEE divisions, compiled with --fmad=false, so every entry is the value
 * the operators would form at each point of each step.
 */
#include "context.h"
#include "kernels.cuh"

namespace game {
namespace {

__global__ void k_reciprocal(long long n, const double *x, double *r)
{
    const long long i = gtid();
    if (i < n) r[i] = 1.0 / x[i];
}

/* of z_h(k-1) - z_h(k), the edge heights' differences (vorticities.c:200-214) */
__global__ void k_r_dz_h(HGrid<double> g, double *r)
{
    const LayerPoint p = layer_point(g.ne);
    if (!p.in || p.l == 0 || p.l == g.nl) return;
    r[p.i] = 1.0 / (g.z_h[p.i - g.ne] - g.z_h[p.i]);
}

/* the rhombus's area: the sum of its two triangles' (vorticities.c:104-165) */
__global__ void k_rhombus_area(HGrid<double> g, double *a, double *r)
{
    const LayerPoint p = layer_point(g.ne);
    if (!p.in) return;
    const double *at = g.dual_area_t + (long long)p.l * g.nt;
    const double s = at[g.dual_from[p.x]] + at[g.dual_to[p.x]];
    a[p.i] = s;
    r[p.i] = 1.0 / s;
}

/* circulation weights of the triangles' edges: the edge length rescaled to
 * the triangle's height in the orography layers, times the sign
 * (vorticities.c:167-222) */
__global__ void k_tri_circ(HGrid<double> g, double *w)
{
    const LayerPoint p = layer_point(g.nt);
    if (!p.in) return;
    const long long n = (long long)g.nl * g.nt;
    for (int j = 0; j < 3; ++j) {
        const int e = g.vort_i[j * g.nt + p.x];
        const long long le = (long long)p.l * g.ne + e;
        double rescale = 1.0;
        if (p.l >= g.nl - g.n_oro) rescale = (g.radius + g.dual_z_t[p.i]) / (g.radius + g.z_h[le]);
        w[j * n + p.i] = rescale * g.nd_h[le] * double(g.vort_s[j * g.nt + p.x]);
    }
}

/* weights of the terrain corrections (averaging.c:41-95) */
__global__ void k_corr_w(HGrid<double> g, double *w)
{
    const LayerPoint p = layer_point(g.nc);
    if (!p.in) return;
    const long long ns = (long long)g.nl * g.nc;
    const int n_edges = p.x < N_PENT ? 5 : 6;
    for (int j = 0; j < 6; ++j)
        w[j * ns + p.i] =
            j < n_edges ? -0.5 * ipw_at(g, j, p.l, p.x) * g.slope_h[(long long)p.l * g.ne + g.adj[j * g.nc + p.x]] : 0.0;
}

}  // namespace

int make_f64_tables(Context *c)
{
    const HGrid<double> &g = c->hg64;
    cudaStream_t st = c->stream;
    const long long nwc = (long long)(c->nl + 1) * c->nc, nze = (long long)(c->nl + 1) * c->ne;
    const long long nue = (long long)c->nl * c->ne, ntt = (long long)c->nl * c->nt;
    auto rcp = [&](long long n, const double *x, const double *r) {
        k_reciprocal<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, x, const_cast<double *>(r));
    };
    rcp(nwc, g.nd_v, g.r_nd_v);
    rcp(nue, g.nd_h, g.r_nd_h);
    rcp(nze, g.dual_area_h, g.r_dual_area_h);
    rcp(ntt, g.dual_area_t, g.r_dual_area_t);
    k_r_dz_h<<<layer_grid(c->nl + 1, c->ne, 256), 256, 0, st>>>(g, const_cast<double *>(g.r_dz_h));
    k_rhombus_area<<<layer_grid(c->nl, c->ne, 256), 256, 0, st>>>(g, const_cast<double *>(g.rhombus_area),
                                                                  const_cast<double *>(g.r_rhombus_area));
    k_tri_circ<<<layer_grid(c->nl, c->nt, 256), 256, 0, st>>>(g, const_cast<double *>(g.tri_circ));
    CK(cudaGetLastError());
    return 0;
}

int make_f64_corr_weights(Context *c)
{
    k_corr_w<<<layer_grid(c->nl, c->nc, 256), 256, 0, c->stream>>>(c->hg64, const_cast<double *>(c->hg64.corr_w));
    CK(cudaGetLastError());
    return 0;
}

}  // namespace game
