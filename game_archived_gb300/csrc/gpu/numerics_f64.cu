/*
 * game_gpu_numerics' operations of the FP64 path (numeric.cuh, kernels.cuh),
 * in a translation unit compiled like that path's (--fmad=false).
 */
#include "context.h"
#include "kernels.cuh"
#include "numerics.h"

namespace game {
namespace {

__global__ void k_numerics_f64(int op, const double *x, double *out, long long n)
{
    const long long i = gtid();
    if (i >= n) return;
    const double a = x[i], y = numerics_two_inputs(op) ? x[n + i] : 0.0;
    double z = 0.0;
    switch (op) {
    case 11: z = div_rcp(a, y, 1.0 / y); break;
    case 12: z = div_rcp(a, y, rcp_nr<2>(y)); break;
    case 13: z = a / y; break;
    case 14: {
        const double r = 1.0 / y;
        z = div_rcp(a, y * y, r * r);
        break;
    }
    case 15: z = a / (y * y); break;
    case 16: z = rcp_full(a); break;
    case 17: z = half_of(a); break;
    case 18: z = 0.5 * a; break;
    case 19: z = cube(a); break;
    case 20: z = fourth(a); break;
    case 21: z = div_sweep(a, y, rcp_sweep(y)); break;
    default: break;
    }
    out[i] = z;
}

}  // namespace

void launch_numerics_f64(int op, const double *in, double *out, long long n)
{
    k_numerics_f64<<<(unsigned)((n + 255) / 256), 256>>>(op, in, out, n);
}

}  // namespace game
