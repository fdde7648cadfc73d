/*
 * Numeric helpers shared by the step kernels: thread index, the mixed path's
 * FP64 reciprocal and sign test, and conversions between FP64 and FP32 by
 * integer operations (kept off GB300's FP64 pipe, which runs at 1/64 of the
 * FP32 rate and also executes comparisons and conversions of doubles).
 */
#pragma once

#include <cuda_runtime.h>

namespace game {
/* internal linkage: each translation unit compiles its own copy with its own
 * contraction flags */
namespace {

/* ------------------------------------------------------------ utilities */
__device__ __forceinline__ long long gtid() { return (long long)blockIdx.x * blockDim.x + threadIdx.x; }

/* The point of a kernel over [layer][entity] fields with a two-dimensional
 * grid (layer_grid): y is the layer, x the entity, so no thread divides its
 * index by the row length (a 64-bit division, some seventy instructions
 * before the first load).  RES_ID 6, mixed: k_momentum_h 89.4 -> 78.7 us,
 * k_edge_vort 63.9 -> 56.2 us, k_cell_kinetic 24.7 -> 21.7 us.  k_waves_apply
 * and the sedimentation heat lose with it (43.7 -> 47.1, 43.4 -> 46.8 us: the
 * shorter last block of every layer) and take row_of. */
struct LayerPoint {
    int l, x;    /* layer (or level), entity */
    long long i; /* l * n + x */
    bool in;
};
__device__ __forceinline__ LayerPoint layer_point(int n)
{
    const int x = (int)(blockIdx.x * blockDim.x + threadIdx.x), l = (int)blockIdx.y;
    return {l, x, (long long)l * n + x, x < n};
}
inline dim3 layer_grid(int layers, int n, int bs) { return dim3((unsigned)((n + bs - 1) / bs), (unsigned)layers); }
/* the row of index i in rows of n, for the kernels with a one-dimensional
 * grid: a 32-bit division (every index is below 2^31: the index maps are
 * 32-bit).  kd_sdiff_div 345 -> 216 us, kd_fric_h 197 -> 168 us, kd_n2_adv
 * 104 -> 80 us (RES_ID 6, mixed).  The column kernels keep the 64-bit form,
 * once per column: k_tracers_pcr was slower with the other (181 -> 216 us). */
__device__ __forceinline__ int row_of(long long i, int n) { return (int)((unsigned)i / (unsigned)n); }

/* x == +-0 by an integer test (an FP64 comparison would issue on the FP64
 * pipe) */
__device__ __forceinline__ bool is_zero(double x) { return ((unsigned long long)__double_as_longlong(x) << 1) == 0ULL; }

/* FP64 reciprocal for the mixed path, and for the FP64 path's quotients that
 * div_rcp and div_sweep correct.  The seed is the hardware's approximate reciprocal (PTX
 * rcp.approx.ftz.f64; relative error below 2^-20, measured on GB300 over
 * 2^20 inputs spanning 1e-300..1e300), refined by Newton-Raphson steps
 * r <- r + r (1 - x r), each of which squares the relative error: one step
 * leaves about 2^-40, two steps are within one ulp of the correctly rounded
 * reciprocal and equal to it on all but a few inputs (tested against IEEE
 * 1.0 / x on 2^20 sampled inputs and edge values: only x = 1 - 2^-53, whose
 * reciprocal lies just above the midpoint of two doubles, came out one ulp
 * off).  One multiply-add pair per step
 * instead of the several FP64 operations of an IEEE division, on a GPU whose
 * FP64 rate is 1/64 of FP32.
 * x must be a normal number whose reciprocal is normal (ftz). */
template <int STEPS>
__device__ __forceinline__ double rcp_nr(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
#pragma unroll
    for (int s = 0; s < STEPS; ++s) r = fma(r, fma(-x, r, 1.0), r);
    return r;
}

/* x / y for a y whose reciprocal r = 1 / y is at hand (a grid quantity's from
 * its table, or one reciprocal shared by several quotients): the quotient
 * x r corrected once with its exact remainder (Markstein, "Computation of
 * elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
 * Dev. 34, 1990; Brisebarre, Muller and Raina, "Accelerating correctly
 * rounded floating-point division when the divisor is known in advance",
 * IEEE Trans. Computers 53, 2004), in three FP64 issues instead of the
 * division's eight or more, without its branch.  The theorem holds while
 * dividend and quotient are far from the ends of the exponent range (their
 * exponents within 500 of 0; the divisor's is then within 1000); elsewhere,
 * so for subnormal, infinite and NaN operands, divisors of 0 and overflows,
 * the call divides.  The test is four integer instructions beside FP64 ones
 * that issue at 1/64 of their rate: no kernel's time moved with it, but for
 * the column sweeps' (div_sweep).  Equal to x / y bit for bit where r is the
 * correctly rounded reciprocal (tested on the device).  With a reciprocal an
 * ulp off (rcp_nr<2>, a product of two) the same but for quotients as close
 * to the middle of two doubles as any, by divisors next to the end of their
 * binade, where one ulp is possible. */
__device__ __noinline__ double div_ieee(double x, double y) { return x / y; }
__device__ __forceinline__ bool mid_range(double x)
{
    return ((unsigned)__double2hiint(x) & 0x7ff00000u) - (523u << 20) <= 1000u << 20;
}
__device__ __forceinline__ double div_rcp(double x, double y, double r)
{
    const double q = __dmul_rn(x, r);
    double z = __fma_rn(__fma_rn(-q, y, x), r, q);
    if (!mid_range(q) || !mid_range(x)) z = is_zero(q) && is_zero(x) ? q : div_ieee(x, y);
    return z;
}
/* 1 / x as div_rcp gives it, from the hardware's seed.  Where the reciprocal
 * only serves div_rcp, whose correction absorbs its last bits, rcp_nr<2>
 * alone does. */
__device__ __forceinline__ double rcp_full(double x) { return div_rcp(1.0, x, rcp_nr<2>(x)); }
/* The same in the column sweeps, whose unrolled rows hold a column in
 * registers: a call at every quotient costs them (RES_ID 6, k_tracers_solve
 * 102 -> 177 us, k_waves_thomas 53 -> 86 us), so a selection takes its place:
 * x r itself where it is zero, subnormal, infinite or NaN, and the seed as the
 * reciprocal of a pivot that is zero, infinite or NaN.  IEEE's result for
 * those too (a subnormal pivot counts as 0, one above 2^1022 as infinite);
 * one ulp is possible where the quotient is subnormal or the dividend below
 * 2^-900. */
__device__ __forceinline__ double div_sweep(double x, double y, double r)
{
    const double q = __dmul_rn(x, r);
    const double z = __fma_rn(__fma_rn(-q, y, x), r, q);
    return ((unsigned)__double2hiint(q) & 0x7ff00000u) - 0x100000u <= 0x7fd00000u ? z : q;
}
__device__ __forceinline__ double rcp_sweep(double x)
{
    const double seed = rcp_nr<0>(x), r = rcp_nr<2>(x);
    return ((unsigned)__double2hiint(seed) & 0x7ff00000u) - 0x100000u <= 0x7fd00000u ? r : seed;
}
/* x / tab[i] with the reciprocals of tab in rtab on the FP64 path; the mixed
 * path divides in FP32 */
__device__ __forceinline__ double div_tab(double x, const double *tab, const double *rtab, long long i)
{
    return div_rcp(x, tab[i], rtab[i]);
}
__device__ __forceinline__ float div_tab(float x, const float *tab, const float *, long long i) { return x / tab[i]; }

/* x >= 0 for the solvers' branch and clip tests.  The FP64 path compares as
 * the reference does; the mixed path reads the sign bit on the integer pipe
 * instead of issuing an FP64 comparison (FP64 issues at 1/64 of the FP32
 * rate on this GPU).  The two differ only at -0, where every branch they
 * select between yields the same values up to the sign of a zero term. */
template <bool EXACT>
__device__ __forceinline__ bool nonneg(double x)
{
    return EXACT ? x >= 0.0 : __double2hiint(x) >= 0;
}

/* double -> float rounded to nearest even, by integer operations alone: the same
 * bits as float(x), zeros, subnormal results, overflows, infinities and NaNs
 * included (tested).  Used by the mixed path where it writes its FP32 shadow
 * from FP64 results, to keep the conversion off the FP64 pipe (one warp
 * instruction per 16 cycles).  No case may use the conversion instruction: the
 * compiler runs it ahead of the test that guards it, so a fallback costs every
 * value its FP64 issue.  RES_ID 6, against the form with a fallback in the same
 * tree: k_make_shadow 39.0 -> 36.1 us, k_cell_prepare_f32 58.7 -> 56.6 us.
 * Where a kernel converts a value or two per point beside gathers that wait
 * for L2, the instruction's issue hides and the longer code does not: most of
 * the diffusion kernels convert by the instruction (diff.cuh). */
__device__ __forceinline__ float to_float(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x), m = b & 0xfffffffffffffULL;
    const unsigned e = (unsigned)(b >> 52) & 0x7ffu, sign = (unsigned)(b >> 63) << 31;
    if (e - 897u <= 253u) { /* float exponent field e - 896 in [1, 254] */
        unsigned r = sign | ((e - 896u) << 23) | (unsigned)(m >> 29);
        const unsigned rem = (unsigned)(m & 0x1fffffffULL), half = 0x10000000u;
        r += (rem > half || (rem == half && (r & 1u))) ? 1u : 0u;
        return __uint_as_float(r);
    }
    if (e > 896u) /* beyond the float range, infinity, NaN */
        return __uint_as_float(sign | 0x7f800000u | (e == 0x7ffu && m != 0ULL ? 0x400000u | (unsigned)(m >> 29) : 0u));
    const unsigned shift = 926u - e; /* to units of the smallest subnormal float */
    if (shift > 54u) return __uint_as_float(sign);
    const unsigned long long v = m | 0x10000000000000ULL, rem = v & ((1ULL << shift) - 1ULL), half = 1ULL << (shift - 1u);
    unsigned r = (unsigned)(v >> shift);
    r += (rem > half || (rem == half && (r & 1u))) ? 1u : 0u;
    return __uint_as_float(sign | r);
}

/* float -> double (exact) by integer operations alone, for the same reason:
 * the same bits as double(x) except a NaN's payload.  The mixed path widens
 * its FP32 sums and products with it before the FP64 accumulation.  wide() is
 * the identity on double. */
__device__ __forceinline__ double to_double(float x)
{
    const unsigned u = __float_as_uint(x), sign = u & 0x80000000u;
    const unsigned fe = (u >> 23) & 0xffu;
    if (fe - 1u <= 253u) /* normal */
        return __hiloint2double((int)(sign | ((fe + 896u) << 20) | ((u >> 3) & 0xfffffu)), (int)(u << 29));
    const unsigned m = u & 0x7fffffu;
    if (fe != 0u) /* infinity, NaN */
        return __hiloint2double((int)(sign | 0x7ff00000u | (m ? 0x80000u : 0u) | (m >> 3)), (int)(m << 29));
    if (m == 0u) return __hiloint2double((int)sign, 0);
    const int p = 31 - __clz((int)m); /* m 2^-149 = 1.f 2^(p - 149) */
    const unsigned long long f = ((unsigned long long)m << (52 - p)) & 0xfffffffffffffULL;
    return __hiloint2double((int)(sign | ((unsigned)(p + 874) << 20) | (unsigned)(f >> 32)), (int)(unsigned)f);
}

/* FP64 operations that stay behind the test that guards them: the compiler runs
 * plain ones ahead of it and selects, and each issue holds the FP64 pipe for 16
 * cycles */
__device__ __forceinline__ double guarded_mul(double a, double b)
{
    double r;
    asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
    return r;
}
__device__ __forceinline__ double guarded_add(double a, double b)
{
    double r;
    asm volatile("add.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
    return r;
}
__device__ __forceinline__ double guarded_fma(double a, double b, double c)
{
    double r;
    asm volatile("fma.rn.f64 %0, %1, %2, %3;" : "=d"(r) : "d"(a), "d"(b), "d"(c));
    return r;
}

/* half of x exactly, without an FP64 instruction for normal numbers whose half
 * is normal, and zeros */
__device__ __forceinline__ double half_of(double x)
{
    const int hi = __double2hiint(x);
    if (((unsigned)(hi >> 20) & 0x7ffu) - 2u <= 2044u) return __hiloint2double(hi - 0x100000, __double2loint(x));
    return is_zero(x) ? x : guarded_mul(0.5, x);
}

/* a double passed to either conversion would be narrowed silently */
double to_double(double) = delete;
float to_float(float) = delete;
__device__ __forceinline__ double wide(float x) { return to_double(x); }
__device__ __forceinline__ double wide(double x) { return x; }
/* x in the horizontal precision R (to_float from double to float) */
template <typename R, typename F>
__device__ __forceinline__ R as(F x)
{
    if constexpr (sizeof(R) == sizeof(float) && sizeof(F) == sizeof(double)) return to_float(x);
    else return x;
}

}  // namespace
}  // namespace game
