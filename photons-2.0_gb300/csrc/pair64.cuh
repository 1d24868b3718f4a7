// The FP64 pair force of the P2P kernels and the direct sums: with
// u = r / 2rs and q = u^2,
//     m g(u) / max(r, eps)^3 dx = m / (2rs)^3 f(q) dx,
//     f(q) = (erfc(u) + (2/sqrt(pi)) u exp(-u^2)) / u^3        (r >= eps)
// (src/fmm.c:823-855).
//
// GB300's FP64 pipe runs at 1/64 of the FP32 rate: one FP64 instruction
// costs a warp scheduler about 64 issue slots, more than a whole 64-bit
// fixed-point polynomial on the integer pipe.  So f is evaluated in
// integers from q's bits (tables of fit_pair_fp64.py: 1280 intervals of
// degree 7, the largest error of the rounded double 1.5e-16 relative for
// q < 4 and 2.2e-17 of the Newtonian factor beyond), and a pair costs 13
// FP64 instructions: 3 differences, 3 for r^2, one for q, 3 sums, and 3
// reaction sums where both particles are wanted.  With 1/r from rsqrt and g
// by Horner's rule in FP64 it was 33.
#pragma once

#include <cmath>

#include "fmm_internal.cuh"
#include "split_fp64_table.h"
#include "pair_fp64_table.h"

namespace ph {
namespace {

// ---------------------------------------------------------------------
// g(u) = erfc(u) + (2/sqrt(pi)) u exp(-u^2) (src/fmm.c:846-848) in FP64:
// piecewise polynomials of degree 8 on intervals of 1/16 (coefficients by
// fit_split_fp64.py, within 5.3e-17 of g on [0, 8)), erfc and exp beyond.
// tab: the coefficients k-major, [k][interval].
__device__ const double g_split64[SPLIT64_DEG + 1][SPLIT64_NI] = SPLIT64_C_INIT;

__device__ __forceinline__ double split_g_fp64(double u, const double *tab, double coeff)
{
    if (u < SPLIT64_NI * SPLIT64_W) {
        const int i = (int)(u * SPLIT64_INVW);
        const double d = u - ((double)i + 0.5) * SPLIT64_W;
        double acc = tab[SPLIT64_DEG * SPLIT64_NI + i];
#pragma unroll
        for (int k = SPLIT64_DEG - 1; k >= 0; k--) acc = fma(acc, d, tab[k * SPLIT64_NI + i]);
        return acc;
    }
    return erfc(u) + coeff * u * exp(-u * u);
}

// ---------------------------------------------------------------------
// f(q)'s tables, 66.5 KB: component-major, so that lanes on different
// intervals read different shared-memory banks
__device__ const longlong2 g_pair64_p01[PAIR64_NI] = PAIR64_P01_INIT;
__device__ const longlong2 g_pair64_p23[PAIR64_NI] = PAIR64_P23_INIT;
__device__ const int4 g_pair64_t[PAIR64_NI] = PAIR64_T_INIT;
__device__ const int g_pair64_e[PAIR64_NI] = PAIR64_E_INIT;

struct Pair64Tab {
    const longlong2 *p01, *p23;
    const int4 *t;
    const int *e;
};
#define PAIR64_BYTES (PAIR64_NI * (2 * 16 + 16 + 4))

__device__ __forceinline__ Pair64Tab pair64_global() { return Pair64Tab{g_pair64_p01, g_pair64_p23, g_pair64_t, g_pair64_e}; }

// a block's copy of the tables in shared memory (16-byte aligned, PAIR64_BYTES)
__device__ __forceinline__ Pair64Tab pair64_load(unsigned char *smem)
{
    longlong2 *p01 = reinterpret_cast<longlong2 *>(smem), *p23 = p01 + PAIR64_NI;
    int4 *t = reinterpret_cast<int4 *>(p23 + PAIR64_NI);
    int *e = reinterpret_cast<int *>(t + PAIR64_NI);
    for (int i = threadIdx.x; i < PAIR64_NI; i += blockDim.x) {
        p01[i] = g_pair64_p01[i];
        p23[i] = g_pair64_p23[i];
        t[i] = g_pair64_t[i];
        e[i] = g_pair64_e[i];
    }
    __syncthreads();
    return Pair64Tab{p01, p23, t, e};
}

// interval of q's high word; outside [2^-14, 2^6) (and for negative q,
// infinities and NaN) not below PAIR64_NI
__device__ __forceinline__ unsigned pair64_index(int qhi)
{
    return ((unsigned)qhi >> (20 - PAIR64_MB)) - ((1023 + PAIR64_LO) << PAIR64_MB);
}

// f(q) on interval i, in integers: 32-bit Horner for P[7..4], 64-bit for
// P[3..0], then the double's bits (rounded to nearest)
__device__ __forceinline__ double pair64_poly(unsigned i, double q, const Pair64Tab &tab)
{
    const unsigned hi = (unsigned)__double2hiint(q), lo = (unsigned)__double2loint(q);
    const int4 t = tab.t[i];
    const longlong2 p01 = tab.p01[i], p23 = tab.p23[i];
    const int es = tab.e[i];
    // the mantissa bits below the interval's, as d in [-1/2, 1/2) with 64 fraction bits
    const int dh = (int)(__funnelshift_l(lo, hi, 12 + PAIR64_MB) ^ 0x80000000u);
    const long long d = (long long)(((unsigned long long)(unsigned)dh << 32) | (lo << (12 + PAIR64_MB)));
    int v = t.w;
    v = t.z + __mulhi(v, dh);
    v = t.y + __mulhi(v, dh);
    v = t.x + __mulhi(v, dh);
    long long acc = p23.y + (((long long)v * dh) >> (es >> 16));
    acc = p23.x + __mul64hi(acc, d);
    acc = p01.y + __mul64hi(acc, d);
    acc = p01.x + __mul64hi(acc, d);
    // acc > 0 with 62 fraction bits, near [1/2, 1): normalise, round to 53 bits
    const int lz = __clz((int)(acc >> 32));
    const unsigned long long m = (((unsigned long long)acc << lz) + (1ull << 10)) >> 11;
    return __longlong_as_double((long long)(m + ((unsigned long long)(unsigned)((es & 0xffff) - lz) << 52)));
}

// f where the tables do not reach (r < eps, q outside their range): 1/r
// from rsqrt and g from its own polynomials; two coincident particles get
// the softened factor.  Rare: not inlined.
__device__ __noinline__ double pair64_slow(double r2, double eps, double rs)
{
    const double hrs = 0.5 / rs, cube = 8.0 * rs * rs * rs;
    const double rinv = r2 > 0.0 ? rsqrt(r2) : 0.0;
    const double dr = r2 * rinv;
    const double w = dr < eps ? 1.0 / (eps * eps * eps) : rinv * rinv * rinv;
    return w * split_g_fp64(dr * hrs, &g_split64[0][0], 2.0 / sqrt(M_PI)) * cube;
}

// Per-box constants: f's argument is r^2 ia2, the tables serve r^2 >= eps^2
// (compared as bit patterns: r^2 is not negative), and sums of f dx are
// multiplied by scale
struct Pair64 {
    double ia2, eps, rs;
    long long eps2_bits;
};

__device__ __forceinline__ Pair64 pair64_consts(double eps, double rs)
{
    Pair64 c;
    const double ia = 0.5 / rs;
    c.ia2 = ia * ia;
    c.eps = eps;
    c.rs = rs;
    c.eps2_bits = __double_as_longlong(eps * eps);
    return c;
}

__device__ __forceinline__ double pair64_scale(double mass, double rs)
{
    const double ia = 0.5 / rs;
    return mass * (ia * ia * ia);
}

// f for a source dx away; 0 where !on
__device__ __forceinline__ double pair64_f(double dx, double dy, double dz, bool on, const Pair64 &c,
                                           const Pair64Tab &tab)
{
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double q = r2 * c.ia2;
    const unsigned i = pair64_index(__double2hiint(q));
    const bool fast = i < PAIR64_NI && __double_as_longlong(r2) >= c.eps2_bits;
    double f = pair64_poly(fast ? i : 0u, q, tab);
    if (on && !fast) f = pair64_slow(r2, c.eps, c.rs);
    return on ? f : 0.0;
}

}  // namespace
}  // namespace ph
