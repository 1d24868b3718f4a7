// The FP64 pair force of the P2P kernels and the direct sums: with
// u = r / 2rs and q = u^2,
//     m g(u) / max(r, eps)^3 dx = m / (2rs)^3 f(q) dx,
//     f(q) = (erfc(u) + (2/sqrt(pi)) u exp(-u^2)) / u^3        (r >= eps)
// (src/fmm.c:823-855).
//
// GB300's FP64 pipe runs at 1/64 of the FP32 rate: one FP64 instruction
// costs a warp scheduler about 64 issue slots, more than a whole 64-bit
// fixed-point polynomial on the integer pipe.  So q is formed and f
// evaluated in integers (tables of fit_pair_fp64.py: 1280 intervals of
// degree 7, the largest error of the rounded double 1.5e-16 relative for
// q < 4 and 2.2e-17 of the Newtonian factor beyond), and a pair costs 9 FP64
// instructions: 3 differences, 3 sums, and 3 reaction sums where both
// particles are wanted.  With 1/r from rsqrt and g by Horner's rule in FP64
// it was 33; with only f in integers, 13.
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
// fit_split_fp64.py, within 5.3e-17 of g on [0, 8)), erfc and exp elsewhere
// (below 0 too: a negative split scale is not refused everywhere).
// tab: the coefficients k-major, [k][interval].
__device__ const double g_split64[SPLIT64_DEG + 1][SPLIT64_NI] = SPLIT64_C_INIT;

__device__ __forceinline__ double split_g_fp64(double u, const double *tab, double coeff)
{
    if (__double2hiint(u) >= 0 && u < SPLIT64_NI * SPLIT64_W) {
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

// the high 64 bits of a product, up to a few units in the last place
__device__ __forceinline__ unsigned long long mulhi64_near(unsigned long long a, unsigned long long b)
{
    const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a, bh = (unsigned)(b >> 32), bl = (unsigned)b;
    return (unsigned long long)ah * bh + __umulhi(ah, bl) + __umulhi(al, bh);
}

// |v| with 62 fraction bits below 2^(e + 1), e the biased exponent of the
// largest component (v below 2^-1022 counts as 0, bits below 2^(e - 61) are
// cut off)
__device__ __forceinline__ unsigned long long pair64_fixed(double v, int e)
{
    const unsigned hi = (unsigned)__double2hiint(v) & 0x7fffffffu, lo = (unsigned)__double2loint(v);
    const int ev = (int)(hi >> 20);
    const unsigned h = ev ? (hi & 0xfffffu) | 0x100000u : 0u;
    const unsigned long long m = ((unsigned long long)__funnelshift_l(lo, h, 10) << 32) | (lo << 10);
    return m >> min(e - ev, 63);
}

// f(q) on interval i, in integers: 32-bit Horner for P[7..4], 64-bit for
// P[3..0], then the double's bits (rounded to nearest).  d: the position in
// the interval, in [-1/2, 1/2) with 64 fraction bits.
__device__ __forceinline__ double pair64_poly(unsigned i, long long d, const Pair64Tab &tab)
{
    const int4 t = tab.t[i];
    const longlong2 p01 = tab.p01[i], p23 = tab.p23[i];
    const int es = tab.e[i];
    const int dh = (int)(d >> 32);
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
// from rsqrt and g from its own polynomials, ~30 FP64 instructions; two
// coincident particles get the softened factor.  Not inlined; its constants
// are read from memory, so that they take no registers of the callers, and
// ahead of their use (volatile: read where they are needed, behind a branch,
// they cost a halo's one-way lists 8 %).
__device__ __noinline__ double pair64_slow(double dx, double dy, double dz, const volatile Pair64Box *b)
{
    const double eps = b->eps, ieps3 = b->ieps3, hrs = b->hrs, cube = b->cube;
    const double r2 = dx * dx + dy * dy + dz * dz;
    const double rinv = r2 > 0.0 ? rsqrt(r2) : 0.0;
    const double dr = r2 * rinv;
    const double w = dr < eps ? ieps3 : rinv * rinv * rinv;
    return w * split_g_fp64(dr * hrs, &g_split64[0][0], 1.1283791670955126) * cube;
}

// what a pair needs of the constants in registers
struct Pair64 {
    unsigned long long k;
    int ke, qeps;
    const Pair64Box *box;
};

__device__ __forceinline__ Pair64 pair64_consts(const Pair64Box &b) { return Pair64{b.k, b.ke, b.qeps, &b}; }

// f for a source dx away; 0 where !on.  q = r^2 ia2 in fixed point too (the
// squares of the components aligned to the largest, good to 2^-58), which
// takes r^2's three FP64 instructions and the product off the FP64 pipe.
__device__ __forceinline__ double pair64_f(double dx, double dy, double dz, bool on, const Pair64 &c,
                                           const Pair64Tab &tab)
{
    const unsigned hx = (unsigned)__double2hiint(dx) & 0x7fffffffu, hy = (unsigned)__double2hiint(dy) & 0x7fffffffu,
                   hz = (unsigned)__double2hiint(dz) & 0x7fffffffu;
    const int e = (int)(max(hx, max(hy, hz)) >> 20);
    const unsigned long long x = pair64_fixed(dx, e), y = pair64_fixed(dy, e), z = pair64_fixed(dz, e);
    unsigned long long s = mulhi64_near(x, x) + mulhi64_near(y, y) + mulhi64_near(z, z);  // < 3 2^62
    const int ls = __clzll((long long)s);
    s = mulhi64_near(s << ls, c.k);
    const int l2 = (long long)s < 0 ? 0 : 1;
    s <<= l2;  // q's mantissa, leading one at bit 63 (s = 0 only for r = 0)
    // r^2 = s 2^(2 (e - 1023) - 60) before the shifts
    const int eq = 2 * (e - 1023) + 4 - ls - l2 + c.ke;
    const int qhi = ((eq + 1022) << 20) + (int)(s >> 43);
    const unsigned i = ((unsigned)(eq - PAIR64_LO) << PAIR64_MB) + ((unsigned)(s >> (63 - PAIR64_MB)) & ((1u << PAIR64_MB) - 1u));
    const bool fast = i < PAIR64_NI && qhi > c.qeps;
    double f = pair64_poly(fast ? i : 0u, (long long)((s << (PAIR64_MB + 1)) ^ (1ull << 63)), tab);
    if (on && !fast) f = pair64_slow(dx, dy, dz, c.box);
    return on ? f : 0.0;
}

}  // namespace
}  // namespace ph
