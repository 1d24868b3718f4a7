// PM long-range force on an N^3 periodic mesh, the other half of the
// reference's force split (src/partmesh.c:18-800 for one rank,
// src/conv.f90:128-247 for the convolution):
//   1. cloud-in-cell deposit of the particle mass, scaled to a density by
//      (N/L)^3 (src/partmesh.c:86-180);
//   2. FFT, multiplication by the long-range Green's function
//      G(k) = L^2 / (pi N^3) exp(-|k|^2 (2 pi rs / L)^2) / |k|^2 / W(k)^2,
//      W = prod sinc(pi k_d / N) (the CIC window, deconvolved twice), and the
//      inverse FFT: the potential psi with G-free units (conv.f90:171-227);
//   3. a 4-point finite-difference gradient of psi per mesh cell
//      (src/partmesh.c:524-735) and its CIC interpolation to the particles:
//      acc_pm = grad psi (src/partmesh.c:574-587).
// The Green's function and the transforms are FP64; the weights, the gradient
// and the interpolation sums are 64-bit integers that resolve more than a
// double's 53 bits of what they are added to.  The constant pi is the
// reference's: conv.f90 declares `real*8, parameter :: M_PI = 3.1415926`, a
// default (single-precision) real literal, so its value is 3.1415926 rounded
// to FP32 (3.141592502593994).
// The deposit adds with FP64 atomics, so its summation order (and the last
// bits of the density) varies from run to run.
#include <cufft.h>

#include <cmath>
#include <cstring>

#include "api_internal.cuh"

namespace {

constexpr double PM_PI = (double)3.1415926f;  // src/conv.f90:171

__device__ __forceinline__ int wrap(int a, int N) { return a < 0 ? a + N : (a >= N ? a - N : a); }

// nearest cell, neighbour cell on the particle's side and the two weights
// per axis (src/partmesh.c:91-132)
__device__ __forceinline__ void cic_axis(double x, double norm, double delta, int N, int &c, int &cn, double &w,
                                         double &wn)
{
    c = (int)__dmul_rn(x, norm);
    w = __dmul_rn(__dsub_rn(x, __dmul_rn((double)c + 0.5, delta)), norm);
    if (w > 0) {
        cn = c + 1;
    } else {
        w = -w;
        cn = c - 1;
    }
    wn = __dsub_rn(1.0, w);
    c = wrap(c, N);
    cn = wrap(cn, N);
}

__device__ __forceinline__ size_t cell(int i, int j, int k, int N) { return ((size_t)i * N + j) * N + k; }


// The same in 64-bit integers.  GB300 issues one warp instruction on doubles
// in the time of about 35 on integers, and the deposit and the interpolation
// were bound by them.  Weights in units of 2^-63.  The cell's centre is the
// reference's (c + 1/2) delta rounded to a double; the distance to it and its
// product with N / L are held to 2^-53 of a cell, a product of weights to
// 2^-62.  (The exact centre instead took 8 us less and halved the error
// against extended precision, but left the reference's rounding: 2.2e-15
// against 1.4e-15 of the FP64 evaluation's forces.)
// A particle more than half a cell below the box has weights the reference
// leaves outside [0, 1] (its cell index is truncated towards zero, so the
// distance to the centre is up to 1.5 cells and the neighbour's weight
// negative): its weights are doubles, held as bit patterns.
enum { CIC_FIXED = 0, CIC_SIGNED = 1, CIC_NAN = 2 };

struct CicFix {
    int i, j, k, ii, jj, kk;
    unsigned long long wi, wj, wk, win, wjn, wkn;
    int kind;
};

// N / L and its inverse: mantissas (64 bits with the top one set, 53 bits)
// and exponent fields; ok: both are ordinary doubles
struct Norm64 {
    unsigned long long mant, dmant;
    int expo, dexpo;
    double norm, delta;
    bool ok;
};

__device__ __forceinline__ void cic_axis_fix(double x, const Norm64 &q, int N, int &c, int &cn, unsigned long long &w,
                                             unsigned long long &wn, int &kind)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)(b >> 52);  // with the sign: negative x has ex >= 2048
    const int sh = 2056 - ex - q.expo;
    const unsigned long long mx = (b & ((1ULL << 52) - 1)) | (ex ? 1ULL << 52 : 0);
    // u = x N / L in units of 2^-52, rounded
    const unsigned long long hi = __umul64hi(mx << 11, q.mant);
    const unsigned long long half = sh > 0 && sh <= 64 ? (hi >> ((sh - 1) & 63)) & 1 : 0;
    const unsigned long long u = (sh >= 0 && sh < 64 ? hi >> sh : 0) + half;
    c = (int)(u >> 52);
    if (q.ok && ex < 2047 && sh >= 0 && c < 1024) {
        // (2 c + 1) delta in units of half delta's last place, rounded to 53
        // bits, half to even
        unsigned long long m = (unsigned long long)(2 * c + 1) * q.dmant;
        const int cut = 11 - __clzll((long long)m);
        if (cut > 0) m = (m + ((1ULL << (cut - 1)) - 1) + ((m >> cut) & 1)) & ~((1ULL << cut) - 1);
        // x in the same units: below delta its last bits may be cut off
        const int up = ex - q.dexpo + 1;
        const unsigned long long xm = up >= 0 ? mx << up : (up > -64 ? mx >> -up : 0);
        const long long t = (long long)(xm - m);
        const unsigned long long d = (unsigned long long)(t > 0 ? t : -t);
        cn = t > 0 ? c + 1 : c - 1;
        w = __umul64hi(d << 10, q.mant) << (q.expo + q.dexpo - 2045);
        w = min(w, 1ULL << 63);
        wn = (1ULL << 63) - w;
        c = wrap(c, N);
        cn = wrap(cn, N);
    } else if (isfinite(x)) {  // below the box, or many cells above its lower edge
        double v, vn;
        cic_axis(x, q.norm, q.delta, N, c, cn, v, vn);
        if (vn < 0.0) kind = max(kind, (int)CIC_SIGNED);
        w = __double2ull_rn(v * 9223372036854775808.0);  // 2^63
        wn = __double2ull_rn(vn * 9223372036854775808.0);
    } else {
        c = cn = 0;
        w = wn = 0;
        kind = CIC_NAN;
    }
}

__device__ __forceinline__ CicFix cic_fix(const double *pos, int p, const Norm64 &q, int N)
{
    CicFix s;
    s.kind = CIC_FIXED;
    const double x = pos[3 * (size_t)p], y = pos[3 * (size_t)p + 1], z = pos[3 * (size_t)p + 2];
    cic_axis_fix(x, q, N, s.i, s.ii, s.wi, s.win, s.kind);
    cic_axis_fix(y, q, N, s.j, s.jj, s.wj, s.wjn, s.kind);
    cic_axis_fix(z, q, N, s.k, s.kk, s.wk, s.wkn, s.kind);
    if (s.kind == CIC_SIGNED) {
        double w[3], wn[3];
        cic_axis(x, q.norm, q.delta, N, s.i, s.ii, w[0], wn[0]);
        cic_axis(y, q.norm, q.delta, N, s.j, s.jj, w[1], wn[1]);
        cic_axis(z, q.norm, q.delta, N, s.k, s.kk, w[2], wn[2]);
        s.wi = __double_as_longlong(w[0]);
        s.wj = __double_as_longlong(w[1]);
        s.wk = __double_as_longlong(w[2]);
        s.win = __double_as_longlong(wn[0]);
        s.wjn = __double_as_longlong(wn[1]);
        s.wkn = __double_as_longlong(wn[2]);
    }
    return s;
}

// product of two weights
__device__ __forceinline__ unsigned long long wmul(unsigned long long a, unsigned long long b)
{
    return __umul64hi(a, b) << 1;
}

// of two weights of a CIC_SIGNED particle
__device__ __forceinline__ unsigned long long wmul_signed(unsigned long long a, unsigned long long b)
{
    return __double_as_longlong(__dmul_rn(__longlong_as_double(a), __longlong_as_double(b)));
}

// a weight (2^-63 units, at most 2^63) as a double, rounded to nearest
__device__ __forceinline__ double weight_d(unsigned long long v)
{
    const int lz = __clzll((long long)v);
    const unsigned long long m = v << (lz & 63);
    const unsigned long long r = (m >> 11) + ((m >> 10) & 1);  // with the leading bit
    return v ? __longlong_as_double((long long)(((unsigned long long)(1022 - lz) << 52) + r)) : 0.0;
}

// a corner's weight from its xy and z parts
__device__ __forceinline__ double corner_d(unsigned long long xy, unsigned long long z, int kind)
{
    if (kind == CIC_FIXED) return weight_d(wmul(xy, z));
    return kind == CIC_SIGNED ? __longlong_as_double(wmul_signed(xy, z)) : __longlong_as_double(0x7ff8000000000000LL);
}

// A warp takes 32 particles; two lanes then add one particle's corners, one
// lane the four at its nearest plane in z and one those at the next, so that
// the two addresses of a pair lie in one 32-byte sector three times in four.
// Bound by the atomics now: 10^6 clustered particles, 128 cells a side,
// 136 -> 90 us (a lane per particle and FP64 weights before).
__global__ void k_pm_deposit(const double *__restrict__ pos, int n, int N, Norm64 q, double *rho)
{
    const int lane = warp_lane(), odd = lane & 1;
    const int step = gridDim.x * blockDim.x;
    for (int p0 = blockIdx.x * blockDim.x + threadIdx.x - lane; p0 < n; p0 += step) {
        const int p = p0 + lane;
        CicFix s{};
        if (p < n) s = cic_fix(pos, p, q, N);
        unsigned long long nn = wmul(s.win, s.wjn), in = wmul(s.wi, s.wjn), nj = wmul(s.win, s.wj), ij = wmul(s.wi, s.wj);
        if (s.kind == CIC_SIGNED) {
            nn = wmul_signed(s.win, s.wjn);
            in = wmul_signed(s.wi, s.wjn);
            nj = wmul_signed(s.win, s.wj);
            ij = wmul_signed(s.wi, s.wj);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int src = (lane & ~1) | h;
            const int pi = __shfl_sync(0xffffffffu, s.i, src), pii = __shfl_sync(0xffffffffu, s.ii, src);
            const int pj = __shfl_sync(0xffffffffu, s.j, src), pjj = __shfl_sync(0xffffffffu, s.jj, src);
            // each lane of the pair needs its plane of the source particle
            const int k0 = __shfl_sync(0xffffffffu, s.k, src), k1 = __shfl_sync(0xffffffffu, s.kk, src);
            const unsigned long long z0 = __shfl_sync(0xffffffffu, s.wkn, src), z1 = __shfl_sync(0xffffffffu, s.wk, src);
            const unsigned long long a = __shfl_sync(0xffffffffu, nn, src), b = __shfl_sync(0xffffffffu, in, src);
            const unsigned long long c = __shfl_sync(0xffffffffu, nj, src), d = __shfl_sync(0xffffffffu, ij, src);
            const int kind = __shfl_sync(0xffffffffu, s.kind, src);
            if (p0 + src >= n) continue;
            const int k = odd ? k1 : k0;
            const unsigned long long z = odd ? z1 : z0;
            atomicAdd(rho + cell(pi, pj, k, N), corner_d(a, z, kind));
            atomicAdd(rho + cell(pii, pj, k, N), corner_d(b, z, kind));
            atomicAdd(rho + cell(pi, pjj, k, N), corner_d(c, z, kind));
            atomicAdd(rho + cell(pii, pjj, k, N), corner_d(d, z, kind));
        }
    }
}

// sinc(pi q / N), 1 at q = 0, as the reference forms it
__device__ __forceinline__ double pm_sinc(int q, int N)
{
    if (q == 0) return 1.0;
    const double f = __ddiv_rn(__dmul_rn(PM_PI, (double)q), (double)N);
    return __ddiv_rn(sin(f), f);
}

// the Green's function on the half spectrum [N][N][N/2+1]; it depends only
// on the mesh size, L and rs, so a context computes it once per set
__global__ void k_pm_green_table(double *G, int N, double pref, double ismth2)
{
    const int nz = N / 2 + 1, nhalf = N / 2;
    const size_t m = (size_t)N * N * nz;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < m; t += (size_t)gridDim.x * blockDim.x) {
        int a = (int)(t / ((size_t)N * nz)), b = (int)((t / nz) % N), c = (int)(t % nz);
        if (a > nhalf) a -= N;
        if (b > nhalf) b -= N;
        if (c > nhalf) c -= N;
        double gf;
        if (a == 0 && b == 0 && c == 0) {
            gf = pref;
        } else {
            const double fx = pm_sinc(a, N), fy = pm_sinc(b, N), fz = pm_sinc(c, N);
            const double k2 = (double)(a * a + b * b + c * c);
            const double ff = __ddiv_rn(1.0, __dmul_rn(__dmul_rn(fx, fy), fz));
            gf = __dmul_rn(pref, exp(__dmul_rn(-k2, ismth2)));
            gf = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(gf, ff), ff), ff), ff);
            gf = __ddiv_rn(gf, k2);
        }
        G[t] = gf;
    }
}

// the half spectrum times the Green's function and the density of one
// particle's mass in one cell, m (N/L)^3 (the deposit adds weights)
__global__ void k_pm_green(cufftDoubleComplex *rk, const double *__restrict__ G, size_t m, double mass_density)
{
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < m; t += (size_t)gridDim.x * blockDim.x) {
        const double gf = __dmul_rn(G[t], mass_density);
        rk[t].x = __dmul_rn(rk[t].x, gf);
        rk[t].y = __dmul_rn(rk[t].y, gf);
    }
}

// 4-point derivative along each axis (src/partmesh.c:524-531):
// f1 invx (psi+1 - psi-1) - f2 invx (psi+2 - psi-2), f1 = 4/3, f2 = 1/6, invx = N / (2 L)
// = invx / 6 (8 (psi+1 - psi-1) - (psi+2 - psi-2)).
// The bracket is formed in 64-bit integers from the twelve potentials, in
// units of 2^-58 of the power of two above the largest of them (exact where
// they are within a factor of 32 of it, and better than one rounded
// difference elsewhere); the interpolation multiplies by invx / 6.
// (x, y, z, exponent) per cell, one 32-byte record, so that the
// interpolation's eight corners are eight sector loads.  128 cells a side:
// 65 -> 42 us.
using GradCell = longlong4_32a;  // w: exponent field of the largest potential, 2047 if one is not finite

__device__ __forceinline__ int d_expo(double v) { return (int)((__double_as_longlong(v) >> 52) & 2047); }

// v in units of 2^(e - 1023 - 57), e the largest exponent field around
__device__ __forceinline__ long long d_fix(double v, int e)
{
    const long long b = __double_as_longlong(v);
    const int ev = (int)((b >> 52) & 2047);
    const long long m = ((b & ((1LL << 52) - 1)) | (ev ? 1LL << 52 : 0)) << 5;
    const int sh = e - (ev ? ev : 1);
    const long long r = sh < 64 ? m >> sh : 0;
    return b < 0 ? -r : r;
}

__global__ void k_pm_gradient(const double *__restrict__ psi, int N, GradCell *__restrict__ g)
{
    const unsigned m2 = (unsigned)N * N;
    const size_t m = (size_t)m2 * N;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < m; t += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(t / m2);
        const unsigned r = (unsigned)(t - (size_t)i * m2);
        const int j = (int)(r / (unsigned)N), k = (int)(r % (unsigned)N);
        double v[12];  // +1, -1, +2, -2 along x, y, z
#pragma unroll
        for (int o = 0; o < 4; o++) {
            const int d = (o & 1) ? -(o / 2 + 1) : o / 2 + 1;
            v[o] = psi[cell(wrap(i + d, N), j, k, N)];
            v[4 + o] = psi[cell(i, wrap(j + d, N), k, N)];
            v[8 + o] = psi[cell(i, j, wrap(k + d, N), N)];
        }
        int e = 1;
#pragma unroll
        for (int o = 0; o < 12; o++) e = max(e, d_expo(v[o]));
        long long d[3];
#pragma unroll
        for (int a = 0; a < 3; a++)
            d[a] = 8 * (d_fix(v[4 * a], e) - d_fix(v[4 * a + 1], e)) - (d_fix(v[4 * a + 2], e) - d_fix(v[4 * a + 3], e));
        g[t] = make_longlong4_32a(d[0], d[1], d[2], e);
    }
}

// the eight weighted cell values, the three components at once: 64-bit
// integer products summed at the largest corner's exponent, to 2^-56 of the
// largest potential around it (the potential itself is known to 2^-53).
// 10^6 particles, 128 cells a side: 132 -> 68 us.
__global__ void k_pm_interp(const double *__restrict__ pos, int n, int N, Norm64 q, double invx6,
                            const GradCell *__restrict__ g, double *acc)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const CicFix s = cic_fix(pos, p, q, N);
        GradCell c[8];
#pragma unroll
        for (int o = 0; o < 8; o++)
            c[o] = g[cell((o & 1) ? s.ii : s.i, (o & 2) ? s.jj : s.j, (o & 4) ? s.kk : s.k, N)];
        int e = 1;
#pragma unroll
        for (int o = 0; o < 8; o++) e = max(e, (int)c[o].w);
        // sums are in units of 2^(e - 1078); two factors stay inside the range of doubles
        const int h = (e - 1078) >> 1, h2 = e - 1078 - h;
        const double f2 = __longlong_as_double((long long)(h2 + 1023) << 52);
        const double f = s.kind != CIC_NAN && e < 2047 ? invx6 * __longlong_as_double((long long)(h + 1023) << 52)
                                                       : __longlong_as_double(0x7ff8000000000000LL);
        if (s.kind == CIC_SIGNED) {
            double v[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int o = 0; o < 8; o++) {
                const unsigned long long xy = wmul_signed((o & 1) ? s.wi : s.win, (o & 2) ? s.wj : s.wjn);
                const double w = __longlong_as_double(wmul_signed(xy, (o & 4) ? s.wk : s.wkn));
                const int up = (int)c[o].w - e - 2;
                v[0] = fma(w, ldexp((double)c[o].x, up), v[0]);
                v[1] = fma(w, ldexp((double)c[o].y, up), v[1]);
                v[2] = fma(w, ldexp((double)c[o].z, up), v[2]);
            }
            for (int d = 0; d < 3; d++) acc[3 * (size_t)p + d] = v[d] * f * f2;
            continue;
        }
        const unsigned long long xy[4] = {wmul(s.win, s.wjn), wmul(s.wi, s.wjn), wmul(s.win, s.wj), wmul(s.wi, s.wj)};
        long long ax = 4, ay = 4, az = 4;  // eight products are cut off below: half a unit each
#pragma unroll
        for (int o = 0; o < 8; o++) {
            const long long w = (long long)__umul64hi(xy[o & 3], (o & 4) ? s.wk : s.wkn);  // 2^-62 units
            const int sh = min(63, e - (int)c[o].w);
            ax += __mul64hi(c[o].x, w) >> sh;
            ay += __mul64hi(c[o].y, w) >> sh;
            az += __mul64hi(c[o].z, w) >> sh;
        }
        acc[3 * (size_t)p] = (double)ax * f * f2;
        acc[3 * (size_t)p + 1] = (double)ay * f * f2;
        acc[3 * (size_t)p + 2] = (double)az * f * f2;
    }
}

int cufft_error(cufftResult r, const char *what)
{
    return ph_set_error(PH_ERR_CUDA, "%s failed (cuFFT status %d)", what, (int)r);
}

}  // namespace

// mesh buffers and FFT plans of one mesh size, kept in the context
int ph_pm_prepare(photons_ctx *c, int N)
{
    if (c->pm_n == N) return 0;
    if (c->pm_plan_r2c) cufftDestroy(c->pm_plan_r2c);
    if (c->pm_plan_c2r) cufftDestroy(c->pm_plan_c2r);
    c->pm_plan_r2c = c->pm_plan_c2r = 0;
    cudaFree(c->pm_rho); cudaFree(c->pm_rk); cudaFree(c->pm_grad); cudaFree(c->pm_green);
    c->pm_rho = nullptr; c->pm_rk = nullptr; c->pm_grad = nullptr; c->pm_green = nullptr;
    c->pm_n = 0;
    c->pm_green_pref = c->pm_green_ismth2 = 0.0;
    const size_t m = (size_t)N * N * N, mk = (size_t)N * N * (N / 2 + 1);
    cudaError_t e = cudaMalloc(&c->pm_rho, sizeof(double) * m);
    if (e == cudaSuccess) e = cudaMalloc(&c->pm_rk, sizeof(cufftDoubleComplex) * mk);
    if (e == cudaSuccess) e = cudaMalloc(&c->pm_grad, 4 * sizeof(double) * m);
    if (e == cudaSuccess) e = cudaMalloc(&c->pm_green, sizeof(double) * mk);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return ph_set_error(PH_ERR_NOMEM, "PM mesh of %d^3 cells does not fit", N);
    }
    cufftResult r = cufftPlan3d(&c->pm_plan_r2c, N, N, N, CUFFT_D2Z);
    if (r != CUFFT_SUCCESS) return cufft_error(r, "cufftPlan3d (forward)");
    r = cufftPlan3d(&c->pm_plan_c2r, N, N, N, CUFFT_Z2D);
    if (r != CUFFT_SUCCESS) return cufft_error(r, "cufftPlan3d (inverse)");
    c->pm_n = N;
    return 0;
}

void ph_pm_release(photons_ctx *c)
{
    if (c->pm_plan_r2c) cufftDestroy(c->pm_plan_r2c);
    if (c->pm_plan_c2r) cufftDestroy(c->pm_plan_c2r);
    cudaFree(c->pm_rho); cudaFree(c->pm_rk); cudaFree(c->pm_grad); cudaFree(c->pm_green);
    c->pm_plan_r2c = c->pm_plan_c2r = 0;
    c->pm_rho = nullptr; c->pm_rk = nullptr; c->pm_grad = nullptr; c->pm_green = nullptr;
    c->pm_n = 0;
    c->pm_green_pref = c->pm_green_ismth2 = 0.0;
}

// enqueue the PM force on device positions pos[3n] into acc_pm[3n]
int ph_pm_enqueue(photons_ctx *c, const photons_params *p, int N, int n, const double *pos, double *acc_pm)
{
    PH_TRY(ph_pm_prepare(c, N));
    cudaStream_t st = c->stream;
    const size_t m = (size_t)N * N * N, mk = (size_t)N * N * (N / 2 + 1);
    const int blocks = ph::device_sm_count() * 8;
    const double L = p->boxsize;
    const double norm = (double)N / L, delta = 1.0 / norm;  // src/partmesh.c:85-86
    PH_CUDA_CHECK(cudaMemsetAsync(c->pm_rho, 0, sizeof(double) * m, st));
    Norm64 q;
    q.norm = norm;
    q.delta = delta;
    unsigned long long nb, db;
    memcpy(&nb, &norm, sizeof nb);
    memcpy(&db, &delta, sizeof db);
    q.mant = ((nb & ((1ULL << 52) - 1)) | 1ULL << 52) << 11;
    q.dmant = (db & ((1ULL << 52) - 1)) | 1ULL << 52;
    q.expo = (int)(nb >> 52);
    q.dexpo = (int)(db >> 52);
    q.ok = std::isnormal(norm) && std::isnormal(delta);  // otherwise weights are formed in FP64
    ph::note_launch(), k_pm_deposit<<<blocks, 256, 0, st>>>(pos, n, N, q, c->pm_rho);
    double renormal = (double)N / L;
    renormal = renormal * renormal * renormal;
    cufftResult r = cufftSetStream(c->pm_plan_r2c, st);
    if (r == CUFFT_SUCCESS) r = cufftSetStream(c->pm_plan_c2r, st);
    if (r == CUFFT_SUCCESS) r = cufftExecD2Z(c->pm_plan_r2c, c->pm_rho, c->pm_rk);
    if (r != CUFFT_SUCCESS) return cufft_error(r, "cufftExecD2Z");
    // conv.f90:175-177: ismth2 = (2 pi rs / L)^2, pref = L^2 / (pi N^3)
    double ismth2 = 2 * PM_PI * p->rs / L;
    ismth2 = ismth2 * ismth2;
    const double pref = L * L / (PM_PI * (double)N * (double)N * (double)N);
    if (c->pm_green_pref != pref || c->pm_green_ismth2 != ismth2) {
        ph::note_launch(), k_pm_green_table<<<blocks, 256, 0, st>>>(c->pm_green, N, pref, ismth2);
        c->pm_green_pref = pref;
        c->pm_green_ismth2 = ismth2;
    }
    ph::note_launch(), k_pm_green<<<blocks, 256, 0, st>>>(c->pm_rk, c->pm_green, mk, p->mass * renormal);
    r = cufftExecZ2D(c->pm_plan_c2r, c->pm_rk, c->pm_rho);
    if (r != CUFFT_SUCCESS) return cufft_error(r, "cufftExecZ2D");
    const double invx = 0.5 * N / L;  // src/partmesh.c:458
    GradCell *g = reinterpret_cast<GradCell *>(c->pm_grad);
    ph::note_launch(), k_pm_gradient<<<blocks, 256, 0, st>>>(c->pm_rho, N, g);
    ph::note_launch(), k_pm_interp<<<blocks, 256, 0, st>>>(pos, n, N, q, invx / 6.0, g, acc_pm);
    PH_CUDA_CHECK(cudaGetLastError());
    return 0;
}

extern "C" int photons_pm_force(photons_ctx *c, const photons_params *p, int nside, int n, const double *pos,
                                double *acc_pm)
{
    photons_gpu_clear_error();
    if (!c || !p || !pos || !acc_pm) return ph_set_error(PH_ERR_ARG, "null argument");
    if (n < 1 || nside < 4 || nside > 2048) return ph_set_error(PH_ERR_ARG, "bad PM arguments (n %d, mesh %d)", n, nside);
    if (!(p->boxsize > 0) || !(p->rs > 0)) return ph_set_error(PH_ERR_ARG, "invalid PM parameters");
    cudaSetDevice(c->device);
    cudaStream_t st = c->stream;
    const int dio = p->flags & PHOTONS_F_DEVICE_IO;
    const double *dpos = pos;
    double *dacc = acc_pm;
    if (!dio) {
        if (n > c->pm_cap_io) {
            cudaFree(c->pm_io);
            c->pm_io = nullptr;
            c->pm_cap_io = 0;
            if (cudaMalloc(&c->pm_io, sizeof(double) * 6 * (size_t)n) != cudaSuccess) {
                cudaGetLastError();
                return ph_set_error(PH_ERR_NOMEM, "PM staging for %d particles does not fit", n);
            }
            c->pm_cap_io = n;
        }
        PH_CUDA_CHECK(cudaMemcpyAsync(c->pm_io, pos, sizeof(double) * 3 * (size_t)n, cudaMemcpyHostToDevice, st));
        dpos = c->pm_io;
        dacc = c->pm_io + 3 * (size_t)n;
    }
    PH_TRY(ph_pm_enqueue(c, p, nside, n, dpos, dacc));
    if (!dio)
        PH_CUDA_CHECK(cudaMemcpyAsync(acc_pm, dacc, sizeof(double) * 3 * (size_t)n, cudaMemcpyDeviceToHost, st));
    PH_CUDA_CHECK(cudaStreamSynchronize(st));
    return 0;
}
