// Measurement helpers that run on the GPU:
//  * photons_direct_sum: FP64 direct sum of the untruncated short-range
//    kernel m g(r/2rs) dx / max(r,eps)^3 over all sources within rmax
//    (minimum image), for a subset of targets.  This is the error
//    reference for the force pass (the pass truncates by tree cells, this
//    does not).  Sources are binned into cells of side >= rmax on the host.
//  * photons_fp32_fma_peak: FFMA throughput probe, the denominator of the
//    P2P roofline fraction; photons_fp64_fma_peak: the DFMA one, for the
//    FP64 drop-in pass.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "api_internal.cuh"
#include "pair64.cuh"

namespace {

// FP32 copies of the binned sources, for the distance filter below
__global__ void k_direct_f32(const double *__restrict__ sx, const double *__restrict__ sy,
                             const double *__restrict__ sz, int n, float4 *__restrict__ s4)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        s4[j] = make_float4((float)sx[j], (float)sy[j], (float)sz[j], 0.f);
}

// Minimum image of a coordinate difference: |d| > L/2 (compared as bit
// patterns, on the integer pipe) takes one side off
__device__ __forceinline__ double nearest_image(double d, double L, long long half_bits)
{
    const long long b = __double_as_longlong(d);
    if ((b & 0x7fffffffffffffffLL) > half_bits) d = b < 0 ? d + L : d - L;
    return d;
}

// One block per target.  What bounds the sum is the FP64 pipe (1/64 of the
// FP32 rate on GB300), and most candidates of the 27 cells lie beyond rmax:
// a warp tests 32 candidates in FP32, with a margin above the FP32 error,
// and queues those that may be within rmax; full batches of 32 queued
// sources get the exact FP64 distance, the rmax test and the pair force
// (pair64.cuh), so no FP64 lane idles.  A candidate then costs the FP64 pipe
// nothing and a source within rmax 12 instructions (15 and ~130 with the
// whole test and erfc, exp, sqrt and division in FP64), and a target in a
// halo, with ten times the sources of the others, is spread over 8 warps.
// 262,144 particles half in halos, 2,000 targets, rmax 2 rcut: the call 39.4
// ms with a warp per target (the kernel 34.3), 4.6 now.  Warps take the candidates in a fixed order, so sums
// are deterministic.
#define DIRECT_TB 256
#define DIRECT_WARPS (DIRECT_TB / 32)

// squared FP32 distance up to which a source may be within rmax.  With every
// coordinate and L at most `most`: an FP32 coordinate is within 2^-24 most of
// its double, a difference (at most 2 most) and its image shift round by
// 2^-23 most each, so 4 units of 2^-23 most bound a component's error and 8
// the distance's; the square's rounding is 2^-21 of itself
__device__ __forceinline__ float direct_limit(double rmax2, double most)
{
    const float reach = (float)sqrt(rmax2) * 1.000001f + 8.f * 1.1920929e-7f * (float)most;
    return reach * reach * 1.000001f;
}

// m g / r^3 factor (without m / (2rs)^3) of a source dx away: 0 beyond rmax
// (!(r2 >= rmax2) on bit patterns: a NaN stays in)
__device__ __forceinline__ double direct_factor(double dx, double dy, double dz, bool on, long long rmax2_bits,
                                                const ph::Pair64 &pc, const ph::Pair64Tab &tab)
{
    const double r2 = dx * dx + dy * dy + dz * dz;
    const long long rb = __double_as_longlong(r2);
    const bool near = on && (rb < rmax2_bits || rb > 0x7ff0000000000000LL);
    double f = ph::pair64_f(dx, dy, dz, near, pc, tab);
    if (near && rb == 0 && pc.box->eps == 0.0) f = INFINITY;  // coincident and unsoftened: m / r^3
    return f;
}

__global__ void __launch_bounds__(DIRECT_TB) k_direct(const double *__restrict__ sx, const double *__restrict__ sy,
                                                      const double *__restrict__ sz, const float4 *__restrict__ s4,
                                                      const int *__restrict__ cell_start, int ncell, double cellw,
                                                      const double *__restrict__ tx, const double *__restrict__ ty,
                                                      const double *__restrict__ tz, const int *__restrict__ tself,
                                                      int nt, double L, double most, double rmax2,
                                                      const __grid_constant__ Pair64Box box, double *out)
{
    __shared__ int s_queue[DIRECT_WARPS][64];
    __shared__ double s_sum[DIRECT_WARPS][3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    int *queue = s_queue[warp];
    const ph::Pair64Tab tab = ph::pair64_global();
    const ph::Pair64 pc = ph::pair64_consts(box);
    const long long half_bits = __double_as_longlong(0.5 * L), rmax2_bits = __double_as_longlong(rmax2);
    const float Lf = (float)L, halff = 0.5f * Lf;
    const float limit = direct_limit(rmax2, most);
    const int span = ncell >= 3 ? 1 : 0;
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const double px = tx[t], py = ty[t], pz = tz[t];
        const float fx = (float)px, fy = (float)py, fz = (float)pz;
        const int self = tself[t];
        int ci[3] = {(int)(px / cellw), (int)(py / cellw), (int)(pz / cellw)};
        for (int d = 0; d < 3; d++) ci[d] = min(max(ci[d], 0), ncell - 1);
        double ax = 0, ay = 0, az = 0;
        int waiting = 0;
        auto evaluate = [&](int count) {
            const bool on = lane < count;
            const int j = queue[on ? lane : 0];
            const double dx = nearest_image(sx[j] - px, L, half_bits), dy = nearest_image(sy[j] - py, L, half_bits),
                         dz = nearest_image(sz[j] - pz, L, half_bits);
            const double f = direct_factor(dx, dy, dz, on, rmax2_bits, pc, tab);
            ax = fma(dx, f, ax);
            ay = fma(dy, f, ay);
            az = fma(dz, f, az);
        };
        for (int o = 0; o < (span ? 27 : 1); o++) {
            int c = 0;
            if (span) {
                const int cx = (ci[0] + o / 9 - 1 + ncell) % ncell, cy = (ci[1] + o / 3 % 3 - 1 + ncell) % ncell,
                          cz = (ci[2] + o % 3 - 1 + ncell) % ncell;
                c = (cx * ncell + cy) * ncell + cz;
            }
            const int b = span ? cell_start[c] : 0;
            const int e = span ? cell_start[c + 1] : cell_start[ncell * ncell * ncell];
            for (int j0 = b + 32 * warp; j0 < e; j0 += DIRECT_TB) {
                const int j = j0 + lane;
                bool in = j < e && j != self;
                if (in) {
                    const float4 s = s4[j];
                    float dx = fabsf(s.x - fx), dy = fabsf(s.y - fy), dz = fabsf(s.z - fz);
                    if (dx > halff) dx = fabsf(dx - Lf);
                    if (dy > halff) dy = fabsf(dy - Lf);
                    if (dz > halff) dz = fabsf(dz - Lf);
                    in = !(dx * dx + dy * dy + dz * dz > limit);  // (a NaN goes on to the exact test)
                }
                const unsigned m = __ballot_sync(0xffffffffu, in);
                if (in) queue[waiting + __popc(m & lt)] = j;
                waiting += __popc(m);
                __syncwarp();
                if (waiting >= 32) {
                    evaluate(32);
                    __syncwarp();
                    const int rest = waiting - 32, moved = lane < rest ? queue[32 + lane] : 0;
                    __syncwarp();
                    if (lane < rest) queue[lane] = moved;
                    waiting = rest;
                    __syncwarp();
                }
            }
        }
        if (waiting) evaluate(waiting);
        ax = warp_sum_d(ax);
        ay = warp_sum_d(ay);
        az = warp_sum_d(az);
        if (lane == 0) { s_sum[warp][0] = ax; s_sum[warp][1] = ay; s_sum[warp][2] = az; }
        __syncthreads();
        if (threadIdx.x < 3) {
            double v = 0.0;
            for (int w = 0; w < DIRECT_WARPS; w++) v += s_sum[w][threadIdx.x];
            out[3 * (size_t)t + threadIdx.x] = v * box.scale;
        }
        __syncthreads();
    }
}

// The sum without binning, for few targets: every source is tested against
// DIRECT_TG targets at a time (one load for four tests), which costs less
// than binning the sources on the host did up to thousands of targets, and
// sources keep the caller's order.  An item is a group of targets and a
// slice of the sources; a block takes items from a counter and leaves each
// one's partial sums in its slot, which k_direct_reduce adds in slice order.
// The pair tables are in shared memory.
#define DIRECT_TG 4
#define DIRECT_ALL_TARGETS 4096

// positions as they are, and in FP32; *outside is set if one lies outside [0, L]
__global__ void k_direct_sources(const double *__restrict__ pos, int n, double L, double4 *__restrict__ s8,
                                 float4 *__restrict__ s4, int *outside)
{
    bool out = false;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const double x = pos[3 * (size_t)j], y = pos[3 * (size_t)j + 1], z = pos[3 * (size_t)j + 2];
        out = out || !(x >= 0.0 && x <= L && y >= 0.0 && y <= L && z >= 0.0 && z <= L);
        s8[j] = make_double4(x, y, z, 0.0);
        s4[j] = make_float4((float)x, (float)y, (float)z, 0.f);
    }
    if (__any_sync(0xffffffffu, out) && (threadIdx.x & 31) == 0) *outside = 1;
}

__global__ void __launch_bounds__(DIRECT_TB, 3) k_direct_all(const double4 *__restrict__ s8,
                                                             const float4 *__restrict__ s4, int n,
                                                             const int *__restrict__ targets, int nt, int slice,
                                                             int nslice, double L, double rmax2,
                                                             const __grid_constant__ Pair64Box box, int *work,
                                                             const int *outside, double *part)
{
    extern __shared__ __align__(16) unsigned char direct_smem[];
    __shared__ int s_queue[DIRECT_WARPS][DIRECT_TG][64];
    __shared__ double s_sum[DIRECT_WARPS][3 * DIRECT_TG];
    __shared__ double s_target[3 * DIRECT_TG];
    __shared__ int s_item;
    if (*outside) return;
    const ph::Pair64Tab tab = ph::pair64_load(direct_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const ph::Pair64 pc = ph::pair64_consts(box);
    const long long half_bits = __double_as_longlong(0.5 * L), rmax2_bits = __double_as_longlong(rmax2);
    const float Lf = (float)L, halff = 0.5f * Lf, limit = direct_limit(rmax2, L);
    const int groups = (nt + DIRECT_TG - 1) / DIRECT_TG, items = groups * nslice;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(work, 1);
        __syncthreads();
        const int item = s_item;
        if (item >= items) break;
        const int group = item / nslice, j_end = min(n, (item % nslice + 1) * slice);
        int self[DIRECT_TG], waiting[DIRECT_TG];
        float fx[DIRECT_TG], fy[DIRECT_TG], fz[DIRECT_TG];
        double ax[DIRECT_TG], ay[DIRECT_TG], az[DIRECT_TG];
#pragma unroll
        for (int g = 0; g < DIRECT_TG; g++) {
            // a group's missing targets repeat its first; their sums are not written
            const int t = DIRECT_TG * group + g;
            self[g] = targets[t < nt ? t : DIRECT_TG * group];
            const double4 p = s8[self[g]];
            if (threadIdx.x == 0) { s_target[3 * g] = p.x; s_target[3 * g + 1] = p.y; s_target[3 * g + 2] = p.z; }
            fx[g] = (float)p.x; fy[g] = (float)p.y; fz[g] = (float)p.z;
            ax[g] = ay[g] = az[g] = 0.0;
            waiting[g] = 0;
        }
        __syncthreads();
        auto evaluate = [&](int g, int count) {
            const bool on = lane < count;
            const double4 s = s8[s_queue[warp][g][on ? lane : 0]];
            const double dx = nearest_image(s.x - s_target[3 * g], L, half_bits),
                         dy = nearest_image(s.y - s_target[3 * g + 1], L, half_bits),
                         dz = nearest_image(s.z - s_target[3 * g + 2], L, half_bits);
            const double f = direct_factor(dx, dy, dz, on, rmax2_bits, pc, tab);
            ax[g] = fma(dx, f, ax[g]);
            ay[g] = fma(dy, f, ay[g]);
            az[g] = fma(dz, f, az[g]);
        };
        for (int j0 = (item % nslice) * slice + 32 * warp; j0 < j_end; j0 += DIRECT_TB) {
            const int j = j0 + lane;
            const float4 s = s4[min(j, n - 1)];
#pragma unroll
            for (int g = 0; g < DIRECT_TG; g++) {
                float dx = fabsf(s.x - fx[g]), dy = fabsf(s.y - fy[g]), dz = fabsf(s.z - fz[g]);
                if (dx > halff) dx = fabsf(dx - Lf);
                if (dy > halff) dy = fabsf(dy - Lf);
                if (dz > halff) dz = fabsf(dz - Lf);
                const bool in = j < j_end && j != self[g] && !(dx * dx + dy * dy + dz * dz > limit);
                const unsigned m = __ballot_sync(0xffffffffu, in);
                if (m == 0) continue;
                int *queue = s_queue[warp][g];
                if (in) queue[waiting[g] + __popc(m & lt)] = j;
                waiting[g] += __popc(m);
                __syncwarp();
                if (waiting[g] >= 32) {
                    evaluate(g, 32);
                    __syncwarp();
                    const int rest = waiting[g] - 32, moved = lane < rest ? queue[32 + lane] : 0;
                    __syncwarp();
                    if (lane < rest) queue[lane] = moved;
                    waiting[g] = rest;
                    __syncwarp();
                }
            }
        }
#pragma unroll
        for (int g = 0; g < DIRECT_TG; g++) {
            if (waiting[g]) evaluate(g, waiting[g]);
            const double x = warp_sum_d(ax[g]), y = warp_sum_d(ay[g]), z = warp_sum_d(az[g]);
            if (lane == 0) { s_sum[warp][3 * g] = x; s_sum[warp][3 * g + 1] = y; s_sum[warp][3 * g + 2] = z; }
        }
        __syncthreads();
        if (threadIdx.x < 3 * DIRECT_TG) {
            double v = 0.0;
            for (int w = 0; w < DIRECT_WARPS; w++) v += s_sum[w][threadIdx.x];
            part[(size_t)item * (3 * DIRECT_TG) + threadIdx.x] = v;
        }
    }
}

__global__ void k_direct_reduce(const double *__restrict__ part, int nt, int nslice, double scale, double *out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * nt; i += gridDim.x * blockDim.x) {
        const int t = i / 3, group = t / DIRECT_TG, k = 3 * (t % DIRECT_TG) + i % 3;
        double v = 0.0;
        for (int sl = 0; sl < nslice; sl++) v += part[((size_t)group * nslice + sl) * (3 * DIRECT_TG) + k];
        out[i] = v * scale;
    }
}

__global__ void k_fma_probe(float *out, int iters, float seed)
{
    float a0 = seed + threadIdx.x, a1 = a0 + 1.f, a2 = a0 + 2.f, a3 = a0 + 3.f, a4 = a0 + 4.f, a5 = a0 + 5.f,
          a6 = a0 + 6.f, a7 = a0 + 7.f;
    const float m = 0.999999f, c = 1e-7f;
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 16; k++) {
            a0 = fmaf(a0, m, c); a1 = fmaf(a1, m, c); a2 = fmaf(a2, m, c); a3 = fmaf(a3, m, c);
            a4 = fmaf(a4, m, c); a5 = fmaf(a5, m, c); a6 = fmaf(a6, m, c); a7 = fmaf(a7, m, c);
        }
    }
    float s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s == 1234.5f) out[0] = s;  // keeps the chains live
}

__global__ void k_dfma_probe(double *out, int iters, double seed)
{
    double a0 = seed + threadIdx.x, a1 = a0 + 1.0, a2 = a0 + 2.0, a3 = a0 + 3.0, a4 = a0 + 4.0, a5 = a0 + 5.0,
           a6 = a0 + 6.0, a7 = a0 + 7.0;
    const double m = 0.999999999, c = 1e-12;
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 16; k++) {
            a0 = fma(a0, m, c); a1 = fma(a1, m, c); a2 = fma(a2, m, c); a3 = fma(a3, m, c);
            a4 = fma(a4, m, c); a5 = fma(a5, m, c); a6 = fma(a6, m, c); a7 = fma(a7, m, c);
        }
    }
    double s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s == 1234.5) out[0] = s;  // keeps the chains live
}

__global__ void k_fma2_probe(float *out, int iters, float seed)
{
    float2 a0 = make_float2(seed + threadIdx.x, seed - threadIdx.x), a1 = make_float2(a0.x + 1.f, a0.y + 1.f),
           a2 = make_float2(a0.x + 2.f, a0.y + 2.f), a3 = make_float2(a0.x + 3.f, a0.y + 3.f);
    float2 a4 = make_float2(a0.x + 4.f, a0.y + 4.f), a5 = make_float2(a0.x + 5.f, a0.y + 5.f),
           a6 = make_float2(a0.x + 6.f, a0.y + 6.f), a7 = make_float2(a0.x + 7.f, a0.y + 7.f);
    const float2 m = make_float2(0.999999f, 0.999999f), c = make_float2(1e-7f, 1e-7f);
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 16; k++) {
            a0 = __ffma2_rn(a0, m, c); a1 = __ffma2_rn(a1, m, c); a2 = __ffma2_rn(a2, m, c); a3 = __ffma2_rn(a3, m, c);
            a4 = __ffma2_rn(a4, m, c); a5 = __ffma2_rn(a5, m, c); a6 = __ffma2_rn(a6, m, c); a7 = __ffma2_rn(a7, m, c);
        }
    }
    float s = a0.x + a1.x + a2.x + a3.x + a4.x + a5.x + a6.x + a7.x + a0.y + a1.y + a2.y + a3.y + a4.y + a5.y +
              a6.y + a7.y;
    if (s == 1234.5f) out[0] = s;
}

}  // namespace

// Test hook: with PHOTONS_TEST_DIRECT_NO_ROOM=1 the allocation below counts as failed
static bool direct_no_room()
{
    const char *v = getenv("PHOTONS_TEST_DIRECT_NO_ROOM");
    return v && !strcmp(v, "1");
}

// few targets (see k_direct_all); *done = 0 if a position lies outside the
// box or the device has no room
static int direct_all(const photons_params *p, int n, const double *pos, int nt, const int *targets, double rmax,
                      double *acc, int *done)
{
    static std::atomic<bool> set[64];
    int dev = 0;
    PH_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !set[dev].load()) {
        PH_CUDA_CHECK(cudaFuncSetAttribute(k_direct_all, cudaFuncAttributeMaxDynamicSharedMemorySize, PAIR64_BYTES));
        if (dev >= 0 && dev < 64) set[dev].store(true);
    }
    // slices of the sources: about eight items a block
    const int blocks = ph::device_sm_count() * 3, groups = (nt + DIRECT_TG - 1) / DIRECT_TG;
    int nslice = (8 * blocks + groups - 1) / groups;
    const int most = (n + 4095) / 4096;
    nslice = nslice < 1 ? 1 : (nslice > most ? most : nslice);
    const int slice = ((n + nslice - 1) / nslice + 31) & ~31;
    nslice = (n + slice - 1) / slice;
    // one allocation: sources (FP64, FP32), positions in and sums out, partial sums, targets, two counters
    const size_t b8 = sizeof(double4) * (size_t)n, b4 = sizeof(float4) * (size_t)n, bp = 8 * (((size_t)3 * n + 3) & ~(size_t)3),
                 bs = sizeof(double) * 3 * DIRECT_TG * (size_t)groups * nslice, bo = 8 * (((size_t)3 * nt + 1) & ~(size_t)1),
                 bt = sizeof(int) * (((size_t)nt + 3) & ~(size_t)3);
    // where there is no room for it, the binned sum (40 bytes a source) may still fit
    unsigned char *d = nullptr;
    if (direct_no_room() || cudaMalloc(reinterpret_cast<void **>(&d), b8 + b4 + bp + bs + bo + bt + 16) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    double4 *s8 = reinterpret_cast<double4 *>(d);
    float4 *s4 = reinterpret_cast<float4 *>(d + b8);
    double *dpos = reinterpret_cast<double *>(d + b8 + b4), *part = reinterpret_cast<double *>(d + b8 + b4 + bp),
           *out = reinterpret_cast<double *>(d + b8 + b4 + bp + bs);
    int *tgt = reinterpret_cast<int *>(d + b8 + b4 + bp + bs + bo), *ctl = reinterpret_cast<int *>(d + b8 + b4 + bp + bs + bo + bt);
    const Pair64Box box = pair64_box(p->eps, p->rs, p->mass);
    int outside = 0;
    cudaMemsetAsync(ctl, 0, 2 * sizeof(int));
    cudaMemcpyAsync(tgt, targets, sizeof(int) * (size_t)nt, cudaMemcpyHostToDevice);
    cudaMemcpyAsync(dpos, pos, sizeof(double) * 3 * (size_t)n, cudaMemcpyHostToDevice);
    ph::note_launch(), k_direct_sources<<<ph::device_sm_count() * 8, 256>>>(dpos, n, p->boxsize, s8, s4, ctl + 1);
    ph::note_launch(), k_direct_all<<<blocks, DIRECT_TB, PAIR64_BYTES>>>(s8, s4, n, tgt, nt, slice, nslice, p->boxsize,
                                                                        rmax * rmax, box, ctl, ctl + 1, part);
    ph::note_launch(), k_direct_reduce<<<(3 * nt + 255) / 256, 256>>>(part, nt, nslice, box.scale, out);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&outside, ctl + 1, sizeof(int), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(acc, out, sizeof(double) * 3 * (size_t)nt, cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return ph_set_cuda_error(e, "direct sum", __FILE__, __LINE__);
    *done = !outside;
    return 0;
}

extern "C" int photons_direct_sum(const photons_params *p, int n, const double *pos, int nt, const int *targets,
                                  double rmax, double *acc)
{
    photons_gpu_clear_error();
    if (!p || n < 1 || nt < 0 || !pos || (nt > 0 && (!targets || !acc)) || !(rmax > 0))
        return ph_set_error(PH_ERR_ARG, "bad direct-sum arguments");
    if (nt == 0) return 0;
    for (int t = 0; t < nt; t++)
        if (targets[t] < 0 || targets[t] >= n) return ph_set_error(PH_ERR_ARG, "target index out of range");
    // Up to here testing every source costs less than binning the sources on
    // the host (~8 ns a source; a test 1.5 ps).  Calls, binned -> not: 262,144
    // sources half in halos, 2,000 targets 4.4 -> 3.1 ms, 200 targets 3.1 ->
    // 0.7; 2,097,152 sources, 2,000 targets 22.9 -> 11.3 (16,000: 34.1 -> 81)
    if (nt <= DIRECT_ALL_TARGETS) {
        int done = 0;
        const int rc = direct_all(p, n, pos, nt, targets, rmax, acc, &done);
        if (rc || done) return rc;
    }
    const double L = p->boxsize;
    int ncell = (int)(L / rmax);
    if (ncell > 512) ncell = 512;
    if (ncell < 3) ncell = 1;
    const double cw = L / ncell;
    const size_t nc3 = (size_t)ncell * ncell * ncell;
    std::vector<int> cnt(nc3 + 1, 0), cellof(n);
    double most = L;  // largest coordinate, for the distance filter's margin
    for (int j = 0; j < n; j++) {
        int c[3];
        for (int d = 0; d < 3; d++) {
            most = std::max(most, std::fabs(pos[3 * (size_t)j + d]));
            c[d] = (int)(pos[3 * (size_t)j + d] / cw);
            if (c[d] < 0) c[d] = 0;
            if (c[d] >= ncell) c[d] = ncell - 1;
        }
        cellof[j] = (int)(((size_t)c[0] * ncell + c[1]) * ncell + c[2]);
        cnt[cellof[j] + 1]++;
    }
    for (size_t c = 0; c < nc3; c++) cnt[c + 1] += cnt[c];
    std::vector<int> fill(cnt.begin(), cnt.end() - 1), slot(n);
    std::vector<double> sx(n), sy(n), sz(n);
    for (int j = 0; j < n; j++) {
        int s = fill[cellof[j]]++;
        slot[j] = s;
        sx[s] = pos[3 * (size_t)j];
        sy[s] = pos[3 * (size_t)j + 1];
        sz[s] = pos[3 * (size_t)j + 2];
    }
    std::vector<double> tx(nt), ty(nt), tz(nt);
    std::vector<int> ts(nt);
    for (int t = 0; t < nt; t++) {
        int j = targets[t];
        tx[t] = pos[3 * (size_t)j];
        ty[t] = pos[3 * (size_t)j + 1];
        tz[t] = pos[3 * (size_t)j + 2];
        ts[t] = slot[j];
    }
    double *d_sx = nullptr, *d_sy = nullptr, *d_sz = nullptr, *d_tx = nullptr, *d_ty = nullptr, *d_tz = nullptr,
           *d_out = nullptr;
    float4 *d_s4 = nullptr;
    int *d_cell = nullptr, *d_ts = nullptr;
    int rc = 0;
    auto al = [&](void **ptr, size_t bytes) {
        if (rc) return;
        if (cudaMalloc(ptr, bytes) != cudaSuccess) {
            cudaGetLastError();
            rc = ph_set_error(PH_ERR_NOMEM, "direct-sum allocation failed");
        }
    };
    al((void **)&d_sx, sizeof(double) * n); al((void **)&d_sy, sizeof(double) * n); al((void **)&d_sz, sizeof(double) * n);
    al((void **)&d_tx, sizeof(double) * nt); al((void **)&d_ty, sizeof(double) * nt); al((void **)&d_tz, sizeof(double) * nt);
    al((void **)&d_out, sizeof(double) * 3 * nt); al((void **)&d_cell, sizeof(int) * (nc3 + 1));
    al((void **)&d_ts, sizeof(int) * nt); al((void **)&d_s4, sizeof(float4) * n);
    if (!rc) {
        cudaMemcpy(d_sx, sx.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
        cudaMemcpy(d_sy, sy.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
        cudaMemcpy(d_sz, sz.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
        cudaMemcpy(d_tx, tx.data(), sizeof(double) * nt, cudaMemcpyHostToDevice);
        cudaMemcpy(d_ty, ty.data(), sizeof(double) * nt, cudaMemcpyHostToDevice);
        cudaMemcpy(d_tz, tz.data(), sizeof(double) * nt, cudaMemcpyHostToDevice);
        cudaMemcpy(d_ts, ts.data(), sizeof(int) * nt, cudaMemcpyHostToDevice);
        cudaMemcpy(d_cell, cnt.data(), sizeof(int) * (nc3 + 1), cudaMemcpyHostToDevice);
        const int blocks = ph::device_sm_count() * 8;
        ph::note_launch(), k_direct_f32<<<blocks, 256>>>(d_sx, d_sy, d_sz, n, d_s4);
        ph::note_launch(), k_direct<<<nt, DIRECT_TB>>>(d_sx, d_sy, d_sz, d_s4, d_cell, ncell, cw, d_tx, d_ty, d_tz, d_ts, nt, L, most, rmax * rmax,
                                  pair64_box(p->eps, p->rs, p->mass), d_out);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpy(acc, d_out, sizeof(double) * 3 * nt, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) rc = ph_set_cuda_error(e, "direct sum", __FILE__, __LINE__);
    }
    cudaFree(d_sx); cudaFree(d_sy); cudaFree(d_sz); cudaFree(d_tx); cudaFree(d_ty); cudaFree(d_tz);
    cudaFree(d_out); cudaFree(d_cell); cudaFree(d_ts); cudaFree(d_s4);
    return rc;
}

static double fma_probe(int iters, bool packed)
{
    photons_gpu_clear_error();
    if (iters < 1) iters = 4096;
    float *d = nullptr;
    if (cudaMalloc(&d, sizeof(float)) != cudaSuccess) { cudaGetLastError(); return -1.0; }
    int blocks = ph::device_sm_count() * 8, threads = 256;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    if (packed) ph::note_launch(), k_fma2_probe<<<blocks, threads>>>(d, iters / 8 + 1, 1.0f);  // warm-up
    else ph::note_launch(), k_fma_probe<<<blocks, threads>>>(d, iters / 8 + 1, 1.0f);
    cudaEventRecord(a);
    if (packed) ph::note_launch(), k_fma2_probe<<<blocks, threads>>>(d, iters, 1.0f);
    else ph::note_launch(), k_fma_probe<<<blocks, threads>>>(d, iters, 1.0f);
    cudaEventRecord(b);
    cudaEventSynchronize(b);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(d);
    if (cudaGetLastError() != cudaSuccess || ms <= 0.f) return -1.0;
    double flops = (packed ? 2.0 : 1.0) * 2.0 * 8.0 * 16.0 * (double)iters * blocks * threads;
    return flops / (ms * 1e-3) / 1e12;
}

extern "C" double photons_fp32_fma_peak(int iters)
{
    photons_gpu_clear_error();
    if (iters < 1) iters = 4096;
    return fma_probe(iters, false);
}

// TFLOP/s of DFMA chains (2 flops each) over the whole device
extern "C" double photons_fp64_fma_peak(int iters)
{
    photons_gpu_clear_error();
    if (iters < 1) iters = 256;
    double *d = nullptr;
    if (cudaMalloc(&d, sizeof(double)) != cudaSuccess) { cudaGetLastError(); return -1.0; }
    const int blocks = ph::device_sm_count() * 8, threads = 256;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    ph::note_launch(), k_dfma_probe<<<blocks, threads>>>(d, iters / 8 + 1, 1.0);  // warm-up
    cudaEventRecord(a);
    ph::note_launch(), k_dfma_probe<<<blocks, threads>>>(d, iters, 1.0);
    cudaEventRecord(b);
    cudaEventSynchronize(b);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(d);
    if (cudaGetLastError() != cudaSuccess || ms <= 0.f) return -1.0;
    const double flops = 2.0 * 8.0 * 16.0 * (double)iters * blocks * threads;
    return flops / (ms * 1e-3) / 1e12;
}

extern "C" double photons_fp32x2_fma_peak(int iters)
{
    photons_gpu_clear_error();
    if (iters < 1) iters = 4096;
    return fma_probe(iters, true);
}

// the FP64 pair factor's split term erfc(u) + (2/sqrt(pi)) u exp(-u^2) at n
// host points: the piecewise polynomials of the FP64 kernels, or (exact)
// erfc and exp as src/fmm.c:846-848 writes them
extern "C" int photons_split_factor_fp64(const double *u, int n, int exact, double *g)
{
    photons_gpu_clear_error();
    if (n < 0 || (n > 0 && (!u || !g))) return ph_set_error(PH_ERR_ARG, "bad split-factor arguments");
    if (n == 0) return 0;
    double *d = nullptr;
    PH_CUDA_CHECK(cudaMalloc(&d, sizeof(double) * 2 * (size_t)n));
    int rc = 0;
    cudaError_t e = cudaMemcpy(d, u, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        rc = ph::launch_split_factor_fp64(d, n, exact, d + n, 0);
        if (!rc) e = cudaMemcpy(g, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    }
    if (!rc && e != cudaSuccess) rc = ph_set_cuda_error(e, "split factor", __FILE__, __LINE__);
    cudaFree(d);
    return rc;
}
