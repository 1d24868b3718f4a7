// kd-tree build on the device.
//
// Restates src/fmm.c:30-264 (bksort_inplace, build_kdtree, center_kdtree,
// build_localtree) in two parts.
//
// Wide nodes (more than BuildBufs::mid particles) are split level-synchronously:
// every wide node of one depth in the same set of launches (the per-node
// bookkeeping of the first, small levels in single blocks).  Per level:
//   1. each node's particle range is cut into chunks of CHUNK particles;
//   2. chunk sums of the split coordinate (axis = depth mod 3) and a
//      fixed-order reduction give the node's mean;
//   3. the reference's two-ended swap partition (src/fmm.c:58-72) is
//      reproduced exactly: with S particles not above the mean, the k-th
//      particle above the mean counted from the left among positions < S
//      trades places with the k-th particle not above the mean counted from
//      the right among positions >= S.  Ranks come from chunk counts, so the
//      swaps are independent and run in parallel;
//   4. children with <= MAXLEAF particles become leaves, the others nodes
//      of the next level; child boxes come from the split plane.
// A node of at most mid particles (PH_MID, or CHUNK in large builds) is not
// split by the levels: one block holds its particles in shared memory and
// splits it down to nodes of at most sub, CHUNK (k_mid_build), and each of
// those roots a subtree that one block builds whole (k_subtree_build), every
// node of it split by one warp.  Both
// use the arithmetic of the levels (sums over chunks of CHUNK in the same
// order), so the tree is the one a build that splits every depth level by
// level makes.
// Special cases follow the reference: a pair splits at its midpoint and is
// ordered (src/fmm.c:38-47); if no particle lies above the mean the last
// one goes to the upper child.
// Afterwards leaves take the reference's depth-first order and nodes preorder
// (src/fmm.c:101-118), both read off the particle ranges, and geometry is
// written in the unified index space.
//
// The mean is a deterministic parallel sum, not the reference's sequential
// one, so a mean can differ from the reference's in the last bits; that
// changes the partition only for a particle within those bits of the mean.
#include <atomic>
#include <cstdio>
#include <vector>

#include "fmm_context.cuh"

#define CHUNK 1024
#define TB 256

// subtree blocks: one warp per node of the subtree level being split
#define SUB_TB 256
#define SUB_NW (SUB_TB / 32)
#define SUB_FAIL (1 << 20)  // failure mark in a subtree's node counters (above any node count)

// levels of at most this many nodes run their bookkeeping in one block
#define SMALL_LEVEL 32

// depth lists: unified ids per block (one warp) of the counting sort (4096,
// a load at a time: k_depth_place 66-75 us whatever the size of the tree)
#define DEPTH_R 1024

// temp-node modes: 0-2 the kinds of a split node (two-ended swap, nothing
// above the mean, a pair), then the two states of a node not yet split
#define MODE_DEFERRED 3  // at most CHUNK particles: split by k_subtree_build
#define MODE_PENDING 4   // wide: split by the levels
#define MODE_MID 5       // at most PH_MID particles: split by k_mid_build

// blocks of k_mid_build
#define MID_TB 512
#define MID_NW (MID_TB / 32)
#define MID_SEG 256  // positions a warp ranks at a time

namespace ph {
namespace {

__host__ __device__ __forceinline__ const double *axis_ptr(const double *x, const double *y, const double *z, int D)
{
    return D == 0 ? x : (D == 1 ? y : z);
}

// An integer key that orders doubles as the FP64 comparison does (both
// zeros equal), so that !(x > mean) is key(x) <= key(mean) on the integer
// pipe; GB300's FP64 pipe runs at 1/64 of the FP32 rate.  Exact for every
// non-NaN x.
__device__ __forceinline__ long long order_key(double x)
{
    const long long b = __double_as_longlong(x);
    if ((b & 0x7FFFFFFFFFFFFFFFLL) == 0) return 0;
    return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFLL);
}

// the state of a node of len particles not yet split
__device__ __forceinline__ int open_mode(const BuildBufs &b, int len)
{
    return len <= b.sub ? MODE_DEFERRED : (len <= b.mid ? MODE_MID : MODE_PENDING);
}

// one root per box: its particle range and the box [0, L]^3 as
// src/fmm.c:194-197 derives the root from the domain box (centre 0.5*(L+0),
// width L-0, src/toptree.c:150-159)
__global__ void k_init_roots(BuildBufs b, int n, int top)
{
    ph::chain_begin();
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < b.nbox; t += gridDim.x * blockDim.x) {
        const BoxParams &B = b.boxes[t];
        b.tn_start[t] = B.first;
        b.tn_len[t] = B.count;
        b.tn_depth[t] = 0;
        b.tn_parent[t] = -1;
        b.tn_boxid[t] = t;
        b.tn_mode[t] = open_mode(b, B.count);
        for (int d = 0; d < 3; d++) {
            // a rank's domain: its top-tree node's centre and width
            // (src/toptree.c:150-159) give the bounds of src/fmm.c:189-197
            const double lo = B.domain ? B.dom_lo[d] : 0.0, hi = B.domain ? B.dom_hi[d] : B.boxsize;
            const double c = 0.5 * (hi + lo), w = hi - lo;
            b.tn_box[d * b.cap_nodes + t] = c - 0.5 * w;
            b.tn_box[(3 + d) * b.cap_nodes + t] = c + 0.5 * w;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        for (int i = 0; i < BC_NCOUNTERS; i++) b.cnt[i] = 0;
        // top = 0: no box has a wide root
        b.cnt[top ? BC_LEVEL_COUNT : BC_LEVEL_BEGIN] = b.nbox;
        b.cnt[BC_NLEVELS] = top ? 0 : 1;
        b.cnt[BC_WORDS] = (n + 31) / 32;
    }
}

__global__ void k_init_particles(const double *__restrict__ pos, int n, BuildBufs b)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        b.x[i] = pos[3 * i];
        b.y[i] = pos[3 * i + 1];
        b.z[i] = pos[3 * i + 2];
        b.perm[i] = i;
    }
}

// chunks per node; a node that is not wide has none and makes no children here
__device__ __forceinline__ void level_nch_node(BuildBufs &b, int lb, int i)
{
    const int t = lb + i;
    if (b.tn_mode[t] != MODE_PENDING) {
        b.tn_nch[i] = 0;
        b.tn_nodeflag[i] = 0;
        b.tn_leafflag[i] = 0;
    } else {
        b.tn_nch[i] = (b.tn_len[t] + CHUNK - 1) / CHUNK;
    }
}

__global__ void k_level_nch(BuildBufs b)
{
    ph::chain_begin();
    const int lb = b.cnt[BC_LEVEL_BEGIN], C = b.cnt[BC_LEVEL_COUNT];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < C; i += gridDim.x * blockDim.x) level_nch_node(b, lb, i);
}

// chunk -> level-local node index, written once per level (a warp per node)
__device__ __forceinline__ void chunk_map_node(BuildBufs &b, int i, int lane)
{
    const int c0 = b.tn_chunk_base[i], nc = b.tn_nch[i];
    for (int k = lane; k < nc; k += 32) b.ch_node[c0 + k] = i;
}

__global__ void k_chunk_map(BuildBufs b)
{
    ph::chain_begin();
    const int C = b.cnt[BC_LEVEL_COUNT];
    int lane = warp_lane();
    int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int i = gw; i < C; i += nw) chunk_map_node(b, i, lane);
}

// Chunk sums: lane l adds positions l, l+32, l+64, ... of the chunk in that
// order, then the warp butterfly.  Loads are issued eight at a time ahead
// of the adds, which keep their order.
__global__ void k_chunk_sum(BuildBufs b, int D)
{
    ph::chain_begin();
    const int lb = b.cnt[BC_LEVEL_BEGIN];
    const double *coord = axis_ptr(b.x, b.y, b.z, D);
    int W = b.cnt[BC_W];
    int lane = warp_lane();
    int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int w = gw; w < W; w += nw) {
        int i = b.ch_node[w];
        int t = lb + i;
        int start = b.tn_start[t], len = b.tn_len[t];
        int s0 = (w - b.tn_chunk_base[i]) * CHUNK;
        int s1 = min(len, s0 + CHUNK);
        const double *cp = coord + start;
        double s = 0.0;
        int k = s0 + lane;
        for (; k + 224 < s1; k += 256) {
            double v[8];
#pragma unroll
            for (int q = 0; q < 8; q++) v[q] = cp[k + 32 * q];
#pragma unroll
            for (int q = 0; q < 8; q++) s += v[q];
        }
        for (; k < s1; k += 32) s += cp[k];
        s = warp_sum_d(s);
        if (lane == 0) b.ch_partial[w] = s;
    }
}

// Node means, a warp each: lane-strided sums of the chunk sums, then the
// warp reduction (fixed order)
__global__ void k_node_mean(BuildBufs b, int D)
{
    ph::chain_begin();
    const int lb = b.cnt[BC_LEVEL_BEGIN], C = b.cnt[BC_LEVEL_COUNT];
    int lane = warp_lane();
    int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int i = gw; i < C; i += nw) {
        const int nc = b.tn_nch[i];
        if (nc == 0) continue;
        const int t = lb + i;
        const int c0 = b.tn_chunk_base[i];
        double s = 0.0;
        for (int k = lane; k < nc; k += 32) s += b.ch_partial[c0 + k];
        s = warp_sum_d(s);
        if (lane == 0) b.tn_split[t] = s / (double)b.tn_len[t];
    }
}

__global__ void k_chunk_count(BuildBufs b, int D)
{
    ph::chain_begin();
    const int lb = b.cnt[BC_LEVEL_BEGIN];
    const double *coord = axis_ptr(b.x, b.y, b.z, D);
    int W = b.cnt[BC_W];
    int lane = warp_lane();
    int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int w = gw; w < W; w += nw) {
        int i = b.ch_node[w];
        int t = lb + i;
        int start = b.tn_start[t], len = b.tn_len[t];
        const long long km = order_key(b.tn_split[t]);
        int s0 = (w - b.tn_chunk_base[i]) * CHUNK;
        int s1 = min(len, s0 + CHUNK);
        const double *cp = coord + start;
        int c = 0;
        int k = s0 + lane;
        for (; k + 224 < s1; k += 256) {
            double v[8];
#pragma unroll
            for (int q = 0; q < 8; q++) v[q] = cp[k + 32 * q];
#pragma unroll
            for (int q = 0; q < 8; q++) c += order_key(v[q]) <= km;
        }
        for (; k < s1; k += 32) c += order_key(cp[k]) <= km;
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) b.ch_cnt[w] = c;
    }
}

// the split kind and lower-child size of a node of len particles, S of them
// not above the mean
__device__ __forceinline__ void split_sizes(int len, int S, int &mode, int &left)
{
    if (len == 2) { mode = 2; left = 1; }
    else if (S == len) { mode = 1; left = len - 1; }
    else { mode = 0; left = S; }
}

// per node: the child kinds and sizes from the count of particles not above
// the mean
__device__ __forceinline__ void node_split_finish(BuildBufs &b, int i, int t, int len, int S, int maxleaf)
{
    int mode, left;
    split_sizes(len, S, mode, left);
    b.tn_S[t] = S;
    b.tn_mode[t] = mode;
    int right = len - left;
    // child sizes are stashed in child codes until the children exist
    b.tn_child0[t] = left;
    b.tn_child1[t] = right;
    b.tn_nodeflag[i] = (left > maxleaf) + (right > maxleaf);
    b.tn_leafflag[i] = (left <= maxleaf) + (right <= maxleaf);
}

// per wide node of the level, a warp each: prefix of chunk counts,
// partition sizes, child kinds.  Each lane sums a contiguous block of chunk
// counts (the prefix is exact integer arithmetic, so the blocking does not
// change it).
__device__ __forceinline__ void node_split_node(BuildBufs &b, int lb, int i, int lane, int maxleaf)
{
    const int nc = b.tn_nch[i];
    if (nc == 0) return;
    const int t = lb + i, c0 = b.tn_chunk_base[i];
    const int per = (nc + 31) / 32;
    const int kb = min(nc, lane * per), ke = min(nc, kb + per);
    int own = 0;
#pragma unroll 8
    for (int k = kb; k < ke; k++) own += b.ch_cnt[c0 + k];
    const int incl = warp_incl_scan(own);
    int run = incl - own;
    for (int k = kb; k < ke; k++) {
        b.ch_small_base[c0 + k] = run;
        run += b.ch_cnt[c0 + k];
    }
    const int S = shfl(incl, 31);
    if (lane == 0) node_split_finish(b, i, t, b.tn_len[t], S, maxleaf);
}

__global__ void k_node_split(BuildBufs b, int maxleaf)
{
    ph::chain_begin();
    const int lb = b.cnt[BC_LEVEL_BEGIN], C = b.cnt[BC_LEVEL_COUNT];
    int lane = warp_lane();
    int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int i = gw; i < C; i += nw) node_split_node(b, lb, i, lane, maxleaf);
}

__device__ __forceinline__ void make_children_node(BuildBufs &b, int lb, int C, int leaves_before, int i, int maxleaf,
                                                   int D)
{
    {
        int t = lb + i;
        if (b.tn_mode[t] == MODE_DEFERRED || b.tn_mode[t] == MODE_MID) return;
        int start = b.tn_start[t];
        int depth = b.tn_depth[t];
        int sizes[2] = {b.tn_child0[t], b.tn_child1[t]};
        double split = b.tn_split[t];
        double lo[3], hi[3];
        for (int d = 0; d < 3; d++) {
            lo[d] = b.tn_box[d * b.cap_nodes + t];
            hi[d] = b.tn_box[(3 + d) * b.cap_nodes + t];
        }
        int nid = lb + C + b.tn_nodebase[i];
        int lid = leaves_before + b.tn_leafbase[i];
        int code[2];
        int ip = start;
        int wide = 0;
        for (int c = 0; c < 2; c++) {
            double clo[3] = {lo[0], lo[1], lo[2]}, chi[3] = {hi[0], hi[1], hi[2]};
            if (c == 0) chi[D] = split;
            else clo[D] = split;
            if (sizes[c] <= maxleaf) {
                if (lid >= b.rule_cap) {
                    atomicOr(&b.cnt[BC_FLAGS], PH_FLAG_LEAF_CAPACITY);
                    code[c] = ~0;
                } else {
                    b.tl_start[lid] = ip;
                    b.tl_len[lid] = sizes[c];
                    b.tl_depth[lid] = depth + 1;
                    b.tl_parent[lid] = t;
                    b.tl_boxid[lid] = b.tn_boxid[t];
                    for (int d = 0; d < 3; d++) {
                        b.tl_box[d * b.cap_leaves + lid] = clo[d];
                        b.tl_box[(3 + d) * b.cap_leaves + lid] = chi[d];
                    }
                    code[c] = ~lid;
                }
                lid++;
            } else {
                if (nid >= b.rule_cap) {
                    atomicOr(&b.cnt[BC_FLAGS], PH_FLAG_NODE_CAPACITY);
                    code[c] = 0;
                } else {
                    b.tn_start[nid] = ip;
                    b.tn_len[nid] = sizes[c];
                    b.tn_depth[nid] = depth + 1;
                    b.tn_parent[nid] = t;
                    b.tn_boxid[nid] = b.tn_boxid[t];
                    b.tn_mode[nid] = open_mode(b, sizes[c]);
                    wide += sizes[c] > b.mid;
                    for (int d = 0; d < 3; d++) {
                        b.tn_box[d * b.cap_nodes + nid] = clo[d];
                        b.tn_box[(3 + d) * b.cap_nodes + nid] = chi[d];
                    }
                    code[c] = nid;
                }
                nid++;
            }
            ip += sizes[c];
        }
        b.tn_child0[t] = code[0];
        b.tn_child1[t] = code[1];
        if (wide) atomicAdd(&b.cnt[BC_NEXT_WIDE], wide);
    }
}

__global__ void k_make_children(BuildBufs b, int maxleaf, int D)
{
    ph::chain_begin();
    const int lb = b.cnt[BC_LEVEL_BEGIN], C = b.cnt[BC_LEVEL_COUNT];
    const int leaves_before = b.cnt[BC_LEAVES];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < C; i += gridDim.x * blockDim.x)
        make_children_node(b, lb, C, leaves_before, i, maxleaf, D);
}

// Close level d and advance.  When the last launched level (d = top - 1)
// made no wide node, its children are counted in too.  After a capacity
// overflow no further level is built.
__device__ void level_finish(BuildBufs &b, int d, int top)
{
    {
        const int C = b.cnt[BC_LEVEL_COUNT], lb = b.cnt[BC_LEVEL_BEGIN];
        if (C == 0) return;
        if (b.cnt[BC_FLAGS] & (PH_FLAG_LEAF_CAPACITY | PH_FLAG_NODE_CAPACITY)) {
            b.cnt[BC_LEVEL_COUNT] = 0;
            return;
        }
        b.cnt[BC_LEAVES] += b.cnt[BC_NEW_LEAVES];
        b.cnt[BC_LEVEL_BEGIN] = lb + C;
        const int next = b.cnt[BC_NEXT_NODES];
        b.cnt[BC_LEVEL_COUNT] = next;
        b.cnt[BC_NLEVELS] = d + 1;
        if (d == top - 1 && next > 0 && b.cnt[BC_NEXT_WIDE] == 0) {
            b.cnt[BC_LEVEL_BEGIN] = lb + C + next;
            b.cnt[BC_LEVEL_COUNT] = 0;
            b.cnt[BC_NLEVELS] = d + 2;
        }
        b.cnt[BC_NEXT_WIDE] = 0;
    }
}

__global__ void k_level_finish(BuildBufs b, int d, int top)
{
    ph::chain_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) level_finish(b, d, top);
}

// ---------------- one block for the bookkeeping of a small level ----------------
// A level of at most SMALL_LEVEL nodes (the first levels) runs its per-node
// bookkeeping in single-block kernels: the same per-node work as the
// kernels above, the scans in one block.  k_level_plan closes the level
// before (when that was small too), then counts chunks, numbers them and
// maps them to nodes; k_level_close splits the nodes, numbers the children
// and makes them.  Integer work throughout, so the tree is unchanged.
#define SMALL_TB 1024

// exclusive scan of in[0, n) into out by the whole block; returns the total
__device__ int block_scan_excl(const int *in, int *out, int n, int *s_warp)
{
    const int lane = warp_lane(), warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int carry = 0;
    for (int base = 0; base < n; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const int v = i < n ? in[i] : 0;
        const int incl = warp_incl_scan(v);
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const int w = lane < nwarps ? s_warp[lane] : 0;
            const int wi = warp_incl_scan(w);
            s_warp[lane] = wi - w;
            if (lane == 31) s_warp[32] = wi;
        }
        __syncthreads();
        if (i < n) out[i] = carry + s_warp[warp] + incl - v;
        carry += s_warp[32];
        __syncthreads();
    }
    return carry;
}

__global__ void __launch_bounds__(SMALL_TB) k_level_plan(BuildBufs b, int finish_prev, int top)
{
    ph::chain_begin();
    __shared__ int s_warp[33];
    if (finish_prev >= 0 && threadIdx.x == 0) level_finish(b, finish_prev, top);
    __syncthreads();
    const int lb = b.cnt[BC_LEVEL_BEGIN], C = b.cnt[BC_LEVEL_COUNT];
    for (int i = threadIdx.x; i < C; i += blockDim.x) level_nch_node(b, lb, i);
    __syncthreads();
    const int W = block_scan_excl(b.tn_nch, b.tn_chunk_base, C, s_warp);
    if (threadIdx.x == 0) b.cnt[BC_W] = W;
    const int lane = warp_lane();
    for (int i = threadIdx.x >> 5; i < C; i += blockDim.x >> 5) chunk_map_node(b, i, lane);
}

__global__ void __launch_bounds__(SMALL_TB) k_level_close(BuildBufs b, int maxleaf, int D)
{
    ph::chain_begin();
    __shared__ int s_warp[33];
    const int lb = b.cnt[BC_LEVEL_BEGIN], C = b.cnt[BC_LEVEL_COUNT];
    const int lane = warp_lane();
    for (int i = threadIdx.x >> 5; i < C; i += blockDim.x >> 5) node_split_node(b, lb, i, lane, maxleaf);
    __syncthreads();
    const int next = block_scan_excl(b.tn_nodeflag, b.tn_nodebase, C, s_warp);
    const int fresh = block_scan_excl(b.tn_leafflag, b.tn_leafbase, C, s_warp);
    if (threadIdx.x == 0) {
        b.cnt[BC_NEXT_NODES] = next;
        b.cnt[BC_NEW_LEAVES] = fresh;
    }
    const int leaves_before = b.cnt[BC_LEAVES];
    for (int i = threadIdx.x; i < C; i += blockDim.x) make_children_node(b, lb, C, leaves_before, i, maxleaf, D);
}

// After k_subtree_build: totals, and PH_FLAG_TOP if wide nodes remain
// unsplit after the last launched level.  A failed build (capacity, depth
// or levels) reports an empty tree, so every later stage of the pass has
// no work and reads nothing stale.
__global__ void k_tree_totals(BuildBufs b)
{
    ph::chain_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (b.cnt[BC_LEVEL_COUNT] > 0) b.cnt[BC_FLAGS] |= PH_FLAG_TOP;
        b.cnt[BC_NODES] = b.cnt[BC_LEVEL_BEGIN] + b.cnt[BC_MID_NODES] + b.cnt[BC_SUB_NODES];
        b.cnt[BC_LEAVES] += b.cnt[BC_MID_LEAVES] + b.cnt[BC_SUB_LEAVES];
        if (b.cnt[BC_FLAGS] & PH_FLAGS_TREE) {
            b.cnt[BC_NODES] = 0;
            b.cnt[BC_LEAVES] = 0;
            b.cnt[BC_NLEVELS] = 0;
            b.cnt[BC_SUB_NODES] = 0;
            b.cnt[BC_SUB_LEAVES] = 0;
        }
    }
}

// Ranks for the swap partition.  A particle not above the mean that sits in
// the right region (p >= S) publishes its position under slot S-1-r (r =
// its rank among such particles, counted from the left); a particle above
// the mean in the left region (p < S) publishes its position under slot
// p-r (its rank among particles above the mean).  Slot k pairs the k-th
// from the left with the k-th from the right, which is the order
// src/fmm.c:60-72 swaps them in.  ch_swap records each chunk's slots
// (the left-region particles above the mean), so k_swap reads one record
// per chunk.
__global__ void k_rank(BuildBufs b, int D)
{
    ph::chain_begin();
    const int lb = b.cnt[BC_LEVEL_BEGIN];
    const double *coord = axis_ptr(b.x, b.y, b.z, D);
    int W = b.cnt[BC_W];
    int lane = warp_lane();
    unsigned lt = (1u << lane) - 1u;
    int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int w = gw; w < W; w += nw) {
        int i = b.ch_node[w];
        int t = lb + i;
        if (b.tn_mode[t] != 0) {
            if (lane == 0) b.ch_swap[w] = make_int4(0, 0, 0, 0);
            continue;
        }
        int start = b.tn_start[t], len = b.tn_len[t];
        const long long km = order_key(b.tn_split[t]);
        int S = b.tn_S[t];
        int s0 = (w - b.tn_chunk_base[i]) * CHUNK;
        int s1 = min(len, s0 + CHUNK);
        const double *cp = coord + start;
        int *bigpos = b.bigpos + start, *smallpos = b.smallpos + start;
        const int small_before = b.ch_small_base[w];
        int run = small_before;
        int nbig = 0;
        for (int k0 = s0; k0 < s1; k0 += 128) {
            double v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int p = k0 + 32 * q + lane;
                v[q] = p < s1 ? cp[p] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int p = k0 + 32 * q + lane;
                const bool in = p < s1;
                const bool small = in && order_key(v[q]) <= km;
                const unsigned m = __ballot_sync(0xffffffffu, small);
                const int r = run + __popc(m & lt);
                if (in) {
                    if (p < S) { if (!small) bigpos[p - r] = p; }
                    else if (small) smallpos[S - 1 - r] = p;
                }
                nbig += __popc(__ballot_sync(0xffffffffu, in && p < S && !small));
                run += __popc(m);
            }
        }
        // the chunk's swaps for k_swap: its node's first particle, its first
        // slot and its number of slots (none once s0 >= S)
        if (lane == 0) b.ch_swap[w] = make_int4(start, s0 - small_before, s0 < S ? nbig : 0, 0);
    }
}

// The swaps of a chunk's slots: its left-region particles above the mean
// hold slots [s0 - (particles not above the mean before s0), + their
// number), as k_rank recorded in ch_swap; each slot's two particles trade
// places.  Pairs are disjoint; a lane loads four slots' particles before it
// stores any.
__global__ void k_swap(BuildBufs b, int D)
{
    ph::chain_begin();
    int W = b.cnt[BC_W];
    int lane = warp_lane();
    int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int w = gw; w < W; w += nw) {
        const int4 c = b.ch_swap[w];
        const int start = c.x, kb = c.y, nb = c.z;
        if (nb == 0) continue;
        const int *bigpos = b.bigpos + start + kb, *smallpos = b.smallpos + start + kb;
        for (int k0 = 0; k0 < nb; k0 += 128) {
            int pi[4], pj[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int k = k0 + 32 * q + lane;
                pi[q] = k < nb ? start + bigpos[k] : -1;
                pj[q] = k < nb ? start + smallpos[k] : -1;
            }
            double xi[4], yi[4], zi[4], xj[4], yj[4], zj[4];
            int qi[4], qj[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (pi[q] >= 0) {
                    xi[q] = b.x[pi[q]]; yi[q] = b.y[pi[q]]; zi[q] = b.z[pi[q]]; qi[q] = b.perm[pi[q]];
                    xj[q] = b.x[pj[q]]; yj[q] = b.y[pj[q]]; zj[q] = b.z[pj[q]]; qj[q] = b.perm[pj[q]];
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (pi[q] >= 0) {
                    b.x[pi[q]] = xj[q]; b.y[pi[q]] = yj[q]; b.z[pi[q]] = zj[q]; b.perm[pi[q]] = qj[q];
                    b.x[pj[q]] = xi[q]; b.y[pj[q]] = yi[q]; b.z[pj[q]] = zi[q]; b.perm[pj[q]] = qi[q];
                }
            }
        }
    }
}

// ---------------- nodes of CHUNK + 1 to PH_MID particles ----------------
// One block per such node: its particles in shared memory, it and its
// descendants of more than CHUNK particles split one after another by the
// whole block, with the sums, counts, ranks and swaps of the level kernels
// (chunk sums by one warp each in the same lane order), and the particles
// written back once.  New nodes and leaves go after the level-built ones, in
// any order (the numbering reads particle ranges).  What a level costs here
// is a few barriers (~4 us a node) instead of 7 or 19 launches (~25-40 us).
// With the numbering below, build of 4,096 grid particles 0.222 -> 0.130 ms,
// 32,768 0.361 -> 0.269, 110,591 half in halos 0.767 -> 0.517.
struct MidTree {
    double x[PH_MID], y[PH_MID], z[PH_MID];
    // a node's slots while it is split; at the end the original permutation
    unsigned short bigpos[PH_MID], smallpos[PH_MID];
    unsigned short loc[PH_MID];
    double part[PH_MID / CHUNK + 1], mean;
    int seg[PH_MID / MID_SEG + 1];
    int nbig, fail;
    // nodes still to split: at most PH_MID / CHUNK - 1 at a time (disjoint, more than CHUNK particles each)
    int head, tail;
    int q_id[8], q_start[8], q_len[8], q_depth[8];
};
static_assert(PH_MID / CHUNK <= 8 && PH_MID / MID_SEG <= 32, "one warp holds a node's chunk sums and segment counts");

// Whether the build has failed so far (wide nodes left, too little room or
// too few levels): node numbers may then have been taken without a record
// written, so no block goes on from them.  One thread reads, since blocks
// of the same launch may raise a flag meanwhile, and the block returns as a
// whole.
__device__ __forceinline__ bool build_failed(const BuildBufs &b)
{
    __shared__ int s_failed;
    if (threadIdx.x == 0)
        s_failed = b.cnt[BC_LEVEL_COUNT] > 0 ||
                   (b.cnt[BC_FLAGS] & (PH_FLAG_LEAF_CAPACITY | PH_FLAG_NODE_CAPACITY | PH_FLAG_DEPTH | PH_FLAG_SUBTREE));
    __syncthreads();
    return s_failed != 0;
}

__global__ void __launch_bounds__(MID_TB, 1) k_mid_build(BuildBufs b, int axis0, int maxleaf, int levels)
{
    ph::chain_begin();
    extern __shared__ __align__(16) unsigned char mid_smem[];
    MidTree &s = *reinterpret_cast<MidTree *>(mid_smem);
    if (build_failed(b)) return;
    const int T0 = b.cnt[BC_LEVEL_BEGIN], L0 = b.cnt[BC_LEAVES];
    const int tid = threadIdx.x, lane = warp_lane(), warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    for (int t = blockIdx.x; t < T0; t += gridDim.x) {
        if (b.tn_mode[t] != MODE_MID) continue;  // the same for the whole block
        const int start = b.tn_start[t], len = b.tn_len[t], boxid = b.tn_boxid[t];
        __syncthreads();  // the last node's particles and state have been read
        for (int k = tid; k < len; k += MID_TB) {
            s.x[k] = b.x[start + k];
            s.y[k] = b.y[start + k];
            s.z[k] = b.z[start + k];
            s.loc[k] = (unsigned short)k;
        }
        if (tid == 0) {
            s.head = 0;
            s.tail = 1;
            s.q_id[0] = t;
            s.q_start[0] = 0;
            s.q_len[0] = len;
            s.q_depth[0] = b.tn_depth[t];
            s.fail = b.tn_depth[t] >= levels ? PH_FLAG_DEPTH : 0;
        }
        __syncthreads();
        while (s.head < s.tail && !s.fail) {
            const int q = s.head & 7, id = s.q_id[q], ns = s.q_start[q], ln = s.q_len[q], depth = s.q_depth[q];
            const int D = (axis0 + depth) % 3;
            const double *cd = axis_ptr(s.x, s.y, s.z, D) + ns;
            const int nc = (ln + CHUNK - 1) / CHUNK, nseg = (ln + MID_SEG - 1) / MID_SEG;
            // chunk sums, then the node's mean
            if (warp < nc) {
                const int s1 = min(ln, (warp + 1) * CHUNK);
                double sum = 0.0;
#pragma unroll 8
                for (int k = warp * CHUNK + lane; k < s1; k += 32) sum += cd[k];
                sum = warp_sum_d(sum);
                if (lane == 0) s.part[warp] = sum;
            }
            if (tid == 0) s.nbig = 0;
            __syncthreads();
            if (warp == 0) {
                double sum = 0.0;
                if (lane < nc) sum += s.part[lane];
                sum = warp_sum_d(sum);
                if (lane == 0) s.mean = sum / (double)ln;
            }
            __syncthreads();
            const double mean = s.mean;
            const long long km = order_key(mean);
            for (int g = warp; g < nseg; g += MID_NW) {
                int c = 0;
#pragma unroll
                for (int k = 0; k < MID_SEG; k += 32) {
                    const int p = g * MID_SEG + k + lane;
                    c += p < ln && order_key(cd[p]) <= km;
                }
                c = __reduce_add_sync(0xffffffffu, c);
                if (lane == 0) s.seg[g] = c;
            }
            __syncthreads();
            const int own = lane < nseg ? s.seg[lane] : 0, incl = warp_incl_scan(own);
            const int S = __shfl_sync(0xffffffffu, incl, 31);
            int mode, left;
            split_sizes(ln, S, mode, left);
            unsigned short *bigpos = s.bigpos + ns, *smallpos = s.smallpos + ns;
            if (mode == 0) {
                int nbig = 0;
                for (int g = warp; g < nseg; g += MID_NW) {
                    int run = __shfl_sync(0xffffffffu, incl - own, g);
                    for (int k = 0; k < MID_SEG; k += 32) {
                        const int p = g * MID_SEG + k + lane;
                        const bool in = p < ln;
                        const bool small = in && order_key(cd[p]) <= km;
                        const unsigned m = __ballot_sync(0xffffffffu, small);
                        const int r = run + __popc(m & lt);
                        if (in) {
                            if (p < S) { if (!small) bigpos[p - r] = (unsigned short)p; }
                            else if (small) smallpos[S - 1 - r] = (unsigned short)p;
                        }
                        nbig += __popc(__ballot_sync(0xffffffffu, in && p < S && !small));
                        run += __popc(m);
                    }
                }
                if (lane == 0 && nbig) atomicAdd(&s.nbig, nbig);
            }
            __syncthreads();
            if (mode == 0) {
                for (int k = tid; k < s.nbig; k += MID_TB) {
                    const int i = ns + bigpos[k], j = ns + smallpos[k];
                    double v;
                    v = s.x[i]; s.x[i] = s.x[j]; s.x[j] = v;
                    v = s.y[i]; s.y[i] = s.y[j]; s.y[j] = v;
                    v = s.z[i]; s.z[i] = s.z[j]; s.z[j] = v;
                    const unsigned short w = s.loc[i]; s.loc[i] = s.loc[j]; s.loc[j] = w;
                }
            }
            // the children, a thread each, beside the swaps
            if (tid >= MID_TB - 2) {
                const int c = tid - (MID_TB - 2);
                const int size = c ? ln - left : left, first = start + ns + (c ? left : 0);
                double *box = b.tn_box;
                double bound[6];
                for (int d = 0; d < 6; d++) bound[d] = box[d * b.cap_nodes + id];
                bound[c ? D : 3 + D] = mean;
                int code = 0;
                if (size <= maxleaf) {
                    const int lid = L0 + atomicAdd(&b.cnt[BC_MID_LEAVES], 1);
                    if (lid >= b.rule_cap) {
                        atomicOr(&s.fail, PH_FLAG_LEAF_CAPACITY);
                    } else {
                        b.tl_start[lid] = first;
                        b.tl_len[lid] = size;
                        b.tl_depth[lid] = depth + 1;
                        b.tl_parent[lid] = id;
                        b.tl_boxid[lid] = boxid;
                        for (int d = 0; d < 6; d++) b.tl_box[d * b.cap_leaves + lid] = bound[d];
                        code = ~lid;
                    }
                } else {
                    const int nid = T0 + atomicAdd(&b.cnt[BC_MID_NODES], 1);
                    if (nid >= b.rule_cap) {
                        atomicOr(&s.fail, PH_FLAG_NODE_CAPACITY);
                    } else if (depth + 1 >= levels) {
                        atomicOr(&s.fail, PH_FLAG_DEPTH);
                    } else {
                        b.tn_start[nid] = first;
                        b.tn_len[nid] = size;
                        b.tn_depth[nid] = depth + 1;
                        b.tn_parent[nid] = id;
                        b.tn_boxid[nid] = boxid;
                        b.tn_mode[nid] = open_mode(b, size);
                        for (int d = 0; d < 6; d++) box[d * b.cap_nodes + nid] = bound[d];
                        code = nid;
                        if (size > CHUNK) {
                            const int w = atomicAdd(&s.tail, 1) & 7;
                            s.q_id[w] = nid;
                            s.q_start[w] = first - start;
                            s.q_len[w] = size;
                            s.q_depth[w] = depth + 1;
                        }
                    }
                }
                if (c == 0) {
                    b.tn_child0[id] = code;
                    b.tn_split[id] = mean;
                    b.tn_mode[id] = mode;
                    s.head++;
                } else {
                    b.tn_child1[id] = code;
                }
            }
            __syncthreads();
        }
        if (s.fail) {
            if (tid == 0) atomicOr(&b.cnt[BC_FLAGS], s.fail);
            continue;
        }
        int *operm = reinterpret_cast<int *>(s.bigpos);
        for (int k = tid; k < len; k += MID_TB) {
            operm[k] = b.perm[start + k];
            b.x[start + k] = s.x[k];
            b.y[start + k] = s.y[k];
            b.z[start + k] = s.z[k];
        }
        __syncthreads();
        for (int k = tid; k < len; k += MID_TB) b.perm[start + k] = operm[s.loc[k]];
    }
}

// ---------------- subtrees of at most CHUNK particles ----------------
// Shared memory of one subtree block, 53.3 KB: four blocks per SM.  The
// arrays hold CHUNK nodes and leaves.  Subtrees with empty leaves can have
// more (a line of particles: up to three nodes a particle, two of the three
// axes splitting nothing off); the build is then repeated with subtrees of
// at most PH_SUB_SMALL particles, the rest split by the levels.
struct SubTree {
    // the subtree's particles; once written back, the region holds the
    // original permutation (bytes 0-4095) and the parents
    double x[CHUNK], y[CHUNK], z[CHUNK];
    unsigned short loc[CHUNK];                      // subtree-local index of the particle at each position
    unsigned short bigpos[CHUNK], smallpos[CHUNK];  // a node's slots, over its own local range
    // nodes by level in creation order (node 0 the subtree root): local
    // range, child codes (>= 0 node, < 0 ~leaf), split
    unsigned short n_start[CHUNK], n_len[CHUNK];
    short n_c0[CHUNK], n_c1[CHUNK];
    double n_split[CHUNK];
    unsigned short l_start[CHUNK], l_len[CHUNK];
    unsigned short lev[CHUNK + 2];  // first node of each level of the subtree
    // nodes made by a level are numbered after the level's end through
    // counter (L + 1) mod 3, which also records a failure (see
    // k_subtree_build)
    int nalloc[3];
    int nleaves, fail, nbase, lbase;
    int large;  // more nodes or leaves than the arrays hold
};

__device__ __forceinline__ void sub_swap(SubTree &s, int i, int j)
{
    double t;
    t = s.x[i]; s.x[i] = s.x[j]; s.x[j] = t;
    t = s.y[i]; s.y[i] = s.y[j]; s.y[j] = t;
    t = s.z[i]; s.z[i] = s.z[j]; s.z[j] = t;
    const unsigned short q = s.loc[i]; s.loc[i] = s.loc[j]; s.loc[j] = q;
}

// One warp splits node i of the subtree (at depth `depth`, level L of the
// subtree whose nodes end at lend): the mean, count, ranks and swaps a node
// of one chunk gets, with the same lane order and reductions (the sum is
// lane 0's butterfly result added to 0.0, as the one-term reduction of
// k_node_mean does), then its two children.
__device__ void sub_split_node(SubTree &s, int i, int depth, int L, int lend, int axis0, int maxleaf, int levels)
{
    const int lane = warp_lane();
    const unsigned lt = (1u << lane) - 1u;
    const int ns = s.n_start[i], len = s.n_len[i];
    const int D = (axis0 + depth) % 3;
    const double *cd = axis_ptr(s.x, s.y, s.z, D) + ns;
    double mean;
    if (len == 2) {
        mean = 0.5 * (cd[0] + cd[1]);
    } else {
        double sum = 0.0;
        for (int k = lane; k < len; k += 32) sum += cd[k];
        sum = __shfl_sync(0xffffffffu, warp_sum_d(sum), 0);
        double m = 0.0;
        m += sum;
        mean = m / (double)len;
    }
    const long long km = order_key(mean);
    int c = 0;
    for (int k = lane; k < len; k += 32) c += order_key(cd[k]) <= km;
    const int S = __reduce_add_sync(0xffffffffu, c);
    int mode, left;
    split_sizes(len, S, mode, left);
    if (len == 2) {
        if (lane == 0 && cd[0] > cd[1]) sub_swap(s, ns, ns + 1);
    } else if (mode == 0) {
        unsigned short *bigpos = s.bigpos + ns, *smallpos = s.smallpos + ns;
        int run = 0, nbig = 0;
        for (int k0 = 0; k0 < len; k0 += 32) {
            const int p = k0 + lane;
            const bool in = p < len;
            const bool small = in && order_key(cd[p]) <= km;
            const unsigned m = __ballot_sync(0xffffffffu, small);
            const int r = run + __popc(m & lt);
            if (in) {
                if (p < S) { if (!small) bigpos[p - r] = (unsigned short)p; }
                else if (small) smallpos[S - 1 - r] = (unsigned short)p;
            }
            nbig += __popc(__ballot_sync(0xffffffffu, in && p < S && !small));
            run += __popc(m);
        }
        __syncwarp();
        for (int k = lane; k < nbig; k += 32) sub_swap(s, ns + bigpos[k], ns + smallpos[k]);
    }
    __syncwarp();
    if (lane == 0) {
        s.n_split[i] = mean;
        const int sizes[2] = {left, len - left};
        int off = ns;
        for (int ch = 0; ch < 2; ch++) {
            int code;
            // a node below the launched depths fails the subtree, and so does
            // a node or leaf beyond the arrays
            if (sizes[ch] <= maxleaf) {
                const int j = atomicAdd(&s.nleaves, 1);
                code = ~j;
                if (j < CHUNK) {
                    s.l_start[j] = (unsigned short)off;
                    s.l_len[j] = (unsigned short)sizes[ch];
                } else {
                    atomicAdd(&s.nalloc[(L + 1) % 3], SUB_FAIL);
                    s.large = 1;
                }
            } else {
                const bool deep = depth + 1 >= levels;
                const int j = lend + (atomicAdd(&s.nalloc[(L + 1) % 3], deep ? SUB_FAIL + 1 : 1) & (SUB_FAIL - 1));
                code = j;
                if (j < CHUNK) {
                    s.n_start[j] = (unsigned short)off;
                    s.n_len[j] = (unsigned short)sizes[ch];
                } else {
                    atomicAdd(&s.nalloc[(L + 1) % 3], SUB_FAIL);
                    s.large = 1;
                }
            }
            if (ch == 0) s.n_c0[i] = (short)code;
            else s.n_c1[i] = (short)code;
            off += sizes[ch];
        }
    }
}

// One block per deferred node: load its particles into shared memory, split
// its subtree level by level (a warp per node), write the particles back,
// then write the nodes and leaves into the temp arrays after those made
// before, with boxes from the split planes.
// Every barrier is reached by all threads of the block: loop bounds and
// failure flags are read after a barrier and not written again before the
// next one.  Level L numbers its new nodes through counter (L + 1) mod 3
// (a failure adds SUB_FAIL to it), which thread 0 cleared during level
// L - 1; counter (L + 2) mod 3, last read after level L - 2, is cleared
// during level L.  So one barrier per level.
__global__ void __launch_bounds__(SUB_TB) k_subtree_build(BuildBufs b, int axis0, int maxleaf, int levels)
{
    ph::chain_begin();
    extern __shared__ __align__(16) unsigned char sub_smem[];
    SubTree &s = *reinterpret_cast<SubTree *>(sub_smem);
    if (build_failed(b)) return;
    const int T0 = b.cnt[BC_LEVEL_BEGIN] + b.cnt[BC_MID_NODES], L0 = b.cnt[BC_LEAVES] + b.cnt[BC_MID_LEAVES];
    const int tid = threadIdx.x, warp = tid >> 5;
    int *operm = reinterpret_cast<int *>(s.x);
    unsigned short *npar = reinterpret_cast<unsigned short *>(s.x) + 2 * CHUNK, *lpar = npar + CHUNK;
    for (int t = blockIdx.x; t < T0; t += gridDim.x) {
        if (b.tn_mode[t] != MODE_DEFERRED) continue;
        const int start = b.tn_start[t], len = b.tn_len[t], rd = b.tn_depth[t];
        for (int k = tid; k < len; k += SUB_TB) {
            s.x[k] = b.x[start + k];
            s.y[k] = b.y[start + k];
            s.z[k] = b.z[start + k];
            s.loc[k] = (unsigned short)k;
        }
        if (tid == 0) {
            s.nalloc[1] = 0;
            s.nleaves = 0;
            s.n_start[0] = 0;
            s.n_len[0] = (unsigned short)len;
            s.lev[0] = 0;
            s.fail = 0;
            s.large = 0;
        }
        __syncthreads();
        int failed = rd >= levels;
        int nlev = 0, lbeg = 0, lend = 1;
        while (lbeg < lend && !failed) {
            if (tid == 0) s.nalloc[(nlev + 2) % 3] = 0;
            for (int i = lbeg + warp; i < lend; i += SUB_NW)
                sub_split_node(s, i, rd + nlev, nlev, lend, axis0, maxleaf, levels);
            __syncthreads();
            const int got = s.nalloc[(nlev + 1) % 3];
            lbeg = lend;
            lend += got & (SUB_FAIL - 1);
            failed = got >= SUB_FAIL;
            nlev++;
            if (tid == 0) s.lev[nlev] = (unsigned short)lbeg;
        }
        __syncthreads();  // lev[] complete
        if (failed) {
            if (tid == 0) atomicOr(&b.cnt[BC_FLAGS], s.large ? PH_FLAG_SUBTREE : PH_FLAG_DEPTH);
            continue;  // the next subtree's first writes follow a barrier all threads passed
        }
        for (int k = tid; k < len; k += SUB_TB) {
            b.x[start + k] = s.x[k];
            b.y[start + k] = s.y[k];
            b.z[start + k] = s.z[k];
        }
        __syncthreads();  // x, y, z read: their region now takes the original permutation
        for (int k = tid; k < len; k += SUB_TB) operm[k] = b.perm[start + k];
        __syncthreads();
        for (int k = tid; k < len; k += SUB_TB) b.perm[start + k] = operm[s.loc[k]];
        // parents from the child codes
        for (int i = tid; i < lend; i += SUB_TB) {
            const int c0 = s.n_c0[i], c1 = s.n_c1[i];
            if (c0 >= 0) npar[c0] = (unsigned short)i; else lpar[~c0] = (unsigned short)i;
            if (c1 >= 0) npar[c1] = (unsigned short)i; else lpar[~c1] = (unsigned short)i;
        }
        if (tid == 0) {
            const int ltot = s.nleaves;
            const int nb = atomicAdd(&b.cnt[BC_SUB_NODES], lend - 1);
            const int lbg = atomicAdd(&b.cnt[BC_SUB_LEAVES], ltot);
            s.nbase = T0 + nb;
            s.lbase = L0 + lbg;
            if (T0 + nb + lend - 1 > b.rule_cap) {
                atomicOr(&b.cnt[BC_FLAGS], PH_FLAG_NODE_CAPACITY);
                s.fail = 1;
            }
            if (L0 + lbg + ltot > b.rule_cap) {
                atomicOr(&b.cnt[BC_FLAGS], PH_FLAG_LEAF_CAPACITY);
                s.fail = 1;
            }
        }
        __syncthreads();
        failed = s.fail;
        __syncthreads();
        if (failed) continue;
        // node i of the subtree becomes temp node nbase + i - 1, leaf j temp leaf lbase + j
        const int nbase = s.nbase - 1, lbase = s.lbase, boxid = b.tn_boxid[t];
        // nodes level by level: a node's box is its parent's, written a level earlier, cut at the parent's split
        for (int L = 0; L < nlev; L++) {
            for (int i = s.lev[L] + tid; i < s.lev[L + 1]; i += SUB_TB) {
                const int ti = i == 0 ? t : nbase + i;
                const int c0 = s.n_c0[i], c1 = s.n_c1[i];
                b.tn_child0[ti] = c0 >= 0 ? nbase + c0 : ~(lbase + ~c0);
                b.tn_child1[ti] = c1 >= 0 ? nbase + c1 : ~(lbase + ~c1);
                b.tn_split[ti] = s.n_split[i];
                if (i == 0) continue;
                const int par = npar[i];
                const int tp = par == 0 ? t : nbase + par;
                b.tn_start[ti] = start + s.n_start[i];
                b.tn_len[ti] = s.n_len[i];
                b.tn_depth[ti] = rd + L;
                b.tn_parent[ti] = tp;
                b.tn_boxid[ti] = boxid;
                const int Dp = (axis0 + rd + L - 1) % 3;
                const bool upper = s.n_c0[par] != i;
                for (int d = 0; d < 3; d++) {
                    double lo = b.tn_box[d * b.cap_nodes + tp], hi = b.tn_box[(3 + d) * b.cap_nodes + tp];
                    if (d == Dp) {
                        if (upper) lo = s.n_split[par];
                        else hi = s.n_split[par];
                    }
                    b.tn_box[d * b.cap_nodes + ti] = lo;
                    b.tn_box[(3 + d) * b.cap_nodes + ti] = hi;
                }
            }
            __syncthreads();
        }
        for (int j = tid; j < s.nleaves; j += SUB_TB) {
            const int tl = lbase + j;
            const int par = lpar[j];
            const int tp = par == 0 ? t : nbase + par;
            const int pd = b.tn_depth[tp];
            b.tl_start[tl] = start + s.l_start[j];
            b.tl_len[tl] = s.l_len[j];
            b.tl_depth[tl] = pd + 1;
            b.tl_parent[tl] = tp;
            b.tl_boxid[tl] = boxid;
            const int Dp = (axis0 + pd) % 3;
            const bool upper = s.n_c0[par] != ~j;
            for (int d = 0; d < 3; d++) {
                double lo = b.tn_box[d * b.cap_nodes + tp], hi = b.tn_box[(3 + d) * b.cap_nodes + tp];
                if (d == Dp) {
                    if (upper) lo = s.n_split[par];
                    else hi = s.n_split[par];
                }
                b.tl_box[d * b.cap_leaves + tl] = lo;
                b.tl_box[(3 + d) * b.cap_leaves + tl] = hi;
            }
        }
        __syncthreads();
    }
}

// ---------------- numbering ----------------
// Leaves partition the particles in depth-first order, so a leaf's number is
// the number of leaves before its own start: a bit per particle where a leaf
// with particles starts, counted by words, plus the empty leaves before.
// Nodes that start where such a leaf does are its ancestors from the
// topmost one starting there (a right child or a root) down to its parent,
// and nodes in preorder are those of the first leaf, those of the second and
// so on: a node's number is the nodes of the leaves before plus its depth
// below that topmost one.  (The reference numbers them while it recurses,
// src/fmm.c:101-118.)
// An empty leaf is a left child: where the mean of equal coordinates rounds
// below them, the lower half of the split holds nothing (sheets, lines and
// lattices; a right child always holds something).  It starts where its
// sibling does and comes before what the sibling holds, so the empty leaves
// of one start are ordered by depth and precede the leaf with particles.
__global__ void k_mark_leaves(BuildBufs b)
{
    ph::chain_begin();
    const int nleaves = b.cnt[BC_LEAVES];
    for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < nleaves; l += gridDim.x * blockDim.x) {
        b.lf_empty[l] = 0;
        if (b.tl_len[l] > 0) {
            const int p = b.tl_start[l];
            atomicOr(reinterpret_cast<unsigned *>(b.words) + (p >> 5), 1u << (p & 31));
        } else {
            atomicAdd(&b.cnt[BC_EMPTY], 1);
        }
    }
}

// starts before particle p
__device__ __forceinline__ int start_rank(const BuildBufs &b, int p)
{
    return b.wordpre[p >> 5] + __popc((unsigned)b.words[p >> 5] & ((1u << (p & 31)) - 1u));
}

// scan inputs: the starts of word i; per start, the nodes there and, in the
// upper half, the empty leaves
__device__ __forceinline__ void scan_value(const BuildBufs &b, int i, int &v) { v = __popc((unsigned)b.words[i]); }
__device__ __forceinline__ void scan_value(const BuildBufs &b, int i, long long &v)
{
    v = (b.lf_depth[i] - b.lf_top[i]) | ((long long)b.lf_empty[i] << 32);
}

template <class V>
__global__ void k_scan_input(BuildBufs b, const int *n_ptr, V *out)
{
    ph::chain_begin();
    const int n = *n_ptr;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) scan_value(b, i, out[i]);
}

template <class V>
__device__ __forceinline__ V warp_incl(V v)
{
    const int lane = warp_lane();
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const V t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// the exclusive scan of up to ONE_SCAN_MAX of them in one block
#define ONE_SCAN_TB 1024
#define ONE_SCAN_MAX (1 << 16)
template <class V>
__global__ void __launch_bounds__(ONE_SCAN_TB) k_scan_one(BuildBufs b, const int *n_ptr, V *out)
{
    ph::chain_begin();
    __shared__ V s_warp[33];
    const int lane = warp_lane(), warp = threadIdx.x >> 5, n = *n_ptr;
    V carry = 0;
    for (int base = 0; base < n; base += 4 * ONE_SCAN_TB) {
        const int i0 = base + 4 * (int)threadIdx.x;
        V v[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = 0;
            if (i0 + k < n) scan_value(b, i0 + k, v[k]);
            sum += v[k];
        }
        const V incl = warp_incl(sum);
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const V x = s_warp[lane], xi = warp_incl(x);
            s_warp[lane] = xi - x;
            if (lane == 31) s_warp[32] = xi;
        }
        __syncthreads();
        V at = carry + s_warp[warp] + incl - sum;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i0 + k < n) out[i0 + k] = at;
            at += v[k];
        }
        carry += s_warp[32];
        __syncthreads();
    }
}

// per start: the depth of the leaf with particles, the depth of the topmost
// node or leaf that starts there, and the empty leaves
__global__ void k_leaf_ranks(BuildBufs b)
{
    ph::chain_begin();
    const int nleaves = b.cnt[BC_LEAVES], nnodes = b.cnt[BC_NODES];
    if (blockIdx.x == 0 && threadIdx.x == 0) b.cnt[BC_STARTS] = nleaves - b.cnt[BC_EMPTY];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nleaves + nnodes; i += gridDim.x * blockDim.x) {
        const bool leaf = i < nleaves;
        const int t = leaf ? i : i - nleaves;
        const int start = leaf ? b.tl_start[t] : b.tn_start[t], parent = leaf ? b.tl_parent[t] : b.tn_parent[t],
                  depth = leaf ? b.tl_depth[t] : b.tn_depth[t];
        const int r = start_rank(b, start);
        if (leaf && b.tl_len[t] == 0) {
            atomicAdd(&b.lf_empty[r], 1);
            continue;
        }
        if (leaf) b.lf_depth[r] = depth;
        if (parent < 0 || b.tn_start[parent] != start) b.lf_top[r] = depth;
    }
}

__device__ __forceinline__ void write_geom(TreeBufs &T, int u, const double *box, int cap, int idx)
{
    double lo0 = box[0 * cap + idx], lo1 = box[1 * cap + idx], lo2 = box[2 * cap + idx];
    double hi0 = box[3 * cap + idx], hi1 = box[4 * cap + idx], hi2 = box[5 * cap + idx];
    // width = right - left, centre = 0.5*(right + left), src/fmm.c:126-131
    double w0 = hi0 - lo0, w1 = hi1 - lo1, w2 = hi2 - lo2;
    T.wx[u] = w0; T.wy[u] = w1; T.wz[u] = w2;
    T.cx[u] = 0.5 * (hi0 + lo0); T.cy[u] = 0.5 * (hi1 + lo1); T.cz[u] = 0.5 * (hi2 + lo2);
    T.wsum[u] = w0 + w1 + w2;
}

// preorder number of the node of depth `depth` that starts at particle p
__device__ __forceinline__ int node_number(const BuildBufs &b, int p, int depth)
{
    const int r = start_rank(b, p);
    return (int)b.lf_base[r] + depth - b.lf_top[r];
}

// depth-first number of temp leaf l
__device__ __forceinline__ int leaf_number(const BuildBufs &b, int l)
{
    const int start = b.tl_start[l], r = start_rank(b, start), empty = b.lf_empty[r];
    int id = r + (int)(b.lf_base[r] >> 32);
    if (empty == 0) return id;
    if (b.tl_len[l] > 0) return id + empty;
    // after the empty leaves of the nodes above its parent that start here too
    for (int t = b.tl_parent[l];;) {
        t = b.tn_parent[t];
        if (t < 0 || b.tn_start[t] != start) return id;
        const int c = b.tn_child0[t];
        id += PH_IS_LEAF_CODE(c) && b.tl_len[~c] == 0;
    }
}

// a child's unified id: a leaf's number, or a node's preorder number after the leaves
__device__ __forceinline__ int child_id(const BuildBufs &b, int code, int nleaves)
{
    return PH_IS_LEAF_CODE(code) ? leaf_number(b, ~code)
                                 : nleaves + node_number(b, b.tn_start[code], b.tn_depth[code]);
}

// temp nodes and leaves into the unified index space
__global__ void k_scatter_tree(BuildBufs b, TreeBufs T)
{
    ph::chain_begin();
    const int nnodes = b.cnt[BC_NODES], nleaves = b.cnt[BC_LEAVES];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nleaves + nnodes; i += gridDim.x * blockDim.x) {
        if (i < nleaves) {
            const int l = i, u = leaf_number(b, l), par = b.tl_parent[l];
            T.ipart[u] = b.tl_start[l];
            T.npart[u] = b.tl_len[l];
            T.depth[u] = b.tl_depth[l];
            T.parent[u] = nleaves + node_number(b, b.tn_start[par], b.tn_depth[par]);
            T.son0[u] = -1;
            T.son1[u] = -1;
            T.split[u] = 0.0;
            T.boxid[u] = b.tl_boxid[l];
            write_geom(T, u, b.tl_box, b.cap_leaves, l);
        } else {
            const int t = i - nleaves, u = nleaves + node_number(b, b.tn_start[t], b.tn_depth[t]), par = b.tn_parent[t];
            T.ipart[u] = b.tn_start[t];
            T.npart[u] = b.tn_len[t];
            T.depth[u] = b.tn_depth[t];
            T.parent[u] = par < 0 ? -1 : nleaves + node_number(b, b.tn_start[par], b.tn_depth[par]);
            T.son0[u] = child_id(b, b.tn_child0[t], nleaves);
            T.son1[u] = child_id(b, b.tn_child1[t], nleaves);
            T.split[u] = b.tn_split[t];
            T.boxid[u] = b.tn_boxid[t];
            if (t < b.nbox) b.boxes[t].root = u;
            write_geom(T, u, b.tn_box, b.cap_nodes, t);
        }
    }
}

// ---------------- depth lists ----------------
// A stable counting sort of the unified ids by depth: depth d's list holds
// its leaves (depth-first order) then its nodes (preorder).  Block k counts
// the depths of ids [k R, (k+1) R) into cells (depth, block), stored depth
// by depth; an exclusive scan of the cells gives each block its first slot
// per depth.
__global__ void __launch_bounds__(32) k_depth_count(BuildBufs b, TreeBufs T, int ndepth)
{
    ph::chain_begin();
    __shared__ int h[PH_MAX_DEPTH_CAP + 2];
    const int nu = b.cnt[BC_NODES] + b.cnt[BC_LEAVES], nblk = gridDim.x, k = blockIdx.x, lane = threadIdx.x;
    for (int d = lane; d < ndepth; d += 32) h[d] = 0;
    __syncwarp();
    const int u0 = k * DEPTH_R, u1 = min(nu, u0 + DEPTH_R);
#pragma unroll 8
    for (int u = u0 + lane; u < u1; u += 32) {
        const int d = T.depth[u];
        if (d >= 0 && d < ndepth) atomicAdd(&h[d], 1);
    }
    __syncwarp();
    for (int d = lane; d < ndepth; d += 32) T.depth_blk[d * nblk + k] = h[d];
    if (k == 0 && lane == 0) b.cnt[BC_DEPTH_CELLS] = ndepth * nblk;
}

__global__ void __launch_bounds__(32) k_depth_place(BuildBufs b, TreeBufs T, int ndepth)
{
    ph::chain_begin();
    __shared__ int cur[PH_MAX_DEPTH_CAP + 2];
    const int nu = b.cnt[BC_NODES] + b.cnt[BC_LEAVES], nblk = gridDim.x, k = blockIdx.x, lane = threadIdx.x;
    const unsigned lt = (1u << lane) - 1u;
    const int *first = T.depth_blk + (size_t)ndepth * nblk;  // the scanned cells
    for (int d = lane; d < ndepth; d += 32) cur[d] = first[d * nblk + k];
    if (k == 0) {
        // per-depth offsets and counts, and the deepest depth holding an id
        int deepest = 0;
        for (int d = lane; d < ndepth; d += 32) {
            const int o = first[d * nblk], e = d + 1 < ndepth ? first[(d + 1) * nblk] : nu;
            T.depth_off[d] = o;
            T.depth_cnt[d] = e - o;
            if (e > o) deepest = d;
        }
        deepest = __reduce_max_sync(0xffffffffu, deepest);
        if (lane == 0) {
            T.depth_off[ndepth] = nu;
            b.cnt[BC_DEPTH] = deepest;
        }
    }
    __syncwarp();
    const int u0 = k * DEPTH_R, u1 = min(nu, u0 + DEPTH_R);
    for (int b0 = u0; b0 < u1; b0 += 256) {
        int dd[8];  // eight loads ahead of the placing, which is serial
#pragma unroll
        for (int q = 0; q < 8; q++) dd[q] = b0 + 32 * q + lane < u1 ? T.depth[b0 + 32 * q + lane] : -1;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int u = b0 + 32 * q + lane;
            int d = dd[q];
            if (d >= ndepth) d = -1;
            const unsigned same = __match_any_sync(0xffffffffu, d);
            if (d >= 0) T.depth_list[cur[d] + __popc(same & lt)] = u;
            __syncwarp();
            if (d >= 0 && (same & lt) == 0) cur[d] += __popc(same);
            __syncwarp();
        }
    }
}

}  // namespace

int launch_init_particles(BuildBufs &b, const double *pos, int n, cudaStream_t st)
{
    ph::note_launch(), k_init_particles<<<device_sm_count() * 8, TB, 0, st>>>(pos, n, b);
    PH_CUDA_CHECK(cudaGetLastError());
    return 0;
}

int depth_sort_blocks(int cap_u) { return (cap_u + DEPTH_R - 1) / DEPTH_R; }

// Enqueue the whole build, no host sync: at most `top` levels of wide
// nodes, then the subtrees, with nodes at depths < `levels`.  Levels past
// the last wide node exit at once.  Wide nodes left after `top` levels
// raise PH_FLAG_TOP in b.cnt[BC_FLAGS] and a node at depth `levels` raises
// PH_FLAG_DEPTH (the caller grows the count and builds again); capacity
// overflows raise their flags there too.  Depth lists cover depths
// 0..levels.
int build_tree(BuildBufs &b, TreeBufs &T, const PassParams &p, int n, int levels, int top, cudaStream_t st)
{
    const int maxb = device_sm_count() * 8;
    if (levels < 1 || levels + 1 > T.max_depth_cap || T.max_depth_cap > PH_MAX_DEPTH_CAP)
        return ph_set_error(7, "tree deeper than %d levels", T.max_depth_cap - 1);
    if (top < 0 || top > levels) top = levels;
    const int ndepth = levels + 1;  // leaves can sit one level below the deepest nodes
    // blocks for as many nodes and leaves as this pass can have
    const int nblk = depth_sort_blocks(2 * b.rule_cap);
    if (nblk < 1 || nblk > T.depth_nblk) return ph_set_error(7, "depth-sort buffers not allocated");
    // shared memory above the 48 KB default, allowed once per device
    static std::atomic<bool> done[64];
    int dev = 0;
    PH_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !done[dev].load()) {
        PH_CUDA_CHECK(cudaFuncSetAttribute(k_subtree_build, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sizeof(SubTree)));
        PH_CUDA_CHECK(cudaFuncSetAttribute(k_mid_build, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sizeof(MidTree)));
        if (dev >= 0 && dev < 64) done[dev].store(true);
    }
    PH_CUDA_CHECK(cudaMemsetAsync(b.words, 0, sizeof(int) * (size_t)((n + 31) / 32), st));
    ph::chain(k_init_roots, (b.nbox + TB - 1) / TB, TB, 0, st, b, n, top);
    // a level has at most nbox 2^d nodes: the first levels are small enough for
    // single-block bookkeeping (7 launches a level instead of 19)
    bool pending = false;  // a small level whose k_level_finish is still to come
    // nodes of one level: the roots, or the children of the level above's
    // wide nodes (more than b.mid particles each, so at most N / b.mid)
    const long long lvl_bound = 2LL * (b.cap_n / b.mid) + 2LL * b.nbox + 2;
    const int lvl_max = lvl_bound < b.cap_nodes ? (int)lvl_bound : b.cap_nodes;
    for (int d = 0; d < top; d++) {
        const int D = (p.axis0 + d) % 3;  // from direct_local_start; the axis cycles (src/fmm.c:99)
        const bool small = d < 24 && ((long long)b.nbox << d) <= SMALL_LEVEL;
        if (small) {
            ph::chain(k_level_plan, 1, SMALL_TB, 0, st, b, pending ? d - 1 : -1, top);
        } else {
            if (pending) ph::chain(k_level_finish, 1, 1, 0, st, b, d - 1, top);
            ph::chain(k_level_nch, maxb, TB, 0, st, b);
            scan_exclusive_i32_bounded(b.tn_nch, b.tn_chunk_base, b.cnt + BC_LEVEL_COUNT, b.cap_nodes, lvl_max,
                                       b.cnt + BC_W, b.scan_scratch, b.scan_scratch_elems, st);
            ph::chain(k_chunk_map, maxb, TB, 0, st, b);
        }
        ph::chain(k_chunk_sum, maxb, TB, 0, st, b, D);
        ph::chain(k_node_mean, maxb, TB, 0, st, b, D);
        ph::chain(k_chunk_count, maxb, TB, 0, st, b, D);
        if (small) {
            ph::chain(k_level_close, 1, SMALL_TB, 0, st, b, p.maxleaf, D);
        } else {
            ph::chain(k_node_split, maxb, TB, 0, st, b, p.maxleaf);
            scan_exclusive_i32_bounded(b.tn_nodeflag, b.tn_nodebase, b.cnt + BC_LEVEL_COUNT, b.cap_nodes, lvl_max,
                                       b.cnt + BC_NEXT_NODES, b.scan_scratch, b.scan_scratch_elems, st);
            scan_exclusive_i32_bounded(b.tn_leafflag, b.tn_leafbase, b.cnt + BC_LEVEL_COUNT, b.cap_nodes, lvl_max,
                                       b.cnt + BC_NEW_LEAVES, b.scan_scratch, b.scan_scratch_elems, st);
            ph::chain(k_make_children, maxb, TB, 0, st, b, p.maxleaf, D);
        }
        ph::chain(k_rank, maxb, TB, 0, st, b, D);
        ph::chain(k_swap, maxb, TB, 0, st, b, D);
        if (small) {
            pending = true;
        } else {
            ph::chain(k_level_finish, 1, 1, 0, st, b, d, top);
            pending = false;
        }
    }
    if (pending) ph::chain(k_level_finish, 1, 1, 0, st, b, top - 1, top);
    if (b.mid > CHUNK)
        ph::chain(k_mid_build, device_sm_count(), MID_TB, sizeof(MidTree), st, b, p.axis0, p.maxleaf, levels);
    ph::chain(k_subtree_build, device_sm_count() * 4, SUB_TB, sizeof(SubTree), st, b, p.axis0, p.maxleaf,
                                                                                                levels);
    ph::chain(k_tree_totals, 1, 1, 0, st, b);
    ph::chain(k_mark_leaves, maxb, TB, 0, st, b);
    // starts before each word of 32 positions, then nodes and empty leaves before each start
    const int nwords = (n + 31) / 32;
    if (nwords <= ONE_SCAN_MAX) {
        ph::chain(k_scan_one<int>, 1, ONE_SCAN_TB, 0, st, b, b.cnt + BC_WORDS, b.wordpre);
    } else {
        ph::chain(k_scan_input<int>, maxb, TB, 0, st, b, b.cnt + BC_WORDS, b.bigpos);
        scan_exclusive_i32(b.bigpos, b.wordpre, b.cnt + BC_WORDS, nwords, b.cnt + BC_SCAN_TOTAL, b.scan_scratch,
                           b.scan_scratch_elems, st);
    }
    ph::chain(k_leaf_ranks, maxb, TB, 0, st, b);
    if (b.rule_cap <= ONE_SCAN_MAX) {
        ph::chain(k_scan_one<long long>, 1, ONE_SCAN_TB, 0, st, b, b.cnt + BC_STARTS, b.lf_base);
    } else {
        ph::chain(k_scan_input<long long>, maxb, TB, 0, st, b, b.cnt + BC_STARTS, b.lf_in);
        scan_exclusive_i64(b.lf_in, b.lf_base, b.cnt + BC_STARTS, b.rule_cap, nullptr, b.lf_scan, st);
    }
    ph::chain(k_scatter_tree, maxb, TB, 0, st, b, T);
    ph::chain(k_depth_count, nblk, 32, 0, st, b, T, ndepth);
    scan_exclusive_i32(T.depth_blk, T.depth_blk + (size_t)ndepth * nblk, b.cnt + BC_DEPTH_CELLS, ndepth * nblk,
                       b.cnt + BC_DEPTH_TOTAL, b.scan_scratch, b.scan_scratch_elems, st);
    ph::chain(k_depth_place, nblk, 32, 0, st, b, T, ndepth);
    PH_CUDA_CHECK(cudaGetLastError());
    return 0;
}

// host view of the finished build (after the stream has been synchronised)
int read_tree_info(const BuildBufs &b, const TreeBufs &T, int levels, TreeInfo &info)
{
    int h[BC_NCOUNTERS];
    PH_CUDA_CHECK(cudaMemcpy(h, b.cnt, sizeof(h), cudaMemcpyDeviceToHost));
    info.nleaf = h[BC_LEAVES];
    info.nnode = h[BC_NODES];
    info.depth = h[BC_DEPTH];
    info.levels = h[BC_NLEVELS];
    info.flags = h[BC_FLAGS];
    info.depth_off.resize(levels + 2);
    PH_CUDA_CHECK(cudaMemcpy(info.depth_off.data(), T.depth_off, sizeof(int) * (levels + 2), cudaMemcpyDeviceToHost));
    return 0;
}

}  // namespace ph
