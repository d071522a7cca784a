// GPU binned-SAH BVH builder: the same binary BVH (BVHNode layout, leaf order)
// as build_bvh2 in bvh_build.cpp, for a whole set of meshes at once (a forest:
// one tree per mesh, all in the same launches), built top down one tree level
// per round of kernels, and the meshes' device arrays.
//
// A task is an inner node to split: a range of positions in the primitive
// order array and its primitives' centroid bounds. Per level:
//   k_bin        every primitive of every task adds its box and centroid to
//                32 bins per axis of its task (shared-memory bins when a whole
//                block of positions belongs to one task, global atomics else)
//   k_split      one warp per task, one lane per bin: SAH over the 31
//                candidate planes per axis (surface area x count on both
//                sides), or the median when all centroids coincide
//   k_partition  every primitive moves to its side (per-task cursors)
//   k_emit       the task's node is written (both children's boxes and links);
//                children of more than 32 primitives become next-level tasks
// Ranges of at most 32 primitives are left to one launch at the end (k_small:
// a warp per range, a lane per primitive, every split of the sorted centroids
// tried), which also ends the levels early: binning 96 bins per task pays for
// hundreds of primitives, not for a few. The host only reads the task count
// per level. Positions inside a leaf keep the order the partition left them
// in, so the build is not deterministic across runs; traversal results do not
// depend on it (exact closest hit under the (t, instance, primitive) order).
//
// Bound by atomics and latency at the top levels (few tasks, all primitives in
// one) and by launches below. Building eight meshes of 124,820 triangles one
// after the other, a thread per split, took 60 ms; together, with the boxes
// and the packing on the device, the whole scene uploads in 7.4 ms instead
// of 107 (k_bin 1.7 ms in all, k_small 1.1).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "bvh_build.h"
#include "internal.h"

namespace vvpt {

namespace {

constexpr int kBins = 32;
constexpr int kSmall = 32; // ranges up to this size are finished by one warp

struct GBox {
    float lo[3], hi[3];
};

struct Task {
    int begin, end, node, depth;
    int mesh; // its root's node index; links are relative to it
    float cmin[3], cmax[3];
};

// A range for k_small: link and count go to node `parent`, child `side`; side
// -1: the range is a whole tree and `parent` its root.
struct SmallTask {
    int begin, n, parent, side, depth, mesh;
};

enum { kNodes = 0, kNextTasks = 1, kMaxDepth = 2, kSmallTasks = 3, kCounters = 4 };

// per task, axis, bin: count, box lo/hi, centroid lo/hi (float bits as
// order-preserving ints for atomic min/max)
struct BinStat {
    int count;
    int blo[3], bhi[3];
    int clo[3], chi[3];
};

struct Split {
    int axis, bin;       // left = bins [0, bin], right = (bin, 31]; axis -1: median split
    int nl;              // primitives on the left
    GBox lbox, rbox;     // children's boxes
    float lcmin[3], lcmax[3], rcmin[3], rcmax[3]; // children's centroid bounds
};

__device__ __forceinline__ int f2o(float f)
{
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float o2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }

__device__ __forceinline__ int bin_of(float c, float lo, float hi)
{
    const float ext = hi - lo;
    if (!(ext > 0.0f))
        return 0;
    const int b = (int)((c - lo) * ((float)kBins / ext));
    return min(max(b, 0), kBins - 1);
}

// Per mesh: bounds of the centroids, then of the boxes (lo, hi; ordered ints).
constexpr int kBoundInts = 12;
__global__ void k_clear_bounds(int *bounds, int meshes)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kBoundInts * meshes; i += gridDim.x * blockDim.x)
        bounds[i] = i % 6 < 3 ? f2o(FLT_MAX) : f2o(-FLT_MAX);
}

// The primitives of one mesh: boxes (of its triangles, or given), centroids,
// start order, the mesh's bounds.
__global__ void __launch_bounds__(256) k_primitives(const vvpt_vertex *verts, const uint32_t *tri, const GBox *given,
                                                    int n, int begin, int mesh, GBox *boxes, float4 *cent, int *idx,
                                                    int *side, int *bounds)
{
    __shared__ int sb[kBoundInts];
    if (threadIdx.x < kBoundInts)
        sb[threadIdx.x] = threadIdx.x % 6 < 3 ? f2o(FLT_MAX) : f2o(-FLT_MAX);
    __syncthreads();
    int mine[kBoundInts];
    for (int k = 0; k < kBoundInts; k++)
        mine[k] = k % 6 < 3 ? f2o(FLT_MAX) : f2o(-FLT_MAX);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        GBox b;
        if (given) {
            b = given[i];
        } else {
            for (int a = 0; a < 3; a++) {
                b.lo[a] = INFINITY;
                b.hi[a] = -INFINITY;
            }
            for (int c = 0; c < 3; c++) {
                const float *p = verts[tri[3 * (size_t)i + c]].position;
                for (int a = 0; a < 3; a++) { // a NaN coordinate leaves the box as it is
                    b.lo[a] = fminf(b.lo[a], p[a]);
                    b.hi[a] = fmaxf(b.hi[a], p[a]);
                }
            }
        }
        const float c[3] = {0.5f * (b.lo[0] + b.hi[0]), 0.5f * (b.lo[1] + b.hi[1]), 0.5f * (b.lo[2] + b.hi[2])};
        boxes[begin + i] = b;
        cent[begin + i] = make_float4(c[0], c[1], c[2], 0.0f);
        idx[begin + i] = begin + i;
        side[begin + i] = mesh;
        for (int a = 0; a < 3; a++) {
            if (c[a] == c[a]) {
                mine[a] = min(mine[a], f2o(c[a]));
                mine[3 + a] = max(mine[3 + a], f2o(c[a]));
            }
            mine[6 + a] = min(mine[6 + a], f2o(b.lo[a]));
            mine[9 + a] = max(mine[9 + a], f2o(b.hi[a]));
        }
    }
    for (int k = 0; k < kBoundInts; k++) {
        const int v = k % 6 < 3 ? __reduce_min_sync(0xFFFFFFFFu, mine[k]) : __reduce_max_sync(0xFFFFFFFFu, mine[k]);
        if ((threadIdx.x & 31u) == 0) {
            if (k % 6 < 3)
                atomicMin(&sb[k], v);
            else
                atomicMax(&sb[k], v);
        }
    }
    __syncthreads();
    if (threadIdx.x < kBoundInts) {
        if (threadIdx.x % 6 < 3)
            atomicMin(&bounds[kBoundInts * mesh + threadIdx.x], sb[threadIdx.x]);
        else
            atomicMax(&bounds[kBoundInts * mesh + threadIdx.x], sb[threadIdx.x]);
    }
}

// The root task of every mesh (node index = mesh index).
__global__ void k_roots(const int2 *ranges, int meshes, const int *bounds, Task *tasks, SmallTask *small, int *counters,
                        int *child_task)
{
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < meshes; m += gridDim.x * blockDim.x) {
        const int begin = ranges[m].x, n = ranges[m].y;
        child_task[m] = -1;
        if (n <= kSmall) {
            small[atomicAdd(&counters[kSmallTasks], 1)] = SmallTask{begin, n, m, -1, 0, m};
            continue;
        }
        Task t;
        t.begin = begin;
        t.end = begin + n;
        t.node = t.mesh = m;
        t.depth = 0;
        for (int j = 0; j < 3; j++) {
            t.cmin[j] = o2f(bounds[kBoundInts * m + j]);
            t.cmax[j] = o2f(bounds[kBoundInts * m + 3 + j]);
        }
        const int id = atomicAdd(&counters[kNextTasks], 1);
        tasks[id] = t;
        child_task[m] = id;
    }
}

__global__ void k_clear_bins(BinStat *bins, int nstats)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nstats; i += gridDim.x * blockDim.x) {
        BinStat &b = bins[i];
        b.count = 0;
        for (int a = 0; a < 3; a++) {
            b.blo[a] = b.clo[a] = f2o(FLT_MAX);
            b.bhi[a] = b.chi[a] = f2o(-FLT_MAX);
        }
    }
}

__device__ __forceinline__ void add_to_bin(BinStat &s, const GBox &b, const float4 &c)
{
    atomicAdd(&s.count, 1);
    const float cc[3] = {c.x, c.y, c.z};
    for (int a = 0; a < 3; a++) {
        atomicMin(&s.blo[a], f2o(b.lo[a]));
        atomicMax(&s.bhi[a], f2o(b.hi[a]));
        if (cc[a] == cc[a]) {
            atomicMin(&s.clo[a], f2o(cc[a]));
            atomicMax(&s.chi[a], f2o(cc[a]));
        }
    }
}

// Blocks of 256 positions; a block whose positions all belong to one task
// bins in shared memory and flushes once.
__global__ void __launch_bounds__(256) k_bin(const GBox *boxes, const float4 *cent, const int *idx, const int *task_of,
                                             int n, const Task *tasks, BinStat *bins)
{
    __shared__ BinStat sb[3 * kBins];
    __shared__ int first_task, uniform;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = p < n ? task_of[p] : -1;
    if (threadIdx.x == 0) {
        first_task = t;
        uniform = 1;
    }
    __syncthreads();
    if (t != first_task)
        uniform = 0;
    __syncthreads();
    const bool use_shared = uniform && first_task >= 0;
    if (use_shared) {
        for (int i = threadIdx.x; i < 3 * kBins; i += blockDim.x) {
            BinStat &b = sb[i];
            b.count = 0;
            for (int a = 0; a < 3; a++) {
                b.blo[a] = b.clo[a] = f2o(FLT_MAX);
                b.bhi[a] = b.chi[a] = f2o(-FLT_MAX);
            }
        }
        __syncthreads();
    }
    if (t >= 0) {
        const Task &T = tasks[t];
        const int prim = idx[p];
        const GBox b = boxes[prim];
        const float4 c = cent[prim];
        const float cc[3] = {c.x, c.y, c.z};
        for (int a = 0; a < 3; a++) {
            const int k = a * kBins + bin_of(cc[a], T.cmin[a], T.cmax[a]);
            add_to_bin(use_shared ? sb[k] : bins[(size_t)t * 3 * kBins + k], b, c);
        }
    }
    if (use_shared) {
        __syncthreads();
        for (int i = threadIdx.x; i < 3 * kBins; i += blockDim.x) {
            const BinStat &s = sb[i];
            if (s.count == 0)
                continue;
            BinStat &g = bins[(size_t)first_task * 3 * kBins + i];
            atomicAdd(&g.count, s.count);
            for (int a = 0; a < 3; a++) {
                atomicMin(&g.blo[a], s.blo[a]);
                atomicMax(&g.bhi[a], s.bhi[a]);
                atomicMin(&g.clo[a], s.clo[a]);
                atomicMax(&g.chi[a], s.chi[a]);
            }
        }
    }
}

__device__ __forceinline__ float half_area(const float lo[3], const float hi[3])
{
    const float dx = fmaxf(hi[0] - lo[0], 0.0f), dy = fmaxf(hi[1] - lo[1], 0.0f), dz = fmaxf(hi[2] - lo[2], 0.0f);
    return dx * dy + dy * dz + dz * dx;
}

// Inclusive min / max scans over the lanes, from the first lane up (UP) or
// from the last one down; `from` and `to` bound the lanes that take part.
template <bool UP>
__device__ __forceinline__ void scan_box(float (&lo)[3], float (&hi)[3], int from, int to)
{
    const int lane = (int)(threadIdx.x & 31u);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const bool ok = UP ? lane - d >= from : lane + d < to;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const float l = UP ? __shfl_up_sync(0xFFFFFFFFu, lo[j], d) : __shfl_down_sync(0xFFFFFFFFu, lo[j], d);
            const float h = UP ? __shfl_up_sync(0xFFFFFFFFu, hi[j], d) : __shfl_down_sync(0xFFFFFFFFu, hi[j], d);
            if (ok) {
                lo[j] = fminf(lo[j], l);
                hi[j] = fmaxf(hi[j], h);
            }
        }
    }
}

// Cost of the cut after this lane, the left box scanned up and the right one
// down: area x count on both sides.
__device__ __forceinline__ float cut_cost(const float (&llo)[3], const float (&lhi)[3], int lc, const float (&rlo)[3],
                                          const float (&rhi)[3], int rc)
{
    float nlo[3], nhi[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        nlo[j] = __shfl_down_sync(0xFFFFFFFFu, rlo[j], 1);
        nhi[j] = __shfl_down_sync(0xFFFFFFFFu, rhi[j], 1);
    }
    return half_area(llo, lhi) * (float)lc + half_area(nlo, nhi) * (float)rc;
}

__global__ void __launch_bounds__(256) k_split(const Task *tasks, int ntasks, const BinStat *bins, Split *splits)
{
    const int t = (int)((blockIdx.x * blockDim.x + threadIdx.x) / 32u), lane = (int)(threadIdx.x & 31u);
    if (t >= ntasks)
        return;
    const BinStat *B = bins + (size_t)t * 3 * kBins;
    const int total = tasks[t].end - tasks[t].begin;
    float best = INFINITY;
    int best_axis = -1, best_left = 0;
    for (int a = 0; a < 3; a++) {
        if (!(tasks[t].cmax[a] > tasks[t].cmin[a]))
            continue;
        const BinStat s = B[a * kBins + lane];
        float llo[3], lhi[3], rlo[3], rhi[3];
        for (int j = 0; j < 3; j++) {
            llo[j] = rlo[j] = o2f(s.blo[j]);
            lhi[j] = rhi[j] = o2f(s.bhi[j]);
        }
        int lc = s.count;
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xFFFFFFFFu, lc, d);
            lc += lane >= d ? o : 0;
        }
        scan_box<true>(llo, lhi, 0, 32);
        scan_box<false>(rlo, rhi, 0, 32);
        const float cost = cut_cost(llo, lhi, lc, rlo, rhi, total - lc);
        if (lc > 0 && lc < total && lane < kBins - 1 && cost < best) {
            best = cost;
            best_axis = a;
            best_left = lc;
        }
    }
    const int low = __reduce_min_sync(0xFFFFFFFFu, best_axis >= 0 ? f2o(best) : 0x7FFFFFFF);
    const uint32_t at = __ballot_sync(0xFFFFFFFFu, best_axis >= 0 && f2o(best) == low);
    const int from = at ? __ffs((int)at) - 1 : 0;
    Split S;
    S.axis = at ? __shfl_sync(0xFFFFFFFFu, best_axis, from) : -1;
    S.bin = from;
    S.nl = at ? __shfl_sync(0xFFFFFFFFu, best_left, from) : total / 2;
    // children's boxes and centroid bounds from the bins (for a median split
    // k_partition and k_emit fill them in)
    const BinStat s = B[(S.axis < 0 ? 0 : S.axis) * kBins + lane];
    for (int side = 0; side < 2; side++) {
        const bool in = S.axis >= 0 && s.count && (lane <= S.bin) == (side == 0);
        GBox &bx = side == 0 ? S.lbox : S.rbox;
        float *cl = side == 0 ? S.lcmin : S.rcmin, *ch = side == 0 ? S.lcmax : S.rcmax;
        for (int j = 0; j < 3; j++) {
            bx.lo[j] = o2f(__reduce_min_sync(0xFFFFFFFFu, in ? s.blo[j] : f2o(FLT_MAX)));
            bx.hi[j] = o2f(__reduce_max_sync(0xFFFFFFFFu, in ? s.bhi[j] : f2o(-FLT_MAX)));
            cl[j] = o2f(__reduce_min_sync(0xFFFFFFFFu, in ? s.clo[j] : f2o(FLT_MAX)));
            ch[j] = o2f(__reduce_max_sync(0xFFFFFFFFu, in ? s.chi[j] : f2o(-FLT_MAX)));
        }
    }
    if (lane == 0)
        splits[t] = S;
}

// Median splits (all centroids equal) keep the order: the first nl
// positions go left. Otherwise each primitive moves to its side.
__global__ void k_partition(const GBox *boxes, const float4 *cent, const int *idx_in, const int *task_of_in, int n,
                            const Task *tasks, const Split *splits, int *cursors, int *idx_out, int *side_out,
                            GBox *median_boxes)
{
    const uint32_t lane = threadIdx.x & 31u;
    for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const int p = base + (int)threadIdx.x;
        const int t = p < n ? task_of_in[p] : -1;
        const int prim = p < n ? idx_in[p] : 0;
        bool left = false;
        if (t >= 0) {
            const Task &T = tasks[t];
            const Split &S = splits[t];
            if (S.axis < 0) {
                left = p - T.begin < S.nl;
            } else {
                const float4 c = cent[prim];
                const float cc = S.axis == 0 ? c.x : (S.axis == 1 ? c.y : c.z);
                left = bin_of(cc, T.cmin[S.axis], T.cmax[S.axis]) <= S.bin;
            }
        }
        // one atomic per warp for the primitives of a task and side
        const int key = t >= 0 ? 2 * t + (left ? 0 : 1) : -1;
        const uint32_t same = __match_any_sync(0xFFFFFFFFu, key);
        const int leader = __ffs((int)same) - 1;
        int at = 0;
        if (key >= 0 && (int)lane == leader)
            at = atomicAdd(&cursors[key], __popc(same));
        at = __shfl_sync(0xFFFFFFFFu, at, leader) + __popc(same & ((1u << lane) - 1u));
        if (p >= n)
            continue;
        if (key < 0) {
            idx_out[p] = prim;
            side_out[p] = -1;
            continue;
        }
        const int dst = tasks[t].begin + (left ? 0 : splits[t].nl) + at;
        idx_out[dst] = prim;
        side_out[dst] = key;
        if (splits[t].axis < 0) {
            // median split: children boxes accumulated here
            const GBox b = boxes[prim];
            int *mi = reinterpret_cast<int *>(&median_boxes[key]);
            for (int j = 0; j < 3; j++) {
                atomicMin(&mi[j], f2o(b.lo[j]));
                atomicMax(&mi[3 + j], f2o(b.hi[j]));
            }
        }
    }
}

__global__ void k_clear_median(GBox *m, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int *mi = reinterpret_cast<int *>(&m[i]);
        for (int j = 0; j < 3; j++) {
            mi[j] = f2o(FLT_MAX);
            mi[3 + j] = f2o(-FLT_MAX);
        }
    }
}

// One thread per task: the node record, child tasks for children of more than
// kSmall primitives, entries for k_small for the others; child task ids go to
// child_task[2t + side].
__global__ void k_emit(const Task *tasks, int ntasks, Split *splits, const GBox *median_boxes, BVHNode *nodes,
                       int *counters, Task *next, SmallTask *small, int *child_task, int max_depth,
                       const int2 *ranges, uint8_t *last)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntasks)
        return;
    const Task &T = tasks[t];
    Split &S = splits[t];
    if (S.axis < 0) {
        // median: boxes from the partition's atomics; centroid bounds equal
        for (int side = 0; side < 2; side++) {
            const int *mi = reinterpret_cast<const int *>(&median_boxes[2 * t + side]);
            GBox &bx = side == 0 ? S.lbox : S.rbox;
            for (int j = 0; j < 3; j++) {
                bx.lo[j] = o2f(mi[j]);
                bx.hi[j] = o2f(mi[3 + j]);
            }
        }
        for (int j = 0; j < 3; j++) {
            S.lcmin[j] = S.rcmin[j] = T.cmin[j];
            S.lcmax[j] = S.rcmax[j] = T.cmax[j];
        }
    }
    int link[2] = {0, 0}, cnt[2] = {0, 0};
    for (int side = 0; side < 2; side++) {
        const int b = side == 0 ? T.begin : T.begin + S.nl;
        const int e = side == 0 ? T.begin + S.nl : T.end;
        const int n = e - b;
        child_task[2 * t + side] = -1;
        if (T.depth + 1 >= max_depth) {
            link[side] = b - ranges[T.mesh].x;
            cnt[side] = n;
            last[e - 1] = 1;
        } else if (n <= kSmall) {
            // link and count: k_small
            small[atomicAdd(&counters[kSmallTasks], 1)] = SmallTask{b, n, T.node, side, T.depth + 1, T.mesh};
        } else {
            const int node = atomicAdd(&counters[kNodes], 1);
            const int nt = atomicAdd(&counters[kNextTasks], 1);
            Task c;
            c.begin = b;
            c.end = e;
            c.node = node;
            c.mesh = T.mesh;
            c.depth = T.depth + 1;
            for (int j = 0; j < 3; j++) {
                c.cmin[j] = side == 0 ? S.lcmin[j] : S.rcmin[j];
                c.cmax[j] = side == 0 ? S.lcmax[j] : S.rcmax[j];
            }
            next[nt] = c;
            link[side] = node - T.mesh;
            child_task[2 * t + side] = nt;
        }
    }
    atomicMax(&counters[kMaxDepth], T.depth + 1);
    BVHNode nd;
    nd.lxy = make_float4(S.lbox.lo[0], S.lbox.lo[1], S.lbox.hi[0], S.lbox.hi[1]);
    nd.rxy = make_float4(S.rbox.lo[0], S.rbox.lo[1], S.rbox.hi[0], S.rbox.hi[1]);
    nd.lrz = make_float4(S.lbox.lo[2], S.lbox.hi[2], S.rbox.lo[2], S.rbox.hi[2]);
    nd.c = make_int4(link[0], link[1], cnt[0], cnt[1]);
    nodes[T.node] = nd;
}

// The rest of the tree over at most 32 primitives: a warp, one lane per
// primitive. Every cut of the centroids sorted along each axis is a candidate
// plane; a range of at most max_leaf primitives stays a leaf unless the SAH
// says a split is cheaper (traversal cost 1, intersection cost 1 per
// primitive), the host builder's rule.
constexpr int kSmallWarps = 4;
__global__ void __launch_bounds__(32 * kSmallWarps)
    k_small(const SmallTask *tasks, int ntasks, int *idx, const GBox *boxes, const float4 *cent, BVHNode *nodes,
            int *counters, int max_leaf, int max_depth, const int2 *ranges, uint8_t *last)
{
    struct Seg {
        int off, n, parent, side, depth;
    };
    __shared__ Seg segs[kSmallWarps][kSmall + 1];
    __shared__ int source[kSmallWarps][32];
    const uint32_t all = 0xFFFFFFFFu;
    const int lane = (int)(threadIdx.x & 31u), w = (int)(threadIdx.x >> 5);
    const int t = (int)(blockIdx.x * kSmallWarps) + w;
    if (t >= ntasks)
        return;
    const SmallTask T = tasks[t];
    const int mesh_begin = ranges[T.mesh].x;
    int prim = lane < T.n ? idx[T.begin + lane] : 0;
    GBox b = boxes[prim];
    float c[3];
    {
        const float4 c4 = cent[prim];
        c[0] = c4.x;
        c[1] = c4.y;
        c[2] = c4.z;
    }
    int sp = 0;
    if (lane == 0)
        segs[w][0] = Seg{0, T.n, T.parent, T.side, T.depth};
    sp = 1;
    __syncwarp();
    while (sp > 0) {
        const Seg g = segs[w][--sp];
        const int end = g.off + g.n;
        const bool in = lane >= g.off && lane < end;
        int node = -1; // this range's inner node, -1: a leaf
        int cut = g.n / 2, order = lane;
        if (g.side < 0 || g.n > max_leaf || g.n > 1) {
            float best = INFINITY, area = 0.0f;
            int best_k = 0;
            for (int a = 0; a < 3; a++) {
                int rank = 0;
                for (int k = g.off; k < end; k++) {
                    const float o = __shfl_sync(all, c[a], k);
                    rank += o < c[a] || (!(c[a] < o) && k < lane) ? 1 : 0;
                }
                // NaN centroids compare as equal to everything: keep a permutation
                const uint32_t seen = __reduce_or_sync(all, in && rank < g.n ? 1u << rank : 0u);
                if (seen != (g.n == 32 ? all : (1u << g.n) - 1u))
                    rank = lane - g.off;
                if (in)
                    source[w][g.off + rank] = lane;
                __syncwarp();
                const int from = in ? source[w][lane] : lane;
                __syncwarp();
                float llo[3], lhi[3], rlo[3], rhi[3];
                for (int j = 0; j < 3; j++) {
                    llo[j] = rlo[j] = __shfl_sync(all, b.lo[j], from);
                    lhi[j] = rhi[j] = __shfl_sync(all, b.hi[j], from);
                }
                scan_box<true>(llo, lhi, g.off, end);
                scan_box<false>(rlo, rhi, g.off, end);
                const int k = lane - g.off + 1;
                const float cost = cut_cost(llo, lhi, k, rlo, rhi, g.n - k);
                area = half_area(llo, lhi); // of the whole range on its last lane
                const bool ok = in && k < g.n && cost < INFINITY;
                const int low = __reduce_min_sync(all, ok ? f2o(cost) : 0x7FFFFFFF);
                const uint32_t at = __ballot_sync(all, ok && f2o(cost) == low);
                if (at && o2f(low) < best) {
                    best = o2f(low);
                    best_k = __ffs((int)at) - g.off;
                    order = from;
                }
            }
            area = __shfl_sync(all, area, end - 1);
            if (best_k > 0)
                cut = best_k;
            const float split_cost = 1.0f + (area > 0.0f ? best / area : (float)g.n);
            const bool leaf = g.side >= 0 && (g.depth >= max_depth ||
                                              (g.n <= max_leaf && (best_k == 0 || (float)g.n <= split_cost)));
            if (!leaf) {
                if (g.side < 0) {
                    node = g.parent; // the root's node is given
                } else {
                    if (lane == 0)
                        node = atomicAdd(&counters[kNodes], 1);
                    node = __shfl_sync(all, node, 0);
                }
            }
        }
        if (g.side >= 0 && lane == 0) {
            int *link = reinterpret_cast<int *>(&nodes[g.parent].c);
            link[g.side] = node >= 0 ? node - T.mesh : T.begin + g.off - mesh_begin;
            link[2 + g.side] = node >= 0 ? 0 : g.n;
        }
        if (node < 0) {
            if (lane == 0)
                last[T.begin + end - 1] = 1;
            continue;
        }
        // the range in the order of the best axis, its children's boxes
        prim = __shfl_sync(all, prim, order);
        for (int j = 0; j < 3; j++) {
            b.lo[j] = __shfl_sync(all, b.lo[j], order);
            b.hi[j] = __shfl_sync(all, b.hi[j], order);
            c[j] = __shfl_sync(all, c[j], order);
        }
        float box[2][6];
        for (int side = 0; side < 2; side++) {
            const bool mine = in && (lane < g.off + cut) == (side == 0);
            for (int j = 0; j < 3; j++) {
                box[side][j] = o2f(__reduce_min_sync(all, mine ? f2o(b.lo[j]) : f2o(FLT_MAX)));
                box[side][3 + j] = o2f(__reduce_max_sync(all, mine ? f2o(b.hi[j]) : f2o(-FLT_MAX)));
            }
        }
        if (lane == 0) {
            BVHNode &nd = nodes[node];
            nd.lxy = make_float4(box[0][0], box[0][1], box[0][3], box[0][4]);
            nd.rxy = make_float4(box[1][0], box[1][1], box[1][3], box[1][4]);
            nd.lrz = make_float4(box[0][2], box[0][5], box[1][2], box[1][5]);
            segs[w][sp] = Seg{g.off, cut, node, 0, g.depth + 1};
            segs[w][sp + 1] = Seg{g.off + cut, g.n - cut, node, 1, g.depth + 1};
            atomicMax(&counters[kMaxDepth], g.depth + 1);
        }
        sp += 2;
        __syncwarp();
    }
    if (lane < T.n)
        idx[T.begin + lane] = prim;
}

// positions of child tasks get their new task id; leaf positions -1
__global__ void k_retask(const int *side_in, const int *child_task, int n, int *task_of_out)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const int s = side_in[p];
        task_of_out[p] = s < 0 ? -1 : child_task[s];
    }
}

// One mesh's triangles in leaf order.
__global__ void k_gather(const vvpt_vertex *verts, const uint32_t *tri, const int *idx, const uint8_t *last, int n,
                         int begin, TriVerts *out)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int prim = idx[begin + k] - begin;
        float4 v[3];
        for (int c = 0; c < 3; c++) {
            const float *p = verts[tri[3 * (size_t)prim + c]].position;
            v[c] = make_float4(p[0], p[1], p[2], 0.0f);
        }
        v[0].w = __int_as_float(prim);
        v[2].w = __int_as_float((int)last[begin + k]);
        out[begin + k] = TriVerts{v[0], v[1], v[2]};
    }
}

__global__ void k_shade_verts(const vvpt_vertex *verts, size_t n, ShadeVertex *out)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const vvpt_vertex &x = verts[i];
        ShadeVertex v;
        v.pos_u = make_float4(x.position[0], x.position[1], x.position[2], x.uv[0]);
        v.nrm_v = make_float4(x.normal[0], x.normal[1], x.normal[2], x.uv[1]);
        v.tan_ = make_float4(x.tangent[0], x.tangent[1], x.tangent[2], 0.0f);
        out[i] = v;
    }
}

int grid_of(long n) { return (int)std::max<long>(1, std::min<long>((n + 255) / 256, 152L * 32)); }

bool ck(std::string &err, cudaError_t e, const char *what)
{
    if (e == cudaSuccess)
        return true;
    cudaGetLastError();
    err = std::string("GPU BVH build: ") + what + ": " + cudaGetErrorString(e);
    return false;
}

// The device arrays of a forest build, carved from one allocation.
struct Forest {
    int n = 0, meshes = 0, cap = 0; // primitives, trees, tasks of a level
    DevBuf mem;
    GBox *boxes = nullptr, *median = nullptr;
    float4 *cent = nullptr;
    int *idx[2] = {}, *task_of[2] = {}, *side = nullptr, *cursors = nullptr, *child = nullptr, *counters = nullptr;
    int *bounds = nullptr;
    int2 *ranges = nullptr;
    uint8_t *last = nullptr;
    BVHNode *nodes = nullptr;
    Task *tasks[2] = {};
    SmallTask *small = nullptr;
    BinStat *bins = nullptr;
    Split *splits = nullptr;
    std::vector<int2> ranges_h;
    int counters_h[kCounters] = {};

    size_t carve(char *base)
    {
        size_t off = 0;
        auto take = [&](auto *&p, size_t count) {
            p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + off);
            off += aligned256(count * sizeof(*p));
        };
        take(boxes, n);
        take(cent, n);
        for (int k = 0; k < 2; k++) {
            take(idx[k], n);
            take(task_of[k], n);
            take(tasks[k], cap);
        }
        take(side, n);
        take(last, n);
        take(nodes, (size_t)n + meshes); // a tree whose leaves hold >= 1 primitive has < n inner nodes
        take(small, (size_t)n + meshes);
        take(bins, (size_t)3 * kBins * cap);
        take(splits, cap);
        take(cursors, (size_t)2 * cap);
        take(child, std::max<size_t>((size_t)2 * cap, meshes));
        take(median, (size_t)2 * cap);
        take(bounds, (size_t)kBoundInts * meshes);
        take(ranges, meshes);
        take(counters, kCounters);
        return off;
    }

    cudaError_t alloc(const std::vector<int> &counts)
    {
        n = 0;
        meshes = (int)counts.size();
        ranges_h.clear();
        for (int c : counts) {
            ranges_h.push_back(make_int2(n, c));
            n += c;
        }
        cap = n / (kSmall + 1) + 1; // a task has more than kSmall primitives
        const cudaError_t e = mem.alloc(carve(nullptr));
        if (e == cudaSuccess)
            carve(mem.as<char>());
        return e;
    }

    bool begin(cudaStream_t s, std::string &err)
    {
        const int start[kCounters] = {meshes, 0, 0, 0};
        if (!ck(err, cudaMemcpyAsync(ranges, ranges_h.data(), sizeof(int2) * meshes, cudaMemcpyHostToDevice, s),
                "upload") ||
            !ck(err, cudaMemcpyAsync(counters, start, sizeof(start), cudaMemcpyHostToDevice, s), "upload") ||
            !ck(err, cudaMemsetAsync(last, 0, n, s), "clear"))
            return false;
        k_clear_bounds<<<grid_of((long)kBoundInts * meshes), 256, 0, s>>>(bounds, meshes);
        return true;
    }

    void add(int mesh, const vvpt_vertex *verts, const uint32_t *tri, const GBox *given, cudaStream_t s)
    {
        const int2 r = ranges_h[mesh];
        k_primitives<<<std::min(grid_of(r.y), 304), 256, 0, s>>>(verts, tri, given, r.y, r.x, mesh, boxes, cent, idx[0],
                                                                 side, bounds);
    }

    // Builds every tree: nodes (roots first), idx[0] the leaf order.
    bool build(int max_leaf, int max_depth, cudaStream_t s, std::string &err)
    {
        auto counters_back = [&] {
            return ck(err, cudaGetLastError(), "launch") &&
                   ck(err, cudaMemcpyAsync(counters_h, counters, sizeof(counters_h), cudaMemcpyDeviceToHost, s),
                      "download") &&
                   ck(err, cudaStreamSynchronize(s), "sync");
        };
        k_roots<<<grid_of(meshes), 256, 0, s>>>(ranges, meshes, bounds, tasks[0], small, counters, child);
        k_retask<<<grid_of(n), 256, 0, s>>>(side, child, n, task_of[0]);
        if (!counters_back())
            return false;
        int ntasks = counters_h[kNextTasks];
        for (int level = 0, cur = 0; ntasks > 0; level++, cur ^= 1) {
            if (level > max_depth + 1) {
                err = "GPU BVH build: depth bound exceeded";
                return false;
            }
            k_clear_bins<<<grid_of(3L * kBins * ntasks), 256, 0, s>>>(bins, 3 * kBins * ntasks);
            k_bin<<<(n + 255) / 256, 256, 0, s>>>(boxes, cent, idx[0], task_of[0], n, tasks[cur], bins);
            k_split<<<(ntasks + 7) / 8, 256, 0, s>>>(tasks[cur], ntasks, bins, splits);
            cudaMemsetAsync(cursors, 0, 8ull * ntasks, s);
            k_clear_median<<<grid_of(2L * ntasks), 256, 0, s>>>(median, 2 * ntasks);
            k_partition<<<grid_of(n), 256, 0, s>>>(boxes, cent, idx[0], task_of[0], n, tasks[cur], splits, cursors,
                                                   idx[1], side, median);
            cudaMemsetAsync(counters + kNextTasks, 0, 4, s);
            k_emit<<<(ntasks + 127) / 128, 128, 0, s>>>(tasks[cur], ntasks, splits, median, nodes, counters,
                                                        tasks[cur ^ 1], small, child, max_depth, ranges, last);
            k_retask<<<grid_of(n), 256, 0, s>>>(side, child, n, task_of[1]);
            std::swap(idx[0], idx[1]);
            std::swap(task_of[0], task_of[1]);
            if (!counters_back())
                return false;
            ntasks = counters_h[kNextTasks];
        }
        const int ns = counters_h[kSmallTasks];
        if (ns > 0)
            k_small<<<(ns + kSmallWarps - 1) / kSmallWarps, 32 * kSmallWarps, 0, s>>>(
                small, ns, idx[0], boxes, cent, nodes, counters, max_leaf, max_depth, ranges, last);
        if (!counters_back())
            return false;
        if (counters_h[kNodes] > n + meshes) {
            err = "GPU BVH build: node bound exceeded";
            return false;
        }
        return true;
    }
};

}  // namespace

bool build_bvh2_gpu(const std::vector<Box3> &boxes, const BVHBuildOptions &opt, cudaStream_t s, BVHBuildResult &out,
                    std::string &err)
{
    const int n = (int)boxes.size();
    if (n <= opt.max_leaf)
        return false; // the host builder handles trivial trees
    static_assert(sizeof(GBox) == sizeof(Box3), "box layout");
    Forest f;
    DevBuf given;
    if (!ck(err, f.alloc({n}), "alloc") || !f.begin(s, err) || !ck(err, given.alloc(sizeof(GBox) * n), "alloc") ||
        !ck(err, cudaMemcpyAsync(given.ptr, boxes.data(), sizeof(GBox) * n, cudaMemcpyHostToDevice, s), "upload"))
        return false;
    f.add(0, nullptr, nullptr, given.as<GBox>(), s);
    if (!f.build(opt.max_leaf, opt.max_depth, s, err))
        return false;
    const int nnodes = f.counters_h[kNodes];
    out.nodes.resize(nnodes);
    out.order.resize(n);
    out.depth = f.counters_h[kMaxDepth];
    return ck(err, cudaMemcpyAsync(out.nodes.data(), f.nodes, sizeof(BVHNode) * nnodes, cudaMemcpyDeviceToHost, s),
              "download") &&
           ck(err, cudaMemcpyAsync(out.order.data(), f.idx[0], 4ull * n, cudaMemcpyDeviceToHost, s), "download") &&
           ck(err, cudaStreamSynchronize(s), "sync");
}

// The device part of a scene, in the scene's own arrays. Meshes are taken in
// groups of at most VVPT_GROUP_TRIANGLES triangles (or one mesh): the working
// memory, about 310 bytes a triangle beside the group's vertices as they were
// given, is a group's and not the scene's. Only the nodes, whose number a build
// finds out, are there twice at the end.
#ifndef VVPT_GROUP_TRIANGLES
#define VVPT_GROUP_TRIANGLES (16u << 20)
#endif
bool build_meshes_gpu(const vvpt_scene_desc *desc, const std::vector<uint32_t> &meshes, const BVHBuildOptions &opt,
                      cudaStream_t s, DeviceMeshes &out, std::string &err)
{
    out.placed.assign(meshes.size(), DeviceMeshes::Placed{});
    uint64_t nt = 0, nv = 0;
    for (size_t k = 0; k < meshes.size(); k++) {
        const vvpt_mesh_desc &md = desc->meshes[meshes[k]];
        out.placed[k].tri_offset = (uint32_t)nt;
        out.placed[k].vertex_offset = (uint32_t)nv;
        nt += md.num_triangles;
        nv += md.num_vertices;
    }
    out.num_tris = (uint32_t)nt;
    out.num_verts = (uint32_t)nv;
    auto room = [&](cudaError_t e) {
        out.no_room |= e == cudaErrorMemoryAllocation;
        return ck(err, e, "alloc");
    };
    if (!room(out.tris.alloc(sizeof(TriVerts) * (nt + out.host_tris))) ||
        !room(out.verts.alloc(sizeof(ShadeVertex) * (nv + out.host_verts))) ||
        !room(out.indices.alloc(12ull * (nt + out.host_index_tris))))
        return false;
    for (size_t first = 0; first < meshes.size();) {
        size_t end = first;
        std::vector<int> counts;
        uint64_t tris = 0, verts = 0;
        while (end < meshes.size()) {
            const vvpt_mesh_desc &md = desc->meshes[meshes[end]];
            if (end > first && tris + md.num_triangles > VVPT_GROUP_TRIANGLES)
                break;
            tris += md.num_triangles;
            verts += md.num_vertices;
            counts.push_back((int)md.num_triangles);
            end++;
        }
        Forest f;
        DevBuf raw;
        if (!room(f.alloc(counts)) || !room(raw.alloc(sizeof(vvpt_vertex) * verts)) || !f.begin(s, err))
            return false;
        vvpt_vertex *rv = raw.as<vvpt_vertex>();
        const uint32_t t0 = out.placed[first].tri_offset, v0 = out.placed[first].vertex_offset;
        auto mesh_verts = [&](size_t k) { return rv + (out.placed[k].vertex_offset - v0); };
        auto mesh_tris = [&](size_t k) { return out.indices.as<uint32_t>() + 3ull * out.placed[k].tri_offset; };
        for (size_t k = first; k < end; k++) {
            const vvpt_mesh_desc &md = desc->meshes[meshes[k]];
            if (!ck(err, cudaMemcpyAsync(mesh_verts(k), md.vertices, sizeof(vvpt_vertex) * (size_t)md.num_vertices,
                                         cudaMemcpyHostToDevice, s), "upload") ||
                !ck(err, cudaMemcpyAsync(mesh_tris(k), md.indices, 12ull * md.num_triangles, cudaMemcpyHostToDevice, s),
                    "upload"))
                return false;
            f.add((int)(k - first), mesh_verts(k), mesh_tris(k), nullptr, s);
        }
        k_shade_verts<<<grid_of((long)verts), 256, 0, s>>>(rv, verts, out.verts.as<ShadeVertex>() + v0);
        if (!f.build(opt.max_leaf, opt.max_depth, s, err))
            return false;
        for (size_t k = first; k < end; k++) {
            const int2 r = f.ranges_h[k - first];
            k_gather<<<grid_of(r.y), 256, 0, s>>>(mesh_verts(k), mesh_tris(k), f.idx[0], f.last, r.y, r.x,
                                                  out.tris.as<TriVerts>() + t0);
        }
        const int nnodes = f.counters_h[kNodes];
        out.nodes.emplace_back(new DevBuf());
        DevBuf &nb = *out.nodes.back();
        std::vector<int> bounds((size_t)kBoundInts * f.meshes);
        if (!room(nb.alloc(sizeof(BVHNode) * (size_t)nnodes)) ||
            !ck(err, cudaMemcpyAsync(nb.ptr, f.nodes, sizeof(BVHNode) * (size_t)nnodes, cudaMemcpyDeviceToDevice, s),
                "copy") ||
            !ck(err, cudaMemcpyAsync(bounds.data(), f.bounds, 4 * bounds.size(), cudaMemcpyDeviceToHost, s), "download") ||
            !ck(err, cudaStreamSynchronize(s), "sync"))
            return false;
        auto back = [](int i) {
            const int b = i >= 0 ? i : i ^ 0x7FFFFFFF;
            float x;
            std::memcpy(&x, &b, 4);
            return x;
        };
        for (size_t k = first; k < end; k++) {
            DeviceMeshes::Placed &p = out.placed[k];
            p.node_offset = out.num_nodes + (uint32_t)(k - first);
            for (int a = 0; a < 3; a++) {
                p.root.lo[a] = back(bounds[kBoundInts * (k - first) + 6 + a]);
                p.root.hi[a] = back(bounds[kBoundInts * (k - first) + 9 + a]);
            }
        }
        out.num_nodes += (uint32_t)nnodes;
        out.depth = std::max(out.depth, f.counters_h[kMaxDepth]);
        first = end;
    }
    return true;
}

}  // namespace vvpt
