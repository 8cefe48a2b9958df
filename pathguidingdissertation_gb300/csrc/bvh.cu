// GPU binned-SAH BVH build (BVHNode::build, Geometry.h:419-446) and the
// conversion of any tree in the reference layout into the traversal layout.
//
// The build reproduces the reference's decisions exactly: centroids with
// the 0.3333f factor (Geometry.h:96-98), 16 bins over the centroid bounds
// of each axis, the left/right sweep and cost 1 + A_L/A_P*N_L*1.5 +
// A_R/A_P*N_R*1.5 against N*1.5 (Geometry.h:293-365), the partition test
// centroid[axis] < split position and the failed-split rule
// (Geometry.h:384-395), leaves at <= 4 triangles.  All of these are
// order-independent (counts, min/max, comparisons) and computed with
// unfused float ops, so every node owns the same triangle set as in the
// reference; only node numbering and the order of triangles inside a leaf
// differ (the reference partitions in place by swapping).
//
// Phase A (nodes with more than kSmall triangles) runs level by level with two
// launches a level and no host round trip: CTAs take 1024-triangle chunks of
// the active nodes.  k_bin bins a chunk in shared memory, and the block that
// finishes a node's last chunk sweeps the SAH; k_partition splits the chunks
// of such a node into the other record buffer and reduces the children's
// boxes, and the node's last block creates its children.  A node of one chunk
// is split by k_bin itself.  A triangle travels as one 48-byte
// record (box, centroid, id), so every pass reads and writes runs.  Phase B
// gives each node of at most kSmall triangles to one warp, which finishes its
// subtree in shared memory.
#include <algorithm>
#include <chrono>
#include <cstddef>
#include <vector>

#include "pgx_ctx.h"
#include "pgx_trace.cuh"

namespace {

constexpr int kBins = 16;          // BUILD_BINS, Geometry.h:20
constexpr int kMaxLeaf = 4;        // MAXNODE_TRIANGLES, Geometry.h:17
constexpr int kSmall = 128;        // phase-B threshold
constexpr int kThreads = 256;
// Triangles per CTA chunk in phase A (2,093,058 triangles, whole build: 3.99 ms
// with 512, 3.48 with 1024, 3.50 with 2048, 4.04 with 4096: smaller ones merge
// more bins, larger ones leave a nearly empty last wave).
constexpr int kChunk = 1024;
constexpr int kPerThread = kChunk / kThreads;
constexpr int kBinInts = 3 * kBins * 7;
// Bins of a node: count, box minimum and maximum, each for all (axis, bin).
constexpr int kField = 3 * kBins;
// Neighbouring triangles fall into the same bins, and updates of one bin by
// one warp take turns, so neighbouring lanes use copies of their own, which
// are merged before the sweep (2,093,058 triangles: k_bin 1213 us with one
// copy, 3.40 / 3.22 / 3.15 / 3.14 / 3.21 ms of build with 1 / 2 / 4 / 8 / 16
// copies; phase B 3.15 / 3.10 / 3.22 with 1 / 2 / 3, where more shared memory
// costs warps).
constexpr int kBinCopies = 4, kSmallCopies = 2;
// (copies 8 banks apart: 2.91 ms; in the same banks 3.29, 16 apart 2.96)
constexpr int kCopyInts = kBinInts + 8;
constexpr int kMaxLevels = 200;

struct BuildItem {
    int node;
    int start, count;
    int slot;              // global bins of a node of more than one chunk
    int cmin[3], cmax[3];  // centroid bounds, ordered-int encoded
    int axis;
    float pos;
    int split;
    int lcur, rcur;
    unsigned done;         // chunks of the running pass that have finished
    int acc[2][12];  // per side: tbox min[3], tbox max[3], cent min[3], cent max[3] (ordered ints)
};

struct BuildMisc {
    unsigned long long counts;  // nodes in the low word, interior records in the high word
    int nsmall;
    int overflow;
    int root_acc[12];
    int nitems[kMaxLevels + 1];
    int nchunks[kMaxLevels + 1];
    int nslots[kMaxLevels + 1];
};

// A triangle on its way through the build: vertex bounds, centroid, id.
struct RecView {
    float4* lo;  // w = triangle id bits
    float4* hi;
    float4* cent;
};

// Work for phase B: node, and which record buffer holds its triangles; a
// leaf of one chunk only has its triangle ids copied.
constexpr int kSmallBuf = 1, kSmallLeaf = 2;

__device__ __forceinline__ float area_x(float mnx, float mny, float mnz, float mxx, float mxy, float mxz) {
    // AABB::area, Geometry.h:212-215
    float sx = x_sub(mxx, mnx), sy = x_sub(mxy, mny), sz = x_sub(mxz, mnz);
    return x_mul(x_add(x_add(x_mul(sx, sy), x_mul(sy, sz)), x_mul(sx, sz)), 2.f);
}

// Box, centroid (Triangle::centre) and id of every triangle, and the root's
// bounds (one set of 12 atomics per block).
__global__ void __launch_bounds__(kThreads) k_prep(const pgx_triangle* __restrict__ tris, int64_t n, RecView out,
                                                   BuildMisc* misc) {
    grid_begin();
    __shared__ int s_acc[12];
    if (threadIdx.x < 12) s_acc[threadIdx.x] = ((threadIdx.x % 6) < 3) ? INT_MAX : INT_MIN;
    __syncthreads();
    int acc[12];
#pragma unroll
    for (int k = 0; k < 12; k++) acc[k] = ((k % 6) < 3) ? INT_MAX : INT_MIN;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const pgx_triangle& t = tris[i];
        xv3 p0 = mk(t.v[0].p[0], t.v[0].p[1], t.v[0].p[2]);
        xv3 p1 = mk(t.v[1].p[0], t.v[1].p[1], t.v[1].p[2]);
        xv3 p2 = mk(t.v[2].p[0], t.v[2].p[1], t.v[2].p[2]);
        xv3 c = x_scale(x_add(x_add(p0, p1), p2), 0.3333f);
        const float v[9] = {s_min(s_min(p0.x, p1.x), p2.x), s_min(s_min(p0.y, p1.y), p2.y),
                            s_min(s_min(p0.z, p1.z), p2.z), s_max(s_max(p0.x, p1.x), p2.x),
                            s_max(s_max(p0.y, p1.y), p2.y), s_max(s_max(p0.z, p1.z), p2.z), c.x, c.y, c.z};
        out.lo[i] = make_float4(v[0], v[1], v[2], __int_as_float((int)i));
        out.hi[i] = make_float4(v[3], v[4], v[5], 0.f);
        out.cent[i] = make_float4(c.x, c.y, c.z, 0.f);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            acc[k] = min(acc[k], f2o(v[k]));
            acc[3 + k] = max(acc[3 + k], f2o(v[3 + k]));
            acc[6 + k] = min(acc[6 + k], f2o(v[6 + k]));
            acc[9 + k] = max(acc[9 + k], f2o(v[6 + k]));
        }
    }
#pragma unroll
    for (int k = 0; k < 12; k++) {
        const bool is_min = (k % 6) < 3;
        const int v = is_min ? __reduce_min_sync(0xFFFFFFFFu, acc[k]) : __reduce_max_sync(0xFFFFFFFFu, acc[k]);
        if ((threadIdx.x & 31) == 0) {
            if (is_min)
                atomicMin(&s_acc[k], v);
            else
                atomicMax(&s_acc[k], v);
        }
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        if ((threadIdx.x % 6) < 3)
            atomicMin(&misc->root_acc[threadIdx.x], s_acc[threadIdx.x]);
        else
            atomicMax(&misc->root_acc[threadIdx.x], s_acc[threadIdx.x]);
    }
}

// Fills an item and its chunk list; called by one thread.
__device__ __forceinline__ void add_item(BuildItem* items, int2* chunks, BuildMisc* misc, int level, int item_cap,
                                         int chunk_cap, int slot_cap, int node, int start, int count, const int* cmin,
                                         const int* cmax) {
    const int q = atomicAdd(&misc->nitems[level], 1);
    const int nch = (count + kChunk - 1) / kChunk;
    const int base = atomicAdd(&misc->nchunks[level], nch);
    const int slot = nch > 1 ? atomicAdd(&misc->nslots[level], 1) : 0;
    if (q >= item_cap || base + nch > chunk_cap || slot >= slot_cap) {
        atomicExch(&misc->overflow, 1);
        return;
    }
    BuildItem& it = items[q];
    it.node = node;
    it.start = start;
    it.count = count;
    it.slot = slot;
    for (int k = 0; k < 3; k++) {
        it.cmin[k] = cmin[k];
        it.cmax[k] = cmax[k];
    }
    it.split = 0;
    it.lcur = it.rcur = 0;
    it.done = 0;
    for (int s = 0; s < 2; s++)
        for (int k = 0; k < 12; k++) it.acc[s][k] = ((k % 6) < 3) ? INT_MAX : INT_MIN;
    for (int c = 0; c < nch; c++) chunks[base + c] = make_int2(q, c * kChunk);
}

__device__ __forceinline__ void add_small(int2* small, int small_cap, BuildMisc* misc, int node, int flags) {
    const int s = atomicAdd(&misc->nsmall, 1);
    if (s < small_cap)
        small[s] = make_int2(node, flags);
    else
        atomicExch(&misc->overflow, 1);
}

__global__ void k_root_init(pgx_bvh_node* nodes, int* node_rec, BuildItem* items, int2* chunks, int2* small,
                            BuildMisc* misc, int64_t n, int item_cap, int chunk_cap, int slot_cap, int small_cap) {
    grid_begin();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    pgx_bvh_node& r = nodes[0];
    for (int k = 0; k < 3; k++) {
        r.bmin[k] = o2f(misc->root_acc[k]);
        r.bmax[k] = o2f(misc->root_acc[3 + k]);
    }
    r.left_first = 0;
    r.used = (int)n;
    node_rec[0] = -1;
    misc->counts = 1;
    if (n <= kSmall)
        add_small(small, small_cap, misc, 0, 0);
    else
        add_item(items, chunks, misc, 0, item_cap, chunk_cap, slot_cap, 0, 0, (int)n, misc->root_acc + 6,
                 misc->root_acc + 9);
}

__device__ __forceinline__ void reset_bins(int* b, int i) {
    b[i] = i < kField ? 0 : (i < 4 * kField ? INT_MAX : INT_MIN);
}

__global__ void k_bins_reset(int* bins, int64_t n) {
    grid_begin();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const int f = (int)(i % kBinInts) / kField;
        bins[i] = (f == 0) ? 0 : (f < 4 ? INT_MAX : INT_MIN);
    }
}

// Adds one triangle's box to its bin of one axis (findBestSplitPlane's
// binning loop, Geometry.h:313-323).  Neighbouring triangles usually share a
// bin; a warp whose lanes all do reduces first and updates the bin once,
// instead of 32 conflicting updates of each of its 7 fields.  Whole warps;
// bi < 0: no triangle.
__device__ __forceinline__ void bin_add(int* bins, int ax, int bi, const int* lo, const int* hi) {
    int same;
    __match_all_sync(0xFFFFFFFFu, bi, &same);
    if (same) {
        if (bi < 0) return;
        int* bn = bins + ax * kBins + bi;
        int v[6];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            v[k] = __reduce_min_sync(0xFFFFFFFFu, lo[k]);
            v[3 + k] = __reduce_max_sync(0xFFFFFFFFu, hi[k]);
        }
        const int lane = threadIdx.x & 31;
        if (lane == 0) {
            atomicAdd(bn, 32);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                atomicMin(bn + (1 + k) * kField, v[k]);
                atomicMax(bn + (4 + k) * kField, v[3 + k]);
            }
        }
    } else if (bi >= 0) {
        int* bn = bins + ax * kBins + bi;
        atomicAdd(bn, 1);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            atomicMin(bn + (1 + k) * kField, lo[k]);
            atomicMax(bn + (4 + k) * kField, hi[k]);
        }
    }
}

__device__ __forceinline__ int bin_of(float c, float lo, float scale) {
    const int bi = (int)x_mul(x_sub(c, lo), scale);
    return (bi < kBins - 1) ? bi : kBins - 1;
}

// Sweep of findBestSplitPlane (Geometry.h:325-362) by one warp, an axis at a
// time: lanes 0-15 scan the bins upwards (the left sides), lanes 16-31
// downwards (the right sides), each lane works out its side's cost term, and
// one exchange per axis brings the terms of a plane together.  The smallest
// cost wins, the first one in the reference's order (axis, then plane) on
// ties.  Returns the axis (-1: none) with its plane and cost.  Minima and
// maxima commute, so the result is the sequential sweep's.
//   Shuffles bound it (one a cycle and SM): 87 a node.  Both scans in every
// lane, two axes at once, took 126 and two more divisions.
template <int COPIES>
__device__ __forceinline__ int warp_sweep(const int* bins, const float* lo, const float* hi, float parent_area,
                                          float& best, float& pos) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, i = lane & 15;
    const int b = lane < 16 ? i : 15 - i;
    float cost[3];
    int key[3];
#pragma unroll
    for (int ax = 0; ax < 3; ax++) {
        cost[ax] = FLT_MAX;
        key[ax] = INT_MAX;
        if (lo[ax] == hi[ax]) continue;  // uniform
        const int* bn = bins + ax * kBins + b;
        int c = bn[0], m[6];
#pragma unroll
        for (int k = 0; k < 6; k++) m[k] = bn[(1 + k) * kField];
#pragma unroll
        for (int v = 1; v < COPIES; v++) {
            const int* o = bn + v * kCopyInts;
            c += o[0];
#pragma unroll
            for (int k = 0; k < 6; k++) m[k] = k < 3 ? min(m[k], o[(1 + k) * kField]) : max(m[k], o[(1 + k) * kField]);
        }
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            // (a lane without a source gets its own value: no change to a minimum)
            const int t = __shfl_up_sync(kFull, c, o, 16);
            if (i >= o) c += t;
#pragma unroll
            for (int k = 0; k < 6; k++) {
                const int v = __shfl_up_sync(kFull, m[k], o, 16);
                m[k] = k < 3 ? min(m[k], v) : max(m[k], v);
            }
        }
        const float area = c > 0 ? area_x(o2f(m[0]), o2f(m[1]), o2f(m[2]), o2f(m[3]), o2f(m[4]), o2f(m[5])) : 0.f;
        const float term = x_mul(x_mul(x_div(area, parent_area), (float)c), 1.5f);
        // the right side of plane b starts at bin b + 1, in lane 30 - b
        const float right = __shfl_sync(kFull, term, (30 - lane) & 31);
        cost[ax] = x_add(x_add(1.f, term), right);
        // costs are ordered as ordered ints (a cost that is not below FLT_MAX, or NaN, is no candidate)
        if (lane < kBins - 1 && cost[ax] < FLT_MAX) key[ax] = f2o(cost[ax]);
    }
    best = FLT_MAX;
    pos = -FLT_MAX;
    const int mn = __reduce_min_sync(kFull, min(min(key[0], key[1]), key[2]));
    if (mn == INT_MAX) return -1;
    int axis = -1;
#pragma unroll
    for (int ax = 0; ax < 3; ax++) {
        const unsigned who = __ballot_sync(kFull, key[ax] == mn);
        if (axis < 0 && who) {
            axis = ax;
            const int win = __ffs(who) - 1;
            best = __shfl_sync(kFull, cost[ax], win);
            pos = x_add(lo[ax], x_mul(x_div(x_sub(hi[ax], lo[ax]), (float)kBins), (float)(win + 1)));
        }
    }
    return axis;
}

// True in the block that finishes an item's last chunk: everything the other
// blocks wrote for the item before their arrival is then visible to it.
__device__ __forceinline__ bool last_chunk(BuildItem& it, unsigned nchunks, int* flag) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const bool last = atomicAdd(&it.done, 1u) == nchunks - 1;
        if (last) it.done = 0;  // ready for the next pass
        *flag = last ? 1 : 0;
    }
    __syncthreads();
    const bool last = *flag != 0;
    if (last) __threadfence();
    return last;
}

// Scratch of a block's partition pass.
struct PartShared {
    int warp_l[kThreads / 32], warp_r[kThreads / 32];
    int base_l, base_r, flag;
    int acc[24];
};

// Where a level's children go: the other record buffer, the next level's
// items, the phase-B list, the nodes.
struct BuildOut {
    RecView rec;
    int buf;
    BuildItem* items;
    int2* chunks;
    int item_cap, chunk_cap, slot_cap;
    int2* small;
    int small_cap;
    pgx_bvh_node* nodes;
    int* node_rec;
};

// Partition of a chunk by centroid[axis] < pos (Geometry.h:384-391) into the
// other record buffer, with the children's box and centroid bounds; the
// block of the node's last chunk creates its children (Geometry.h:393-412).
// SINGLE: the chunk is the whole node, so positions and boxes stay in the
// block and no other block is waited for.  Whole blocks.
//   Bound: 96 bytes moved a triangle, 30 us a level of 2,093,058; takes 51.  A
// run of positions per thread instead of per warp (stores in pieces of 16
// bytes) took 100.
template <bool SINGLE>
__device__ __forceinline__ void partition_chunk(BuildItem& it, int first, int axis, float pos, BuildMisc* misc, int level,
                                                const RecView& rec, const BuildOut& out, PartShared& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int start = it.start, count = it.count;
    if (threadIdx.x < 24) sh.acc[threadIdx.x] = ((threadIdx.x % 6) < 3) ? INT_MAX : INT_MIN;
    const int end = min(count, first + kChunk);
    // Thread t reads positions first + k*kThreads + t; a warp's records go to
    // one run per side, so that stores are as coalesced as loads.
    unsigned left[kPerThread];
    int wl = 0, wn = 0;
#pragma unroll
    for (int k = 0; k < kPerThread; k++) {
        const int j = first + k * kThreads + threadIdx.x;
        float cv = 0.f;
        if (j < end) {
            const float4 cc = rec.cent[start + j];
            cv = axis == 0 ? cc.x : (axis == 1 ? cc.y : cc.z);
        }
        left[k] = __ballot_sync(0xFFFFFFFFu, j < end && cv < pos);
        wl += __popc(left[k]);
        wn += max(0, min(32, end - (j - lane)));
    }
    if (lane == 0) {
        sh.warp_l[warp] = wl;
        sh.warp_r[warp] = wn - wl;
    }
    __syncthreads();
    int before_l = 0, before_r = 0, all_l = 0, all_r = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; w++) {
        if (w == warp) before_l = all_l, before_r = all_r;
        all_l += sh.warp_l[w];
        all_r += sh.warp_r[w];
    }
    int base_l = 0, base_r = 0;
    if (!SINGLE) {
        if (threadIdx.x == 0) {
            sh.base_l = atomicAdd(&it.lcur, all_l);
            sh.base_r = atomicAdd(&it.rcur, all_r);
        }
        __syncthreads();
        base_l = sh.base_l;
        base_r = sh.base_r;
    }
    int offl = start + base_l + before_l;
    int offr = start + count - 1 - (base_r + before_r);
    int acc[2][12];
#pragma unroll
    for (int k = 0; k < 24; k++) acc[k / 12][k % 12] = ((k % 6) < 3) ? INT_MAX : INT_MIN;
#pragma unroll
    for (int k = 0; k < kPerThread; k++) {
        const int j = first + k * kThreads + threadIdx.x;
        const unsigned below = (1u << lane) - 1u;
        if (j < end) {
            const float4 a = rec.lo[start + j], b = rec.hi[start + j], cc = rec.cent[start + j];
            const int side = (left[k] >> lane) & 1u ? 0 : 1;
            const int to = side ? offr - __popc(~left[k] & below) : offl + __popc(left[k] & below);
            out.rec.lo[to] = a;
            out.rec.hi[to] = b;
            out.rec.cent[to] = cc;
            const int v[9] = {f2o(a.x), f2o(a.y), f2o(a.z), f2o(b.x), f2o(b.y), f2o(b.z), f2o(cc.x), f2o(cc.y), f2o(cc.z)};
#pragma unroll
            for (int s = 0; s < 2; s++)
                if (s == side) {
#pragma unroll
                    for (int x = 0; x < 3; x++) {
                        acc[s][x] = min(acc[s][x], v[x]);
                        acc[s][3 + x] = max(acc[s][3 + x], v[3 + x]);
                        acc[s][6 + x] = min(acc[s][6 + x], v[6 + x]);
                        acc[s][9 + x] = max(acc[s][9 + x], v[6 + x]);
                    }
                }
        }
        const int nk = __popc(left[k]);
        offl += nk;
        offr -= max(0, min(32, end - (j - lane))) - nk;
    }
    if (first + warp * 32 < end) {  // a warp without triangles has nothing to add
#pragma unroll
        for (int k = 0; k < 24; k++) {
            const bool is_min = (k % 6) < 3;
            const int v = is_min ? __reduce_min_sync(0xFFFFFFFFu, acc[k / 12][k % 12])
                                 : __reduce_max_sync(0xFFFFFFFFu, acc[k / 12][k % 12]);
            if (lane == 0) {
                if (is_min)
                    atomicMin(&sh.acc[k], v);
                else
                    atomicMax(&sh.acc[k], v);
            }
        }
    }
    __syncthreads();
    bool commit = true;
    if (!SINGLE) {
        if (threadIdx.x < 24) {
            const int k = threadIdx.x;
            int* dst = &it.acc[k / 12][k % 12];
            if ((k % 6) < 3)
                atomicMin(dst, sh.acc[k]);
            else
                atomicMax(dst, sh.acc[k]);
        }
        commit = last_chunk(it, (unsigned)((count + kChunk - 1) / kChunk), &sh.flag);
        if (commit) {
            if (threadIdx.x < 24) sh.acc[threadIdx.x] = __ldcg(&it.acc[threadIdx.x / 12][threadIdx.x % 12]);
            __syncthreads();
        }
    }
    // One lane per child: the two chains of list atomics run side by side.
    if (commit && threadIdx.x < 2) {
        const int side = threadIdx.x;
        pgx_bvh_node& nd = out.nodes[it.node];
        const int L = SINGLE ? all_l : __ldcg(&it.lcur);
        const int from = out.buf ? kSmallBuf : 0;
        if (L == 0 || L == count) {
            if (side == 0) {
                nd.left_first = start;
                nd.used = count;
                add_small(out.small, out.small_cap, misc, it.node, kSmallLeaf | from);
            }
        } else {
            unsigned long long at = 0;
            if (side == 0) at = atomicAdd(&misc->counts, 2ull | (1ull << 32));
            at = __shfl_sync(3u, at, 0);
            const int child = (int)(unsigned)at;
            if (side == 0) {
                out.node_rec[it.node] = (int)(at >> 32);
                nd.left_first = child;
                nd.used = 0;
            }
            const int cs = side ? start + L : start;
            const int cn = side ? count - L : L;
            const int* box = sh.acc + 12 * side;
            pgx_bvh_node& cnd = out.nodes[child + side];
            for (int k = 0; k < 3; k++) {
                cnd.bmin[k] = o2f(box[k]);
                cnd.bmax[k] = o2f(box[3 + k]);
            }
            cnd.left_first = cs;
            cnd.used = cn;
            out.node_rec[child + side] = -1;
            if (cn <= kSmall)
                add_small(out.small, out.small_cap, misc, child + side, from);
            else
                add_item(out.items, out.chunks, misc, level + 1, out.item_cap, out.chunk_cap, out.slot_cap, child + side,
                         cs, cn, box + 6, box + 9);
        }
    }
    __syncthreads();
}

// Bins of each chunk in shared memory, merged into the node's global bins
// when it has several chunks; the last chunk's block decides the split
// (subdivide, Geometry.h:367-381).  A node that stays a leaf goes to phase B
// for its triangle ids.  A node of one chunk is partitioned here as well,
// while the block holds its split.
__global__ void __launch_bounds__(kThreads) k_bin(BuildItem* __restrict__ items, const int2* __restrict__ chunks,
                                                  BuildMisc* __restrict__ misc, int level, RecView rec, int buf,
                                                  int* __restrict__ gbins, BuildOut out) {
    grid_begin();
    __shared__ int sb[kBinCopies * kCopyInts];
    int* mine = sb + (threadIdx.x % kBinCopies) * kCopyInts;
    __shared__ PartShared sh;
    __shared__ int s_split, s_axis;
    __shared__ float s_pos;
    const int nchunks = misc->nchunks[level];
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const int2 ch = chunks[c];
        BuildItem& it = items[ch.x];
        const int start = it.start, count = it.count;
        for (int k = threadIdx.x; k < kBinInts; k += kThreads)
            for (int v = 0; v < kBinCopies; v++) reset_bins(sb + v * kCopyInts, k);
        __syncthreads();
        float lo[3], hi[3], scale[3];
#pragma unroll
        for (int ax = 0; ax < 3; ax++) {
            lo[ax] = o2f(it.cmin[ax]);
            hi[ax] = o2f(it.cmax[ax]);
            scale[ax] = x_div((float)kBins, x_sub(hi[ax], lo[ax]));
        }
        const int end = min(count, ch.y + kChunk);
        for (int b = ch.y; b < end; b += kThreads) {  // whole warps
            const int j = b + threadIdx.x;
            const bool in = j < end;
            float cv[3] = {0.f, 0.f, 0.f};
            int l[3] = {INT_MAX, INT_MAX, INT_MAX}, h[3] = {INT_MIN, INT_MIN, INT_MIN};
            if (in) {
                const float4 a = rec.lo[start + j], bb = rec.hi[start + j], cc = rec.cent[start + j];
                cv[0] = cc.x, cv[1] = cc.y, cv[2] = cc.z;
                l[0] = f2o(a.x), l[1] = f2o(a.y), l[2] = f2o(a.z);
                h[0] = f2o(bb.x), h[1] = f2o(bb.y), h[2] = f2o(bb.z);
            }
#pragma unroll
            for (int ax = 0; ax < 3; ax++)
                if (!(lo[ax] == hi[ax])) bin_add(mine, ax, in ? bin_of(cv[ax], lo[ax], scale[ax]) : -1, l, h);
        }
        __syncthreads();
        for (int k = threadIdx.x; k < kBinInts; k += kThreads) {
            const int f = k / kField;
            int r = sb[k];
#pragma unroll
            for (int v = 1; v < kBinCopies; v++) {
                const int o = sb[v * kCopyInts + k];
                r = f == 0 ? r + o : (f < 4 ? min(r, o) : max(r, o));
            }
            sb[k] = r;
        }
        __syncthreads();
        const unsigned nch = (unsigned)((count + kChunk - 1) / kChunk);
        bool decide = true;
        if (nch > 1) {
            int* g = gbins + (size_t)it.slot * kBinInts;
            for (int k = threadIdx.x; k < kBinInts; k += kThreads) {
                if (sb[k % kField] == 0) continue;
                const int f = k / kField;
                if (f == 0)
                    atomicAdd(g + k, sb[k]);
                else if (f < 4)
                    atomicMin(g + k, sb[k]);
                else
                    atomicMax(g + k, sb[k]);
            }
            decide = last_chunk(it, nch, &sh.flag);
            if (decide) {
                for (int k = threadIdx.x; k < kBinInts; k += kThreads) {
                    sb[k] = __ldcg(g + k);
                    reset_bins(g, k);  // for the next level's node in this slot
                }
                __syncthreads();
            }
        }
        if (decide && threadIdx.x < 32) {
            pgx_bvh_node& nd = out.nodes[it.node];
            const float parent_area = area_x(nd.bmin[0], nd.bmin[1], nd.bmin[2], nd.bmax[0], nd.bmax[1], nd.bmax[2]);
            float best, pos;
            const int axis = warp_sweep<1>(sb, lo, hi, parent_area, best, pos);
            if (threadIdx.x == 0) {
                const float no_split = x_mul((float)count, 1.5f);
                s_split = 0;
                if (best >= no_split || axis == -1) {
                    it.split = 0;
                    nd.left_first = start;
                    nd.used = count;
                    // (the chunks of a larger leaf: k_partition)
                    if (nch == 1) add_small(out.small, out.small_cap, misc, it.node, kSmallLeaf | (buf ? kSmallBuf : 0));
                } else if (nch > 1) {
                    it.split = 1;
                    it.axis = axis;
                    it.pos = pos;
                } else {
                    s_split = 1;
                    s_axis = axis;
                    s_pos = pos;
                }
            }
        }
        __syncthreads();  // the shared bins are reused
        if (nch == 1 && s_split) partition_chunk<true>(it, 0, s_axis, s_pos, misc, level, rec, out, sh);
    }
}

// Partition of the chunks of the nodes that have several; where such a node
// stays a leaf (triangles no plane separates), the chunks' triangle ids go to
// the leaf order here, by all its blocks: 2,000,000 coincident triangles are
// one leaf, and the build takes 15.4 ms with one warp of k_small for it, 0.27
// with these.
__global__ void __launch_bounds__(kThreads) k_partition(BuildItem* __restrict__ items, const int2* __restrict__ chunks,
                                                        BuildMisc* __restrict__ misc, int level, RecView rec,
                                                        int* __restrict__ idx, BuildOut out) {
    grid_begin();
    __shared__ PartShared sh;
    if (misc->nslots[level] == 0) return;  // no such node on this level
    const int nchunks = misc->nchunks[level];
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const int2 ch = chunks[c];
        BuildItem& it = items[ch.x];
        if (!it.split) {  // uniform per block
            const int start = it.start, end = it.count > kChunk ? min(it.count, ch.y + kChunk) : 0;
            for (int j = ch.y + threadIdx.x; j < end; j += kThreads) idx[start + j] = __float_as_int(rec.lo[start + j].w);
            continue;
        }
        partition_chunk<false>(it, ch.y, it.axis, it.pos, misc, level, rec, out, sh);
    }
}

// Phase B: one warp finishes the subtree of a node of at most kSmall
// triangles (Geometry.h:274-417), its records in shared memory, depth first.
// The subtree's nodes go to a scratch block first (a subtree of c triangles
// needs at most 2c - 2 of them, and those of the position range
// [first, first + c) are scratch[2 first ...)), so that one atomic reserves a
// contiguous run of nodes and traversal records per subtree.
//   Bound: issue of dependent warp steps and the sweep's shuffles.  2,093,058
// triangles: 0.82 ms; one thread per subtree, with its bins in local memory
// and two atomics a node, took 7.4.
constexpr int kSmallWarps = 4;
struct SmallWarp {
    float v[9][kSmall];    // box min, box max, centroid
    int id[kSmall];
    int bins[kSmallCopies * kCopyInts];
    int2 stack[kSmall];    // (first | count << 8 | scratch node << 16, parent area)
    unsigned char perm[kSmall];
};

__global__ void __launch_bounds__(32 * kSmallWarps) k_small(const int2* __restrict__ small,
                                                            BuildMisc* __restrict__ misc, RecView rec0, RecView rec1,
                                                            int* __restrict__ idx, pgx_bvh_node* __restrict__ nodes,
                                                            int* __restrict__ node_rec,
                                                            pgx_bvh_node* __restrict__ scratch) {
    grid_begin();
    extern __shared__ __align__(16) uint8_t s_dyn[];
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    SmallWarp& W = reinterpret_cast<SmallWarp*>(s_dyn)[threadIdx.x >> 5];
    const int nsmall = misc->nsmall;
    for (int job = blockIdx.x * kSmallWarps + (threadIdx.x >> 5); job < nsmall; job += gridDim.x * kSmallWarps) {
        const int2 jb = small[job];
        const pgx_bvh_node root = nodes[jb.x];
        const int first = root.left_first, total = root.used;
        const RecView rec = (jb.y & kSmallBuf) ? rec1 : rec0;
        if ((jb.y & kSmallLeaf) || total <= kMaxLeaf) {
            for (int k = lane; k < total; k += 32) idx[first + k] = __float_as_int(rec.lo[first + k].w);
            continue;
        }
        __syncwarp();
        for (int k = lane; k < total; k += 32) {
            const float4 a = rec.lo[first + k], b = rec.hi[first + k], c = rec.cent[first + k];
            W.v[0][k] = a.x, W.v[1][k] = a.y, W.v[2][k] = a.z;
            W.v[3][k] = b.x, W.v[4][k] = b.y, W.v[5][k] = b.z;
            W.v[6][k] = c.x, W.v[7][k] = c.y, W.v[8][k] = c.z;
            W.id[k] = __float_as_int(a.w);
            W.perm[k] = (unsigned char)k;
        }
        __syncwarp();
        pgx_bvh_node* tmp = scratch + 2 * (size_t)first;
        int nn = 0, ni = 0, sp = 0;    // scratch nodes, interior nodes, stack height
        int s0 = 0, cnt = total, self = -1;  // current node: [s0, s0 + cnt), its scratch node (-1: the root)
        float area = area_x(root.bmin[0], root.bmin[1], root.bmin[2], root.bmax[0], root.bmax[1], root.bmax[2]);
        for (;;) {
            bool split = cnt > kMaxLeaf;
            if (split) {
                const int rounds = (cnt + 31) >> 5;
                int p[kSmall / 32];
                float lo[3], hi[3], scale[3];
                {
                    int mn[3] = {INT_MAX, INT_MAX, INT_MAX}, mx[3] = {INT_MIN, INT_MIN, INT_MIN};
#pragma unroll
                    for (int k = 0; k < kSmall / 32; k++) {
                        p[k] = -1;
                        if (k < rounds && k * 32 + lane < cnt) {
                            p[k] = W.perm[s0 + k * 32 + lane];
#pragma unroll
                            for (int x = 0; x < 3; x++) {
                                const int o = f2o(W.v[6 + x][p[k]]);
                                mn[x] = min(mn[x], o);
                                mx[x] = max(mx[x], o);
                            }
                        }
                    }
#pragma unroll
                    for (int x = 0; x < 3; x++) {
                        lo[x] = o2f(__reduce_min_sync(kFull, mn[x]));
                        hi[x] = o2f(__reduce_max_sync(kFull, mx[x]));
                        scale[x] = x_div((float)kBins, x_sub(hi[x], lo[x]));
                    }
                }
#pragma unroll
                for (int r = 0; r < (kBinInts + 31) / 32; r++) {
                    const int k = r * 32 + lane;
                    if (k >= kBinInts) break;
#pragma unroll
                    for (int v = 0; v < kSmallCopies; v++) reset_bins(W.bins + v * kCopyInts, k);
                }
                __syncwarp();
#pragma unroll
                for (int k = 0; k < kSmall / 32; k++) {
                    if (k >= rounds || p[k] < 0) continue;
                    int l[3], h[3];
#pragma unroll
                    for (int x = 0; x < 3; x++) {
                        l[x] = f2o(W.v[x][p[k]]);
                        h[x] = f2o(W.v[3 + x][p[k]]);
                    }
#pragma unroll
                    for (int ax = 0; ax < 3; ax++) {
                        if (lo[ax] == hi[ax]) continue;
                        int* bn = W.bins + (lane % kSmallCopies) * kCopyInts + ax * kBins +
                                  bin_of(W.v[6 + ax][p[k]], lo[ax], scale[ax]);
                        atomicAdd(bn, 1);
#pragma unroll
                        for (int x = 0; x < 3; x++) {
                            atomicMin(bn + (1 + x) * kField, l[x]);
                            atomicMax(bn + (4 + x) * kField, h[x]);
                        }
                    }
                }
                __syncwarp();
                float best, pos;
                const int axis = warp_sweep<kSmallCopies>(W.bins, lo, hi, area, best, pos);
                split = !(best >= x_mul((float)cnt, 1.5f) || axis == -1);
                int L = 0;
                unsigned left[kSmall / 32];
                if (split) {
#pragma unroll
                    for (int k = 0; k < kSmall / 32; k++) {
                        left[k] = __ballot_sync(kFull, p[k] >= 0 && W.v[6 + axis][max(p[k], 0)] < pos);
                        L += __popc(left[k]);
                    }
                    split = L != 0 && L != cnt;
                }
                if (split) {
                    int at_l = s0, at_r = s0 + L;
                    int box[2][6];
#pragma unroll
                    for (int k = 0; k < 12; k++) box[k / 6][k % 6] = (k % 6) < 3 ? INT_MAX : INT_MIN;
#pragma unroll
                    for (int k = 0; k < kSmall / 32; k++) {
                        const unsigned have = __ballot_sync(kFull, p[k] >= 0);
                        const unsigned right = have & ~left[k];
                        if (p[k] >= 0) {
                            const bool is_l = (left[k] >> lane) & 1u;
                            W.perm[is_l ? at_l + __popc(left[k] & below) : at_r + __popc(right & below)] =
                                (unsigned char)p[k];
#pragma unroll
                            for (int s = 0; s < 2; s++)
                                if ((s == 0) == is_l) {
#pragma unroll
                                    for (int x = 0; x < 3; x++) {
                                        box[s][x] = min(box[s][x], f2o(W.v[x][p[k]]));
                                        box[s][3 + x] = max(box[s][3 + x], f2o(W.v[3 + x][p[k]]));
                                    }
                                }
                        }
                        at_l += __popc(left[k]);
                        at_r += __popc(right);
                    }
#pragma unroll
                    for (int k = 0; k < 12; k++)
                        box[k / 6][k % 6] = (k % 6) < 3 ? __reduce_min_sync(kFull, box[k / 6][k % 6])
                                                        : __reduce_max_sync(kFull, box[k / 6][k % 6]);
                    float ca[2];
#pragma unroll
                    for (int s = 0; s < 2; s++) {
                        const float b[6] = {o2f(box[s][0]), o2f(box[s][1]), o2f(box[s][2]),
                                            o2f(box[s][3]), o2f(box[s][4]), o2f(box[s][5])};
                        ca[s] = area_x(b[0], b[1], b[2], b[3], b[4], b[5]);
                        if (lane == s) {
                            pgx_bvh_node& ch = tmp[nn + s];
                            for (int x = 0; x < 3; x++) {
                                ch.bmin[x] = b[x];
                                ch.bmax[x] = b[3 + x];
                            }
                            ch.left_first = first + (s ? s0 + L : s0);
                            ch.used = s ? cnt - L : L;
                        }
                    }
                    __syncwarp();
                    // an interior node: its left child's scratch node and its
                    // ordinal among the subtree's interior nodes
                    if (lane == 0) {
                        if (self >= 0) {
                            tmp[self].left_first = nn | (ni << 16);
                            tmp[self].used = 0;
                        }
                        W.stack[sp] = make_int2((s0 + L) | ((cnt - L) << 8) | ((nn + 1) << 16), __float_as_int(ca[1]));
                    }
                    sp++;
                    ni++;
                    self = nn;
                    cnt = L;
                    area = ca[0];
                    nn += 2;
                    __syncwarp();
                    continue;
                }
            }
            // a leaf: the next node from the stack
            if (sp == 0) break;
            sp--;
            __syncwarp();
            const int2 e = W.stack[sp];
            __syncwarp();
            s0 = e.x & 0xFF;
            cnt = (e.x >> 8) & 0xFF;
            self = e.x >> 16;
            area = __int_as_float(e.y);
        }
        __syncwarp();
        for (int k = lane; k < total; k += 32) idx[first + k] = W.id[W.perm[k]];
        if (nn == 0) continue;  // the root stays a leaf
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&misc->counts, (unsigned long long)nn | ((unsigned long long)ni << 32));
        at = __shfl_sync(kFull, at, 0);
        const int base = (int)(unsigned)at, rbase = (int)(at >> 32);
        for (int k = lane; k < nn; k += 32) {
            pgx_bvh_node nd = tmp[k];
            int r = -1;
            if (nd.used == 0) {
                r = rbase + (nd.left_first >> 16);
                nd.left_first = base + (nd.left_first & 0xFFFF);
            }
            nodes[base + k] = nd;
            node_rec[base + k] = r;
        }
        if (lane == 0) {
            nodes[jb.x].left_first = base;
            nodes[jb.x].used = 0;
            node_rec[jb.x] = rbase;
        }
        __syncwarp();
    }
}

__device__ __forceinline__ TravChild trav_child(const pgx_bvh_node& c, int rec) {
    TravChild t;
    t.mnx = c.bmin[0], t.mny = c.bmin[1], t.mnz = c.bmin[2];
    t.mxx = c.bmax[0], t.mxy = c.bmax[1], t.mxz = c.bmax[2];
    t.ref = c.used > 0 ? c.left_first : rec;
    t.count = c.used;
    return t;
}
// Traversal records from the reference-layout tree.
__global__ void k_layout(const pgx_bvh_node* __restrict__ nodes, int64_t nnodes, const int* __restrict__ node_rec,
                         TravNode* __restrict__ out) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nnodes) return;
    const pgx_bvh_node& nd = nodes[i];
    if (nd.used > 0) return;
    int rec = node_rec[i];
    if (rec < 0) return;
    const pgx_bvh_node& L = nodes[nd.left_first];
    const pgx_bvh_node& R = nodes[nd.left_first + 1];
    TravNode t;
    t.l = trav_child(L, node_rec[nd.left_first]);
    t.r = trav_child(R, node_rec[nd.left_first + 1]);
    out[rec] = t;
}

// Leaf-ordered triangles: position p holds triangle idx[p] as v0, e0, e1.
__global__ void k_reorder(const pgx_triangle* __restrict__ tris, const int* __restrict__ idx, int64_t n,
                          TravTri* __restrict__ out) {
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    int id = idx[p];
    const pgx_triangle& t = tris[id];
    xv3 v0 = mk(t.v[0].p[0], t.v[0].p[1], t.v[0].p[2]);
    xv3 e0 = x_sub(mk(t.v[1].p[0], t.v[1].p[1], t.v[1].p[2]), v0);
    xv3 e1 = x_sub(mk(t.v[2].p[0], t.v[2].p[1], t.v[2].p[2]), v0);
    TravTri o;
    o.v0 = make_float4(v0.x, v0.y, v0.z, __int_as_float(id));
    o.e0 = make_float4(e0.x, e0.y, e0.z, 0.f);
    o.e1 = make_float4(e1.x, e1.y, e1.z, 0.f);
    o.pad = make_float4(0.f, 0.f, 0.f, 0.f);
    out[p] = o;
}

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

BvhView bvh_view(const pgx_ctx* ctx) {
    BvhView v;
    v.nodes = ctx->trav_nodes.as<TravNode>();
    v.tris = ctx->trav_tris.as<TravTri>();
    v.root = ctx->root;
    if (!ctx->has_bvh) v.root.valid = 0;
    return v;
}

// Builds the traversal layout from ctx->bvh_nodes_ref / bvh_idx and a node ->
// record map (device buffer b_noderec, filled by the caller).
static int finish_layout(pgx_ctx* ctx) {
    cudaStream_t s = ctx->stream;
    int64_t n = ctx->ntris;
    PGX_CUDA_TRY(ctx, ctx->trav_nodes.reserve(sizeof(TravNode) * (size_t)std::max<int64_t>(ctx->n_records, 1)));
    PGX_CUDA_TRY(ctx, ctx->trav_tris.reserve(sizeof(TravTri) * (size_t)std::max<int64_t>(n, 1)));
    if (ctx->n_nodes > 0)
        k_layout<<<blocks_for(ctx->n_nodes, 256), 256, 0, s>>>(ctx->bvh_nodes_ref.as<pgx_bvh_node>(), ctx->n_nodes,
                                                               ctx->b_noderec.as<int>(), ctx->trav_nodes.as<TravNode>());
    if (n > 0)
        k_reorder<<<blocks_for(n, 256), 256, 0, s>>>(ctx->tris_in.as<pgx_triangle>(), ctx->bvh_idx.as<int>(), n,
                                                     ctx->trav_tris.as<TravTri>());
    PGX_CUDA_TRY(ctx, cudaGetLastError());
    pgx_bvh_node root;
    int root_rec = -1;
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(&root, ctx->bvh_nodes_ref.p, sizeof(root), cudaMemcpyDeviceToHost, s));
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(&root_rec, ctx->b_noderec.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    PGX_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    TravRoot r{};
    for (int k = 0; k < 3; k++) {
        r.bmin[k] = root.bmin[k];
        r.bmax[k] = root.bmax[k];
    }
    if (root.used > 0) {
        r.ref = root.left_first;
        r.count = root.used;
    } else {
        r.ref = root_rec;
        r.count = 0;
    }
    r.valid = n > 0 ? 1 : 0;
    ctx->root = r;
    ctx->has_bvh = true;
    return PGX_OK;
}

int bvh_build_gpu(pgx_ctx* ctx) {
    if (!ctx->has_scene) return pgx_fail(ctx, PGX_ERR_STATE, "pgx_bvh_build: no scene uploaded");
    auto t0 = std::chrono::steady_clock::now();
    cudaStream_t s = ctx->stream;
    const int64_t n = ctx->ntris;
    ctx->has_bvh = false;
    if (n == 0) {
        ctx->n_nodes = 0;
        ctx->n_records = 0;
        ctx->root = TravRoot{};
        ctx->has_bvh = true;
        return PGX_OK;
    }
    if (n > (int64_t)INT32_MAX / 2) return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "too many triangles for a BVH");
    const int64_t max_nodes = 2 * n - 1;
    const int64_t item_cap = n / kSmall + 64;       // an item has more than kSmall triangles
    const int64_t slot_cap = n / kChunk + 64;       // a slot's node has more than kChunk
    const int64_t chunk_cap = n / kChunk + item_cap + 64;
    const int64_t small_cap = n + 64;               // disjoint, non-empty position ranges
    PGX_CUDA_TRY(ctx, ctx->b_recs.reserve(3 * sizeof(float4) * n));
    PGX_CUDA_TRY(ctx, ctx->b_recs2.reserve(3 * sizeof(float4) * n));
    PGX_CUDA_TRY(ctx, ctx->b_tmp.reserve(2 * sizeof(pgx_bvh_node) * n));
    PGX_CUDA_TRY(ctx, ctx->bvh_idx.reserve(sizeof(int) * n));
    PGX_CUDA_TRY(ctx, ctx->bvh_nodes_ref.reserve(sizeof(pgx_bvh_node) * max_nodes));
    PGX_CUDA_TRY(ctx, ctx->b_noderec.reserve(sizeof(int) * max_nodes));
    PGX_CUDA_TRY(ctx, ctx->b_items.reserve(sizeof(BuildItem) * item_cap));
    PGX_CUDA_TRY(ctx, ctx->b_items2.reserve(sizeof(BuildItem) * item_cap));
    PGX_CUDA_TRY(ctx, ctx->b_bins.reserve(sizeof(int) * kBinInts * slot_cap));
    PGX_CUDA_TRY(ctx, ctx->b_chunks.reserve(sizeof(int2) * chunk_cap));
    PGX_CUDA_TRY(ctx, ctx->b_chunks2.reserve(sizeof(int2) * chunk_cap));
    PGX_CUDA_TRY(ctx, ctx->b_small.reserve(sizeof(int2) * small_cap));
    PGX_CUDA_TRY(ctx, ctx->b_misc.reserve(sizeof(BuildMisc)));

    auto view = [n](const DevBuf& b) { return RecView{b.as<float4>(), b.as<float4>() + n, b.as<float4>() + 2 * n}; };
    const RecView recs[2] = {view(ctx->b_recs), view(ctx->b_recs2)};
    int* idx = ctx->bvh_idx.as<int>();
    pgx_bvh_node* nodes = ctx->bvh_nodes_ref.as<pgx_bvh_node>();
    int* node_rec = ctx->b_noderec.as<int>();
    BuildItem* items[2] = {ctx->b_items.as<BuildItem>(), ctx->b_items2.as<BuildItem>()};
    int2* chunks[2] = {ctx->b_chunks.as<int2>(), ctx->b_chunks2.as<int2>()};
    int* bins = ctx->b_bins.as<int>();
    int2* small = ctx->b_small.as<int2>();
    BuildMisc* misc = ctx->b_misc.as<BuildMisc>();

    BuildMisc hm{};
    for (int k = 0; k < 12; k++) hm.root_acc[k] = ((k % 6) < 3) ? INT_MAX : INT_MIN;
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(misc, &hm, sizeof(hm), cudaMemcpyHostToDevice, s));
    const unsigned wide = 8 * pgx_num_sms();
    launch_behind(k_prep, std::min<unsigned>(blocks_for(n, kThreads), wide), kThreads, 0, s,
                  ctx->tris_in.as<pgx_triangle>(), n, recs[0], misc);
    launch_behind(k_bins_reset, blocks_for(kBinInts * slot_cap, 256), 256, 0, s, bins, kBinInts * slot_cap);
    launch_behind(k_root_init, 1, 32, 0, s, nodes, node_rec, items[0], chunks[0], small, misc, n, (int)item_cap,
                  (int)chunk_cap, (int)slot_cap, (int)small_cap);
    // A level's work list is on the device, so levels are enqueued ahead: the
    // fewest there can be (splits in halves) at once, then two at a time until
    // the list is empty.
    int ahead = 0;
    for (int64_t c = n; c > kSmall; c = (c + 1) / 2) ahead++;
    const unsigned grid = (unsigned)std::min<int64_t>(chunk_cap, wide);
    for (int level = 0; n > kSmall;) {
        for (const int stop = level + ahead; level < stop && level < kMaxLevels; level++) {
            const int a = level & 1, b = a ^ 1;
            const BuildOut out{recs[b], b, items[b], chunks[b], (int)item_cap, (int)chunk_cap, (int)slot_cap,
                               small, (int)small_cap, nodes, node_rec};
            launch_behind(k_bin, grid, kThreads, 0, s, items[a], chunks[a], misc, level, recs[a], a, bins, out);
            launch_behind(k_partition, grid, kThreads, 0, s, items[a], chunks[a], misc, level, recs[a], idx, out);
        }
        PGX_CUDA_TRY(ctx, cudaGetLastError());
        int left = 0, bad = 0;
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(&left, &misc->nchunks[level], sizeof(int), cudaMemcpyDeviceToHost, s));
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(&bad, &misc->overflow, sizeof(int), cudaMemcpyDeviceToHost, s));
        PGX_CUDA_TRY(ctx, cudaStreamSynchronize(s));
        if (bad) return pgx_fail(ctx, PGX_ERR_OVERFLOW, "BVH build: work list overflow (%d)", bad);
        if (left == 0) break;
        if (level >= kMaxLevels) return pgx_fail(ctx, PGX_ERR_OVERFLOW, "BVH build: too many levels");
        ahead = 2;
    }
    constexpr int kSmallSmem = (int)sizeof(SmallWarp) * kSmallWarps;
    int per_sm = 0;
    PGX_CUDA_TRY(ctx, cudaFuncSetAttribute(k_small, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem));
    PGX_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_small, 32 * kSmallWarps, kSmallSmem));
    // about two triangles a leaf at least: no more warps than subtrees of 8 triangles
    const int64_t small_blocks = std::min<int64_t>(n / (8 * kSmallWarps) + 1, (int64_t)pgx_num_sms() * std::max(per_sm, 1));
    launch_behind(k_small, (unsigned)small_blocks, 32 * kSmallWarps, kSmallSmem, s, small, misc, recs[0], recs[1],
                  idx, nodes, node_rec, ctx->b_tmp.as<pgx_bvh_node>());
    PGX_CUDA_TRY(ctx, cudaGetLastError());
    BuildMisc fin{};
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(&fin, misc, offsetof(BuildMisc, root_acc), cudaMemcpyDeviceToHost, s));
    PGX_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    if (fin.overflow) return pgx_fail(ctx, PGX_ERR_OVERFLOW, "BVH build: work list overflow (%d)", fin.overflow);
    ctx->n_nodes = (int64_t)(unsigned)fin.counts;
    ctx->n_records = (int64_t)(fin.counts >> 32);
    PGX_TRY(finish_layout(ctx));
    auto t1 = std::chrono::steady_clock::now();
    ctx->bvh_build_ms = std::chrono::duration<double, std::milli>(t1 - t0).count();
    return PGX_OK;
}

int bvh_import_ref(pgx_ctx* ctx, const pgx_bvh_node* nodes, int64_t nnodes, const int32_t* idx) {
    if (!ctx->has_scene) return pgx_fail(ctx, PGX_ERR_STATE, "pgx_bvh_import: no scene uploaded");
    const int64_t n = ctx->ntris;
    if (n == 0) {
        ctx->n_nodes = 0;
        ctx->n_records = 0;
        ctx->root = TravRoot{};
        ctx->has_bvh = true;
        return PGX_OK;
    }
    if (!nodes || !idx || nnodes <= 0) return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_bvh_import: empty tree");
    // Validate the tree on the host and number interior nodes in array order.
    std::vector<int> rec((size_t)nnodes, -1);
    int next = 0;
    for (int64_t i = 0; i < nnodes; i++) {
        const pgx_bvh_node& nd = nodes[i];
        if (nd.used < 0) return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_bvh_import: node %lld negative count", (long long)i);
        if (nd.used > 0) {
            if (nd.left_first < 0 || (int64_t)nd.left_first + nd.used > n)
                return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_bvh_import: leaf %lld out of range", (long long)i);
        } else {
            if (nd.left_first <= i || (int64_t)nd.left_first + 1 >= nnodes)
                return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_bvh_import: node %lld bad children", (long long)i);
            rec[(size_t)i] = next++;
        }
    }
    for (int64_t i = 0; i < n; i++)
        if (idx[i] < 0 || idx[i] >= n)
            return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_bvh_import: triangle index %lld out of range", (long long)i);
    cudaStream_t s = ctx->stream;
    PGX_CUDA_TRY(ctx, ctx->bvh_nodes_ref.reserve(sizeof(pgx_bvh_node) * nnodes));
    PGX_CUDA_TRY(ctx, ctx->bvh_idx.reserve(sizeof(int) * n));
    PGX_CUDA_TRY(ctx, ctx->b_noderec.reserve(sizeof(int) * nnodes));
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->bvh_nodes_ref.p, nodes, sizeof(pgx_bvh_node) * nnodes,
                                      cudaMemcpyHostToDevice, s));
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->bvh_idx.p, idx, sizeof(int) * n, cudaMemcpyHostToDevice, s));
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->b_noderec.p, rec.data(), sizeof(int) * nnodes, cudaMemcpyHostToDevice, s));
    ctx->n_nodes = nnodes;
    ctx->n_records = next;
    ctx->has_bvh = false;
    return finish_layout(ctx);
}
