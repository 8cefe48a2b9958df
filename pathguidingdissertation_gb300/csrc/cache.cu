// Radiance cache: the point BVH over path vertices
// (PointBVHNode::buildPointBVHNode, Renderer.h:85-142,189-211) built on the
// GPU, its k-nearest query, and the per-region QuadTree guide (pgx_guide.cuh).
//
// Build semantics follow the reference: a node holding more than 8 records
// splits on the longest axis of its bounds (ties to the lower axis) so that
// the left child receives the used/2 records with the smallest coordinate
// (std::nth_element at offset + used/2) and the right child the rest.  With
// distinct coordinates every node holds the same record set as the
// reference's.  Nodes of more than kSmall records are split level by level
// (radix select on the ordered-int key, then a partition that also reduces
// the children's bounds); the records travel with their positions between two
// buffers, and since every split is at used/2 the sizes of a level are known
// on the host, so no level waits for the device.  A subtree of at most kSmall
// records is finished by one CTA in shared memory (k_psubtree).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <map>
#include <vector>

#include "pgx_ctx.h"
#include "pgx_guide.cuh"

namespace {

constexpr int kLeafMax = 8;      // MAX_CHILDNODE_RECORDS, Renderer.h:78
constexpr int kSmall = 2048;     // one-CTA subtrees at or below this size
constexpr int kChunk = 2048;     // records per CTA of the level-by-level phase
constexpr int kThreads = 256;
constexpr int kPer = kChunk / kThreads;
constexpr int kDigitBits = 11;   // radix select: digits of 11, 11 and 10 bits, from the top
constexpr int kDigits = 1 << kDigitBits;
constexpr int kPasses = 3;
__host__ __device__ constexpr int digit_shift(int pass) { return pass == 0 ? 21 : (pass == 1 ? 10 : 0); }

struct PItem {
    int node;
    int offset, used;
    int axis;
    unsigned prefix;
    int k;
    int lcur, rcur, tie;
    int acc[2][6];      // child bounds: min xyz, max xyz (ordered ints)
    unsigned done;      // chunks of the running pass that have finished
};

struct PMisc {
    int node_count;
    int nitems_next;
    int nsmall;
    int nregions;
    int overflow;
};

struct CacheState {
    DevBuf recs_in, recs, pos, pos2, idx, nodes, trav, items, items2, hist, small, misc, regions, region_of;
    DevBuf wts_in, wts;  // flux weight per record (input order, then leaf order)
    DevBuf qkey;         // quadtree build: Morton key and weight of each record, two buffers of each
    DevBuf qroot, qnodes, knn_q, knn_i, knn_d, node_region;
    int64_t n_records = 0;
    int64_t n_nodes = 0;
    int n_regions = 0;
    uint64_t generation = 0;  // bumped by every build
    bool valid = false;
    bool pss = false;  // quadtrees over the diffuse BSDF's primary samples
    double build_ms = 0.0;
};

__device__ __forceinline__ unsigned key_of(float f) { return (unsigned)f2o(f) ^ 0x80000000u; }
__device__ __forceinline__ float axis_of(float4 p, int ax) { return ax == 0 ? p.x : (ax == 1 ? p.y : p.z); }

// Longest axis of a box (Renderer.h:90-95).
__device__ __forceinline__ int longest_axis(const pgx_cache_node& n) {
    float ex = n.bmax[0] - n.bmin[0], ey = n.bmax[1] - n.bmin[1], ez = n.bmax[2] - n.bmin[2];
    int ax = 0;
    if (ey > ex) ax = 1;
    float e = ax == 0 ? ex : ey;
    if (ez > e) ax = 2;
    return ax;
}

__global__ void k_bounds_init(int* acc) {
    grid_begin();
    if (threadIdx.x < 6) acc[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
}

// Positions of the input records, each with its record index in w, and their
// bounds (ordered ints; one atomic per block and side).
__global__ void __launch_bounds__(256) k_pos(const pgx_path_vertex* __restrict__ r, int64_t n, float4* __restrict__ pos,
                                             int* __restrict__ acc) {
    grid_begin();
    __shared__ int s_acc[6];
    if (threadIdx.x < 6) s_acc[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
    __syncthreads();
    int a[6] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 p = *reinterpret_cast<const float4*>(r + i);  // 48-byte records: 16-byte aligned
        pos[i] = make_float4(p.x, p.y, p.z, __int_as_float((int)i));
        a[0] = min(a[0], f2o(p.x));
        a[1] = min(a[1], f2o(p.y));
        a[2] = min(a[2], f2o(p.z));
        a[3] = max(a[3], f2o(p.x));
        a[4] = max(a[4], f2o(p.y));
        a[5] = max(a[5], f2o(p.z));
    }
#pragma unroll
    for (int k = 0; k < 6; k++) {
        const int v = k < 3 ? __reduce_min_sync(0xFFFFFFFFu, a[k]) : __reduce_max_sync(0xFFFFFFFFu, a[k]);
        if ((threadIdx.x & 31) == 0) {
            if (k < 3)
                atomicMin(&s_acc[k], v);
            else
                atomicMax(&s_acc[k], v);
        }
    }
    __syncthreads();
    if (threadIdx.x < 3)
        atomicMin(&acc[threadIdx.x], s_acc[threadIdx.x]);
    else if (threadIdx.x < 6)
        atomicMax(&acc[threadIdx.x], s_acc[threadIdx.x]);
}

// An item of the level-by-level phase, ready for its first select pass.
__device__ __forceinline__ void start_item(PItem& it, int node, int offset, int used, const pgx_cache_node& nd) {
    it.node = node;
    it.offset = offset;
    it.used = used;
    it.axis = longest_axis(nd);
    it.prefix = 0;
    it.k = used / 2;
    it.lcur = it.rcur = it.tie = 0;
    it.done = 0;
    for (int s = 0; s < 2; s++)
        for (int k = 0; k < 6; k++) it.acc[s][k] = k < 3 ? INT_MAX : INT_MIN;
}

__global__ void k_root(int64_t n, PMisc* misc, pgx_cache_node* nodes, PItem* items, int2* small, int* acc) {
    grid_begin();
    // acc: 6 ordered ints reduced by k_pos
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    pgx_cache_node& r = nodes[0];
    for (int k = 0; k < 3; k++) {
        r.bmin[k] = o2f(acc[k]);
        r.bmax[k] = o2f(acc[3 + k]);
    }
    r.left = r.right = -1;
    r.offset = 0;
    r.used = (int)n;
    misc->node_count = 1;
    misc->nitems_next = 0;
    misc->nsmall = 0;
    misc->nregions = 0;
    misc->overflow = 0;
    if (n <= kSmall) {
        small[0] = make_int2(0, 0);
        misc->nsmall = 1;
        return;
    }
    start_item(items[0], 0, 0, (int)n, r);
}

// True in the block that finishes an item's last chunk: everything the other
// blocks wrote for the item before their arrival is then visible to it.
__device__ __forceinline__ bool last_chunk(PItem& it, unsigned nchunks, int* flag) {
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

// One pass of the radix select, one block per (item, chunk): histogram of the
// pass's digit among the records whose higher digits equal the item's
// prefix; the block that finishes the item's last chunk scans the counts,
// appends the digit holding rank it.k to the prefix and clears the
// histogram.  Separate one-thread scans (34 us a pass) and 8-bit digits (four
// passes) were most of this phase: 1.7 of 2.1 ms for 0.9 M records.
__global__ void __launch_bounds__(kThreads) k_pselect(PItem* __restrict__ items, unsigned per_item,
                                                      const float4* __restrict__ pos, int* __restrict__ hist,
                                                      int pass) {
    grid_begin();
    __shared__ int sh[kDigits];
    __shared__ int s_warp[kThreads / 32];
    __shared__ int s_flag;
    const unsigned item = blockIdx.x / per_item;
    PItem& it = items[item];
    const int begin = (int)(blockIdx.x % per_item) * kChunk;
    if (begin >= it.used) return;
    const unsigned nchunks = (unsigned)((it.used + kChunk - 1) / kChunk);
    const int shift = digit_shift(pass);
    const unsigned mask = pass == 2 ? 1023u : 2047u;
    const unsigned hi_mask = pass == 0 ? 0u : (0xFFFFFFFFu << digit_shift(pass - 1));
    const unsigned prefix = it.prefix;
    const int axis = it.axis;
    for (int i = threadIdx.x; i < kDigits; i += kThreads) sh[i] = 0;
    __syncthreads();
    const int end = min(it.used, begin + kChunk);
    for (int j = begin + threadIdx.x; j < end; j += kThreads) {
        const unsigned key = key_of(axis_of(pos[it.offset + j], axis));
        if ((key & hi_mask) == prefix) atomicAdd(&sh[(key >> shift) & mask], 1);
    }
    __syncthreads();
    int* h = hist + (size_t)item * kDigits;
    if (nchunks > 1) {
        for (int i = threadIdx.x; i < kDigits; i += kThreads)
            if (sh[i]) atomicAdd(&h[i], sh[i]);
        if (!last_chunk(it, nchunks, &s_flag)) return;
        for (int i = threadIdx.x; i < kDigits; i += kThreads) {
            sh[i] = __ldcg(&h[i]);
            h[i] = 0;
        }
        __syncthreads();
    }
    // each thread sums kDigits / kThreads neighbouring digits; a block scan
    // finds the thread, then the digit, holding rank k
    constexpr int kSpan = kDigits / kThreads;
    int sum = 0;
#pragma unroll
    for (int i = 0; i < kSpan; i++) sum += sh[threadIdx.x * kSpan + i];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    for (int w = 0; w < warp; w++) inc += s_warp[w];
    const int k = it.k;
    __syncthreads();  // every thread has read k
    int before = inc - sum;
    if (before <= k && k < inc) {
        for (int i = 0; i < kSpan; i++) {
            const int c = sh[threadIdx.x * kSpan + i];
            if (k < before + c) {
                it.prefix = prefix | ((unsigned)(threadIdx.x * kSpan + i) << shift);
                it.k = k - before;
                break;
            }
            before += c;
        }
    }
}

// Partition of every item around its selected key, one block per (item, chunk):
// < K left, > K right, == K left while the tie budget (it.k after the select)
// lasts.  The block that finishes the item's last chunk creates its children:
// a child of more than kSmall records becomes an item of the next level,
// any other one a subtree of k_psubtree (with the buffer its records are in).
__global__ void __launch_bounds__(kThreads) k_ppart(PItem* __restrict__ items, unsigned per_item,
                                                    const float4* __restrict__ pos, float4* __restrict__ out,
                                                    PItem* __restrict__ next, int next_cap,
                                                    int2* __restrict__ small, int small_cap, int out_buf,
                                                    pgx_cache_node* __restrict__ nodes, int2* __restrict__ regions,
                                                    int* __restrict__ node_region, PMisc* __restrict__ misc,
                                                    int region_max) {
    grid_begin();
    __shared__ int s_wl[kThreads / 32], s_wr[kThreads / 32];
    __shared__ int s_bl, s_br, s_flag;
    __shared__ int s_acc[12];
    const unsigned item = blockIdx.x / per_item;
    PItem& it = items[item];
    const int begin = (int)(blockIdx.x % per_item) * kChunk;
    if (begin >= it.used) return;
    const unsigned nchunks = (unsigned)((it.used + kChunk - 1) / kChunk);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 12) s_acc[threadIdx.x] = (threadIdx.x % 6) < 3 ? INT_MAX : INT_MIN;
    const int end = min(it.used, begin + kChunk);
    const int axis = it.axis, budget = it.k;
    const unsigned pivot = it.prefix;
    float4 p[kPer];
    unsigned sides = 0, have = 0;
    int nl = 0, nr = 0;
    int acc[2][6];
    for (int s = 0; s < 2; s++)
        for (int k = 0; k < 6; k++) acc[s][k] = k < 3 ? INT_MAX : INT_MIN;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const int j = begin + k * kThreads + threadIdx.x;
        if (j >= end) continue;
        have |= 1u << k;
        p[k] = pos[it.offset + j];
        const unsigned key = key_of(axis_of(p[k], axis));
        int side = key < pivot ? 0 : 1;
        if (key == pivot) side = (atomicAdd(&it.tie, 1) < budget) ? 0 : 1;
        sides |= (unsigned)side << k;
        nl += 1 - side;
        nr += side;
        const int o[3] = {f2o(p[k].x), f2o(p[k].y), f2o(p[k].z)};
#pragma unroll
        for (int s = 0; s < 2; s++)
            if (s == side)
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    acc[s][a] = min(acc[s][a], o[a]);
                    acc[s][3 + a] = max(acc[s][3 + a], o[a]);
                }
    }
    int il = nl, ir = nr;
    for (int o = 1; o < 32; o <<= 1) {
        int tl = __shfl_up_sync(0xFFFFFFFFu, il, o);
        int tr = __shfl_up_sync(0xFFFFFFFFu, ir, o);
        if (lane >= o) {
            il += tl;
            ir += tr;
        }
    }
    if (lane == 31) {
        s_wl[warp] = il;
        s_wr[warp] = ir;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int tl = 0, tr = 0;
        for (int w = 0; w < kThreads / 32; w++) {
            int a = s_wl[w], bb = s_wr[w];
            s_wl[w] = tl;
            s_wr[w] = tr;
            tl += a;
            tr += bb;
        }
        s_bl = atomicAdd(&it.lcur, tl);
        s_br = atomicAdd(&it.rcur, tr);
    }
    __syncthreads();
    int offl = it.offset + s_bl + s_wl[warp] + il - nl;
    int offr = it.offset + it.used - 1 - (s_br + s_wr[warp] + ir - nr);
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        if (!((have >> k) & 1u)) continue;
        if (((sides >> k) & 1u) == 0)
            out[offl++] = p[k];
        else
            out[offr--] = p[k];
    }
#pragma unroll
    for (int k = 0; k < 12; k++) {
        const bool mn = (k % 6) < 3;
        const int v = mn ? __reduce_min_sync(0xFFFFFFFFu, acc[k / 6][k % 6]) : __reduce_max_sync(0xFFFFFFFFu, acc[k / 6][k % 6]);
        if (lane == 0) {
            if (mn)
                atomicMin(&s_acc[k], v);
            else
                atomicMax(&s_acc[k], v);
        }
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        const int k = threadIdx.x;
        int* dst = &it.acc[k / 6][k % 6];
        if ((k % 6) < 3)
            atomicMin(dst, s_acc[k]);
        else
            atomicMax(dst, s_acc[k]);
    }
    if (!last_chunk(it, nchunks, &s_flag) || threadIdx.x != 0) return;
    const int half = it.used / 2;
    if (__ldcg(&it.lcur) != half) atomicExch(&misc->overflow, 3);
    const int c = atomicAdd(&misc->node_count, 2);
    pgx_cache_node& nd = nodes[it.node];
    nd.left = c;
    nd.right = c + 1;
    nd.used = 0;
    for (int side = 0; side < 2; side++) {
        pgx_cache_node ch;
        for (int k = 0; k < 3; k++) {
            ch.bmin[k] = o2f(__ldcg(&it.acc[side][k]));
            ch.bmax[k] = o2f(__ldcg(&it.acc[side][3 + k]));
        }
        ch.left = ch.right = -1;
        ch.offset = side ? it.offset + half : it.offset;
        ch.used = side ? it.used - half : half;
        nodes[c + side] = ch;
        if (ch.used <= region_max && it.used > region_max) {
            const int r = atomicAdd(&misc->nregions, 1);
            regions[r] = make_int2(ch.offset, ch.used);
            node_region[c + side] = r;
        }
        if (ch.used <= kSmall) {
            const int s = atomicAdd(&misc->nsmall, 1);
            if (s < small_cap)
                small[s] = make_int2(c + side, out_buf);
            else
                atomicExch(&misc->overflow, 1);
            continue;
        }
        const int q = atomicAdd(&misc->nitems_next, 1);
        if (q >= next_cap) {
            atomicExch(&misc->overflow, 2);
            continue;
        }
        start_item(next[q], c + side, ch.offset, ch.used, ch);
    }
}

// One CTA finishes the subtree of a node with at most kSmall records.  Level
// l of the subtree has 2^l slots of S = P / 2^l record places (P the power of
// two >= the record count): a slot holds one node, its records first, +inf
// keys behind them.  Per level every slot is sorted by (coordinate on the
// node's longest axis, place) with one bitonic network in shared memory; the
// first used/2 records are the left child and stay, the rest move to the
// slot's upper half (used - used/2 <= S/2, so both always fit).  A slot whose
// node is a leaf (at most 8 records) sorts too, which keeps the network
// uniform, and keeps its records in its lower places.
//   A thread holds four neighbouring places in registers: strides of 1 and 2
// stay in the thread, 4 to 64 are shuffles, and only the 20 of 276 compare
// steps with longer strides go through shared memory.
//   Bound: issue of the network (0.9 M records: 0.26 ms, and 0.33 with every
// step in shared memory).  One thread per <= 256-record subtree with an in-place
// quickselect took 5.1 ms.
constexpr int kSubThreads = 512;
constexpr int kSubSlots = kSmall / 8;  // slots of the deepest level
constexpr int kSubEach = kSmall / kSubThreads;
constexpr int kSubSmem = kSmall * (int)(sizeof(unsigned long long) + sizeof(float4));

struct SubSlot {
    int node;   // -1: empty
    int offset, used;
    int axis;   // -1: leaf or empty
};

__global__ void __launch_bounds__(kSubThreads, 3) k_psubtree(const int2* __restrict__ small, PMisc* __restrict__ misc,
                                                          const float4* __restrict__ pos0,
                                                          const float4* __restrict__ pos1, int* __restrict__ idx,
                                                          pgx_cache_node* __restrict__ nodes,
                                                          int2* __restrict__ regions, int* __restrict__ node_region,
                                                          int region_max) {
    grid_begin();
    extern __shared__ __align__(16) uint8_t s_dyn[];
    unsigned long long* xchg = reinterpret_cast<unsigned long long*>(s_dyn);  // [kSmall]: long strides, then source places
    float4* rec = reinterpret_cast<float4*>(s_dyn + sizeof(unsigned long long) * kSmall);  // [kSmall]
    __shared__ SubSlot slot[2][kSubSlots];
    __shared__ int s_acc[kSubSlots][6];
    __shared__ int s_base, s_nsplit, s_nregion, s_rbase;
    const int tid = threadIdx.x;
    const int2 job = small[blockIdx.x];
    const pgx_cache_node root = nodes[job.x];
    if (root.used <= kLeafMax) {
        const float4* src = (job.y ? pos1 : pos0) + root.offset;
        if (tid < root.used) idx[root.offset + tid] = __float_as_int(src[tid].w);
        return;
    }
    int P = 16;
    while (P < root.used) P <<= 1;
    {
        const float4* src = (job.y ? pos1 : pos0) + root.offset;
        for (int i = tid; i < P; i += kSubThreads)
            if (i < root.used) rec[i] = src[i];
    }
    if (tid == 0) slot[0][0] = SubSlot{job.x, root.offset, root.used, longest_axis(root)};
    __syncthreads();
    int cur = 0;
    for (int S = P, nslots = 1; S >= 16; S >>= 1, nslots <<= 1) {
        // Splitting nodes of this level: node ids and region ids for their children.
        if (tid == 0) {
            s_nsplit = 0;
            s_nregion = 0;
        }
        __syncthreads();
        int rank = -1, my_regions = 0, region_rank = 0;
        if (tid < nslots && slot[cur][tid].axis >= 0) {
            rank = atomicAdd(&s_nsplit, 1);
            const int used = slot[cur][tid].used;
            if (used > region_max) my_regions = (used / 2 <= region_max ? 1 : 0) + (used - used / 2 <= region_max ? 1 : 0);
            if (my_regions) region_rank = atomicAdd(&s_nregion, my_regions);
        }
        __syncthreads();
        if (s_nsplit == 0) break;  // only leaves are left
        if (tid == 0) {
            s_base = atomicAdd(&misc->node_count, 2 * s_nsplit);
            s_rbase = s_nregion ? atomicAdd(&misc->nregions, s_nregion) : 0;
        }
        // Sort keys of the slots that split; the others keep their order.
        unsigned long long key[kSubEach];
#pragma unroll
        for (int e = 0; e < kSubEach; e++) {
            const int i = tid * kSubEach + e;
            key[e] = ~0ull;
            if (i < P) {
                const SubSlot& sl = slot[cur][i / S];
                const int r = i & (S - 1);
                const unsigned k = sl.axis < 0 ? 0u : (r < sl.used ? key_of(axis_of(rec[i], sl.axis)) : 0xFFFFFFFFu);
                // place breaks ties, and puts records before the empty places
                key[e] = ((unsigned long long)k << 32) | (unsigned)r;
            }
        }
        for (int k2 = 2; k2 <= S; k2 <<= 1) {
            for (int j = k2 >> 1; j > 0; j >>= 1) {
                unsigned long long other[kSubEach];
                if (j >= 32 * kSubEach) {  // thread tid ^ (j / kSubEach), another warp
                    __syncthreads();
#pragma unroll
                    for (int e = 0; e < kSubEach; e++) xchg[e * kSubThreads + tid] = key[e];
                    __syncthreads();
#pragma unroll
                    for (int e = 0; e < kSubEach; e++) other[e] = xchg[e * kSubThreads + (tid ^ (j / kSubEach))];
                } else if (j >= kSubEach) {
#pragma unroll
                    for (int e = 0; e < kSubEach; e++) other[e] = __shfl_xor_sync(0xFFFFFFFFu, key[e], j / kSubEach);
                } else {
#pragma unroll
                    for (int e = 0; e < kSubEach; e++) other[e] = j == 2 ? key[e ^ 2] : key[e ^ 1];
                }
#pragma unroll
                for (int e = 0; e < kSubEach; e++) {
                    const int i = tid * kSubEach + e;
                    // ascending blocks of k2 alternate within a slot; the
                    // slot-wide merge (k2 == S) always ascends
                    const bool up = k2 == S || (i & k2) == 0;
                    const bool keep_min = ((i & j) == 0) == up;
                    if ((other[e] < key[e]) == keep_min) key[e] = other[e];
                }
            }
        }
        int* from_place = reinterpret_cast<int*>(xchg);
        __syncthreads();
#pragma unroll
        for (int e = 0; e < kSubEach; e++) from_place[tid * kSubEach + e] = (int)(unsigned)key[e];
        __syncthreads();
        // Children into the slot halves: place q of a half takes the record
        // ranked q (left) or used/2 + q (right).
        const int H = S >> 1;
        float4 moved[kSmall / kSubThreads];
#pragma unroll
        for (int m = 0; m < kSmall / kSubThreads; m++) {
            const int i = tid + m * kSubThreads;
            if (i >= P) continue;
            const SubSlot& sl = slot[cur][i / S];
            const int r = i & (S - 1);
            int from = -1;
            if (sl.axis >= 0) {
                const int half = sl.used / 2;
                if (r < H)
                    from = r < half ? r : -1;
                else
                    from = r - H < sl.used - half ? half + (r - H) : -1;
                if (from >= 0) moved[m] = rec[(i & ~(S - 1)) + from_place[(i & ~(S - 1)) + from]];
            } else if (r < H) {
                moved[m] = rec[i];  // a leaf (or an empty slot) stays in the lower half
            }
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < kSmall / kSubThreads; m++) {
            const int i = tid + m * kSubThreads;
            if (i < P) rec[i] = moved[m];
        }
        for (int i = tid; i < 2 * nslots; i += kSubThreads)
            for (int k = 0; k < 6; k++) s_acc[i][k] = k < 3 ? INT_MAX : INT_MIN;
        if (tid < nslots) {
            const SubSlot sl = slot[cur][tid];
            SubSlot l = sl, r = SubSlot{-1, 0, 0, -1};
            if (rank >= 0) {
                const int half = sl.used / 2;
                l = SubSlot{s_base + 2 * rank, sl.offset, half, 0};
                r = SubSlot{s_base + 2 * rank + 1, sl.offset + half, sl.used - half, 0};
                pgx_cache_node& nd = nodes[sl.node];
                nd.left = l.node;
                nd.right = r.node;
                nd.used = 0;
                int reg = s_rbase + region_rank;
                if (sl.used > region_max) {
                    if (l.used <= region_max) {
                        regions[reg] = make_int2(l.offset, l.used);
                        node_region[l.node] = reg++;
                    }
                    if (r.used <= region_max) {
                        regions[reg] = make_int2(r.offset, r.used);
                        node_region[r.node] = reg;
                    }
                }
            }
            slot[cur ^ 1][2 * tid] = l;
            slot[cur ^ 1][2 * tid + 1] = r;
        }
        __syncthreads();
        cur ^= 1;
        // Bounds of the new nodes: warp reductions over runs of places of one
        // slot (H >= 8, so a warp covers one slot or 2 or 4 whole ones).
#pragma unroll
        for (int m = 0; m < kSmall / kSubThreads; m++) {
            const int i = tid + m * kSubThreads;
            if (m * kSubThreads + (tid & ~31) >= P) continue;  // whole warps
            const int si = i < P ? i / H : 0;
            const bool in = i < P && slot[cur][si].axis == 0 && (i & (H - 1)) < slot[cur][si].used;
            int o[6];
            for (int k = 0; k < 6; k++) o[k] = k < 3 ? INT_MAX : INT_MIN;
            if (in) {
                const float4 q = rec[i];
                o[0] = o[3] = f2o(q.x);
                o[1] = o[4] = f2o(q.y);
                o[2] = o[5] = f2o(q.z);
            }
            const int width = H < 32 ? H : 32;
            for (int d = width >> 1; d > 0; d >>= 1)
                for (int k = 0; k < 6; k++) {
                    const int w = __shfl_xor_sync(0xFFFFFFFFu, o[k], d);
                    o[k] = k < 3 ? min(o[k], w) : max(o[k], w);
                }
            if ((tid & (width - 1)) == 0 && i < P && slot[cur][si].axis == 0)
                for (int k = 0; k < 6; k++) {
                    if (k < 3)
                        atomicMin(&s_acc[si][k], o[k]);
                    else
                        atomicMax(&s_acc[si][k], o[k]);
                }
        }
        __syncthreads();
        if (tid < 2 * nslots) {
            SubSlot& sl = slot[cur][tid];
            if (sl.axis == 0) {  // a node of this level
                pgx_cache_node ch;
                for (int k = 0; k < 3; k++) {
                    ch.bmin[k] = o2f(s_acc[tid][k]);
                    ch.bmax[k] = o2f(s_acc[tid][3 + k]);
                }
                ch.left = ch.right = -1;
                ch.offset = sl.offset;
                ch.used = sl.used;
                nodes[sl.node] = ch;
                sl.axis = sl.used > kLeafMax ? longest_axis(ch) : -1;
                // a leaf's records are final: its place in the leaf order
                if (sl.axis < 0)
                    for (int q = 0; q < sl.used; q++) idx[sl.offset + q] = __float_as_int(rec[tid * H + q].w);
            }
        }
        __syncthreads();
    }
}

// Default flux weight of a record: the luminance of its Li.  The quadtree
// build clamps weights at clamp_median x the region's median weight
// (pgx_guide_params; 0 = no clamp) so that a few very bright records (the
// sun seen through a specular chain) need not take the whole distribution.
__device__ __forceinline__ float record_lum(const pgx_path_vertex& v) {
    float w = ((0.2126f * v.Li[0]) + (0.7152f * v.Li[1])) + (0.0722f * v.Li[2]);
    return (isfinite(w) && w > 0.f) ? w : 0.f;
}

// Records into leaf order, with their flux weights (the given ones, the
// renderer's Lum(Li) |cos| / pdf, or Lum(Li); non-finite or negative -> 0),
// their positions, and the Morton key of the quadtree cell their wi falls
// into at the depth limit: the cylindrical map of the direction, or the
// diffuse sampler's primary sample (pss; kQtOutside below the hemisphere,
// which no cell contains).
constexpr int kQtBits = 2 * PGX_QT_MAX_DEPTH;  // two bits per level
constexpr unsigned kQtOutside = 1u << 31;

__device__ __forceinline__ unsigned spread_bits(unsigned x) {  // bit i -> bit 2i (16 bits)
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    return (x | (x << 1)) & 0x55555555u;
}

__global__ void k_gather(const pgx_path_vertex* __restrict__ in, const float* __restrict__ w_in,
                         const int* __restrict__ idx, int64_t n, pgx_path_vertex* __restrict__ out,
                         float* __restrict__ w_out, float4* __restrict__ pos, unsigned* __restrict__ key_out, int pss) {
    grid_begin();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int j = idx[i];
    const float4* src = reinterpret_cast<const float4*>(in + j);  // 48-byte records: 16-byte aligned
    const float4 a = src[0], b = src[1], c = src[2];
    float4* dst = reinterpret_cast<float4*>(out + i);
    dst[0] = a;
    dst[1] = b;
    dst[2] = c;
    pos[i] = make_float4(a.x, a.y, a.z, 0.f);  // w: the region (k_regions)
    pgx_path_vertex v;
    v.Li[0] = c.y, v.Li[1] = c.z, v.Li[2] = c.w;
    float w = w_in ? w_in[j] : record_lum(v);
    w_out[i] = (isfinite(w) && w > 0.f) ? w : 0.f;
    const F3 wi = f3(b.z, b.w, c.x);
    float u, vv;
    bool inside = true;
    if (pss)
        inside = pss_uv(f3(a.w, b.x, b.y), wi, u, vv);
    else
        dir_to_uv(wi, u, vv);
    // u, v in [0, 1): the product by a power of two and its truncation are
    // exact, so the key's digits are the comparisons u >= u0 + half of every level
    const float scale = (float)(1 << PGX_QT_MAX_DEPTH);
    key_out[i] = inside ? (spread_bits((unsigned)(u * scale)) | (spread_bits((unsigned)(vv * scale)) << 1)) : kQtOutside;
}

__global__ void k_trav(const pgx_cache_node* __restrict__ nodes, int64_t nn, CacheTravNode* __restrict__ out) {
    grid_begin();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn) return;
    const pgx_cache_node& n = nodes[i];
    CacheTravNode t;
    bool leaf = n.left < 0;
    t.bmin = make_float4(n.bmin[0], n.bmin[1], n.bmin[2], __int_as_float(leaf ? -(n.offset + 1) : n.left));
    t.bmax = make_float4(n.bmax[0], n.bmax[1], n.bmax[2], __int_as_float(leaf ? n.used : n.right));
    out[i] = t;
}

__global__ void k_regions(const int2* __restrict__ regions, int nreg, float4* __restrict__ pos) {
    grid_begin();
    int r = blockIdx.x;
    if (r >= nreg) return;
    int2 g = regions[r];
    for (int i = threadIdx.x; i < g.y; i += blockDim.x) pos[g.x + i].w = __int_as_float(r);
}

// A float sum with its rounding error carried along (Knuth's two-sum), so
// that a cell's flux does not depend on the order of its records and the
// refinement decisions are those of the exact sums.
struct PairSum {
    float s = 0.f, e = 0.f;
    __device__ __forceinline__ void add(float w) {
        const float t = s + w, z = t - s;
        e += (s - (t - z)) + (w - z);
        s = t;
    }
    __device__ __forceinline__ void warp_reduce() {
        for (int o = 16; o > 0; o >>= 1) {
            const float s2 = __shfl_xor_sync(0xFFFFFFFFu, s, o), e2 = __shfl_xor_sync(0xFFFFFFFFu, e, o);
            add(s2);
            e += e2;
        }
    }
    __device__ __forceinline__ float value() const { return s + e; }
};

// One CTA builds one region's quadtree (pgx_guide.cuh).  The records are
// sorted once by the Morton key of their cell at the depth limit (four
// stable 5-bit radix passes), after which every cell of every level is a
// contiguous range: a level sums each child cell's range with one warp, finds
// the next level's ranges by binary search and numbers the children that
// split in breadth-first order.  Work is records x depth; re-reading the
// region's records for each of up to 256 cells with one warp per region took
// 9.5 ms for 78 regions of 16,384 records.
//   Bound: latency (syncs and L2 round trips of one CTA per region).
// THREADS by region size: the regions' count, not their size, fills the GPU
// when they are small.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_quadtree(const int2* __restrict__ regions,
                                                      const unsigned* keys, const float* wts, unsigned* kbuf,
                                                      float* wbuf, int64_t n_all, int* __restrict__ qroot,
                                                      QuadNode* __restrict__ qnodes, int pss, float clamp_median, float refine, float compensate) {
    grid_begin();
    constexpr int kWarps = THREADS / 32;
    __shared__ int s_cnt[kWarps][32];
    __shared__ float s_f[kWarps], s_g[kWarps];
    __shared__ int s_i[kWarps];
    __shared__ int s_beg[PGX_QT_MAX_NODES + 1][5];        // a level's cells: child range bounds
    __shared__ float s_c[PGX_QT_MAX_NODES];
    __shared__ unsigned short s_first[PGX_QT_MAX_DEPTH + 1];  // first node of each level
    __shared__ int2 s_range[PGX_QT_MAX_NODES];
    __shared__ unsigned s_code[PGX_QT_MAX_NODES];         // Morton prefix of each node's cell
    __shared__ float s_flux[PGX_QT_MAX_NODES][4];
    __shared__ __align__(4) unsigned char s_want[PGX_QT_MAX_NODES];
    __shared__ int s_nn;
    const int r = blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned below = (1u << lane) - 1u;
    const int2 g = regions[r];
    const int n = g.y;
    const float* rw = wts + g.x;
    auto block_sum_i = [&](int v) {
        v = __reduce_add_sync(0xFFFFFFFFu, v);
        __syncthreads();
        if (lane == 0) s_i[warp] = v;
        __syncthreads();
        v = 0;
        for (int w = 0; w < kWarps; w++) v += s_i[w];
        return v;
    };
    // Median of the positive weights by bisection on the value (only needed
    // for the clamp).
    float lo = FLT_MAX, hi = 0.f;
    int pos = 0;
    for (int i = tid; i < n; i += THREADS) {
        const float w = rw[i];
        if (w > 0.f) {
            lo = fminf(lo, w);
            hi = fmaxf(hi, w);
            pos++;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
    }
    if (lane == 0) {
        s_f[warp] = lo;
        s_g[warp] = hi;
    }
    pos = block_sum_i(pos);
    for (int w = 0; w < kWarps; w++) {
        lo = fminf(lo, s_f[w]);
        hi = fmaxf(hi, s_g[w]);
    }
    if (pos == 0) {
        if (tid == 0) qroot[r] = -1;
        return;
    }
    const int half_count = (pos + 1) / 2;
    for (int it = 0; it < (clamp_median > 0.f ? 24 : 0); it++) {
        const float mid = 0.5f * (lo + hi);
        int cnt = 0;
        for (int i = tid; i < n; i += THREADS) {
            const float w = rw[i];
            if (w > 0.f && w <= mid) cnt++;
        }
        cnt = block_sum_i(cnt);
        if (cnt >= half_count)
            hi = mid;
        else
            lo = mid;
    }
    const float clamp = clamp_median > 0.f ? clamp_median * hi : FLT_MAX;
    PairSum sum;
    for (int i = tid; i < n; i += THREADS) sum.add(fminf(rw[i], clamp));
    sum.warp_reduce();
    __syncthreads();
    if (lane == 0) {
        s_f[warp] = sum.s;
        s_g[warp] = sum.e;
    }
    __syncthreads();
    sum = PairSum{};
    for (int w = 0; w < kWarps; w++) {
        sum.add(s_f[w]);
        sum.e += s_g[w];
    }
    const float total = sum.value();
    if (!(total > 0.f) || !isfinite(total)) {
        if (tid == 0) qroot[r] = -1;
        return;
    }
    // Stable LSD radix sort of (key, clamped weight); records outside the
    // domain sort last.  Every warp owns one contiguous run of a pass's input.
    const int run = ((n + kWarps - 1) / kWarps + 31) & ~31;
    const int r0 = min(n, warp * run), r1 = min(n, r0 + run);
    const unsigned* ksrc = keys + g.x;
    const float* wsrc = rw;
    bool raw = true;  // first pass: weights are clamped on the way
    // Only primary-sample records can lie outside the domain: one more pass
    // moves those behind the others.
    const int passes = kQtBits / 5 + (pss ? 1 : 0);
    for (int pass = 0; pass < passes; pass++) {
        const int shift = pass < kQtBits / 5 ? 5 * pass : 31;
        unsigned* kdst = kbuf + (size_t)(pass & 1) * n_all + g.x;
        float* wdst = wbuf + (size_t)(pass & 1) * n_all + g.x;
        __syncthreads();
        s_cnt[warp][lane] = 0;
        __syncwarp();
        for (int i = r0 + lane; i < r1; i += 32) atomicAdd(&s_cnt[warp][(ksrc[i] >> shift) & 31u], 1);
        __syncthreads();
        if (warp == 0) {  // lane = digit: exclusive offsets, digit-major then warp-major
            int sum = 0;
            for (int w = 0; w < kWarps; w++) sum += s_cnt[w][lane];
            int inc = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += t;
            }
            int at = inc - sum;
            for (int w = 0; w < kWarps; w++) {
                const int c = s_cnt[w][lane];
                s_cnt[w][lane] = at;
                at += c;
            }
        }
        __syncthreads();
        for (int b = r0; b < r1; b += 32) {
            const int i = b + lane;
            const bool in = i < r1;
            const unsigned k = in ? ksrc[i] : 0u;
            const unsigned d = in ? ((k >> shift) & 31u) : 32u;
            const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
            int at = 0;
            if (in) at = s_cnt[warp][d] + __popc(peers & below);
            __syncwarp();
            if (in) {
                if ((peers & below) == 0u) s_cnt[warp][d] += __popc(peers);
                kdst[at] = k;
                wdst[at] = raw ? fminf(wsrc[i], clamp) : wsrc[i];
            }
            __syncwarp();
        }
        __syncthreads();  // the pass's output is visible to the whole block
        ksrc = kdst;
        wsrc = wdst;
        raw = false;
    }
    // first sorted record whose key is >= bound (records outside the domain have bit 31 set)
    auto lower = [&](int a, int b, unsigned bound) {
        while (a < b) {
            const int m = (a + b) >> 1;
            if (ksrc[m] < bound)
                a = m + 1;
            else
                b = m;
        }
        return a;
    };
    QuadNode* out = qnodes + (size_t)r * PGX_QT_MAX_NODES;
    if (tid == 0) {
        s_range[0] = make_int2(0, lower(0, n, kQtOutside));
        s_code[0] = 0u;
        s_nn = 1;
        s_first[0] = 0;
    }
    __syncthreads();
    const float thresh = refine * total;
    int first = 0, nn = 1, depth = 0;
    while (first < nn) {
        const int count = nn - first;  // this level's nodes: [first, nn)
        const int shift = kQtBits - 2 * (depth + 1);
        for (int i = tid; i < count * 5; i += THREADS) {
            const int node = first + i / 5, c = i % 5;
            const int2 rg = s_range[node];
            s_beg[i / 5][c] = c == 0 ? rg.x : (c == 4 ? rg.y : lower(rg.x, rg.y, ((s_code[node] << 2) | (unsigned)c) << shift));
        }
        for (int i = tid; i < count; i += THREADS) s_want[i] = 0;  // a level can hold more nodes than THREADS
        __syncthreads();
        for (int i = warp; i < 4 * count; i += kWarps) {
            const int ni = i >> 2, c = i & 3;
            const int a = s_beg[ni][c], b = s_beg[ni][c + 1];
            PairSum cell;
            int some = 0;
            for (int k = a + lane; k < b; k += 32) {
                const float w = wsrc[k];
                cell.add(w);
                some += w > 0.f ? 1 : 0;
            }
            cell.warp_reduce();
            const float f = cell.value();
            some = __reduce_add_sync(0xFFFFFFFFu, some);
            if (lane == 0) {
                s_flux[ni][c] = f;
                if (f > thresh && some >= 2 && depth + 1 < PGX_QT_MAX_DEPTH) atomicOr(reinterpret_cast<unsigned*>(&s_want[ni & ~3]), 1u << (8 * (ni & 3) + c));
            }
        }
        __syncthreads();
        if (warp == 0) {  // number the splitting children in order while the node budget lasts
            int next = nn;
            for (int b = 0; b < count; b += 32) {
                const int ni = b + lane;
                const unsigned want = ni < count ? s_want[ni] : 0u;
                const int mine = __popc(want);
                int inc = mine;
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                    if (lane >= o) inc += t;
                }
                int at = next + inc - mine;
                if (ni < count) {
                    QuadNode q;
                    for (int c = 0; c < 4; c++) {
                        q.flux[c] = s_flux[ni][c];
                        q.child[c] = -1;
                        if ((want >> c) & 1u) {
                            if (at < PGX_QT_MAX_NODES) {
                                q.child[c] = at;
                                s_range[at] = make_int2(s_beg[ni][c], s_beg[ni][c + 1]);
                                s_code[at] = (s_code[first + ni] << 2) | (unsigned)c;
                            }
                            at++;
                        }
                    }
                    out[first + ni] = q;
                }
                next += __shfl_sync(0xFFFFFFFFu, inc, 31);
            }
            if (lane == 0) {
                s_nn = min(next, PGX_QT_MAX_NODES);
                s_first[depth + 1] = (unsigned short)nn;
            }
        }
        __syncthreads();
        first = nn;
        nn = s_nn;
        depth++;
    }
    if (compensate > 0.f && tid == 0) {
        // MIS compensation: leaves lose compensate x the mean flux over their
        // area (floored at 0); interior fluxes are the sums of their
        // children, computed leaves-up (reverse breadth-first order).
        auto depth_of = [&](int node) {
            int d = 0;
            while (d + 1 < depth && s_first[d + 1] <= node) d++;
            return d;
        };
        const QuadNode root = out[0];
        const float tot = ((root.flux[0] + root.flux[1]) + root.flux[2]) + root.flux[3];
        float* comp = s_c;
        for (int node = nn - 1; node >= 0; node--) {
            const QuadNode q = out[node];
            const float sub = compensate * tot * ldexpf(1.f, -2 * (depth_of(node) + 1));
            float sum = 0.f;
            for (int c = 0; c < 4; c++) sum += q.child[c] >= 0 ? comp[q.child[c]] : fmaxf(q.flux[c] - sub, 0.f);
            comp[node] = sum;
        }
        if (comp[0] >= 0.05f * tot) {
            for (int node = 0; node < nn; node++) {
                QuadNode q = out[node];
                const float sub = compensate * tot * ldexpf(1.f, -2 * (depth_of(node) + 1));
                for (int c = 0; c < 4; c++) q.flux[c] = q.child[c] >= 0 ? comp[q.child[c]] : fmaxf(q.flux[c] - sub, 0.f);
                out[node] = q;
            }
        }
    }
    if (tid == 0) qroot[r] = r * PGX_QT_MAX_NODES;
    // children inside the region's block of nodes: absolute indexes
    __syncthreads();
    for (int i = tid; i < nn * 4; i += THREADS) {
        int& c = out[i >> 2].child[i & 3];
        if (c >= 0) c += r * PGX_QT_MAX_NODES;
    }
}

// A warp per query shortens each query, a thread per query does more of them at
// once.  Time with a warp over time with a thread, 1 M records on the faces
// of a box, queries near them:
//   queries    k = 1    4     8     12    16    24    32    64
//     16,384   0.75  0.62  0.54  0.47  0.39  0.31  0.25  0.17
//     65,536   1.40  1.13  0.99  0.82  0.71  0.55  0.42  0.22
//    131,072   2.02  1.57  1.26  1.01  0.87  0.67  0.48  0.32
//    262,144   2.31  1.75  1.42  1.15  0.99  0.70  0.60  0.31
//  1,000,000   3.16  2.28  1.06  1.36  1.17  0.85  0.64  0.34
// (records in the box's volume: 1.1 to 1.3 times these; 1,000, 100,000 and
// 4 M records much the same).  The line runs where threads begin to win, and
// leaves lists above 16 to warps.
constexpr int kKnnThreadK = 16;
inline bool knn_per_thread(int64_t nq, int k) { return k <= kKnnThreadK && nq >= 16384 + 6144 * (int64_t)k; }

// The k nearest records of a query, ascending by distance, ties to the lower
// index: (d, i) is behind (d2, i2).
__device__ __forceinline__ bool knn_behind(float d, int i, float d2, int i2) { return d > d2 || (d == d2 && i > i2); }
__device__ __forceinline__ float knn_box(const CacheTravNode& c, float x, float y, float z) {
    const float dx = fmaxf(fmaxf(c.bmin.x - x, x - c.bmax.x), 0.f);
    const float dy = fmaxf(fmaxf(c.bmin.y - y, y - c.bmax.y), 0.f);
    const float dz = fmaxf(fmaxf(c.bmin.z - z, z - c.bmax.z), 0.f);
    return dx * dx + dy * dy + dz * dz;
}

// Many queries of few neighbours: one thread per query with its list and
// stack in local memory.
__global__ void __launch_bounds__(128) k_knn_thread(const CacheTravNode* __restrict__ nodes,
                                                    const float4* __restrict__ pos, int nrec,
                                                    const float* __restrict__ q, int64_t nq, int k,
                                                    int* __restrict__ out_i, float* __restrict__ out_d) {
    grid_begin();
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nq) return;
    const float x = q[3 * t], y = q[3 * t + 1], z = q[3 * t + 2];
    float bd[kKnnThreadK];
    int bi[kKnnThreadK];
    int cnt = 0;
    int stack[64];
    int sp = 0;
    if (nrec > 0) stack[sp++] = 0;
    while (sp > 0) {
        const CacheTravNode n = nodes[stack[--sp]];
        const float lim = cnt < k ? FLT_MAX : bd[k - 1];
        if (knn_box(n, x, y, z) > lim) continue;
        const int l = __float_as_int(n.bmin.w), r = __float_as_int(n.bmax.w);
        if (l < 0) {
            const int off = -l - 1;
            for (int id = off; id < off + r; id++) {
                const float4 p = pos[id];
                const float dx = p.x - x, dy = p.y - y, dz = p.z - z;
                const float d = dx * dx + dy * dy + dz * dz;
                if (cnt == k && !knn_behind(bd[k - 1], bi[k - 1], d, id)) continue;
                int m = cnt < k ? cnt++ : k - 1;
                for (; m > 0 && knn_behind(bd[m - 1], bi[m - 1], d, id); m--) {
                    bd[m] = bd[m - 1];
                    bi[m] = bi[m - 1];
                }
                bd[m] = d;
                bi[m] = id;
            }
        } else if (sp + 2 <= 64) {
            // the nearer child is pushed last and entered first
            const bool left_first = knn_box(nodes[l], x, y, z) < knn_box(nodes[r], x, y, z);
            stack[sp++] = left_first ? r : l;
            stack[sp++] = left_first ? l : r;
        }
    }
    for (int j = 0; j < k; j++) {
        out_i[t * k + j] = j < cnt ? bi[j] : -1;
        out_d[t * k + j] = j < cnt && bd[j] != FLT_MAX ? bd[j] : INFINITY;
    }
}

// One warp per query.  The best list lives in the lanes (entry e of lane l is rank
// 32 e + l, kept sorted); a leaf's records are tested by one lane each and the
// ones that improve the list are inserted in turn: every lane compares its
// entries, the insertion point is a popcount, and the tail moves up one lane.
// The visit order and the comparisons are those of k_knn_thread.  16,384
// queries of 8 among 0.9 M records: 140 us, and 266 with a thread each (128
// blocks of dependent local-memory accesses).
template <int E>
__global__ void __launch_bounds__(128) k_knn(const CacheTravNode* __restrict__ nodes, const float4* __restrict__ pos,
                                             int nrec, const float* __restrict__ q, int64_t nq, int k,
                                             int* __restrict__ out_i, float* __restrict__ out_d) {
    grid_begin();
    constexpr unsigned kFull = 0xFFFFFFFFu;
    __shared__ int s_stack[4][64];
    const int lane = threadIdx.x & 31;
    int* stack = s_stack[threadIdx.x >> 5];
    const int64_t t = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (t >= nq) return;  // whole warps
    const float x = q[3 * t], y = q[3 * t + 1], z = q[3 * t + 2];
    float bd[E];
    int bi[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        bd[e] = FLT_MAX;
        bi[e] = INT_MAX;
    }
    int cnt = 0;
    float worst_d = FLT_MAX;  // rank k - 1 once k records are known
    int worst_i = INT_MAX;
    if (nrec > 0) {
        int sp = 0;
        if (lane == 0) stack[0] = 0;
        sp = 1;
        while (sp > 0) {
            __syncwarp();
            const int ni = stack[--sp];
            const CacheTravNode n = nodes[ni];
            const float lim = cnt < k ? FLT_MAX : worst_d;
            if (knn_box(n, x, y, z) > lim) continue;
            const int l = __float_as_int(n.bmin.w), r = __float_as_int(n.bmax.w);
            if (l < 0) {
                const int off = -l - 1;
                for (int j0 = 0; j0 < r; j0 += 32) {
                    float d = 0.f;
                    const int id = off + j0 + lane;
                    const bool have = j0 + lane < r;
                    if (have) {
                        const float4 p = pos[id];
                        const float dx = p.x - x, dy = p.y - y, dz = p.z - z;
                        d = dx * dx + dy * dy + dz * dz;
                    }
                    unsigned todo = __ballot_sync(kFull, have);
                    while (todo) {
                        const int src = __ffs(todo) - 1;
                        todo &= todo - 1;
                        const float cd = __shfl_sync(kFull, d, src);
                        const int ci = off + j0 + src;
                        if (cnt == k && !knn_behind(worst_d, worst_i, cd, ci)) continue;
                        if (cnt < k) cnt++;
                        // entries that stay in front of the new one
                        int at = 0;
#pragma unroll
                        for (int e = 0; e < E; e++)
                            at += __popc(__ballot_sync(kFull, bi[e] != INT_MAX && !knn_behind(bd[e], bi[e], cd, ci)));
#pragma unroll
                        for (int e = E - 1; e >= 0; e--) {
                            float pd = __shfl_up_sync(kFull, bd[e], 1);
                            int pi = __shfl_up_sync(kFull, bi[e], 1);
                            if (e > 0) {  // rank 32 e takes over from the last lane of the entry before
                                const float cd2 = __shfl_sync(kFull, bd[e > 0 ? e - 1 : 0], 31);
                                const int ci2 = __shfl_sync(kFull, bi[e > 0 ? e - 1 : 0], 31);
                                if (lane == 0) {
                                    pd = cd2;
                                    pi = ci2;
                                }
                            }
                            const int rank = 32 * e + lane;
                            if (rank == at) {
                                bd[e] = cd;
                                bi[e] = ci;
                            } else if (rank > at) {
                                bd[e] = pd;
                                bi[e] = pi;
                            }
                        }
                        if (cnt == k) {
                            const int last = k - 1;
                            worst_d = __shfl_sync(kFull, E > 1 && last >= 32 ? bd[E - 1] : bd[0], last & 31);
                            worst_i = __shfl_sync(kFull, E > 1 && last >= 32 ? bi[E - 1] : bi[0], last & 31);
                        }
                    }
                }
            } else if (sp + 2 <= 64) {
                const float da = knn_box(nodes[l], x, y, z), db = knn_box(nodes[r], x, y, z);
                const bool left_first = da < db;  // the one entered first is pushed last
                __syncwarp();
                if (lane == 0) {
                    stack[sp] = left_first ? r : l;
                    stack[sp + 1] = left_first ? l : r;
                }
                sp += 2;
            }
        }
    }
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int rank = 32 * e + lane;
        if (rank < k) {
            const bool have = rank < cnt;
            out_i[t * k + rank] = have ? bi[e] : -1;
            out_d[t * k + rank] = !have || bd[e] == FLT_MAX ? INFINITY : bd[e];
        }
    }
}

// Guide pdf / sample for explicit positions (pgx_guide_pdf / _sample).
__global__ void k_guide_query(GuideView g, const float* __restrict__ pos, const float* __restrict__ in, int64_t n,
                              int sample, float* __restrict__ dirs, float* __restrict__ pdf) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    F3 x = f3(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2]);
    int root = guide_region_root(g, x);
    const float inv4pi = 1.f / (4.f * 3.14159265f);
    if (sample) {
        F3 w = f3(0.f, 0.f, 1.f);
        float p = 0.f;
        if (root >= 0) {
            float u, v;
            quad_sample(g.qnodes, root, in[2 * i], in[2 * i + 1], u, v);
            w = uv_to_dir(u, v);
            float pu, pv;
            dir_to_uv(w, pu, pv);
            p = quad_pdf(g.qnodes, root, pu, pv) * inv4pi;  // the quadtree alone
        }
        dirs[3 * i] = w.x;
        dirs[3 * i + 1] = w.y;
        dirs[3 * i + 2] = w.z;
        pdf[i] = p;
    } else {
        float p = 0.f;
        if (root >= 0) {
            float u, v;
            dir_to_uv(normalize(f3(in[3 * i], in[3 * i + 1], in[3 * i + 2])), u, v);
            p = quad_pdf(g.qnodes, root, u, v) * inv4pi;
        }
        pdf[i] = p;
    }
}

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

CacheState* cstate(pgx_ctx* ctx) {
    if (!ctx->cache_state) ctx->cache_state = new CacheState();
    return static_cast<CacheState*>(ctx->cache_state);
}

}  // namespace

void cache_state_free(pgx_ctx* ctx) {
    delete static_cast<CacheState*>(ctx->cache_state);
    ctx->cache_state = nullptr;
}

GuideView guide_view(const pgx_ctx* ctx) {
    GuideView g{};
    const CacheState* cs = static_cast<const CacheState*>(ctx->cache_state);
    if (!cs || !cs->valid || cs->n_records == 0) return g;
    g.valid = 1;
    g.n_nodes = (int)cs->n_nodes;
    g.n_records = (int)cs->n_records;
    g.nodes = cs->trav.as<CacheTravNode>();
    g.rec_pos = cs->pos.as<float4>();
    g.region_qroot = cs->qroot.as<int>();
    g.qnodes = cs->qnodes.as<QuadNode>();
    g.node_region = cs->node_region.as<int>();
    g.pss = cs->pss ? 1 : 0;
    g.uniform = ctx->guide.uniform_share;
    g.min_alpha = ctx->guide.glossy_alpha;
    return g;
}

uint64_t guide_generation(const pgx_ctx* ctx) {
    const CacheState* cs = static_cast<const CacheState*>(ctx->cache_state);
    return cs ? cs->generation : 0;
}

int guide_regions(const pgx_ctx* ctx) {
    const CacheState* cs = static_cast<const CacheState*>(ctx->cache_state);
    return (cs && cs->valid && cs->n_records > 0) ? cs->n_regions : 0;
}

bool guide_ready(const pgx_ctx* ctx) {
    const CacheState* cs = static_cast<const CacheState*>(ctx->cache_state);
    return cs && cs->valid && cs->n_records > 0;
}

// Builds the cache from n records already on the device.
int cache_build_device(pgx_ctx* ctx, const pgx_path_vertex* d_records, int64_t n, bool pss,
                       const float* d_weights) {
    CacheState* cs = cstate(ctx);
    cs->valid = false;
    cs->generation++;
    cs->pss = pss;
    if (n < 0 || n > (int64_t)INT32_MAX / 2) return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "cache: bad record count");
    auto t0 = std::chrono::steady_clock::now();
    cudaStream_t s = ctx->stream;
    cs->n_records = n;
    cs->n_nodes = 0;
    cs->n_regions = 0;
    if (n == 0) {
        cs->valid = true;
        return PGX_OK;
    }
    // Every split is at used/2, so the sizes of the nodes of a level are one
    // or two neighbouring numbers, and the counts of nodes, of large nodes per
    // level, of subtrees and of regions follow from n alone.
    const int region_max = ctx->guide.region_records;
    struct Level {
        int64_t items, max_used;
    };
    std::vector<Level> levels;
    int64_t nsmall = n <= kSmall ? 1 : 0, total_nodes = 1, nregions = n <= region_max ? 1 : 0;
    for (std::map<int64_t, int64_t> sizes{{n, 1}}; !sizes.empty();) {
        std::map<int64_t, int64_t> next;
        Level lv{0, 0};
        for (const auto& [used, count] : sizes) {
            if (used <= kLeafMax) continue;
            total_nodes += 2 * count;
            if (used > kSmall) {
                lv.items += count;
                lv.max_used = std::max(lv.max_used, used);
            }
            for (const int64_t child : {used / 2, used - used / 2}) {
                next[child] += count;
                if (used > kSmall && child <= kSmall) nsmall += count;
                if (used > region_max && child <= region_max) nregions += count;
            }
        }
        if (lv.items) levels.push_back(lv);
        sizes.swap(next);
    }
    int64_t item_cap = 1;
    for (const Level& lv : levels) item_cap = std::max(item_cap, lv.items);
    const int64_t max_nodes = total_nodes;
    // Parameters of this build (later pgx_guide_configure calls shape the next one).
    const float clamp_median = ctx->guide.clamp_median, refine = ctx->guide.refine_fraction;
    const float compensate = ctx->guide.compensate;
    PGX_CUDA_TRY(ctx, cs->recs_in.reserve(sizeof(pgx_path_vertex) * n));
    PGX_CUDA_TRY(ctx, cs->recs.reserve(sizeof(pgx_path_vertex) * n));
    PGX_CUDA_TRY(ctx, cs->wts.reserve(sizeof(float) * n));
    PGX_CUDA_TRY(ctx, cs->qkey.reserve(4 * sizeof(float) * n));
    if (d_weights) {
        PGX_CUDA_TRY(ctx, cs->wts_in.reserve(sizeof(float) * n));
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(cs->wts_in.p, d_weights, sizeof(float) * n, cudaMemcpyDeviceToDevice,
                                          ctx->stream));
    }
    PGX_CUDA_TRY(ctx, cs->pos.reserve(sizeof(float4) * n));
    PGX_CUDA_TRY(ctx, cs->pos2.reserve(sizeof(float4) * n));
    PGX_CUDA_TRY(ctx, cs->idx.reserve(sizeof(int) * n));
    PGX_CUDA_TRY(ctx, cs->nodes.reserve(sizeof(pgx_cache_node) * max_nodes));
    PGX_CUDA_TRY(ctx, cs->trav.reserve(sizeof(CacheTravNode) * max_nodes));
    PGX_CUDA_TRY(ctx, cs->items.reserve(sizeof(PItem) * item_cap));
    PGX_CUDA_TRY(ctx, cs->items2.reserve(sizeof(PItem) * item_cap));
    PGX_CUDA_TRY(ctx, cs->hist.reserve(sizeof(int) * kDigits * item_cap));
    PGX_CUDA_TRY(ctx, cs->small.reserve(sizeof(int2) * std::max<int64_t>(nsmall, 1)));
    PGX_CUDA_TRY(ctx, cs->misc.reserve(sizeof(PMisc) + sizeof(int) * 8));
    PGX_CUDA_TRY(ctx, cs->regions.reserve(sizeof(int2) * nregions));
    PGX_CUDA_TRY(ctx, cs->node_region.reserve(sizeof(int) * max_nodes));
    PGX_CUDA_TRY(ctx, cs->qroot.reserve(sizeof(int) * nregions));
    PGX_CUDA_TRY(ctx, cs->qnodes.reserve(sizeof(QuadNode) * PGX_QT_MAX_NODES * (size_t)nregions));
    // -1 everywhere; region roots get their region index (the root: region 0
    // when the whole cache is one region).
    PGX_CUDA_TRY(ctx, cudaMemsetAsync(cs->node_region.p, 0xFF, sizeof(int) * max_nodes, s));
    if (n <= region_max) PGX_CUDA_TRY(ctx, cudaMemsetAsync(cs->node_region.p, 0, sizeof(int), s));
    if (d_records != cs->recs_in.as<pgx_path_vertex>())
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(cs->recs_in.p, d_records, sizeof(pgx_path_vertex) * n,
                                          cudaMemcpyDeviceToDevice, s));
    float4* pos = cs->pos.as<float4>();
    float4* pos2 = cs->pos2.as<float4>();
    int* idx = cs->idx.as<int>();
    pgx_cache_node* nodes = cs->nodes.as<pgx_cache_node>();
    PItem* items = cs->items.as<PItem>();
    PItem* items2 = cs->items2.as<PItem>();
    int* hist = cs->hist.as<int>();
    int2* small = cs->small.as<int2>();
    PMisc* misc = cs->misc.as<PMisc>();
    int* acc = reinterpret_cast<int*>(misc + 1);
    int2* regions = cs->regions.as<int2>();

    launch_behind(k_bounds_init, 1, 32, 0, s, acc);
    launch_behind(k_pos, std::min<unsigned>(blocks_for(n, 256), 8 * pgx_num_sms()), 256, 0, s,
                  cs->recs_in.as<pgx_path_vertex>(), n, pos, acc);
    launch_behind(k_root, 1, 32, 0, s, n, misc, nodes, items, small, acc);
    PGX_CUDA_TRY(ctx, cudaMemsetAsync(hist, 0, sizeof(int) * kDigits * item_cap, s));
    PGX_CUDA_TRY(ctx, cudaGetLastError());
    float4 *src = pos, *dst = pos2;
    int dst_buf = 1;
    for (const Level& lv : levels) {
        const int64_t per_item = (lv.max_used + kChunk - 1) / kChunk;
        if (per_item * lv.items > (int64_t)INT32_MAX) return pgx_fail(ctx, PGX_ERR_OVERFLOW, "cache build: too many records");
        const unsigned grid = (unsigned)(per_item * lv.items);
        PGX_CUDA_TRY(ctx, cudaMemsetAsync(&misc->nitems_next, 0, sizeof(int), s));
        for (int pass = 0; pass < kPasses; pass++)
            launch_behind(k_pselect, grid, kThreads, 0, s, items, (unsigned)per_item, src, hist, pass);
        launch_behind(k_ppart, grid, kThreads, 0, s, items, (unsigned)per_item, src, dst, items2, (int)item_cap,
                      small, (int)nsmall, dst_buf, nodes, regions, cs->node_region.as<int>(), misc, region_max);
        std::swap(items, items2);
        std::swap(src, dst);
        dst_buf ^= 1;
    }
    PGX_CUDA_TRY(ctx, cudaFuncSetAttribute(k_psubtree, cudaFuncAttributeMaxDynamicSharedMemorySize, kSubSmem));
    launch_behind(k_psubtree, (unsigned)nsmall, kSubThreads, kSubSmem, s, small, misc, pos, pos2, idx, nodes, regions,
                  cs->node_region.as<int>(), region_max);
    PGX_CUDA_TRY(ctx, cudaGetLastError());
    cs->n_nodes = total_nodes;
    cs->n_regions = (int)nregions;
    if (n <= region_max) {
        const int2 r0 = make_int2(0, (int)n);
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(regions, &r0, sizeof(r0), cudaMemcpyHostToDevice, s));
    }
    pgx_path_vertex* recs = cs->recs.as<pgx_path_vertex>();
    unsigned* qkey = cs->qkey.as<unsigned>();
    // the keys in leaf order start in the buffer that the sort's second pass
    // overwrites, once its first pass has read them
    unsigned* keys = qkey + n;
    launch_behind(k_gather, blocks_for(n, 256), 256, 0, s, cs->recs_in.as<pgx_path_vertex>(),
                  d_weights ? cs->wts_in.as<float>() : nullptr, idx, n, recs, cs->wts.as<float>(), pos, keys,
                  pss ? 1 : 0);
    launch_behind(k_trav, blocks_for(cs->n_nodes, 256), 256, 0, s, nodes, cs->n_nodes, cs->trav.as<CacheTravNode>());
    // Records carry their region id; leaves below regions are inside them.
    launch_behind(k_regions, (unsigned)nregions, 128, 0, s, regions, cs->n_regions, pos);
    float* wbuf = reinterpret_cast<float*>(qkey + 2 * n);
    // 512 threads keep a region's serial passes short; small regions are many
    // and need no more than 128 (1,024 records: 8 a thread).
    auto quad = region_max <= 2048 ? k_quadtree<128> : k_quadtree<512>;
    launch_behind(quad, (unsigned)nregions, region_max <= 2048 ? 128 : 512, 0, s, regions, keys, cs->wts.as<float>(),
                  qkey, wbuf, n, cs->qroot.as<int>(), cs->qnodes.as<QuadNode>(), pss ? 1 : 0, clamp_median, refine,
                  compensate);
    PGX_CUDA_TRY(ctx, cudaGetLastError());
    PMisc hm{};
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(&hm, misc, sizeof(hm), cudaMemcpyDeviceToHost, s));
    PGX_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    if (hm.overflow || hm.node_count != total_nodes || (n > region_max && hm.nregions != nregions))
        return pgx_fail(ctx, PGX_ERR_OVERFLOW, "cache build: internal overflow (%d)", hm.overflow);
    cs->valid = true;
    cs->build_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return PGX_OK;
}

int64_t render_vertex_count(pgx_ctx* ctx);
const pgx_path_vertex* render_vertices(pgx_ctx* ctx);
const float* render_vertex_weights(pgx_ctx* ctx);

extern "C" int pgx_cache_build(pgx_ctx* ctx, const pgx_path_vertex* records, int64_t n) {
    if (!ctx) return PGX_ERR_INVALID_ARG;
    ctx->err.clear();
    if (n < 0 || (n > 0 && !records)) return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_cache_build: bad arguments");
    PGX_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    CacheState* cs = cstate(ctx);
    PGX_CUDA_TRY(ctx, cs->recs_in.reserve(sizeof(pgx_path_vertex) * std::max<int64_t>(n, 1)));
    if (n > 0)
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(cs->recs_in.p, records, sizeof(pgx_path_vertex) * n, cudaMemcpyHostToDevice,
                                          ctx->stream));
    return cache_build_device(ctx, cs->recs_in.as<pgx_path_vertex>(), n);
}

extern "C" int pgx_cache_build_from_render(pgx_ctx* ctx) {
    if (!ctx) return PGX_ERR_INVALID_ARG;
    ctx->err.clear();
    const pgx_path_vertex* v = render_vertices(ctx);
    int64_t n = render_vertex_count(ctx);
    if (!v) return pgx_fail(ctx, PGX_ERR_STATE, "pgx_cache_build_from_render: no recorded path vertices");
    return cache_build_device(ctx, v, n, false, render_vertex_weights(ctx));
}

extern "C" int pgx_cache_get_stats(pgx_ctx* ctx, pgx_cache_stats* out) {
    if (!ctx || !out) return PGX_ERR_INVALID_ARG;
    ctx->err.clear();
    CacheState* cs = static_cast<CacheState*>(ctx->cache_state);
    if (!cs || !cs->valid) return pgx_fail(ctx, PGX_ERR_STATE, "pgx_cache_get_stats: no cache");
    *out = pgx_cache_stats{};
    out->records = cs->n_records;
    out->nodes = cs->n_nodes;
    out->build_ms = cs->build_ms;
    if (cs->n_nodes == 0) return PGX_OK;
    std::vector<pgx_cache_node> nodes((size_t)cs->n_nodes);
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(nodes.data(), cs->nodes.p, sizeof(pgx_cache_node) * nodes.size(),
                                      cudaMemcpyDeviceToHost, ctx->stream));
    PGX_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    // PointBVHNode::stats (Renderer.h:163-177,219-233).
    std::vector<std::pair<int, int>> st{{0, 0}};
    int mn = INT32_MAX, mx = -INT32_MAX;
    long long sum = 0;
    while (!st.empty()) {
        auto [i, d] = st.back();
        st.pop_back();
        const pgx_cache_node& nd = nodes[(size_t)i];
        if (nd.left < 0) {
            out->leaves++;
            mn = std::min(mn, d);
            mx = std::max(mx, d);
            sum += d;
        } else {
            st.push_back({nd.right, d + 1});
            st.push_back({nd.left, d + 1});
        }
    }
    out->min_leaf_depth = mn;
    out->max_leaf_depth = mx;
    out->mean_leaf_depth = out->leaves ? (double)sum / (double)out->leaves : 0.0;
    return PGX_OK;
}

extern "C" int pgx_cache_export(pgx_ctx* ctx, pgx_cache_node* nodes, int64_t* nnodes, pgx_path_vertex* records,
                                int64_t* nrecords) {
    if (!ctx) return PGX_ERR_INVALID_ARG;
    ctx->err.clear();
    CacheState* cs = static_cast<CacheState*>(ctx->cache_state);
    if (!cs || !cs->valid) return pgx_fail(ctx, PGX_ERR_STATE, "pgx_cache_export: no cache");
    if (nnodes) *nnodes = cs->n_nodes;
    if (nrecords) *nrecords = cs->n_records;
    if (nodes && cs->n_nodes > 0)
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(nodes, cs->nodes.p, sizeof(pgx_cache_node) * cs->n_nodes,
                                          cudaMemcpyDeviceToHost, ctx->stream));
    if (records && cs->n_records > 0)
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(records, cs->recs.p, sizeof(pgx_path_vertex) * cs->n_records,
                                          cudaMemcpyDeviceToHost, ctx->stream));
    PGX_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return PGX_OK;
}

extern "C" int pgx_cache_export_weights(pgx_ctx* ctx, float* weights, int64_t* nrecords) {
    if (!ctx) return PGX_ERR_INVALID_ARG;
    ctx->err.clear();
    CacheState* cs = static_cast<CacheState*>(ctx->cache_state);
    if (!cs || !cs->valid) return pgx_fail(ctx, PGX_ERR_STATE, "pgx_cache_export_weights: no cache");
    if (nrecords) *nrecords = cs->n_records;
    if (weights && cs->n_records > 0) {
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(weights, cs->wts.p, sizeof(float) * cs->n_records, cudaMemcpyDeviceToHost,
                                          ctx->stream));
        PGX_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return PGX_OK;
}

extern "C" int pgx_cache_knn(pgx_ctx* ctx, const float* queries, int64_t nq, int32_t k, int32_t* idx, float* d2) {
    if (!ctx) return PGX_ERR_INVALID_ARG;
    ctx->err.clear();
    if (nq < 0 || k < 1 || k > 64 || (nq > 0 && (!queries || !idx || !d2)))
        return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_cache_knn: bad arguments (1 <= k <= 64)");
    CacheState* cs = static_cast<CacheState*>(ctx->cache_state);
    if (!cs || !cs->valid) return pgx_fail(ctx, PGX_ERR_STATE, "pgx_cache_knn: no cache");
    if (nq == 0) return PGX_OK;
    cudaStream_t s = ctx->stream;
    PGX_CUDA_TRY(ctx, cs->knn_q.reserve(sizeof(float) * 3 * nq));
    PGX_CUDA_TRY(ctx, cs->knn_i.reserve(sizeof(int) * k * nq));
    PGX_CUDA_TRY(ctx, cs->knn_d.reserve(sizeof(float) * k * nq));
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(cs->knn_q.p, queries, sizeof(float) * 3 * nq, cudaMemcpyHostToDevice, s));
    const bool per_thread = knn_per_thread(nq, k);
    auto knn = per_thread ? k_knn_thread : (k <= 32 ? k_knn<1> : k_knn<2>);
    launch_behind(knn, blocks_for(nq, per_thread ? 128 : 4), 128, 0, s, cs->trav.as<CacheTravNode>(), cs->pos.as<float4>(),
                  (int)cs->n_records, cs->knn_q.as<float>(), nq, k, cs->knn_i.as<int>(), cs->knn_d.as<float>());
    PGX_CUDA_TRY(ctx, cudaGetLastError());
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(idx, cs->knn_i.p, sizeof(int) * k * nq, cudaMemcpyDeviceToHost, s));
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(d2, cs->knn_d.p, sizeof(float) * k * nq, cudaMemcpyDeviceToHost, s));
    PGX_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    return PGX_OK;
}

static int guide_query(pgx_ctx* ctx, const float* positions, const float* in, int64_t n, int sample, float* dirs,
                       float* pdf) {
    if (!ctx) return PGX_ERR_INVALID_ARG;
    ctx->err.clear();
    if (n < 0 || (n > 0 && (!positions || !in || !pdf || (sample && !dirs))))
        return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_guide_*: bad arguments");
    if (!guide_ready(ctx)) return pgx_fail(ctx, PGX_ERR_STATE, "pgx_guide_*: no radiance cache");
    if (cstate(ctx)->pss)
        return pgx_fail(ctx, PGX_ERR_STATE,
                        "pgx_guide_*: the cache was built by a PGX_MODE_GUIDED_PSS render (primary-sample trees)");
    if (n == 0) return PGX_OK;
    cudaStream_t s = ctx->stream;
    const size_t in_floats = sample ? 2 : 3;
    DevBuf dp, di, dd, dpdf;
    PGX_CUDA_TRY(ctx, dp.reserve(sizeof(float) * 3 * n));
    PGX_CUDA_TRY(ctx, di.reserve(sizeof(float) * in_floats * n));
    PGX_CUDA_TRY(ctx, dd.reserve(sizeof(float) * 3 * n));
    PGX_CUDA_TRY(ctx, dpdf.reserve(sizeof(float) * n));
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(dp.p, positions, sizeof(float) * 3 * n, cudaMemcpyHostToDevice, s));
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(di.p, in, sizeof(float) * in_floats * n, cudaMemcpyHostToDevice, s));
    k_guide_query<<<blocks_for(n, 128), 128, 0, s>>>(guide_view(ctx), dp.as<float>(), di.as<float>(), n, sample,
                                                      dd.as<float>(), dpdf.as<float>());
    PGX_CUDA_TRY(ctx, cudaGetLastError());
    if (sample) PGX_CUDA_TRY(ctx, cudaMemcpyAsync(dirs, dd.p, sizeof(float) * 3 * n, cudaMemcpyDeviceToHost, s));
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(pdf, dpdf.p, sizeof(float) * n, cudaMemcpyDeviceToHost, s));
    PGX_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    return PGX_OK;
}

extern "C" int pgx_guide_pdf(pgx_ctx* ctx, const float* positions, const float* dirs, int64_t n, float* pdf) {
    return guide_query(ctx, positions, dirs, n, 0, nullptr, pdf);
}

extern "C" int pgx_guide_sample(pgx_ctx* ctx, const float* positions, const float* u2, int64_t n, float* dirs,
                                float* pdf) {
    return guide_query(ctx, positions, u2, n, 1, dirs, pdf);
}

extern "C" int pgx_guide_configure(pgx_ctx* ctx, const pgx_guide_params* params) {
    if (!ctx) return PGX_ERR_INVALID_ARG;
    ctx->err.clear();
    const pgx_guide_params defaults{1024, 0.01f, 10.f, 0.2f, 0.f, 0.f};
    const pgx_guide_params p = params ? *params : defaults;
    if (p.region_records < 256 || p.region_records > (1 << 20))
        return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_guide_configure: region_records %d outside [256, 2^20]",
                        (int)p.region_records);
    if (!(p.refine_fraction > 0.f && p.refine_fraction <= 1.f))
        return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_guide_configure: refine_fraction must be in (0, 1]");
    if (!(p.clamp_median >= 0.f) || !std::isfinite(p.clamp_median))
        return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_guide_configure: clamp_median must be finite and >= 0");
    if (!(p.uniform_share >= 0.f && p.uniform_share < 1.f))
        return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_guide_configure: uniform_share must be in [0, 1)");
    if (!(p.compensate >= 0.f && p.compensate <= 4.f))
        return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_guide_configure: compensate must be in [0, 4]");
    if (!(p.glossy_alpha >= 0.f) || !std::isfinite(p.glossy_alpha))
        return pgx_fail(ctx, PGX_ERR_INVALID_ARG, "pgx_guide_configure: glossy_alpha must be finite and >= 0");
    ctx->guide = p;
    return PGX_OK;
}

extern "C" int pgx_guide_get_params(pgx_ctx* ctx, pgx_guide_params* out) {
    if (!ctx || !out) return PGX_ERR_INVALID_ARG;
    *out = ctx->guide;
    return PGX_OK;
}

extern "C" int pgx_guide_export(pgx_ctx* ctx, pgx_guide_region* regions, int32_t* nregions, pgx_quad_node* qnodes,
                                int32_t* pss) {
    if (!ctx || !nregions) return PGX_ERR_INVALID_ARG;
    ctx->err.clear();
    CacheState* cs = static_cast<CacheState*>(ctx->cache_state);
    if (!cs || !cs->valid) return pgx_fail(ctx, PGX_ERR_STATE, "pgx_guide_export: no cache");
    static_assert(sizeof(pgx_quad_node) == sizeof(QuadNode), "quad node layouts differ");
    static_assert(PGX_QT_MAX_NODES == PGX_GUIDE_MAX_QUAD_NODES, "quad node capacity differs");
    const int nreg = cs->n_records > 0 ? cs->n_regions : 0;
    *nregions = nreg;
    if (pss) *pss = cs->pss ? 1 : 0;
    if (!regions || nreg == 0) return PGX_OK;
    cudaStream_t s = ctx->stream;
    std::vector<int2> rg((size_t)nreg);
    std::vector<int> qr((size_t)nreg);
    std::vector<int> nr((size_t)cs->n_nodes);
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(rg.data(), cs->regions.p, sizeof(int2) * nreg, cudaMemcpyDeviceToHost, s));
    PGX_CUDA_TRY(ctx, cudaMemcpyAsync(qr.data(), cs->qroot.p, sizeof(int) * nreg, cudaMemcpyDeviceToHost, s));
    if (cs->n_nodes > 0)
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(nr.data(), cs->node_region.p, sizeof(int) * nr.size(),
                                          cudaMemcpyDeviceToHost, s));
    if (qnodes)
        PGX_CUDA_TRY(ctx, cudaMemcpyAsync(qnodes, cs->qnodes.p, sizeof(QuadNode) * PGX_QT_MAX_NODES * (size_t)nreg,
                                          cudaMemcpyDeviceToHost, s));
    PGX_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    for (int r = 0; r < nreg; r++) regions[r] = pgx_guide_region{rg[(size_t)r].x, rg[(size_t)r].y, -1, qr[(size_t)r]};
    for (size_t i = 0; i < nr.size(); i++)
        if (nr[i] >= 0 && nr[i] < nreg) regions[nr[i]].node = (int32_t)i;
    return PGX_OK;
}
