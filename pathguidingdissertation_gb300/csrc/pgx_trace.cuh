// Stack traversal of the binary BVH: closest hit (BVHNode::traverse,
// Geometry.h:455-512) and any hit (BVHNode::traverseVisible,
// Geometry.h:514-567).
//
// The visit order is the reference's: at an interior node both child boxes
// are tested, a child whose entry distance is >= the current t (or maxT) is
// dropped, the nearer child is entered (the left one on ties), the farther
// one is pushed, and popped nodes are entered without re-testing their box.
// Triangles of a leaf are tested in index order and a hit replaces the best
// one only when 1e-4 < t < best, so ties keep the first triangle visited.
// Box and triangle arithmetic is exact (pgx_device.cuh), hence hits are
// bit-identical to the reference on the same tree.
//
// The stack's depth is checked against PGX_STACK_SIZE: an overflow ends the
// ray with status 1 instead of writing out of bounds (the reference pushes
// unchecked, Geometry.h:509).
#pragma once

#include "pgx_device.cuh"

struct BvhView {
    const TravNode* __restrict__ nodes;
    const TravTri* __restrict__ tris;
    TravRoot root;
};

// 32 bytes through the read-only path in one 256-bit load (sm_100 and
// later); p must be 32-byte aligned.
__device__ __forceinline__ void ldg_256(const void* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// One child of a node record as the slab test wants it.
struct ChildView {
    P2 mnxy, mxxy, z;
    int ref, cnt;
};

// A child in one 256-bit load of its sector: every lane of a warp reads its
// own node, so the load instructions and L1 requests per node matter.  Records
// are 64 bytes in a cudaMalloc'd (256-byte aligned) array.
__device__ __forceinline__ ChildView load_child(const TravChild* __restrict__ p) {
    ChildView c;
    unsigned long long w;
    asm("ld.global.nc.v4.b64 {%0,%1,%2,%3}, [%4];"
        : "=l"(c.mnxy.v), "=l"(c.mxxy.v), "=l"(c.z.v), "=l"(w)
        : "l"(p));
    c.ref = (int)(unsigned)w;
    c.cnt = (int)(w >> 32);
    return c;
}

// A ray as the packed slab test reads it.
struct RayPack {
    P2 oxy, ozz, ixy, izz;
};
__device__ __forceinline__ RayPack ray_pack(const xv3& o, const xv3& inv) {
    return RayPack{pack2(o.x, o.y), pack2(o.z, o.z), pack2(inv.x, inv.y), pack2(inv.z, inv.z)};
}

// Entry distance of a child's box, FLT_MAX when it is missed or not nearer
// than lim; rays with a finite inverse direction (slab_packed).
__device__ __forceinline__ float child_entry(const ChildView& c, const RayPack& r, float lim) {
    float t;
    const bool hit = slab_packed(c.mnxy, c.mxxy, c.z, r.oxy, r.ozz, r.ixy, r.izz, t);
    return hit && t < lim ? t : FLT_MAX;
}
// The same for any ray, with the reference's order of min/max operands.
__device__ __forceinline__ float child_entry_exact(const ChildView& c, const RayPack& rp, float lim) {
    float v[6], t = 0.f, dup;
    xv3 o, inv;
    unpack2(rp.oxy, o.x, o.y);
    unpack2(rp.ozz, o.z, dup);
    unpack2(rp.ixy, inv.x, inv.y);
    unpack2(rp.izz, inv.z, dup);
    unpack2(c.mnxy, v[0], v[1]);
    unpack2(c.mxxy, v[2], v[3]);
    unpack2(c.z, v[4], v[5]);
    const bool hit = ray_box(v[0], v[1], v[4], v[2], v[3], v[5], o, inv, t);
    return hit && t < lim ? t : FLT_MAX;
}

// One triangle of the leaf-ordered array: 256-bit load of v0 and e0, 128-bit
// load of e1.
__device__ __forceinline__ void load_tri(const TravTri* __restrict__ t, float4& v0, float4& e0, float4& e1) {
    const float4* tp = reinterpret_cast<const float4*>(t);
    ldg_256(tp, v0, e0);
    e1 = __ldg(tp + 2);
}

// Closest hit (ANY = false) or any hit (ANY = true) of one ray by one thread.
// Returns: for ANY, 1 when an occluder was found (not visible); otherwise
// the hit fields are updated.  `status` gets 1 on stack overflow.  Node and
// triangle references need no check: pgx_bvh_build makes them and
// pgx_bvh_import refuses a tree holding one out of range.
template <bool ANY>
__device__ __forceinline__ bool bvh_trace(const BvhView& bvh, const xv3& o, const xv3& d, float tmax, int& hit_id,
                                          float& hit_t, float& hit_u, float& hit_v, int& status) {
    hit_id = -1;
    hit_t = tmax;
    hit_u = hit_v = 0.f;
    status = 0;
    bool occluded = false;
    const xv3 inv = mk(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
    float tb;
    if (bvh.root.valid &&
        ray_box(bvh.root.bmin[0], bvh.root.bmin[1], bvh.root.bmin[2], bvh.root.bmax[0], bvh.root.bmax[1],
                bvh.root.bmax[2], o, inv, tb) &&
        !(tb > tmax)) {
        const bool finite = isfinite(inv.x) && isfinite(inv.y) && isfinite(inv.z);
        const RayPack rp = ray_pack(o, inv);
        int2 stack[PGX_STACK_SIZE];
        int sp = 0;
        int ref = bvh.root.ref;
        int cnt = bvh.root.count;
        for (;;) {
            if (cnt > 0) {
                // Leaf: test its triangles in order.
                for (int k = 0; k < cnt; k++) {
                    float4 a, b, c;
                    load_tri(bvh.tris + ref + k, a, b, c);
                    float t, u, v;
                    if (ray_tri(mk(a), mk(b), mk(c), o, d, t, u, v) && t > PGX_EPSILON && t < hit_t) {
                        hit_id = __float_as_int(a.w);
                        if (ANY) {
                            occluded = true;
                            break;
                        }
                        hit_t = t;
                        hit_u = u;
                        hit_v = v;
                    }
                }
                if ((ANY && occluded) || sp == 0) break;
                const int2 e = stack[--sp];
                ref = e.x;
                cnt = e.y;
                continue;
            }
            const TravNode* node = bvh.nodes + ref;
            const ChildView l = load_child(&node->l), r = load_child(&node->r);
            float dl, dr;
            if (finite) {
                dl = child_entry(l, rp, hit_t);
                dr = child_entry(r, rp, hit_t);
            } else {
                dl = child_entry_exact(l, rp, hit_t);
                dr = child_entry_exact(r, rp, hit_t);
            }
            const bool swap = dl > dr;
            const float dn = swap ? dr : dl, df = swap ? dl : dr;
            if (dn == FLT_MAX) {
                if (sp == 0) break;
                const int2 e = stack[--sp];
                ref = e.x;
                cnt = e.y;
            } else {
                ref = swap ? r.ref : l.ref;
                cnt = swap ? r.cnt : l.cnt;
                if (df != FLT_MAX) {
                    if (sp >= PGX_STACK_SIZE) {
                        status = 1;
                        break;
                    }
                    stack[sp++] = make_int2(swap ? l.ref : r.ref, swap ? l.cnt : r.cnt);
                }
            }
        }
    }
    return occluded;
}

// ---- persistent traversal with lane refill ----------------------------------
// Stack of one lane of the persistent traversal (PGX_STACK_SIZE entries, the
// reference's depth): the top SHORT entries live in shared memory (one column
// per thread of the block, so a warp's accesses fall in distinct banks),
// deeper ones spill to local memory.  SHORT trades shared memory (8 bytes x
// 128 threads per entry, so resident blocks) against local-memory traffic;
// the batch autotuner picks it from kShortStackChoices.
constexpr int kShortStack = 8;
constexpr int kShortStackChoices[] = {4, 8, 16};
constexpr int kTraceMaxBlock = 128;  // block size of every kernel using trace_persistent
template <int SHORT = kShortStack>
struct TraceStack {
    int2* sh;  // this thread's column: entry i at sh[i * kTraceMaxBlock]
    int2 loc[PGX_STACK_SIZE - SHORT];
    __device__ __forceinline__ void put(int i, int2 v) {
        if (i < SHORT)
            sh[i * kTraceMaxBlock] = v;
        else
            loc[i - SHORT] = v;
    }
    __device__ __forceinline__ int2 get(int i) const { return i < SHORT ? sh[i * kTraceMaxBlock] : loc[i - SHORT]; }
};

// What the rays of a launch ask for; a mixed launch holds both kinds and each
// lane knows its own.
enum TraceKind { kTraceClosest, kTraceAny, kTraceMixed };

// The same per-ray algorithm as bvh_trace, cut into steps (interior nodes
// and single triangles) so that a warp can keep stepping while its lanes
// finish at different times: lanes whose ray is done take the next ray index
// from a global counter (warp-aggregated atomicAdd) once enough of them are
// idle.  Each ray still visits its nodes and triangles in exactly bvh_trace's
// order, so results are identical; only which rays share a warp instruction
// changes.
struct TraceLane {
    RayPack rp;   // origin and inverse direction
    xv3 d;
    float tmax;   // any hit: the visibility limit; closest: the current best t
    float hu, hv;
    int hit_id;
    int ref;      // node record, or the next triangle's position (cnt > 0)
    int cnt;      // triangles left in the current leaf; 0: interior node; -1: idle
    int sp;
    int status;
    bool finite;  // every component of the inverse direction is finite (see slab_packed)
    bool any;     // mixed launches: this ray stops at the first hit
    unsigned ni, nt;  // counting launches: this ray's nodes and triangles
};

// The tree's own root for every ray (one scene).
struct SceneRoot {
    __device__ __forceinline__ const TravRoot& operator()(unsigned, const BvhView& bvh) const { return bvh.root; }
};

// Starts a ray at `root`; leaves the lane idle when the root box is missed.
template <TraceKind KIND>
__device__ __forceinline__ void lane_start(const TravRoot& root, TraceLane& L, xv3 o, xv3 d,
                                           float tmax) {
    L.d = d;
    L.tmax = tmax;
    L.hit_id = -1;
    L.hu = 0.f;
    L.hv = 0.f;
    L.sp = 0;
    L.status = 0;
    L.ni = L.nt = 0;
    L.cnt = -1;
    if (!root.valid) return;
    const xv3 inv = mk(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));  // 1 / d, correctly rounded
    L.rp = ray_pack(o, inv);
    L.finite = isfinite(inv.x) && isfinite(inv.y) && isfinite(inv.z);
    float tb;
    if (!ray_box(root.bmin[0], root.bmin[1], root.bmin[2], root.bmax[0], root.bmax[1], root.bmax[2], o, inv, tb)) return;
    if (tb > tmax) return;
    L.ref = root.ref;
    L.cnt = root.count;
}

// Next node from the stack; the lane goes idle when the stack is empty.
template <class Stack>
__device__ __forceinline__ void lane_pop(TraceLane& L, const Stack& stack) {
    if (L.sp == 0) {
        L.cnt = -1;
        return;
    }
    const int2 e = stack.get(--L.sp);
    L.ref = e.x;
    L.cnt = e.y;
}

// One triangle of the current leaf.
template <TraceKind KIND, bool COUNT, class Stack>
__device__ __forceinline__ void lane_tri(const BvhView& bvh, TraceLane& L, Stack& stack) {
    float4 a, b, c;
    load_tri(bvh.tris + L.ref, a, b, c);
    if (COUNT) L.nt++;
    xv3 o;
    unpack2(L.rp.oxy, o.x, o.y);
    float dup;
    unpack2(L.rp.ozz, o.z, dup);
    float t, u, v;
    if (ray_tri(mk(a), mk(b), mk(c), o, L.d, t, u, v) && t > PGX_EPSILON && t < L.tmax) {
        L.hit_id = __float_as_int(a.w);
        if (KIND == kTraceAny || (KIND == kTraceMixed && L.any)) {
            L.cnt = -1;
            return;
        }
        L.tmax = t;
        L.hu = u;
        L.hv = v;
    }
    L.ref++;
    if (--L.cnt == 0) lane_pop(L, stack);
}

// One interior node.
template <TraceKind KIND, bool COUNT, class Stack>
__device__ __forceinline__ void lane_node(const BvhView& bvh, TraceLane& L, Stack& stack) {
    if (COUNT) L.ni++;
    const TravNode* node = bvh.nodes + L.ref;
    const ChildView l = load_child(&node->l), r = load_child(&node->r);
    float dl, dr;
    if (L.finite) {
        dl = child_entry(l, L.rp, L.tmax);
        dr = child_entry(r, L.rp, L.tmax);
    } else {
        dl = child_entry_exact(l, L.rp, L.tmax);
        dr = child_entry_exact(r, L.rp, L.tmax);
    }
    const bool swap = dl > dr;
    const float dn = swap ? dr : dl, df = swap ? dl : dr;
    if (dn == FLT_MAX) {
        lane_pop(L, stack);
        return;
    }
    L.ref = swap ? r.ref : l.ref;
    L.cnt = swap ? r.cnt : l.cnt;
    if (df != FLT_MAX) {
        if (L.sp >= PGX_STACK_SIZE) {
            L.status = 1;
            L.cnt = -1;
            return;
        }
        stack.put(L.sp, make_int2(swap ? l.ref : r.ref, swap ? l.cnt : r.cnt));
        L.sp++;
    }
}

// Persistent warp loop over rays [0, n): `load(i, o, d, tmax)` fetches ray i
// (and returns whether it stops at the first hit; read by mixed launches),
// `store(i, lane)` consumes a finished ray, `root_of(i, bvh)` gives the tree
// root ray i starts from (several trees can share the node and triangle
// arrays).  `next` is a zeroed counter.  n_interior and n_tris get a counting
// launch's visits.  Must be called by whole warps.
template <TraceKind KIND, bool COUNT, class Load, class Store, class RootOf = SceneRoot, int SHORT = kShortStack,
          bool SPREAD = KIND == kTraceMixed>
__device__ __forceinline__ void trace_persistent(const BvhView& bvh, unsigned n, unsigned* next, Load load,
                                                 Store store, unsigned long long& n_interior,
                                                 unsigned long long& n_tris, unsigned& status_or,
                                                 RootOf root_of = RootOf()) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    // 200k-triangle interior at 1280x720 x 32 samples, ms per step (first
    // version: a vote per step, leaves from half of the busy lanes on, stores
    // and refills inside the loop: 91.8):
    //   node steps 1 / 2 / 3 / 4 per vote           84.4 / 81.6 / 81.4 / 81.1
    //   + triangle steps 2 / 4                      77.6 / 76
    //   leaves from 2/3, 1/2, 1/3, 1/4 of the lanes 88.1 / 81.6 / 79.6 / (with the above) worse
    //   refill below 16 / 20 / 24 / 28 lanes        76.6 / 76.1 / 76.4 / 79
    // (2 M random triangles prefer 24 to 20: 5.03 against 5.14 ms per 4 M rays)
    constexpr int kRefillBelow = 24;  // refill when fewer lanes than this are busy
    constexpr int kNodeSteps = 4;     // interior nodes per vote
    constexpr int kTriSteps = 4;      // triangles per vote (a leaf of the builder's holds at most 4)
    constexpr int kLeafShare = 3;     // leaves step when at least 1 / kLeafShare of the busy lanes hold one
    const int lane = threadIdx.x & 31;
    // SPREAD: with fewer rays than lanes, every warp takes its share instead
    // of some warps 32: what remains is the longest rays' chain of steps, and
    // a warp with fewer rays takes each step sooner (frames and adjoints
    // 2-3 %).  Off in the kernels for long queues, where it costs 3 %.
    int cap = 32, refill_below = kRefillBelow;
    if (SPREAD) {
        const unsigned warps = gridDim.x * (blockDim.x >> 5);
        cap = (int)min(32u, max(1u, (n + warps - 1) / warps));
        if (cap < 32) refill_below = max(1, cap * 3 / 4);
    }
    __shared__ int2 s_stack[SHORT * kTraceMaxBlock];
    TraceStack<SHORT> stack;
    stack.sh = s_stack + threadIdx.x;
    TraceLane L;
    L.cnt = -1;
    unsigned ray = 0;
    bool have = false;     // the lane holds a ray (finished or not)
    bool drained = false;  // warp-uniform: the counter has passed n
    for (;;) {
        // Finished rays are stored and idle lanes refilled together, so these
        // stretches run with many lanes (possibly several rounds when roots
        // are missed).
        for (;;) {
            const bool idle = L.cnt < 0 && (!SPREAD || lane < cap);
            if (have && idle) {
                status_or |= (unsigned)L.status;
                if (COUNT) {
                    n_interior += L.ni;
                    n_tris += L.nt;
                }
                store(ray, L);
                have = false;
            }
            const unsigned m = drained ? 0u : __ballot_sync(kFull, idle);
            if (!m) break;
            const int leader = __ffs(m) - 1;
            unsigned base = 0;
            if (lane == leader) base = atomicAdd(next, (unsigned)__popc(m));
            base = __shfl_sync(kFull, base, leader);
            if (idle) {
                const unsigned idx = base + __popc(m & ((1u << lane) - 1u));
                if (idx < n) {
                    xv3 o, d;
                    float tmax;
                    L.any = load(idx, o, d, tmax);
                    ray = idx;
                    have = true;
                    lane_start<KIND>(root_of(idx, bvh), L, o, d, tmax);
                }
            }
            drained = base + (unsigned)__popc(m) >= n;
        }
        // Branch vote: lanes at a leaf (triangle tests) and lanes at an
        // interior node (two slab tests) take different code, so one group
        // takes a few steps while the other waits.  A ray's own sequence of nodes and triangles is unchanged (it
        // only pauses), so results stay bit-identical.
        for (;;) {
            const unsigned nodes = __ballot_sync(kFull, L.cnt == 0);
            const unsigned leaves = __ballot_sync(kFull, L.cnt > 0);
            const int busy = __popc(nodes | leaves);
            if (busy < refill_below && (!drained || busy == 0)) break;
            if (kLeafShare * __popc(leaves) >= busy) {
#pragma unroll
                for (int x = 0; x < kTriSteps; x++)
                    if (L.cnt > 0) lane_tri<KIND, COUNT>(bvh, L, stack);
            } else {
#pragma unroll
                for (int x = 0; x < kNodeSteps; x++)
                    if (L.cnt == 0) lane_node<KIND, COUNT>(bvh, L, stack);
            }
        }
        if (drained && !__any_sync(kFull, L.cnt >= 0 || have)) break;
    }
}
