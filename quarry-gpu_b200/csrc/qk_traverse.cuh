// qk_traverse.cuh -- per-query stack traversals shared by the single-tree kernels
// (qk_query.cu) and the batched persistent kernels (qk_batch.cu).
//
// Each function runs one ray or query point through one tree to completion.  Binary nodes
// are 64-byte BNodes (both child boxes inline, four 16-byte loads); 4-wide nodes are 128-byte
// WideNodes.  Pruning follows the reference's rules exactly: the slab test with its 1e-6
// margins for rays, "bound <= best" for closest / kNN, "dist2 <= r2" for radius
// (src/gpu/raycast.cu:100-139, src/gpu/query.cu:74-116, 415-540), so every result is
// independent of tree shape and visit order.
//
// The stack is a template policy: LocalStack keeps every entry in local memory (the
// single-tree kernels), SplitStack keeps the first `sh` entries of every thread in shared
// memory (entry e of thread t at base[e * stride + t], conflict-free) and the rest in local
// memory -- the short-stack depth the batch autotuner chooses at run time.
#pragma once

#include "qk_internal.cuh"

namespace qk {

struct Trav {
    int nodes = 0;
    int leaves = 0;
    bool overflow = false;
};

// Per-thread stack in local memory: entry i is the pair (node, key bits), so a push is one
// 8-byte store and get() one 8-byte load.
template <int kCap>
struct LocalStack {
    static constexpr int kSize = kCap;
    int2 e[kCap];
    __device__ __forceinline__ void put(int i, int n, float k) { e[i] = make_int2(n, __float_as_int(k)); }
    __device__ __forceinline__ void put_node(int i, int n) { e[i].x = n; }
    __device__ __forceinline__ int get_node(int i) const { return e[i].x; }
    __device__ __forceinline__ float get_key(int i) const { return __int_as_float(e[i].y); }
    __device__ __forceinline__ void get(int i, int& n, float& k) const {
        const int2 v = e[i];
        n = v.x;
        k = __int_as_float(v.y);
    }
};

template <int kCap>
struct SplitStack {
    static constexpr int kSize = kCap;
    int* snode;   // this thread's column of the shared-memory part
    float* skey;
    int sh;       // entries kept in shared memory
    int stride;   // threads per block
    int node[kCap];
    float key[kCap];
    __device__ __forceinline__ void put(int i, int n, float k) {
        if (i < sh) {
            snode[i * stride] = n;
            skey[i * stride] = k;
        } else {
            node[i] = n;
            key[i] = k;
        }
    }
    __device__ __forceinline__ void put_node(int i, int n) {
        if (i < sh) snode[i * stride] = n;
        else node[i] = n;
    }
    __device__ __forceinline__ int get_node(int i) const { return i < sh ? snode[i * stride] : node[i]; }
    __device__ __forceinline__ float get_key(int i) const { return i < sh ? skey[i * stride] : key[i]; }
    __device__ __forceinline__ void get(int i, int& n, float& k) const {
        n = get_node(i);
        k = get_key(i);
    }
};

// ---------------------------------------------------------------------------------------
// node and leaf loads
// ---------------------------------------------------------------------------------------
// 32 bytes as four float pairs through the read-only path, in one 256-bit load or two 128-bit
// ones.  In a divergent warp every lane reads its own node; the ray kernels keep many warps in
// flight, and half as many load instructions pay where nodes come from L2 (1 M rays, city 479 -> 460
// us) though not where they come from L1 (terrain 519 -> 528; 2,048 rays 23.4 -> 24.2),
// while the point queries, a few warps per SM bound by the latency of each step, lose more to
// the longer load (closest of 20,000 points 69 -> 80 us, radius 149 -> 163).  The 256-bit load
// needs a 32-byte boundary.
template <bool kVec256>
__device__ __forceinline__ void ldg32(const void* p, F2& a, F2& b, F2& c, F2& d) {
    if constexpr (kVec256) {
        asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p));
    } else {
        const float4 u = __ldg(static_cast<const float4*>(p)), v = __ldg(static_cast<const float4*>(p) + 1);
        a = f2_pack(u.x, u.y);
        b = f2_pack(u.z, u.w);
        c = f2_pack(v.x, v.y);
        d = f2_pack(v.z, v.w);
    }
}

// traversal node i: both child boxes in stored form, child references, small-subtree codes
// (lsm / rsm: 0, or (first slot << 2) | (leaves - 1) for a child subtree of 2..4 leaves on
// contiguous slots)
struct NodePair {
    BoxQ l, r;
    int lref, rref, lsm, rsm;
};
template <bool kVec256 = false>
__device__ __forceinline__ NodePair load_pair(const BNode* __restrict__ bn, int i) {
    NodePair n;
    F2 refs, small;
    const char* p = reinterpret_cast<const char*>(bn) + 64 * static_cast<size_t>(i);
    ldg32<kVec256>(p, n.l.a, n.l.b, n.l.c, n.r.a);
    ldg32<kVec256>(p + 32, n.r.b, n.r.c, refs, small);
    n.lref = static_cast<int>(static_cast<unsigned>(refs));
    n.rref = static_cast<int>(static_cast<unsigned>(refs >> 32));
    n.lsm = static_cast<int>(static_cast<unsigned>(small));
    n.rsm = static_cast<int>(static_cast<unsigned>(small >> 32));
    return n;
}

__device__ __forceinline__ void load_bnode(const BNode* __restrict__ bn, int i, float3& llo,
                                           float3& lhi, float3& rlo, float3& rhi, int& lref,
                                           int& rref) {
    const NodePair n = load_pair(bn, i);
    llo = boxq_lo(n.l);
    lhi = boxq_hi(n.l);
    rlo = boxq_lo(n.r);
    rhi = boxq_hi(n.r);
    lref = n.lref;
    rref = n.rref;
}

// box of the leaf in slot s; lnodes = the canonical nodes of the leaves (nodes + n - 1)
__device__ __forceinline__ Box leaf_box(const Node* __restrict__ lnodes, int s) {
    const float4* p = reinterpret_cast<const float4*>(lnodes + s);
    const float4 a = __ldg(p), b = __ldg(p + 1);
    Box bx;
    bx.lo = f3(a.x, a.y, a.z);
    bx.hi = f3(a.w, b.x, b.y);
    return bx;
}

__device__ __forceinline__ Box root_box(const Node* __restrict__ nodes) {
    const float4* p = reinterpret_cast<const float4*>(nodes);
    const float4 a = __ldg(p), b = __ldg(p + 1);
    Box bx;
    bx.lo = f3(a.x, a.y, a.z);
    bx.hi = f3(a.w, b.x, b.y);
    return bx;
}

// slot s of wide node `node`: box, child and the slot's primitive count -- max(pad, 1): 1 for
// every leaf slot of quarry's form (pad 0), up to 4 for a leaf range of the leaf-size-4 form
// (the primitives on slots ~child .. ~child + count - 1); meaningless for internal slots.  The
// traversals read the count only when instantiated for the leaf-size-4 form (kRange).
__device__ __forceinline__ BoxQ load_wide_entry(const WideNode* __restrict__ w, int node, int s,
                                                int& child, int& count) {
    BoxQ q;
    F2 refs;
    const char* p = reinterpret_cast<const char*>(w) + 128 * static_cast<size_t>(node) + 32 * s;
    ldg32<false>(p, q.a, q.b, q.c, refs);
    child = static_cast<int>(static_cast<unsigned>(refs));
    count = max(static_cast<int>(static_cast<unsigned>(refs >> 32)), 1);
    return q;
}

// The four slots of a 4-wide node with their keys (entry t or squared distance), in registers:
// a miss or an empty slot holds (+inf, kEmptySlot).  sort() orders them by key, equal keys in slot
// order (a query inside several boxes has equal keys, and the first leaf met decides a NaN answer):
// exchanges of neighbours only, six of them; dynamic indexing would put the arrays in local memory.
struct WideHits {
    float k0, k1, k2, k3;
    int c0, c1, c2, c3;
    int n0, n1, n2, n3;  // primitives of a leaf slot (leaf-size-4 form only)
    template <bool kRange>
    __device__ __forceinline__ static void exchange(float& ka, int& ca, int& na, float& kb, int& cb,
                                                    int& nb) {
        const bool sw = kb < ka;
        const float k = sw ? kb : ka;
        kb = sw ? ka : kb;
        ka = k;
        const int c = sw ? cb : ca;
        cb = sw ? ca : cb;
        ca = c;
        if (kRange) {
            const int n = sw ? nb : na;
            nb = sw ? na : nb;
            na = n;
        }
    }
    template <bool kRange>
    __device__ __forceinline__ void sort() {
        exchange<kRange>(k0, c0, n0, k1, c1, n1);
        exchange<kRange>(k2, c2, n2, k3, c3, n3);
        exchange<kRange>(k1, c1, n1, k2, c2, n2);
        exchange<kRange>(k0, c0, n0, k1, c1, n1);
        exchange<kRange>(k2, c2, n2, k3, c3, n3);
        exchange<kRange>(k1, c1, n1, k2, c2, n2);
    }
    // bit j: slot j holds a leaf
    __device__ __forceinline__ static unsigned leaf(int c) { return c < 0 && c != kEmptySlot ? 1u : 0u; }
    __device__ __forceinline__ unsigned leaves() const {
        return leaf(c0) | leaf(c1) << 1 | leaf(c2) << 2 | leaf(c3) << 3;
    }
    __device__ __forceinline__ int hits() const {
        return (c0 != kEmptySlot) + (c1 != kEmptySlot) + (c2 != kEmptySlot) + (c3 != kEmptySlot);
    }
    __device__ __forceinline__ int child(int j) const {
        return j < 2 ? (j == 0 ? c0 : c1) : (j == 2 ? c2 : c3);
    }
    __device__ __forceinline__ float key(int j) const {
        return j < 2 ? (j == 0 ? k0 : k1) : (j == 2 ? k2 : k3);
    }
    __device__ __forceinline__ int count(int j) const {
        return j < 2 ? (j == 0 ? n0 : n1) : (j == 2 ? n2 : n3);
    }
};

// wide node `node` against point p: slots whose squared box distance `admits` lets in
template <class Admits>
__device__ __forceinline__ WideHits wide_point_hits(const WideNode* __restrict__ wn, int node,
                                                    const Vec3Q& p, Admits admits) {
    WideHits h;
    const BoxQ b0 = load_wide_entry(wn, node, 0, h.c0, h.n0);
    const BoxQ b1 = load_wide_entry(wn, node, 1, h.c1, h.n1);
    const BoxQ b2 = load_wide_entry(wn, node, 2, h.c2, h.n2);
    const BoxQ b3 = load_wide_entry(wn, node, 3, h.c3, h.n3);
    dist2_boxq2(p, b0, b1, h.k0, h.k1);
    dist2_boxq2(p, b2, b3, h.k2, h.k3);
    auto drop = [&](float& k, int& c) {
        if (c == kEmptySlot || !admits(k)) {
            k = kInf;
            c = kEmptySlot;
        }
    };
    drop(h.k0, h.c0);
    drop(h.k1, h.c1);
    drop(h.k2, h.c2);
    drop(h.k3, h.c3);
    return h;
}

// The internal children of sorted hits that `admits` still lets in: the nearest is returned
// (-1: none), the others pushed far-first.
template <class St, class Admits>
__device__ __forceinline__ int wide_next(const WideHits& h, St& st, int& sp, Trav& tv,
                                         Admits admits) {
    int next = -1;
    float key = 0.0f;
    auto visit = [&](float k, int c) {
        if (c < 0 || !admits(k)) return;
        if (next >= 0) {
            if (sp >= St::kSize) tv.overflow = true;
            else st.put(sp++, next, key);
        }
        next = c;
        key = k;
    };
    visit(h.k3, h.c3);
    visit(h.k2, h.c2);
    visit(h.k1, h.c1);
    visit(h.k0, h.c0);
    return next;
}

// pops entries until one whose key `admits` lets in; -1: the stack is empty
template <class St, class Admits>
__device__ __forceinline__ int pop_next(St& st, int& sp, Admits admits) {
    while (sp > 0) {
        --sp;
        int pn;
        float pk;
        st.get(sp, pn, pk);
        if (admits(pk)) return pn;
    }
    return -1;
}

// statistics: warp-aggregated counters (src/gpu/raycast.cu:147-156)
template <bool kStats>
__device__ __forceinline__ void flush_stats(bool active, int nodes, int leaves, bool overflow,
                                            unsigned long long* stats) {
    if (stats == nullptr) return;
    const unsigned mask = __ballot_sync(0xffffffffu, active);
    const unsigned ovf = __ballot_sync(0xffffffffu, overflow);
    if (kStats) {
        const int sn = __reduce_add_sync(0xffffffffu, nodes);
        const int sl = __reduce_add_sync(0xffffffffu, leaves);
        if ((threadIdx.x & 31) == 0 && mask) {
            if (sn) atomicAdd(stats + 0, static_cast<unsigned long long>(sn));
            if (sl) atomicAdd(stats + 1, static_cast<unsigned long long>(sl));
        }
    }
    if ((threadIdx.x & 31) == 0 && ovf) atomicAdd(stats + 2, static_cast<unsigned long long>(__popc(ovf)));
}

// ---------------------------------------------------------------------------------------
// rays
// ---------------------------------------------------------------------------------------
// Leaf test.  The first hit is taken even at t == tMax (the CPU reference accepts t <= tMax,
// src/cpu/bvh.cpp:156-168); later hits only when closer.  Among hits at the same t the
// smallest scene index is kept, so the reported primitive does not depend on visit order.
//
// Only this test reads a ray's direction and tmax, so a traversal keeps them in the thread's
// entry of shared memory (RayTail) instead of in four registers of its loop.
struct RayTail {
    unsigned at;  // shared-memory address of this thread's {d.xyz, tmax}
    __device__ __forceinline__ RayTail(float4* slot, const RayPre& r)
        : at(static_cast<unsigned>(__cvta_generic_to_shared(slot))) {
        // get() does not tell the compiler that it reads the slot: the store stays behind the
        // reads for the ray before and ahead of those for this one
        asm volatile("" ::: "memory");
        *slot = make_float4(r.d.x, r.d.y, r.d.z, r.tmax);
        asm volatile("" ::: "memory");
    }
    __device__ __forceinline__ void get(RayPre& r) const {
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(r.d.x), "=f"(r.d.y), "=f"(r.d.z), "=f"(r.tmax)
                     : "r"(at));
    }
};

template <int kMode = -1>
__device__ __forceinline__ void test_tri(const RayPre& R0, const RayTail& tail,
                                         const float4* __restrict__ leaves, int slot, float& best,
                                         float& bound, bool& any, int& best_id) {
    const float4 a = __ldg(leaves + 3 * slot), b = __ldg(leaves + 3 * slot + 1),
                 c = __ldg(leaves + 3 * slot + 2);
    RayPre R = R0;
    tail.get(R);
    float t;
    if (ray_tri<kMode>(R, f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), f3(c.x, c.y, c.z), t)) {
        const int id = __float_as_int(a.w);
        if (!any || t < best || (t == best && id < best_id)) {
            best = t;
            bound = best * kMarginMul + kMarginAdd;
            any = true;
            best_id = id;
        }
    }
}

__device__ __forceinline__ unsigned long long pack_hit(bool any, float best) {
    return any ? ((1ull << 32) | static_cast<unsigned long long>(__float_as_uint(best))) : 0ull;
}

// First hit in a binary tree: near child followed, far child pushed with its entry bound,
// which is re-checked against the current best when popped (src/cpu/bvh.cpp:147-152).
// kMode >= 0: the ray's RayPre::mode, known at compile time (the slab tests drop their
// branch on parallel axes and use min / max); -1 for any ray.
template <class St, bool kLeaf4 = false, int kMode = -1, bool kVec256 = false>
__device__ __forceinline__ unsigned long long ray_bin_one(const BNode* __restrict__ bn,
                                                          const float4* __restrict__ leaves,
                                                          const Box& rb, const RayPre& R,
                                                          const RayTail& tail, int max_iter, St& st, Trav& tv,
                                                          int& best_id,
                                                          const Node* __restrict__ lnodes = nullptr) {
    float best = R.tmax;
    float bound = best * kMarginMul + kMarginAdd;
    bool any = false;
    best_id = -1;
    float te;
    if (!ray_box<kMode>(R, rb.lo, rb.hi, bound, te)) return 0ull;
    ++tv.nodes;
    const Vec3Q qo = vec3q(R.o), qi = vec3q(R.inv);
    int sp = 0;
    int node = 0;
    for (int iter = 0;; ++iter) {
        if (iter >= max_iter) {
            tv.overflow = true;
            break;
        }
        const NodePair nd = load_pair<kVec256>(bn, node);
        const int lref = nd.lref, rref = nd.rref, lsm = nd.lsm, rsm = nd.rsm;
        float tl, tr;
        bool hl = ray_boxq<kMode>(R, qo, qi, nd.l, bound, tl);
        bool hr = ray_boxq<kMode>(R, qo, qi, nd.r, bound, tr);
        tv.nodes += static_cast<int>(hl) + static_cast<int>(hr);
        // leaf children: one copy of the test, so a warp's left and right leaves are tested
        // together and a second round runs only for lanes with both
        const bool ll = hl && lref < 0, rl = hr && rref < 0;
        if (ll || rl) {
            int leaf = ll ? lref : rref;
            bool more = ll && rl;
            for (;;) {
                ++tv.leaves;
                test_tri<kMode>(R, tail, leaves, ~leaf, best, bound, any, best_id);
                if (!more) break;
                more = false;
                leaf = rref;
            }
            hl = hl && !ll;
            hr = hr && !rl;
        }
        if constexpr (kLeaf4) {
            // subtrees of 2..4 triangles: test them now, the nearer first, the farther only
            // while its entry still passes the current bound
            const bool sl = hl && lsm != 0, sr = hr && rsm != 0;
            if (sl || sr) {
                const bool lnear = tl <= tr;
#pragma unroll
                for (int pass = 0; pass < 2; ++pass) {
                    const bool left = (pass == 0) == lnear;
                    const int code = left ? (sl ? lsm : 0) : (sr ? rsm : 0);
                    const float te = left ? tl : tr;
                    if (code && !(te > bound * kMarginMul + kMarginAdd)) {
                        const int first = code >> 2, cnt = (code & 3) + 1;
                        for (int j = 0; j < cnt; ++j) {
                            // the leaf's own box first, as a descent would test it
                            const Box lb = leaf_box(lnodes, first + j);
                            float tb;
                            if (!ray_box<kMode>(R, lb.lo, lb.hi, bound, tb)) continue;
                            ++tv.leaves;
                            test_tri<kMode>(R, tail, leaves, first + j, best, bound, any, best_id);
                        }
                    }
                }
                if (sl) hl = false;
                if (sr) hr = false;
            }
        }
        if (hl && hr) {
            const bool lnear = tl <= tr;
            if (sp >= St::kSize) {
                tv.overflow = true;
                break;
            }
            st.put(sp, lnear ? rref : lref, lnear ? tr : tl);
            ++sp;
            node = lnear ? lref : rref;
        } else if (hl) {
            node = lref;
        } else if (hr) {
            node = rref;
        } else {
            // pop the next entry whose box could still hold a closer hit
            const float limit = bound * kMarginMul + kMarginAdd;
            node = -1;
            while (sp > 0) {
                --sp;
                int pn;
                float pk;
                st.get(sp, pn, pk);
                if (!(pk > limit)) {
                    node = pn;
                    break;
                }
            }
            if (node < 0) break;
        }
    }
    return pack_hit(any, best);
}

// First hit in a 4-wide tree: hit slots sorted by entry t, leaves tested nearest first,
// the nearest internal child followed and the others pushed far-first.
template <bool kRange = false, int kMode = -1, class St>
__device__ __forceinline__ unsigned long long ray_wide_one(const WideNode* __restrict__ wn,
                                                           const float4* __restrict__ leaves,
                                                           const RayPre& R, const RayTail& tail,
                                                           int max_iter, St& st, Trav& tv,
                                                           int& best_id) {
    float best = R.tmax;
    float bound = best * kMarginMul + kMarginAdd;
    bool any = false;
    best_id = -1;
    int sp = 0;
    int node = 0;  // the 4-wide root has no single box; start inside it (raycast.cu:182)
    const Vec3Q qo = vec3q(R.o), qi = vec3q(R.inv);
    for (int iter = 0;; ++iter) {
        if (iter >= max_iter) {
            tv.overflow = true;
            break;
        }
        WideHits h;
        auto test = [&](int s, float& k, int& c, int& n) {
            const BoxQ q = load_wide_entry(wn, node, s, c, n);
            if (c == kEmptySlot || !ray_boxq<kMode>(R, qo, qi, q, bound, k)) {
                k = kInf;
                c = kEmptySlot;
            }
        };
        test(0, h.k0, h.c0, h.n0);
        test(1, h.k1, h.c1, h.n1);
        test(2, h.k2, h.c2, h.n2);
        test(3, h.k3, h.c3, h.n3);
        tv.nodes += h.hits();
        h.template sort<kRange>();
        // leaves nearest first, while their entry passes the current bound (one copy of the
        // test: lanes with leaves in different slots run it together)
        unsigned lm = h.leaves();
#pragma unroll 1
        while (lm) {
            const int j = __ffs(lm) - 1;
            lm &= lm - 1;
            if (h.key(j) > bound * kMarginMul + kMarginAdd) continue;
            const int first = ~h.child(j);
            const int nq = kRange ? h.count(j) : 1;
            for (int q = 0; q < nq; ++q) {
                ++tv.leaves;
                test_tri<kMode>(R, tail, leaves, first + q, best, bound, any, best_id);
            }
        }
        const float limit = bound * kMarginMul + kMarginAdd;
        const auto admits = [&](float k) { return !(k > limit); };
        node = wide_next(h, st, sp, tv, admits);
        if (tv.overflow) break;
        if (node < 0) node = pop_next(st, sp, admits);
        if (node < 0) break;
    }
    return pack_hit(any, best);
}

// ---------------------------------------------------------------------------------------
// closest
// ---------------------------------------------------------------------------------------
template <class Ops>
__device__ __forceinline__ void leaf_closest(float3 p, const float4* __restrict__ leaves, int slot,
                                             float& best, int& best_id) {
    int id;
    const float d2 = Ops::dist2(p, leaves, slot, id, best);  // best is +inf before the first
    if (best_id < 0 || closer(d2, id, best, best_id)) {
        best = d2;
        best_id = id;
    }
}

__device__ __forceinline__ uint2 pack_closest(float best, int best_id) {
    return best_id >= 0 ? make_uint2(__float_as_uint(best), static_cast<unsigned>(best_id))
                        : make_uint2(0u, 0xffffffffu);
}

template <class Ops, class St, bool kLeaf4 = false>
__device__ __forceinline__ uint2 closest_bin_one(const BNode* __restrict__ bn,
                                                 const float4* __restrict__ leaves, float3 p,
                                                 int max_iter, St& st, Trav& tv,
                                                 const Node* __restrict__ lnodes = nullptr) {
    float best = kInf;
    int best_id = -1;
    int sp = 0;
    int node = 0;
    const Vec3Q qp = vec3q(p);
    for (int iter = 0;; ++iter) {
        if (iter >= max_iter) {
            tv.overflow = true;
            break;
        }
        ++tv.nodes;
        const NodePair nd = load_pair(bn, node);
        const int lref = nd.lref, rref = nd.rref, lsm = nd.lsm, rsm = nd.rsm;
        float dl, dr;
        dist2_boxq2(qp, nd.l, nd.r, dl, dr);
        bool okl = best_id < 0 || dl <= best;
        bool okr = best_id < 0 || dr <= best;
        // leaves in near-first order so the second sees the tighter bound (one copy of the
        // test: a warp's left and right leaves are tested together)
        const bool lfirst = dl <= dr;
        const int lslot = okl && lref < 0 ? ~lref : -1, rslot = okr && rref < 0 ? ~rref : -1;
        int leaf = lfirst ? lslot : rslot, other = lfirst ? rslot : lslot;
        const float dfar = lfirst ? dr : dl;
        if (leaf < 0) {
            leaf = other;
            other = -1;
        }
#pragma unroll 1
        while (leaf >= 0) {
            ++tv.leaves;
            leaf_closest<Ops>(p, leaves, leaf, best, best_id);
            leaf = best_id < 0 || dfar <= best ? other : -1;
            other = -1;
        }
        okl = okl && lref >= 0;
        okr = okr && rref >= 0;
        if constexpr (kLeaf4) {
            const bool sl = okl && lsm != 0, sr = okr && rsm != 0;
            if (sl || sr) {
#pragma unroll
                for (int pass = 0; pass < 2; ++pass) {
                    const bool left = (pass == 0) == lfirst;
                    const int code = left ? (sl ? lsm : 0) : (sr ? rsm : 0);
                    const float dbox = left ? dl : dr;
                    if (code && (best_id < 0 || dbox <= best)) {
                        const int first = code >> 2, cnt = (code & 3) + 1;
                        for (int j = 0; j < cnt; ++j) {
                            const Box lb = leaf_box(lnodes, first + j);
                            if (!(best_id < 0 || dist2_box(p, lb.lo, lb.hi) <= best)) continue;
                            ++tv.leaves;
                            leaf_closest<Ops>(p, leaves, first + j, best, best_id);
                        }
                    }
                }
                if (sl) okl = false;
                if (sr) okr = false;
            }
        }
        if (okl && okr) {
            if (sp >= St::kSize) {
                tv.overflow = true;
                break;
            }
            st.put(sp, lfirst ? rref : lref, lfirst ? dr : dl);
            ++sp;
            node = lfirst ? lref : rref;
        } else if (okl) {
            node = lref;
        } else if (okr) {
            node = rref;
        } else {
            node = -1;
            while (sp > 0) {
                --sp;
                int pn;
                float pk;
                st.get(sp, pn, pk);
                if (best_id < 0 || pk <= best) {
                    node = pn;
                    break;
                }
            }
            if (node < 0) break;
        }
    }
    return pack_closest(best, best_id);
}

template <class Ops, bool kRange = false, class St>
__device__ __forceinline__ uint2 closest_wide_one(const WideNode* __restrict__ wn,
                                                  const float4* __restrict__ leaves, float3 p,
                                                  int max_iter, St& st, Trav& tv) {
    float best = kInf;
    int best_id = -1;
    int sp = 0;
    int node = 0;
    const Vec3Q qp = vec3q(p);
    for (int iter = 0;; ++iter) {
        if (iter >= max_iter) {
            tv.overflow = true;
            break;
        }
        const auto admits = [&](float k) { return best_id < 0 || k <= best; };
        WideHits h = wide_point_hits(wn, node, qp, admits);
        tv.nodes += h.hits();
        h.template sort<kRange>();
        unsigned lm = h.leaves();
#pragma unroll 1
        while (lm) {
            const int j = __ffs(lm) - 1;
            lm &= lm - 1;
            if (!admits(h.key(j))) continue;
            const int first = ~h.child(j);
            const int nq = kRange ? h.count(j) : 1;
            for (int q = 0; q < nq; ++q) {
                ++tv.leaves;
                leaf_closest<Ops>(p, leaves, first + q, best, best_id);
            }
        }
        node = wide_next(h, st, sp, tv, admits);
        if (tv.overflow) break;
        if (node < 0) node = pop_next(st, sp, admits);
        if (node < 0) break;
    }
    return pack_closest(best, best_id);
}

// ---------------------------------------------------------------------------------------
// kNN: the k best (dist2, id) pairs stay sorted in registers (unrolled insertion over a
// compile-time capacity K >= k).  Empty slots hold (+inf, INT_MAX), so "strictly closer than
// the k-th" is one comparison whether or not the table is full -- the reference's max-heap
// replacement rule (src/cpu/bvh.cpp:284-299, src/gpu/query.cu:145-158).
// ---------------------------------------------------------------------------------------
//
// The k entries sit at the end of the table, behind K - k entries that compare below every
// candidate and never move: the k-th entry is then always the last one.  Reading it at index
// k - 1 instead made the compiler keep the whole table in local memory for K <= 16.
template <int K>
struct KnnTable {
    float d[K];
    int id[K];

    __device__ __forceinline__ void init(int k = K) {
#pragma unroll
        for (int j = 0; j < K; ++j) {
            d[j] = j < K - k ? -kInf : kInf;
            id[j] = j < K - k ? -1 : 0x7fffffff;
        }
    }
    // dist2 of the k-th entry (the pruning threshold; +inf until the table is full)
    __device__ __forceinline__ float kth() const { return d[K - 1]; }
    __device__ __forceinline__ void insert(float xd, int xid) {
        bool below = closer(xd, xid, d[K - 1], id[K - 1]);  // x goes before entry j
        if (!below) return;
#pragma unroll
        for (int j = K - 1; j > 0; --j) {
            const bool shift = closer(xd, xid, d[j - 1], id[j - 1]);
            d[j] = shift ? d[j - 1] : (below ? xd : d[j]);
            id[j] = shift ? id[j - 1] : (below ? xid : id[j]);
            below = shift;
        }
        if (below) {
            d[0] = xd;
            id[0] = xid;
        }
    }
    // prune test for a subtree bound: keep while the table is not full or bound <= k-th
    __device__ __forceinline__ bool admits(float bound) const {
        return id[K - 1] == 0x7fffffff || bound <= d[K - 1];
    }
};

template <class Ops, int K>
__device__ __forceinline__ void leaf_knn(float3 p, const float4* __restrict__ leaves, int slot,
                                         KnnTable<K>& tab) {
    int id;
    const float d2 = Ops::dist2(p, leaves, slot, id, tab.kth());
    tab.insert(d2, id);
}

template <int K>
__device__ __forceinline__ void write_knn(const KnnTable<K>& tab, int k, uint2* __restrict__ dst) {
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int e = j - (K - k);
        if (e >= 0) {
            const bool valid = tab.id[j] != 0x7fffffff;
            dst[e] = valid ? make_uint2(__float_as_uint(tab.d[j]), static_cast<unsigned>(tab.id[j]))
                           : make_uint2(0u, 0xffffffffu);
        }
    }
}

template <class Ops, int K, class St, bool kLeaf4 = false>
__device__ __forceinline__ void knn_bin_one(const BNode* __restrict__ bn,
                                            const float4* __restrict__ leaves, float3 p, int k,
                                            int max_iter, St& st, Trav& tv, KnnTable<K>& tab,
                                            const Node* __restrict__ lnodes = nullptr) {
    tab.init(k);
    int sp = 0;
    int node = 0;
    const Vec3Q qp = vec3q(p);
    for (int iter = 0;; ++iter) {
        if (iter >= max_iter) {
            tv.overflow = true;
            break;
        }
        ++tv.nodes;
        const NodePair nd = load_pair(bn, node);
        const int lref = nd.lref, rref = nd.rref, lsm = nd.lsm, rsm = nd.rsm;
        float dl, dr;
        dist2_boxq2(qp, nd.l, nd.r, dl, dr);
        const bool lfirst = dl <= dr;
        bool okl = tab.admits(dl);
        bool okr = tab.admits(dr);
        const int lslot = okl && lref < 0 ? ~lref : -1, rslot = okr && rref < 0 ? ~rref : -1;
        int leaf = lfirst ? lslot : rslot, other = lfirst ? rslot : lslot;
        const float dfar = lfirst ? dr : dl;
        if (leaf < 0) {
            leaf = other;
            other = -1;
        }
#pragma unroll 1
        while (leaf >= 0) {
            ++tv.leaves;
            leaf_knn<Ops, K>(p, leaves, leaf, tab);
            leaf = tab.admits(dfar) ? other : -1;
            other = -1;
        }
        okl = okl && lref >= 0;
        okr = okr && rref >= 0;
        if constexpr (kLeaf4) {
            const bool sl = okl && lsm != 0, sr = okr && rsm != 0;
            if (sl || sr) {
#pragma unroll
                for (int pass = 0; pass < 2; ++pass) {
                    const bool left = (pass == 0) == lfirst;
                    const int code = left ? (sl ? lsm : 0) : (sr ? rsm : 0);
                    const float dbox = left ? dl : dr;
                    if (code && tab.admits(dbox)) {
                        const int first = code >> 2, cnt = (code & 3) + 1;
                        for (int j = 0; j < cnt; ++j) {
                            const Box lb = leaf_box(lnodes, first + j);
                            if (!tab.admits(dist2_box(p, lb.lo, lb.hi))) continue;
                            ++tv.leaves;
                            leaf_knn<Ops, K>(p, leaves, first + j, tab);
                        }
                    }
                }
                if (sl) okl = false;
                if (sr) okr = false;
            }
        }
        if (okl && okr) {
            if (sp >= St::kSize) {
                tv.overflow = true;
                break;
            }
            st.put(sp, lfirst ? rref : lref, lfirst ? dr : dl);
            ++sp;
            node = lfirst ? lref : rref;
        } else if (okl) {
            node = lref;
        } else if (okr) {
            node = rref;
        } else {
            node = -1;
            while (sp > 0) {
                --sp;
                int pn;
                float pk;
                st.get(sp, pn, pk);
                if (tab.admits(pk)) {
                    node = pn;
                    break;
                }
            }
            if (node < 0) break;
        }
    }
}

template <class Ops, int K, bool kRange = false, class St>
__device__ __forceinline__ void knn_wide_one(const WideNode* __restrict__ wn,
                                             const float4* __restrict__ leaves, float3 p, int k,
                                             int max_iter, St& st, Trav& tv, KnnTable<K>& tab) {
    tab.init(k);
    int sp = 0;
    int node = 0;
    const Vec3Q qp = vec3q(p);
    for (int iter = 0;; ++iter) {
        if (iter >= max_iter) {
            tv.overflow = true;
            break;
        }
        const auto admits = [&](float bound) { return tab.admits(bound); };
        WideHits h = wide_point_hits(wn, node, qp, admits);
        tv.nodes += h.hits();
        h.template sort<kRange>();
        unsigned lm = h.leaves();
#pragma unroll 1
        while (lm) {
            const int j = __ffs(lm) - 1;
            lm &= lm - 1;
            if (!admits(h.key(j))) continue;
            const int first = ~h.child(j);
            const int nq = kRange ? h.count(j) : 1;
            for (int q = 0; q < nq; ++q) {
                ++tv.leaves;
                leaf_knn<Ops, K>(p, leaves, first + q, tab);
            }
        }
        node = wide_next(h, st, sp, tv, admits);
        if (tv.overflow) break;
        if (node < 0) node = pop_next(st, sp, admits);
        if (node < 0) break;
    }
}

// ---------------------------------------------------------------------------------------
// radius: a box is entered when its squared distance <= r2, a primitive kept when its
// dist2 <= r2 (src/gpu/query.cu:415-540).  The fill pass writes (bits(d2) << 32 | id) keys
// from `write` on and never past `end`; both passes return the number found.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long radius_key(float d2, int id) {
    return (static_cast<unsigned long long>(__float_as_uint(d2)) << 32) | static_cast<unsigned>(id);
}

// Where a radius traversal puts its keys.  SegmentSink: the query's CSR segment
// keys[write, end) (the fill pass), never past its end.
struct SegmentSink {
    unsigned long long* keys;
    int write;
    int end;
    __device__ __forceinline__ void put(unsigned long long k) {
        if (write < end) keys[write++] = k;
    }
};

// PoolSink: the single-pass radius (QK_TUNE_STASH).  A query's first kRadiusStash keys go to
// its stash slots, later ones to chunks of kPoolChunk keys taken from a shared pool (one
// atomic per chunk) and chained per query: *first holds the query's first chunk, next[c] the
// chunk after c; the chain's length follows from the query's count, so it needs no end mark.
// When the pool runs out, *first becomes kPoolLost and the query's later keys are dropped;
// the fill pass traverses such a query again.  Only the thread that owns the query writes its
// stash, its *first and its chain links.
constexpr int kRadiusStash = 16;
constexpr int kPoolChunk = 32;
constexpr int kPoolLost = -2;

// The single-pass radius's buffers for `count` queries, carved from a workspace: the stash
// (kRadiusStash keys per query), the chain heads, the chunk counter, the chain links and the
// pool itself (kPoolPerQuery keys per query on average, shared by all queries).
constexpr int kPoolPerQuery = 128;

struct RadiusPool {
    unsigned long long* stash;
    int* first;
    int* taken;
    int* next;
    unsigned long long* keys;
    int chunks;
};

inline RadiusPool carve_pool(Carve& c, int count, int per_query = kPoolPerQuery) {
    RadiusPool p{};
    p.chunks = static_cast<int>((static_cast<long long>(count) * per_query + kPoolChunk - 1) /
                                kPoolChunk);
    p.stash = c.take<unsigned long long>(static_cast<size_t>(count) * kRadiusStash);
    p.first = c.take<int>(count);
    p.taken = c.take<int>(1);
    p.next = c.take<int>(p.chunks);
    p.keys = c.take<unsigned long long>(static_cast<size_t>(p.chunks) * kPoolChunk);
    return p;
}

struct PoolSink {
    unsigned long long* stash;   // this query's kRadiusStash slots
    unsigned long long* pool;    // chunks of kPoolChunk keys
    int* next;                   // chain links, one per chunk
    int* taken;                  // chunks handed out so far (shared counter)
    int chunks;                  // pool capacity in chunks
    int* first;                  // this query's first chunk, or kPoolLost
    int n;                       // keys seen so far
    int cur;                     // the chunk being filled, or kPoolLost
    __device__ __forceinline__ void put(unsigned long long k) {
        if (n < kRadiusStash) {
            stash[n++] = k;
            return;
        }
        const int j = (n - kRadiusStash) & (kPoolChunk - 1);
        const bool fresh = n == kRadiusStash;
        ++n;
        if (cur == kPoolLost) return;
        if (j == 0) {
            const int c = atomicAdd(taken, 1);
            if (c >= chunks) {
                cur = kPoolLost;
                *first = kPoolLost;
                return;
            }
            if (fresh) *first = c;
            else next[cur] = c;
            cur = c;
        }
        pool[static_cast<size_t>(cur) * kPoolChunk + j] = k;
    }
};

// Copies query q's keys (its stash, then its pool chain) into keys[begin, begin + cnt), one
// warp per query: lane l moves entry l of the stash and of every 32-key chunk, so the reads and
// writes are coalesced.  Every lane of the warp calls it for the same q.
static_assert(kPoolChunk == 32, "a pool chunk is one key per lane");
__device__ __forceinline__ void copy_pooled_warp(const RadiusPool& pool, int q, int begin, int cnt,
                                                 unsigned long long* __restrict__ keys, int lane) {
    const int head = cnt < kRadiusStash ? cnt : kRadiusStash;
    if (lane < head) keys[begin + lane] = pool.stash[static_cast<size_t>(q) * kRadiusStash + lane];
    int left = cnt - head;
    int w = begin + head;
    int c = left > 0 ? pool.first[q] : -1;
    while (left > 0) {
        const int m = left < kPoolChunk ? left : kPoolChunk;
        if (lane < m) keys[w + lane] = pool.keys[static_cast<size_t>(c) * kPoolChunk + lane];
        w += m;
        left -= m;
        if (left > 0) c = pool.next[c];
    }
}

// The copy pass of the single-pass radius: one warp per query whose keys the pool held (the
// others are traversed again); skipped, as the fill is, when offsets[count] exceeds cap (cap <
// 0: no limit).
static __global__ __launch_bounds__(256) void k_radius_gather(RadiusPool pool,
                                                       const int* __restrict__ offsets, int count,
                                                       unsigned long long* __restrict__ keys,
                                                       long long cap) {
    const int q = static_cast<int>((static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (q >= count) return;
    if (cap >= 0 && static_cast<long long>(offsets[count]) > cap) return;
    const int begin = offsets[q], n = offsets[q + 1] - begin;
    if (n > kRadiusStash && pool.first[q] == kPoolLost) return;
    copy_pooled_warp(pool, q, begin, n, keys, lane);
}

// kFew: the single-tree kernels, whose few warps wait out each step's chain of operations: scalar
// box distances and the leaf test in line (20,000 queries on a 1 M-point shell: 143 us against
// 149); the batched kernels keep every scheduler busy and take the shorter code.
template <class Ops, bool kFill, class St, bool kLeaf4, bool kFew, class Sink>
__device__ __forceinline__ int radius_bin_visit(const BNode* __restrict__ bn,
                                                const float4* __restrict__ leaves, const Box& rb,
                                                float3 p, float r2, Sink& sink, int max_iter,
                                                St& st, Trav& tv,
                                                const Node* __restrict__ lnodes = nullptr) {
    int found = 0;
    if (!(dist2_box(p, rb.lo, rb.hi) <= r2)) return 0;
    const Vec3Q qp = vec3q(p);
    int sp = 0;
    int node = 0;
    for (int iter = 0;; ++iter) {
        if (iter >= max_iter) {
            tv.overflow = true;
            break;
        }
        ++tv.nodes;
        const NodePair nd = load_pair(bn, node);
        const int lref = nd.lref, rref = nd.rref, lsm = nd.lsm, rsm = nd.rsm;
        float dl, dr;
        dist2_boxq2<!kFew>(qp, nd.l, nd.r, dl, dr);
        bool okl = dl <= r2;
        bool okr = dr <= r2;
        const auto test = [&](int slot) {
            ++tv.leaves;
            int id;
            const float d2 = Ops::dist2(p, leaves, slot, id, r2);
            if (d2 <= r2) {
                if (kFill) sink.put(radius_key(d2, id));
                ++found;
            }
        };
        int leaf = okl && lref < 0 ? ~lref : -1;
        int other = okr && rref < 0 ? ~rref : -1;
        if (leaf < 0) {
            leaf = other;
            other = -1;
        }
        if constexpr (kFew) {
            if (leaf >= 0) test(leaf);
            if (other >= 0) test(other);
        } else {
#pragma unroll 1
            while (leaf >= 0) {
                test(leaf);
                leaf = other;
                other = -1;
            }
        }
        okl = okl && lref >= 0;
        okr = okr && rref >= 0;
        if constexpr (kLeaf4) {
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                const int code = pass == 0 ? (okl ? lsm : 0) : (okr ? rsm : 0);
                if (code) {
                    const int first = code >> 2, cnt = (code & 3) + 1;
                    for (int j = 0; j < cnt; ++j) {
                        const Box lb = leaf_box(lnodes, first + j);
                        if (!(dist2_box(p, lb.lo, lb.hi) <= r2)) continue;
                        ++tv.leaves;
                        int id;
                        const float d2 = Ops::dist2(p, leaves, first + j, id, r2);
                        if (d2 <= r2) {
                            if (kFill) sink.put(radius_key(d2, id));
                            ++found;
                        }
                    }
                }
            }
            if (lsm) okl = false;
            if (rsm) okr = false;
        }
        if (okl && okr) {
            if (sp >= St::kSize) {
                tv.overflow = true;
                break;
            }
            st.put_node(sp++, rref);
            node = lref;
        } else if (okl) {
            node = lref;
        } else if (okr) {
            node = rref;
        } else {
            if (sp == 0) break;
            node = st.get_node(--sp);
        }
    }
    return found;
}

template <class Ops, bool kFill, class St, bool kLeaf4 = false, bool kFew = false>
__device__ __forceinline__ int radius_bin_one(const BNode* __restrict__ bn,
                                              const float4* __restrict__ leaves, const Box& rb,
                                              float3 p, float r2, int write, int end,
                                              unsigned long long* __restrict__ keys,
                                              int max_iter, St& st, Trav& tv,
                                              const Node* __restrict__ lnodes = nullptr) {
    SegmentSink sink{keys, write, end};
    return radius_bin_visit<Ops, kFill, St, kLeaf4, kFew>(bn, leaves, rb, p, r2, sink, max_iter, st, tv,
                                                          lnodes);
}

template <class Ops, bool kFill, bool kRange = false, class St, class Sink>
__device__ __forceinline__ int radius_wide_visit(const WideNode* __restrict__ wn,
                                                 const float4* __restrict__ leaves, float3 p,
                                                 float r2, Sink& sink, int max_iter, St& st,
                                                 Trav& tv) {
    const Vec3Q qp = vec3q(p);
    int found = 0;
    int sp = 0;
    int node = 0;
    for (int iter = 0;; ++iter) {
        if (iter >= max_iter) {
            tv.overflow = true;
            break;
        }
        const WideHits h = wide_point_hits(wn, node, qp, [&](float k) { return k <= r2; });
        tv.nodes += h.hits();
        unsigned lm = h.leaves();
#pragma unroll 1
        while (lm) {
            const int j = __ffs(lm) - 1;
            lm &= lm - 1;
            const int first = ~h.child(j);
            const int nq = kRange ? h.count(j) : 1;
            for (int q = 0; q < nq; ++q) {
                ++tv.leaves;
                int id;
                const float d2 = Ops::dist2(p, leaves, first + q, id, r2);
                if (d2 <= r2) {
                    if (kFill) sink.put(radius_key(d2, id));
                    ++found;
                }
            }
        }
        node = wide_next(h, st, sp, tv, [](float) { return true; });
        if (tv.overflow) break;
        if (node < 0) {
            if (sp == 0) break;
            node = st.get_node(--sp);
        }
    }
    return found;
}

template <class Ops, bool kFill, bool kRange = false, class St>
__device__ __forceinline__ int radius_wide_one(const WideNode* __restrict__ wn,
                                               const float4* __restrict__ leaves, float3 p,
                                               float r2, int write, int end,
                                               unsigned long long* __restrict__ keys,
                                               int max_iter, St& st, Trav& tv) {
    SegmentSink sink{keys, write, end};
    return radius_wide_visit<Ops, kFill, kRange>(wn, leaves, p, r2, sink, max_iter, st, tv);
}

// ---------------------------------------------------------------------------------------
// split mode (QK_TUNE_SPLIT): one warp per query point.  The top kSplitLevels levels of the
// binary tree are descended with lane l taking child bit ((l >> level) & 1), so the 32 lanes
// own 32 disjoint subtrees (a leaf met on the way belongs to the lowest lane that reaches
// it); each lane then runs the ordinary depth-first traversal of its subtree.  After every
// step the warp shares its pruning bound by shuffles, so a query whose search touches much of
// the tree (a point near the centre of a spherical shell) is spread over 32 lanes.  The
// subtrees partition the leaves and the shared bound only ever comes from found candidates,
// so results equal the one-thread-per-query kernels bit for bit.
//
// Groups (QK_TUNE_SPLIT8 / QK_TUNE_SPLIT4): the same with G = 8 or 4 lanes per query, the top
// log2(G) levels split, every exchange restricted to the query's G aligned lanes (shuffle
// width G, the group's bits of each ballot).  Few queries then fill more of the GPU without
// 32-fold redundancy.  Warp-wide loop conditions keep every lane of the warp in the same
// collectives; a group past the last query traces query 0 and writes nothing.
// ---------------------------------------------------------------------------------------
constexpr int kSplitLevels = 5;

constexpr int log2_lanes(int g) { return g <= 1 ? 0 : 1 + log2_lanes(g / 2); }

// first lane of this thread's group of G lanes in its warp, and the group's ballot bits
template <int G>
__device__ __forceinline__ int group_base() { return (threadIdx.x & 31) & ~(G - 1); }
template <int G>
__device__ __forceinline__ unsigned group_bits(unsigned ballot) {
    return G == 32 ? ballot : (ballot >> group_base<G>()) & ((1u << G) - 1u);
}
template <int G>
__device__ __forceinline__ bool group_any(bool v) {
    return group_bits<G>(__ballot_sync(0xffffffffu, v)) != 0u;
}

template <int G = 32>
__device__ __forceinline__ void warp_min_lex(float& d, int& id) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        const float od = __shfl_xor_sync(0xffffffffu, d, o);
        const int oi = __shfl_xor_sync(0xffffffffu, id, o);
        if (closer(od, oi, d, id)) {
            d = od;
            id = oi;
        }
    }
}

// Forced descent of lane `lane` from the root: returns the subtree root the lane owns (an
// internal node) or -1; a leaf met on the way is handed to `on_leaf` by its owning lane.
// `keep(box)` decides whether a child box can still hold a result; `on_child(node, right)` sees
// every node the lane passes and the side it takes there.
template <int kLevels = kSplitLevels, class Leaf, class Keep, class Child>
__device__ __forceinline__ int split_descend(const BNode* __restrict__ bn, int lane, Leaf on_leaf,
                                             Keep keep, Child on_child) {
    int node = 0;
    for (int d = 0; d < kLevels; ++d) {
        const NodePair nd = load_pair(bn, node);
        const bool right = ((lane >> d) & 1) != 0;
        const int ref = right ? nd.rref : nd.lref;
        const float3 lo = boxq_lo(right ? nd.r : nd.l);
        const float3 hi = boxq_hi(right ? nd.r : nd.l);
        on_child(nd, right);
        if (ref < 0) {
            if ((lane >> (d + 1)) == 0 && keep(lo, hi)) on_leaf(~ref);
            return -1;
        }
        if (!keep(lo, hi)) return -1;
        node = ref;
    }
    return node;
}
template <int kLevels = kSplitLevels, class Leaf, class Keep>
__device__ __forceinline__ int split_descend(const BNode* __restrict__ bn, int lane, Leaf on_leaf,
                                             Keep keep) {
    return split_descend<kLevels>(bn, lane, on_leaf, keep, [](const NodePair&, bool) {});
}

// kFirst: one thread per query takes the first leaf it meets whatever its distance, so a NaN there
// (a query that is not finite, or a triangle with a = b) is its answer; a NaN met later is never
// closer.  The lane whose subtree holds that leaf then keeps to the one-thread path down to it,
// unpruned, and a NaN there is the group's answer too.
template <class Ops, int G = 32, bool kFirst = false>
__device__ __forceinline__ uint2 closest_split_one(const BNode* __restrict__ bn,
                                                   const float4* __restrict__ leaves, float3 p,
                                                   int lane, int max_iter, Trav& tv,
                                                   bool valid = true) {
    float best = kInf;
    int best_id = 0x7fffffff;
    bool first = kFirst;   // this lane is on the one-thread path and that has met no leaf
    float first_d = 0.0f;  // NaN: the answer is first_id
    int first_id = 0;
    auto on_leaf = [&](int slot) {
        ++tv.leaves;
        int id;
        const float d2 = Ops::dist2(p, leaves, slot, id, kFirst && first ? kInf : best);
        if (kFirst && first) {
            first_d = d2;
            first_id = id;
            first = false;
        }
        if (closer(d2, id, best, best_id)) {
            best = d2;
            best_id = id;
        }
    };
    // a lane leaves the one-thread path when its child is not the one that takes: a leaf before an
    // internal child, the nearer (left of equals) of two alike
    auto on_child = [&](const NodePair& nd, bool right) {
        float dl, dr;
        dist2_boxq2(vec3q(p), nd.l, nd.r, dl, dr);
        const bool ll = nd.lref < 0, rl = nd.rref < 0;
        const bool take_right = ll == rl ? !(dl <= dr) : rl;
        if (take_right != right) first = false;
    };
    int node = -1;
    if (valid) {
        if constexpr (kFirst)
            node = split_descend<log2_lanes(G)>(bn, lane, on_leaf, [](float3, float3) { return true; },
                                                on_child);
        else
            node = split_descend<log2_lanes(G)>(bn, lane, on_leaf, [](float3, float3) { return true; });
    }
    warp_min_lex<G>(best, best_id);
    const Vec3Q qp = vec3q(p);
    LocalStack<kStack> st;
    int sp = 0;
    bool active = node >= 0;
    for (int iter = 0; __any_sync(0xffffffffu, active); ++iter) {
        if (active) {
            if (iter >= max_iter) {
                tv.overflow = true;
                active = false;
            } else {
                ++tv.nodes;
                const NodePair nd = load_pair(bn, node);
                const int lref = nd.lref, rref = nd.rref;
                float dl, dr;
                dist2_boxq2(qp, nd.l, nd.r, dl, dr);
                bool okl = dl <= best || (kFirst && first);
                bool okr = dr <= best || (kFirst && first);
                const bool lfirst = dl <= dr;
                const int lslot = okl && lref < 0 ? ~lref : -1, rslot = okr && rref < 0 ? ~rref : -1;
                int leaf = lfirst ? lslot : rslot, other = lfirst ? rslot : lslot;
                const float dfar = lfirst ? dr : dl;
                if (leaf < 0) {
                    leaf = other;
                    other = -1;
                }
#pragma unroll 1
                while (leaf >= 0) {
                    on_leaf(leaf);
                    leaf = dfar <= best ? other : -1;
                    other = -1;
                }
                okl = okl && lref >= 0;
                okr = okr && rref >= 0;
                if (okl && okr) {
                    if (sp >= kStack) {
                        tv.overflow = true;
                        active = false;
                    } else {
                        st.put(sp++, lfirst ? rref : lref, lfirst ? dr : dl);
                        node = lfirst ? lref : rref;
                    }
                } else if (okl) {
                    node = lref;
                } else if (okr) {
                    node = rref;
                } else {
                    node = -1;
                    while (sp > 0) {
                        --sp;
                        int pn;
                        float pk;
                        st.get(sp, pn, pk);
                        if (pk <= best) {
                            node = pn;
                            break;
                        }
                    }
                    if (node < 0) active = false;
                }
            }
        }
        warp_min_lex<G>(best, best_id);
    }
    if constexpr (kFirst) {
        const unsigned nan = group_bits<G>(__ballot_sync(0xffffffffu, first_d != first_d));
        const int src = nan ? __ffs(nan) - 1 : 0;
        const float nd = __shfl_sync(0xffffffffu, first_d, src, G);
        const int ni = __shfl_sync(0xffffffffu, first_id, src, G);
        if (nan) return make_uint2(__float_as_uint(nd), static_cast<unsigned>(ni));
    }
    return best_id != 0x7fffffff ? make_uint2(__float_as_uint(best), static_cast<unsigned>(best_id))
                                 : make_uint2(0u, 0xffffffffu);
}

// kNN, split: the k best candidates form ONE warp-wide sorted table, entry j held by lane j
// (k <= 32), so every lane prunes with the exact k-th distance of everything found so far.
// After each traversal step the lanes' new leaf candidates (up to two per lane) are inserted
// one at a time: a ballot gives the insertion rank, a shuffle shifts the tail down.
struct WarpTable {
    float d;   // this lane's entry
    int id;
    float kd;  // entry k-1, broadcast
    int kid;
    __device__ __forceinline__ void init() {
        d = kInf;
        id = 0x7fffffff;
        kd = kInf;
        kid = 0x7fffffff;
    }
    __device__ __forceinline__ bool admits(float bound) const {
        return kid == 0x7fffffff || bound <= kd;
    }
    // whole warp; x is the same on every lane of a group, `lane` the lane in the group; a group
    // with doit false keeps its table (every lane still takes part in the exchanges)
    template <int G = 32>
    __device__ __forceinline__ void insert(float xd, int xid, int k, int lane, bool doit = true) {
        if constexpr (G < 32) {
            const bool want = doit && closer(xd, xid, kd, kid);
            const unsigned before = group_bits<G>(
                __ballot_sync(0xffffffffu, lane < k && closer(d, id, xd, xid)));
            const int pos = __popc(before);
            const float pd = __shfl_up_sync(0xffffffffu, d, 1, G);
            const int pid = __shfl_up_sync(0xffffffffu, id, 1, G);
            if (want && lane < k) {
                if (lane == pos) {
                    d = xd;
                    id = xid;
                } else if (lane > pos) {
                    d = pd;
                    id = pid;
                }
            }
            kd = __shfl_sync(0xffffffffu, d, k - 1, G);
            kid = __shfl_sync(0xffffffffu, id, k - 1, G);
            return;
        }
        if (!closer(xd, xid, kd, kid)) return;
        const unsigned before = __ballot_sync(0xffffffffu, lane < k && closer(d, id, xd, xid));
        const int pos = __popc(before);
        const float pd = __shfl_up_sync(0xffffffffu, d, 1);
        const int pid = __shfl_up_sync(0xffffffffu, id, 1);
        if (lane < k) {
            if (lane == pos) {
                d = xd;
                id = xid;
            } else if (lane > pos) {
                d = pd;
                id = pid;
            }
        }
        kd = __shfl_sync(0xffffffffu, d, k - 1);
        kid = __shfl_sync(0xffffffffu, id, k - 1);
    }
};

// the warp's (group's) table holds the query's k best on return (entry j in lane j; k <= G)
template <class Ops, int G = 32>
__device__ __forceinline__ void knn_split_one(const BNode* __restrict__ bn,
                                              const float4* __restrict__ leaves, float3 p, int k,
                                              int lane, int max_iter, Trav& tv, WarpTable& tab,
                                              bool valid = true) {
    tab.init();
    // up to two pending leaf candidates per lane (the first one first), inserted by the group
    float cd0 = 0.0f, cd1 = 0.0f;
    int cid0 = 0, cid1 = 0;
    bool has0 = false, has1 = false;
    auto leaf = [&](int slot) {
        ++tv.leaves;
        int id;
        const float d = Ops::dist2(p, leaves, slot, id, tab.kd);
        // a candidate past the k-th entry cannot enter: the entry only gets closer
        if (!closer(d, id, tab.kd, tab.kid)) return;
        if (has0) {
            cd1 = d;
            cid1 = id;
            has1 = true;
        } else {
            cd0 = d;
            cid0 = id;
            has0 = true;
        }
    };
    // every group inserts its own candidates, lowest lane first, until no group has one left
    auto flush = [&]() {
        if constexpr (G == 32) {
            unsigned m = __ballot_sync(0xffffffffu, has0), m1 = __ballot_sync(0xffffffffu, has1);
            for (; m; m &= m - 1) {
                const int src = __ffs(m) - 1;
                tab.insert(__shfl_sync(0xffffffffu, cd0, src), __shfl_sync(0xffffffffu, cid0, src), k,
                           lane);
            }
            for (; m1; m1 &= m1 - 1) {
                const int src = __ffs(m1) - 1;
                tab.insert(__shfl_sync(0xffffffffu, cd1, src), __shfl_sync(0xffffffffu, cid1, src), k,
                           lane);
            }
            has0 = has1 = false;
        } else {
            for (;;) {
                const unsigned all = __ballot_sync(0xffffffffu, has0);
                if (all == 0u) break;
                const unsigned m = group_bits<G>(all);
                const bool doit = m != 0u;
                const int src = doit ? __ffs(m) - 1 : 0;
                const float xd = __shfl_sync(0xffffffffu, cd0, src, G);
                const int xid = __shfl_sync(0xffffffffu, cid0, src, G);
                tab.insert<G>(xd, xid, k, lane, doit);
                if (doit && lane == src) {
                    cd0 = cd1;
                    cid0 = cid1;
                    has0 = has1;
                    has1 = false;
                }
            }
        }
    };
    int node = valid ? split_descend<log2_lanes(G)>(bn, lane, leaf, [](float3, float3) { return true; })
                     : -1;
    flush();
    const Vec3Q qp = vec3q(p);
    LocalStack<kStack> st;
    int sp = 0;
    bool active = node >= 0;
    for (int iter = 0; __any_sync(0xffffffffu, active); ++iter) {
        if (active) {
            if (iter >= max_iter) {
                tv.overflow = true;
                active = false;
            } else {
                ++tv.nodes;
                const NodePair nd = load_pair(bn, node);
                const int lref = nd.lref, rref = nd.rref;
                float dl, dr;
                // a warp per query keeps the schedulers busy enough for the packed form (city, k 16,
                // 200,000 queries: 5,550 us with scalar distances, 5,491 packed)
                dist2_boxq2<(G == 32)>(qp, nd.l, nd.r, dl, dr);
                const bool lfirst = dl <= dr;
                bool okl = tab.admits(dl);
                bool okr = tab.admits(dr);
                int lslot = okl && lref < 0 ? ~lref : -1;
                int other = okr && rref < 0 ? ~rref : -1;
                if (lslot < 0) {
                    lslot = other;
                    other = -1;
                }
#pragma unroll 1
                while (lslot >= 0) {
                    leaf(lslot);
                    lslot = other;
                    other = -1;
                }
                okl = okl && lref >= 0;
                okr = okr && rref >= 0;
                if (okl && okr) {
                    if (sp >= kStack) {
                        tv.overflow = true;
                        active = false;
                    } else {
                        st.put(sp++, lfirst ? rref : lref, lfirst ? dr : dl);
                        node = lfirst ? lref : rref;
                    }
                } else if (okl) {
                    node = lref;
                } else if (okr) {
                    node = rref;
                } else {
                    node = -1;
                    while (sp > 0) {
                        --sp;
                        int pn;
                        float pk;
                        st.get(sp, pn, pk);
                        if (tab.admits(pk)) {
                            node = pn;
                            break;
                        }
                    }
                    if (node < 0) active = false;
                }
            }
        }
        flush();
    }
}

__device__ __forceinline__ uint2 warp_table_entry(const WarpTable& tab) {
    return tab.id != 0x7fffffff ? make_uint2(__float_as_uint(tab.d), static_cast<unsigned>(tab.id))
                                : make_uint2(0u, 0xffffffffu);
}

// radius, split: hands this lane's keys to `sink` and returns their count.  Groups of 4 and 8 lanes
// take scalar box distances and both leaf tests in line, as radius_bin_visit's kFew (1 M points on a
// noisy shell, 8,000 queries on 4 lanes: 1,879 us packed with one copy of the test, 1,758 this way);
// whole warps the packed form (20,000 queries: 1,724 against 1,830).
template <class Ops, int G, class Sink>
__device__ __forceinline__ int radius_split_visit(const BNode* __restrict__ bn,
                                                  const float4* __restrict__ leaves, float3 p,
                                                  float r2, int lane, Sink& sink, int max_iter,
                                                  Trav& tv, bool valid) {
    int found = 0;
    auto keep = [&](float3 lo, float3 hi) { return dist2_box(p, lo, hi) <= r2; };
    auto on_leaf = [&](int slot) {
        ++tv.leaves;
        int id;
        const float d2 = Ops::dist2(p, leaves, slot, id, r2);
        if (d2 <= r2) {
            sink.put(radius_key(d2, id));
            ++found;
        }
    };
    int node = valid ? split_descend<log2_lanes(G)>(bn, lane, on_leaf, keep) : -1;
    const Vec3Q qp = vec3q(p);
    LocalStack<kStack> st;
    int sp = 0;
    for (int iter = 0; node >= 0; ++iter) {
        if (iter >= max_iter) {
            tv.overflow = true;
            break;
        }
        ++tv.nodes;
        const NodePair nd = load_pair(bn, node);
        const int lref = nd.lref, rref = nd.rref;
        float dl, dr;
        dist2_boxq2<(G == 32)>(qp, nd.l, nd.r, dl, dr);
        bool okl = dl <= r2;
        bool okr = dr <= r2;
        int leaf = okl && lref < 0 ? ~lref : -1;
        int other = okr && rref < 0 ? ~rref : -1;
        if (leaf < 0) {
            leaf = other;
            other = -1;
        }
        if constexpr (G < 32) {
            if (leaf >= 0) on_leaf(leaf);
            if (other >= 0) on_leaf(other);
        } else {
#pragma unroll 1
            while (leaf >= 0) {
                on_leaf(leaf);
                leaf = other;
                other = -1;
            }
        }
        okl = okl && lref >= 0;
        okr = okr && rref >= 0;
        if (okl && okr) {
            if (sp >= kStack) {
                tv.overflow = true;
                break;
            }
            st.put_node(sp++, rref);
            node = lref;
        } else if (okl) {
            node = lref;
        } else if (okr) {
            node = rref;
        } else {
            node = sp > 0 ? st.get_node(--sp) : -1;
        }
    }
    return found;
}

// the same as two passes: the count pass drops the keys, the fill pass writes them from `write` on,
// never past `end` (the query's offset plus the counts of the lower lanes)
template <class Ops, bool kFill, int G = 32>
__device__ __forceinline__ int radius_split_one(const BNode* __restrict__ bn,
                                                const float4* __restrict__ leaves, float3 p,
                                                float r2, int lane, int write, int end,
                                                unsigned long long* __restrict__ keys,
                                                int max_iter, Trav& tv, bool valid = true) {
    SegmentSink sink{keys, write, kFill ? end : write};
    return radius_split_visit<Ops, G>(bn, leaves, p, r2, lane, sink, max_iter, tv, valid);
}

// exclusive prefix over the lanes of `v` (of the group of G lanes; `lane` the lane in it)
template <int G = 32>
__device__ __forceinline__ int warp_exclusive(int v, int lane) {
    int incl = v;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o, G);
        if (lane >= o) incl += u;
    }
    return incl - v;
}

// sum of `v` over the group of G lanes (every lane gets it)
template <int G>
__device__ __forceinline__ int group_sum(int v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace qk
