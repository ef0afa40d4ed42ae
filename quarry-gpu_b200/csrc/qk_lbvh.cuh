// qk_lbvh.cuh -- the LBVH from sorted (code, id) keys in one pass over the leaves: leaf
// scatter, radix-tree links, boxes, traversal nodes, parents and depths.  Shared by the
// single-tree build (qk_build.cu) and the batched build (qk_batch.cu).
//
// The tree is the radix tree over the unique 64-bit keys (code << 32 | index), in Karras'
// numbering: internal node k is the one whose slot range starts (it is a right child) or ends
// (a left child) at slot k; node 0 is the root.  Write gap(g) for the common prefix length of
// keys g and g + 1 (-1 past either end).  A node covering slots [l, r] is a left child exactly
// when gap(r) > gap(l - 1), and then its parent splits at r; otherwise at l - 1 (Apetrei 2014).
// So a climb from the leaves knows every link, number, parent and slot range when two siblings
// meet, and the top-down range and split searches per node (about 2 log n dependent loads of
// the sorted codes), the separate pass for the boxes and the arrays between them are gone.
//
// One block takes 256 leaves.  A node inside the block (its split's gap exceeds some gap of
// the block on either side) is met in shared memory: the first sibling leaves its box and
// bound there, the second goes on.  The block's nodes then go out in whole sectors, and the
// climbs that reach a node spanning blocks (about a dozen per block) are listed for a second
// launch, one thread each, which meets siblings through device-scope exchanges: doing that in
// the first launch kept every block resident behind a device fence and a few threads' climbs
// (67 of the build's 308 us).
//
// Depths need no climb.  The ancestors of slot i have distinct prefix lengths: those at which
// the running minimum of the gaps changes going left from i, and going right.  As a 64-bit mask
// that is a scan: passing gap d keeps the bits below d and sets bit d.  depth(leaf i) is the
// popcount of the two masks, and depth(node k) the popcount below k's own prefix length, which
// is the lowest bit above the smaller of k's two gaps.  k_lbvh_carry finds the masks at block
// boundaries by one binary search per prefix length.
//
// 1,048,576 uniform points, one B200, under ncu: the emit with its searches (62 us), the boxes
// (108) and the depths (40) became this pass (88), the climbs that leave its blocks (46) and the
// masks (16).  The pass is bound by its chain of latencies (key, item, scans, climb), not by
// bytes: without the climb and the node writes the build takes 51 us less, without the scans 10.
#pragma once

#include "qk_build.cuh"

namespace qk {

constexpr int kLbvhSpan = 256;  // leaves (and threads) per block

// the arrays of one tree and its sorted keys
struct LbvhView {
    const float* items;     // scene order
    const uint32_t* codes;  // sorted
    const uint32_t* ids;    // sorted: scene indices
    int n;
    Node* nodes;
    float* sorted;
    int* prim_ids;
    int* slot_of;
    int* parent;
    int* depth;
    BNode* bnodes;
    float4* leaves;
    int* flags;  // n - 1 words, zero on entry and on exit
};

// Climbs left for the second launch: {block of the first launch, first | last slot << 8 inside
// it}.  Half an entry per leaf holds them all.  A climb leaves its block toward a node that spans
// the block's left or right end; the nodes across one end have distinct prefix lengths, of which
// there are 62 (2..63), and each has at most one child inside the block.  So a block hands over at
// most 124 climbs (128 entries for 256 leaves), a tree's first block at most 62 and its last, with
// m leaves, at most min(m, 62), which the first's spare entries cover; a tree of one block none.
struct LbvhPending {
    uint2* list;
    int* count;  // zero before the first launch
};

// block-boundary masks of prefix lengths (see above): to the left of a block's first slot, to
// the right of its last
struct LbvhCarry {
    unsigned long long left, right;
};

__device__ __forceinline__ int key_gap(const LbvhView& v, int g) {
    if (g < 0 || g >= v.n - 1) return -1;
    return __clzll(key64(v.codes, v.ids, g) ^ key64(v.codes, v.ids, g + 1));
}

// first slot of [lo, hi) whose key is at least `target`
__device__ __forceinline__ int key_lower_bound(const LbvhView& v, int lo, int hi, uint64_t target) {
    const uint32_t tc = static_cast<uint32_t>(target >> 32), ti = static_cast<uint32_t>(target);
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const uint32_t c = v.codes[mid];
        if (c < tc || (c == tc && ti != 0u && v.ids[mid] < ti)) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// One warp: the masks at the boundary between slots base - 1 and base.  They share `d0` bits;
// at a shorter prefix length d an ancestor of both splits exactly when some key with the same
// d bits differs in the next one: to the left if that bit of theirs is 1, else to the right.
__device__ __forceinline__ void lbvh_boundary(const LbvhView& v, int base, int lane,
                                              unsigned long long& left,
                                              unsigned long long& right) {
    const uint64_t k0 = key64(v.codes, v.ids, base - 1), k1 = key64(v.codes, v.ids, base);
    const int d0 = __clzll(k0 ^ k1);
    left = right = 1ull << d0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int d = lane + 32 * h;
        bool hit = false;
        const uint64_t bit = 1ull << (63 - d);
        if (d >= 2 && d < d0) {  // codes have 30 bits
            const uint64_t prefix = (k1 >> (64 - d)) << (64 - d);
            if (k1 & bit) {
                const int at = key_lower_bound(v, 0, base, prefix);
                hit = at < base && key64(v.codes, v.ids, at) < (prefix | bit);
            } else {
                const int at = key_lower_bound(v, base, v.n, prefix | bit);
                hit = at < v.n && (key64(v.codes, v.ids, at) >> (64 - d)) == (k1 >> (64 - d));
            }
        }
        const unsigned l = __ballot_sync(0xffffffffu, hit && (k1 & bit) != 0);
        const unsigned r = __ballot_sync(0xffffffffu, hit && (k1 & bit) == 0);
        left |= static_cast<unsigned long long>(l) << (32 * h);
        right |= static_cast<unsigned long long>(r) << (32 * h);
    }
}

// A run of gaps as the mask map x -> (x & below(lo)) | set: lo its smallest gap (64: no gap).
struct GapRun {
    int lo;
    unsigned long long set;
};
__device__ __forceinline__ unsigned long long bits_below(int d) {
    return d >= 64 ? ~0ull : (d <= 0 ? 0ull : (1ull << d) - 1ull);
}
__device__ __forceinline__ GapRun gap_run(int d) { return {d, d < 0 ? 0ull : 1ull << d}; }
// the map of `a` followed by that of `b`
__device__ __forceinline__ GapRun gap_then(const GapRun& a, const GapRun& b) {
    return {min(a.lo, b.lo), (a.set & bits_below(b.lo)) | b.set};
}
__device__ __forceinline__ unsigned long long gap_apply(const GapRun& r, unsigned long long x) {
    return (x & bits_below(r.lo)) | r.set;
}

struct LbvhShared {
    union {
        float box[12][kLbvhSpan + 1];  // by gap: left child lo xyz hi xyz, right child's
        float stage[kLbvhSpan / 32][32 * 12];  // leaf staging, before the climb
    };
    int ref[2][kLbvhSpan];   // by gap: child references (>= 0 internal, else ~slot)
    int code[2][kLbvhSpan];  // ... and small-subtree codes
    int idx[kLbvhSpan];      // by gap: the node's number, -1 until both children arrived
    int bound[kLbvhSpan];    // by gap: 1 + outer end of the first arrival's range
    int par_leaf[kLbvhSpan], par_node[kLbvhSpan];
    int gap[kLbvhSpan + 1];  // gap[j]: gap base - 1 + j
    GapRun run[2][kLbvhSpan / 32];
    unsigned inside[kLbvhSpan / 32];  // bit per gap: its node lies inside the block
};

__device__ __forceinline__ int lbvh_exchange(int* word, int v) {
    int old;
    asm volatile("atom.acq_rel.gpu.global.exch.b32 %0, [%1], %2;"
                 : "=r"(old)
                 : "l"(word), "r"(v)
                 : "memory");
    return old;
}

__device__ __forceinline__ Box box_union(const Box& a, const Box& b) {
    Box u;
    u.lo = f3(fmin_t(a.lo.x, b.lo.x), fmin_t(a.lo.y, b.lo.y), fmin_t(a.lo.z, b.lo.z));
    u.hi = f3(fmax_t(a.hi.x, b.hi.x), fmax_t(a.hi.y, b.hi.y), fmax_t(a.hi.z, b.hi.z));
    return u;
}

// small-subtree code of the internal node covering slots [l, r]
__device__ __forceinline__ int range_code(int l, int r) {
    return r - l < kLeafMax ? (l << 2) | (r - l) : 0;
}

// One climb through nodes that span blocks, from the finished node (or leaf) covering slots
// [L, R], whose box is in device memory.
__device__ __forceinline__ void lbvh_climb_out(const LbvhView& v, int L, int R) {
    const int n = v.n;
    const auto canonical = [&](int c) { return c < 0 ? n - 1 + ~c : c; };
    int dl = key_gap(v, L - 1), dr = key_gap(v, R);
    int ref = L == R ? ~L : (dr > dl ? R : L);
    int code = L == R ? 0 : range_code(L, R);
    Box box = load_box_cg(v.nodes + canonical(ref));
    for (int guard = 0; guard < 64; ++guard) {  // a path has at most 62 nodes
        const bool left = dr > dl;
        const int g = left ? R : L - 1;
        const int far = lbvh_exchange(v.flags + g, (left ? L : R) + 1);
        if (far == 0) return;
        v.flags[g] = 0;
        const int end = far - 1;
        // the sibling: [R + 1, end] on the right, [end, L - 1] on the left
        const int near = left ? R + 1 : L - 1;
        const int sref = end == near ? ~near : near;
        const int scode = end == near ? 0 : range_code(min(near, end), max(near, end));
        const Box hb = load_box_cg(v.nodes + canonical(sref));
        if (left) {
            R = end;
            dr = key_gap(v, R);
        } else {
            L = end;
            dl = key_gap(v, L - 1);
        }
        const bool root = dl < 0 && dr < 0;
        const int idx = root ? 0 : (dr > dl ? R : L);
        const Box a = left ? box : hb, b = left ? hb : box;
        const int lref = left ? ref : sref, rref = left ? sref : ref;
        box = box_union(a, b);
        float4* np = reinterpret_cast<float4*>(v.nodes + idx);
        np[0] = make_float4(box.lo.x, box.lo.y, box.lo.z, box.hi.x);
        np[1] = make_float4(box.hi.y, box.hi.z, __int_as_float(canonical(lref)),
                            __int_as_float(canonical(rref)));
        float4* bp = reinterpret_cast<float4*>(v.bnodes + idx);
        bp[0] = make_float4(a.lo.x, a.lo.y, a.lo.z, a.hi.x);
        bp[1] = make_float4(a.hi.y, a.hi.z, b.lo.x, b.lo.y);
        bp[2] = make_float4(b.lo.z, b.hi.x, b.hi.y, b.hi.z);
        bp[3] = make_float4(__int_as_float(lref), __int_as_float(rref),
                            __int_as_float(left ? code : scode),
                            __int_as_float(left ? scode : code));
        v.parent[canonical(lref)] = idx;
        v.parent[canonical(rref)] = idx;
        if (root) return;
        ref = idx;
        code = range_code(L, R);
    }
}

// Slots [base, base + 256) of one tree, by a block of 256 threads; the tree's largest depth is
// raised in *max_depth and the climbs that leave the block go to `pending` under `block`.
template <class Ops>
__device__ __forceinline__ void lbvh_block(const LbvhView& v, int base, const LbvhCarry& carry,
                                           int* max_depth, const LbvhPending& pending, int block,
                                           LbvhShared& sh) {
    static_assert(emit_stage_floats<Ops>() <= 32 * 12, "leaf staging fits the shared union");
    const int n = v.n, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int k = base + t;
    const bool in = k < n;

    // gaps, and this slot's primitive
    const int d = key_gap(v, k);
    sh.gap[t + 1] = d;
    if (t == 0) sh.gap[0] = key_gap(v, base - 1);
    sh.idx[t] = -1;
    sh.bound[t] = 0;
    sh.par_leaf[t] = -1;
    sh.par_node[t] = -1;
    const int src = in ? static_cast<int>(v.ids[k]) : 0;
    float it[Ops::kFloats];
#pragma unroll
    for (int j = 0; j < Ops::kFloats; ++j)
        it[j] = in ? v.items[static_cast<size_t>(src) * Ops::kFloats + j] : 0.0f;
    if (base + 32 * warp < n)
        store_leaves_warp<Ops>(it, src, n, v.nodes, v.sorted, v.prim_ids, v.slot_of, v.leaves,
                               base + 32 * warp, min(32, n - base - 32 * warp), sh.stage[warp]);
    Box box = Ops::bounds(it);

    // runs of gaps before this slot (exclusive, left to right) and from it on (right to left;
    // the block's last gap is in the carry)
    GapRun lr = gap_run(d), rr = t == kLbvhSpan - 1 ? GapRun{64, 0ull} : gap_run(d);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        GapRun a{__shfl_up_sync(0xffffffffu, lr.lo, o), __shfl_up_sync(0xffffffffu, lr.set, o)};
        GapRun b{__shfl_down_sync(0xffffffffu, rr.lo, o), __shfl_down_sync(0xffffffffu, rr.set, o)};
        if (lane >= o) lr = gap_then(a, lr);
        if (lane + o < 32) rr = gap_then(b, rr);
    }
    if (lane == 31) sh.run[0][warp] = lr;
    if (lane == 0) sh.run[1][warp] = rr;
    GapRun lx{__shfl_up_sync(0xffffffffu, lr.lo, 1), __shfl_up_sync(0xffffffffu, lr.set, 1)};
    if (lane == 0) lx = {64, 0ull};
    const int rx_lo = __shfl_down_sync(0xffffffffu, rr.lo, 1);
    __syncthreads();
    GapRun lw{64, 0ull}, rw{64, 0ull};
    for (int w = 0; w < warp; ++w) lw = gap_then(lw, sh.run[0][w]);
    for (int w = kLbvhSpan / 32 - 1; w > warp; --w) rw = gap_then(rw, sh.run[1][w]);
    lx = gap_then(lw, lx);
    rr = gap_then(rw, rr);
    const unsigned long long anc = gap_apply(lx, carry.left) | gap_apply(rr, carry.right);
    int leaf_depth = 0;
    if (in) {
        leaf_depth = __popcll(anc);
        v.depth[n - 1 + k] = leaf_depth;
        if (k < n - 1) {
            const int dmin = min(sh.gap[t], d);
            const unsigned long long own = anc & ~bits_below(dmin + 1);
            v.depth[k] = __popcll(anc & ((own & (0ull - own)) - 1ull));
        }
    }
    // a gap's node lies inside the block when smaller gaps of the block bound it on both sides
    const int before = min(sh.gap[0], lx.lo);
    const int after = min(sh.gap[kLbvhSpan], min(rw.lo, lane == 31 ? 64 : rx_lo));
    const bool inner = t < kLbvhSpan - 1 && d > before && d > after;
    const unsigned im = __ballot_sync(0xffffffffu, inner);
    if (lane == 0) sh.inside[warp] = im;
    block_max_to(leaf_depth, max_depth);
    __syncthreads();

    // climb inside the block
    int l = t, r = t, dl = sh.gap[l], dr = sh.gap[r + 1], ref = ~k, code = 0;
    bool on = in;  // still climbing
    while (on) {
        const bool left = dr > dl;
        const int g = left ? r : l - 1;
        if (g < 0 || !((sh.inside[g >> 5] >> (g & 31)) & 1u)) break;  // spans blocks
        const int side = left ? 0 : 1, other = 1 - side;
        float(*mine)[kLbvhSpan + 1] = sh.box + 6 * side;
        mine[0][g] = box.lo.x;
        mine[1][g] = box.lo.y;
        mine[2][g] = box.lo.z;
        mine[3][g] = box.hi.x;
        mine[4][g] = box.hi.y;
        mine[5][g] = box.hi.z;
        sh.ref[side][g] = ref;
        sh.code[side][g] = code;
        __threadfence_block();
        const int far = atomicExch(&sh.bound[g], (left ? l : r) + 1);
        __threadfence_block();
        if (far == 0) {
            on = false;
            break;
        }
        const float(*his)[kLbvhSpan + 1] = sh.box + 6 * other;
        Box hb;
        hb.lo = f3(his[0][g], his[1][g], his[2][g]);
        hb.hi = f3(his[3][g], his[4][g], his[5][g]);
        const int href = sh.ref[other][g];
        box = left ? box_union(box, hb) : box_union(hb, box);
        if (left) r = far - 1;
        else l = far - 1;
        dl = sh.gap[l];
        dr = sh.gap[r + 1];
        const int idx = (dl < 0 && dr < 0) ? 0 : base + (dr > dl ? r : l);
        sh.idx[g] = idx;
        if (ref < 0) sh.par_leaf[~ref - base] = idx;
        else sh.par_node[ref - base] = idx;
        if (href < 0) sh.par_leaf[~href - base] = idx;
        else sh.par_node[href - base] = idx;
        ref = idx;
        code = range_code(base + l, base + r);
        if (dl < 0 && dr < 0) on = false;  // the root
    }
    __syncthreads();

    // the block's nodes, in whole sectors
    if (k == 0) v.parent[0] = -1;
    if (sh.par_leaf[t] >= 0) v.parent[n - 1 + k] = sh.par_leaf[t];
    if (sh.par_node[t] >= 0) v.parent[k] = sh.par_node[t];
    const auto canonical = [&](int c) { return c < 0 ? n - 1 + ~c : c; };
#pragma unroll
    for (int i = t; i < 2 * kLbvhSpan; i += kLbvhSpan) {
        const int g = i >> 1, idx = sh.idx[g];
        if (idx < 0) continue;
        const float(*b)[kLbvhSpan + 1] = sh.box;
        float4 q;
        if (i & 1)
            q = make_float4(fmax_t(b[4][g], b[10][g]), fmax_t(b[5][g], b[11][g]),
                            __int_as_float(canonical(sh.ref[0][g])),
                            __int_as_float(canonical(sh.ref[1][g])));
        else
            q = make_float4(fmin_t(b[0][g], b[6][g]), fmin_t(b[1][g], b[7][g]),
                            fmin_t(b[2][g], b[8][g]), fmax_t(b[3][g], b[9][g]));
        reinterpret_cast<float4*>(v.nodes + idx)[i & 1] = q;
    }
#pragma unroll
    for (int i = t; i < 4 * kLbvhSpan; i += kLbvhSpan) {
        const int g = i >> 2, part = i & 3, idx = sh.idx[g];
        if (idx < 0) continue;
        const float(*b)[kLbvhSpan + 1] = sh.box + 4 * part;
        const float4 q = part < 3 ? make_float4(b[0][g], b[1][g], b[2][g], b[3][g])
                                  : make_float4(__int_as_float(sh.ref[0][g]),
                                                __int_as_float(sh.ref[1][g]),
                                                __int_as_float(sh.code[0][g]),
                                                __int_as_float(sh.code[1][g]));
        reinterpret_cast<float4*>(v.bnodes + idx)[part] = q;
    }
    // climbs that left the block
    const unsigned om = __ballot_sync(0xffffffffu, on);
    if (lane == 0) sh.inside[warp] = __popc(om);
    __syncthreads();
    unsigned at = __popc(om & ((1u << lane) - 1u)), all = 0;
#pragma unroll
    for (int w = 0; w < kLbvhSpan / 32; ++w) {
        at += w < warp ? sh.inside[w] : 0u;
        all += sh.inside[w];
    }
    if (all == 0) return;
    if (t == 0) sh.bound[0] = atomicAdd(pending.count, static_cast<int>(all));
    __syncthreads();
    if (on)
        pending.list[sh.bound[0] + static_cast<int>(at)] =
            make_uint2(static_cast<unsigned>(block), static_cast<unsigned>(l | (r << 8)));
}

}  // namespace qk
