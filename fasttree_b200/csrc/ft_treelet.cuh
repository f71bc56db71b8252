// ft_treelet.cuh -- topology, boxes and records of a radix tree over sorted keys, built bottom up
// in blocks of consecutive leaves (src/hlbvh.hpp:852-969: Karras topology and refit).
//
// A node that covers leaves [l, r] joins the neighbour it shares the longer key prefix with: its
// parent's split is the pair (r, r + 1) when delta(r) > delta(l - 1), else (l - 1, l), with
// delta(x) the common prefix of the sorted keys x and x + 1 (the agglomerative form of the binary
// radix tree, Apetrei 2014).  It is therefore the Karras tree of the same keys, and every node
// takes its Karras number: a left child the last leaf it covers, a right child the first, the
// root 0.
//
// A block takes kTreeletLeaves consecutive leaves.  Climbs meet in shared memory as long as both
// sides of a split lie in the block; one whose split or sibling reaches beyond the block's edge
// is left for the end.  Then the block writes every node it formed -- boxes, children, counts and
// heights as coalesced arrays, node records, and the fast walks' records -- all of whose
// descendants are in shared memory.
// The climbs that left their blocks (about one leaf in 25) meet again the same way, the climbs of
// 16 blocks in one block, level by level (treelet_join_kernel).  Climbs that too large groups pass
// on end in global memory, where the second arrival at a split (one acquire-release exchange)
// forms the node; a last launch makes the walk records of the nodes formed outside a block of
// leaves.
//
// Bound: with one climb step per level in global memory the refit alone was bound by the
// latency of its atomics (1.27 ms for 10M uint64 points, after 0.34 ms of binary searches for the
// topology, 0.60 ms of gather and 0.78 ms for the walk records: 3.0 ms).  In shared memory a step
// is some tens of cycles and each array moves once: treelets 1.31, joins 0.19, walk records of the
// nodes outside 0.05 ms.  The treelets move 3.0 TB/s; what holds them back is the L1's share of the
// scattered record stores (32-byte stores: 3.09 -> 2.96 ms for the build) and the barriers between
// their phases.  Leaves / threads of a block: 512 / 256 2.96, 1024 / 512 2.95 (refit of 3M float64
// points 764 against 742 us), 256 / 128 3.09, 512 / 512 3.13 ms.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ft_build_dev.cuh"
#include "ft_common.cuh"
#include "ft_qtree.cuh"

namespace ft {

// Which of a sort's two buffers holds its pairs: the passes that ran (skip: null, or a word per
// pass, set when it moved nothing).
FT_D int sort_parity(const uint32_t *skip, int passes) {
    int p = 0;
    for (int d = 0; d < passes; ++d) p ^= (skip && skip[d]) ? 0 : 1;
    return p;
}

static constexpr int kTreeletLeaves = 512, kTreeletThreads = 256;
static_assert(kTreeletLeaves <= kDenseLeaves, "no node inside a block is dense");

// A point of the sort's input order in one 16- or 32-byte sector: the gather by permutation reads
// one sector a leaf, not three.
template <class T> struct alignas(sizeof(T) * 4) PackedPoint {
    T x, y, z, pad; // pad: the low key word of 64-bit integer positions
};

// Where the leaves come from.
enum TreeletSource {
    LEAVES_PACKED = 0, // pack[perm[i]]: the build; also writes id, ghost, orig
    LEAVES_IN_PLACE = 1, // the leaf slots hold them: points, or boxes of the caller's (QFLAG_BOXES)
    LEAVES_MOVED = 2   // new positions x / y / z of the points in the leaves (refit)
};

template <class T> struct TreeletArgs {
    int                       n, periodic;
    const unsigned long long *klo, *khi; // sorted keys (LEAVES_PACKED: key / perm instead)
    const unsigned long long *key[2];    // LEAVES_PACKED: the sort's buffers; those that hold the
    const uint32_t           *perm[2];   // pairs follow from the passes that ran
    const uint32_t           *skip;
    int                       passes;
    const uint32_t           *stop;      // null, or a word that is set when nothing is to be built
    unsigned long long       *klo_out;   // LEAVES_PACKED, 126-bit keys: the sorted low words
    const PackedPoint<T>     *pack;
    const T                  *x, *y, *z; // LEAVES_MOVED
    int                       leaf_order;
    const uint32_t           *id;
    const int8_t             *ghost;
    const T                  *box; // the points' box (6 coordinates), from which the frame follows
    T                        *soa[6];
    int32_t                  *left, *right, *parent, *orig;
    uint32_t                 *id_out;
    int8_t                   *ghost_out;
    NodeRec<T>               *recs;
    uint8_t                  *height;
    int32_t                  *leaves;
    QRec                     *qrec;
    QPoint                   *qpts;
    uint32_t                 *qflag; // four words, zero: the tree's flag, nodes in `list`, entries of
                                     // `left_over` taken, entries of `left_over`
    int32_t                  *slot;       // n words, -1
    uint32_t                 *pend, *pend_count; // climbs that left a block of leaves: from its first
                                                 // leaf's place on, and their number (null: one block)
    uint32_t                 *left_over;  // climbs that left the joins too
    int32_t                  *list;       // nodes formed outside a block
    uint32_t                 *status;
};

// A child of a node by its leaf range; `right`: a right child (which numbers it).
struct TreeletChild {
    int  l, r;
    bool right;
    FT_D int count() const { return r - l + 1; }
    FT_D int node() const { return right ? l : r; } // internal number (l < r)
};

// The walk record of a node covering [l, r] with split s (dense: see qdense): its two children, then twice the child
// with the most leaves (more than kBucket) replaced by its own two.  split(c): the split of
// internal child c; box(c, b): its box.
template <class T, class Split, class Box>
FT_D void treelet_qrec(int l, int r, int s, bool dense, const QFrame<T> &f, QRec *out, Split split, Box box) {
    TreeletChild ch[4] = {{l, s, false}, {s + 1, r, true}, {0, -1, false}, {0, -1, false}};
    int          c     = 2;
#pragma unroll
    for (int step = 0; step < 2; ++step) {
        int b = -1, most = kBucket;
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (i < c && ch[i].count() > most) {
                b    = i;
                most = ch[i].count();
            }
        if (b < 0) break;
        const TreeletChild o  = b == 0 ? ch[0] : b == 1 ? ch[1] : ch[2];
        const int          os = split(o);
#pragma unroll
        for (int i = 3; i > 0; --i)
            if (i > b + 1) ch[i] = ch[i - 1]; // make room behind the opened child
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i == b) ch[i] = {o.l, os, false};
            else if (i == b + 1) ch[i] = {os + 1, o.r, true};
        }
        ++c;
    }
    uint32_t w[32];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        T b[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
        if (i < c) box(ch[i], b);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const uint32_t lo = (uint32_t)f.pos(b[2 * a], a), hi = (uint32_t)f.pos(b[2 * a + 1], a);
            const uint32_t ce = lo + ((hi - lo) >> 1);
            w[6 * i + a]      = ce;
            w[6 * i + 3 + a]  = (hi - ce) + f.m;
        }
        const int cnt = ch[i].count();
        w[24 + i]     = i >= c || dense ? kQEmpty : cnt <= kBucket ? qref_bucket(ch[i].l, cnt) : (uint32_t)ch[i].node();
        w[28 + i]     = i >= c ? 0u : (uint32_t)cnt;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        unsigned long long v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = (unsigned long long)w[8 * i + 2 * j + 1] << 32 | w[8 * i + 2 * j];
        st_words32(reinterpret_cast<unsigned char *>(out) + 32 * i, v);
    }
}

// A node's record for the exact traversals.
template <class T>
FT_D void treelet_noderec(NodeRec<T> *out, const T lb[6], const T rb[6], int lc, int rc, int nl, int nr, int hl, int hr) {
    NodeRec<T> rec;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        rec.lb[d] = lb[d];
        rec.rb[d] = rb[d];
    }
    rec.l = lc;
    rec.r = rc;
#pragma unroll
    for (int d = 0; d < (int)(sizeof(rec.pad) / 4); ++d) rec.pad[d] = 0;
    rec.pad[0] = (int32_t)rec_child_info((uint32_t)nl, (uint32_t)hl);
    rec.pad[1] = (int32_t)rec_child_info((uint32_t)nr, (uint32_t)hr);
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(&rec);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(rec) / 32); ++i) {
        const unsigned long long v[4] = {src[4 * i], src[4 * i + 1], src[4 * i + 2], src[4 * i + 3]};
        st_words32(reinterpret_cast<unsigned char *>(out) + 32 * i, v);
    }
}

// The root is formed.  The records are in the frame of a.box and a query takes the root box's: the
// two differ when the box was folded over points that are not the leaves (a refit whose original
// indices leave rows of its input out), and the frame does not serve the tree then.
template <class T> FT_D void treelet_root(const TreeletArgs<T> &a, const T box[6]) {
    a.parent[0] = -1;
    bool same   = true;
#pragma unroll
    for (int d = 0; d < 6; ++d) same = same && box[d] == a.box[d];
    if (!same) atomicOr(a.qflag, QFLAG_FRAME);
}

// delta of the adjacent sorted keys x and x + 1 (0 <= x < n - 1), plus one (0 is the border's).
// (not below one: keys wider than the reference's would differ above its prefix)
// lo: the sorted low words, or null (LEAVES_PACKED of 126-bit keys): they are in the packed points.
template <class T> struct TreeletKeys {
    const unsigned long long *lo, *hi;
    const uint32_t           *perm;
};
template <class T, int KIND> FT_D int treelet_delta(const TreeletArgs<T> &a, const TreeletKeys<T> &key, int x) {
    if constexpr (KIND == 2) {
        const unsigned long long p = key.hi[x], q = key.hi[x + 1];
        if (p != q) return max(clz64(p ^ q) - 1, 1);
        const unsigned long long u = key.lo ? key.lo[x] : (unsigned long long)a.pack[key.perm[x]].pad,
                                 v = key.lo ? key.lo[x + 1] : (unsigned long long)a.pack[key.perm[x + 1]].pad;
        if (u != v) return 63 + clz64(u ^ v);
        return 127 + clz64((unsigned long long)x ^ (unsigned long long)(x + 1));
    } else {
        const unsigned long long u = key.lo[x], v = key.lo[x + 1];
        if (u != v) return max(clz64(u ^ v) - (KIND == 1 ? 1 : 0) + 1, 1);
        return 64 + clz64((unsigned long long)x ^ (unsigned long long)(x + 1));
    }
}

template <class T> struct TreeletShared {
    T        lx[3][kTreeletLeaves];    // leaf positions
    T        bx[6][kTreeletLeaves];    // boxes of the nodes formed here, by their number in the block
    int32_t  slot[kTreeletLeaves];     // first arrival's far end at each split
    uint16_t nl[kTreeletLeaves], nr[kTreeletLeaves], ns[kTreeletLeaves]; // a node's leaves and split
    uint8_t  nh[kTreeletLeaves];       // height; 0: no node of this number here
    uint8_t  delta[kTreeletLeaves + 1]; // pairs (j - 1, j)
    uint16_t out[kTreeletLeaves];      // nodes (kTreeletLeaves +: leaves) that climb on outside
    int      outs; // their number
};

template <class T, int KIND, int SRC>
__global__ void __launch_bounds__(kTreeletThreads) treelet_kernel(const TreeletArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TreeletShared<T> &s  = *reinterpret_cast<TreeletShared<T> *>(smem_raw);
    const int         n = a.n, tid = threadIdx.x;
    const int         b0 = blockIdx.x * kTreeletLeaves, m = min(kTreeletLeaves, n - b0);
    if (SRC == LEAVES_PACKED && a.stop && *a.stop) return; // grid-uniform
    TreeletKeys<T> key = {a.klo, a.khi, nullptr};
    if constexpr (SRC == LEAVES_PACKED) {
        const int par = sort_parity(a.skip, a.passes);
        key.perm      = a.perm[par];
        if (KIND == 2) key = {nullptr, a.key[par], a.perm[par]};
        else key.lo = a.key[par];
    }
    QFrame<T>         f;
    f.make(a.box, n, a.periodic != 0);
    if (!f.ok && blockIdx.x == 0 && tid == 0) atomicOr(a.qflag, f.flag());

    // ---- leaves and deltas ----
    if (tid == 0) s.outs = 0;
    for (int j = tid; j < m; j += kTreeletThreads) {
        const int i = b0 + j;
        const int leaf = i + n - 1;
        T         p[3];
        if constexpr (SRC == LEAVES_PACKED) {
            const uint32_t       src = key.perm[i];
            const uint4         *q   = reinterpret_cast<const uint4 *>(a.pack + src);
            uint4                v[sizeof(T) / 4];
#pragma unroll
            for (int c = 0; c < (int)sizeof(T) / 4; ++c) v[c] = __ldg(q + c);
            const PackedPoint<T> &pt = *reinterpret_cast<const PackedPoint<T> *>(v);
            p[0] = pt.x;
            p[1] = pt.y;
            p[2] = pt.z;
            if constexpr (KIND == 2) a.klo_out[i] = (unsigned long long)pt.pad;
            a.id_out[leaf]    = a.id ? a.id[src] : src;
            a.ghost_out[leaf] = a.ghost ? a.ghost[src] : (int8_t)0;
            a.orig[leaf]      = (int32_t)src;
            if (i < n - 1) { // internal slots
                a.id_out[i]    = 0u;
                a.ghost_out[i] = (int8_t)0;
                a.orig[i]      = 0;
            }
        } else if constexpr (SRC == LEAVES_MOVED) {
            int64_t src = a.leaf_order ? (int64_t)i : (int64_t)a.orig[leaf];
            if (src < 0 || src >= (int64_t)n) { // (the slot keeps its position)
                atomicOr(a.status, STATUS_BAD_INPUT);
                atomicOr(a.qflag, QFLAG_FRAME); // (it may lie outside the new positions' box)
                p[0] = a.soa[0][leaf];
                p[1] = a.soa[2][leaf];
                p[2] = a.soa[4][leaf];
            } else {
                p[0] = a.x[src];
                p[1] = a.y[src];
                p[2] = a.z[src];
            }
        } else {
            p[0] = a.soa[0][leaf];
            p[1] = a.soa[2][leaf];
            p[2] = a.soa[4][leaf];
            if (!(a.soa[1][leaf] == p[0] && a.soa[3][leaf] == p[1] && a.soa[5][leaf] == p[2]))
                atomicOr(a.qflag, QFLAG_BOXES);
        }
        if constexpr (SRC != LEAVES_IN_PLACE) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                a.soa[2 * d][leaf]     = p[d];
                a.soa[2 * d + 1][leaf] = p[d];
            }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) s.lx[d][j] = p[d];
        a.qpts[i] = qpoint<T>(p[0], p[1], p[2], f, a.periodic != 0, a.qflag);
        s.slot[j] = -1;
        s.nh[j]   = 0;
    }
    for (int j = tid; j <= m; j += kTreeletThreads) {
        const int x = b0 + j - 1;
        s.delta[j]  = (x < 0 || x >= n - 1) ? 0 : (uint8_t)treelet_delta<T, KIND>(a, key, x);
    }
    __syncthreads();

    // a leaf's box: its point, or what the caller left in its slot
    auto leaf_box = [&](int j, T b[6]) {
        if constexpr (SRC == LEAVES_IN_PLACE) {
#pragma unroll
            for (int d = 0; d < 6; ++d) b[d] = a.soa[d][b0 + j + n - 1];
        } else {
#pragma unroll
            for (int d = 0; d < 3; ++d) b[2 * d] = b[2 * d + 1] = s.lx[d][j];
        }
    };
    // ---- climbs inside the block ----
    for (int j = tid; j < m; j += kTreeletThreads) {
        int l = j, r = j, sp = 0, h = 0;
        T   box[6];
        leaf_box(j, box);
        for (;;) {
            const int  dl = s.delta[l], dr = s.delta[r + 1];
            const bool root     = b0 + l == 0 && b0 + r == n - 1;
            const bool up_right = dr > dl;
            const int  ci       = root ? 0 : (up_right ? r : l);
            if (l < r) { // a node formed by this thread
#pragma unroll
                for (int d = 0; d < 6; ++d) s.bx[d][ci] = box[d];
                s.nl[ci] = (uint16_t)l;
                s.nr[ci] = (uint16_t)r;
                s.ns[ci] = (uint16_t)sp;
                s.nh[ci] = (uint8_t)min(h, 255);
            }
            if (root) break;
            const int split = up_right ? r : l - 1;
            if (split < 0 || split + 1 >= m) { // the split lies on the block's edge
                const int o = atomicAdd(&s.outs, 1);
                s.out[o]    = (uint16_t)(l == r ? kTreeletLeaves + l : ci);
                break;
            }
            __threadfence_block();
            const int prev = atomicExch(&s.slot[split], up_right ? l : r);
            if (prev < 0) break; // first arrival: the sibling forms the parent
            s.slot[split] = -2;  // both have arrived
            __threadfence_block();
            const int sl = up_right ? split + 1 : prev, sr = up_right ? prev : split;
            const int si = up_right ? sl : sr; // the sibling's number
            T         sb[6];
            int       sh = 0;
            if (sl == sr) {
                leaf_box(sl, sb);
            } else {
                const volatile T *q = &s.bx[0][si];
#pragma unroll
                for (int d = 0; d < 6; ++d) sb[d] = q[d * kTreeletLeaves];
                sh = *(const volatile uint8_t *)&s.nh[si];
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) { // (left, right) order, as the refit merges
                box[2 * d]     = up_right ? box_min(box[2 * d], sb[2 * d]) : box_min(sb[2 * d], box[2 * d]);
                box[2 * d + 1] = up_right ? box_max(box[2 * d + 1], sb[2 * d + 1]) : box_max(sb[2 * d + 1], box[2 * d + 1]);
            }
            h  = 1 + max(h, sh);
            sp = split;
            l  = min(l, sl);
            r  = max(r, sr);
        }
    }
    __syncthreads();
    // splits where only one side arrived: the other reaches beyond the block's edge
    for (int j = tid; j < m - 1; j += kTreeletThreads) {
        const int far = s.slot[j];
        if (far < 0) continue;
        const int o  = atomicAdd(&s.outs, 1);
        const int at = far <= j ? j : j + 1; // [far, j] or [j + 1, far]
        s.out[o]     = (uint16_t)(far == at ? kTreeletLeaves + at : at);
    }

    // ---- the nodes formed here ----
    auto child_box = [&](const TreeletChild &c, T b[6]) {
        if (c.l == c.r) {
            leaf_box(c.l - b0, b);
        } else {
#pragma unroll
            for (int d = 0; d < 6; ++d) b[d] = s.bx[d][c.node() - b0];
        }
    };
    for (int j = tid; j < m; j += kTreeletThreads) {
        const int h = s.nh[j];
        if (h == 0) continue;
        const int          v = b0 + j, l = b0 + s.nl[j], r = b0 + s.nr[j], sp = b0 + s.ns[j];
        const TreeletChild cl = {l, sp, false}, cr = {sp + 1, r, true};
        const int          lc = l == sp ? l + n - 1 : sp, rc = sp + 1 == r ? r + n - 1 : sp + 1;
        T                  lb[6], rb[6];
        child_box(cl, lb);
        child_box(cr, rb);
#pragma unroll
        for (int d = 0; d < 6; ++d) a.soa[d][v] = s.bx[d][j];
        a.left[v]   = lc;
        a.right[v]  = rc;
        a.parent[lc] = v;
        a.parent[rc] = v;
        a.leaves[v] = r - l + 1;
        a.height[v] = (uint8_t)h;
        if (v == 0) { // (number 0 is the root's)
            const T rb0[6] = {s.bx[0][0], s.bx[1][0], s.bx[2][0], s.bx[3][0], s.bx[4][0], s.bx[5][0]};
            treelet_root<T>(a, rb0);
        }
        treelet_noderec<T>(a.recs + v, lb, rb, lc, rc, cl.count(), cr.count(), l == sp ? 0 : s.nh[sp - b0],
                           sp + 1 == r ? 0 : s.nh[sp + 1 - b0]);
        if (v == 0 || r - l + 1 > kBucket)
            treelet_qrec<T>(l, r, sp, false, f, a.qrec + v,
                            [&](const TreeletChild &c) { return b0 + (int)s.ns[c.node() - b0]; }, child_box);
    }
    __syncthreads();

    // ---- climbs that leave the block ----
    const int outs = s.outs;
    if (tid == 0 && a.pend_count) a.pend_count[blockIdx.x] = (uint32_t)outs;
    for (int o = tid; o < outs; o += kTreeletThreads) { // (into this block's part of the array)
        const int code = s.out[o];
        uint32_t  w;
        if (code >= kTreeletLeaves) w = ((uint32_t)(b0 + code - kTreeletLeaves) << 2) | 2u;
        else w = ((uint32_t)(b0 + code) << 2) | (code == (int)s.nr[code] ? 1u : 0u);
        a.pend[b0 + o] = w;
    }
}

// Leaf range of a climb that left its block (number << 2 | leaf << 1 | (number is the last leaf)).
template <class T> FT_D void treelet_range(const TreeletArgs<T> &a, uint32_t w, int &l, int &r) {
    const int  v    = (int)(w >> 2);
    const bool leaf = (w & 2u) != 0u;
    const int  c    = leaf ? 1 : a.leaves[v];
    l               = (leaf || !(w & 1u)) ? v : v - c + 1;
    r               = l + c - 1;
}

// The climbs that left kJoinBlocks consecutive blocks, in one block: the same as treelet_kernel's
// with those subtrees in the leaves' place (some 20 a block).  Launched level by level, the blocks
// of one level being the next one's groups, until one block is left; a group of more than
// kJoinItems passes its climbs on as they are.  What the last level leaves goes to
// treelet_climb_kernel (a level takes 12 to 16 us, the climbs of 100K points one by one 44 us).
struct JoinLevel {
    const uint32_t *in, *in_count; // segment b: in_count[b] entries from in + b * stride on
    int             segs;
    size_t          stride;
    uint32_t       *out, *out_count; // this level's segments; out_count null: one list, its length
};                                   // in qflag[3]
static constexpr int kJoinBlocks = 16, kJoinItems = 512, kJoinThreads = 256;
template <class T> struct JoinShared {
    T        ib[6][kJoinItems]; // the items' boxes
    T        bx[6][kJoinItems]; // boxes of the nodes formed here
    int32_t  il[kJoinItems], ir[kJoinItems], slot[kJoinItems];
    uint32_t code[kJoinItems]; // unsorted entries
    uint32_t out[kJoinItems];
    uint16_t nl[kJoinItems], nr[kJoinItems], ns[kJoinItems];
    uint8_t  ih[kJoinItems], nh[kJoinItems], delta[kJoinItems + 1];
    int      start[kJoinBlocks + 1];
    int      outs, base;
};
template <class T, int KIND, int SRC>
__global__ void __launch_bounds__(kJoinThreads) treelet_join_kernel(const TreeletArgs<T> a, const JoinLevel lv) {
    if (SRC == LEAVES_PACKED && a.stop && *a.stop) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    JoinShared<T> &s   = *reinterpret_cast<JoinShared<T> *>(smem_raw);
    const int      tid = threadIdx.x, n = a.n;
    const int      t0 = blockIdx.x * kJoinBlocks, nb = min(kJoinBlocks, lv.segs - t0);
    uint32_t      *out = lv.out + (lv.out_count ? (size_t)t0 * lv.stride : 0);
    TreeletKeys<T> key = {a.klo, a.khi, nullptr};
    if constexpr (SRC == LEAVES_PACKED) {
        const int par = sort_parity(a.skip, a.passes);
        if (KIND == 2) key = {a.klo_out, a.key[par], nullptr}; // (the low words are written out by now)
        else key.lo = a.key[par];
    }
    if (tid == 0) {
        int c = 0;
        for (int b = 0; b < nb; ++b) {
            s.start[b] = c;
            c += (int)lv.in_count[t0 + b];
        }
        s.start[nb] = c;
        s.outs      = 0;
    }
    __syncthreads();
    const int m = s.start[nb];
    auto place = [&](int count) { // where this block's entries go (every thread calls it)
        if (tid == 0) {
            if (lv.out_count) lv.out_count[blockIdx.x] = (uint32_t)count;
            s.base = lv.out_count ? 0 : (int)atomicAdd(a.qflag + 3, (uint32_t)count);
        }
        __syncthreads();
        return out + s.base;
    };
    if (m > kJoinItems) { // block-uniform: passed on as they are
        uint32_t *to = place(m);
        for (int b = 0; b < nb; ++b) {
            const int c = s.start[b + 1] - s.start[b];
            for (int o = tid; o < c; o += kJoinThreads) to[s.start[b] + o] = lv.in[(size_t)(t0 + b) * lv.stride + o];
        }
        return;
    }
    // ---- items in leaf order: by block, and inside a block by rank among its own ----
    for (int i = tid; i < m; i += kJoinThreads) {
        int b = 0;
        while (i >= s.start[b + 1]) ++b;
        const uint32_t w = lv.in[(size_t)(t0 + b) * lv.stride + (i - s.start[b])];
        s.code[i]        = w;
        int l, r;
        treelet_range<T>(a, w, l, r);
        s.slot[i] = l; // (for the ranks)
    }
    __syncthreads();
    for (int i = tid; i < m; i += kJoinThreads) {
        int b = 0;
        while (i >= s.start[b + 1]) ++b;
        const int mine = s.slot[i];
        int       at   = s.start[b];
        for (int o = s.start[b]; o < s.start[b + 1]; ++o) at += s.slot[o] < mine ? 1 : 0;
        const uint32_t w = s.code[i];
        int            l, r;
        treelet_range<T>(a, w, l, r);
        const int id = l == r ? l + n - 1 : (int)(w >> 2);
        s.il[at]     = l;
        s.ir[at]     = r;
        s.ih[at]     = l == r ? (uint8_t)0 : a.height[id];
        s.nh[at]     = 0;
#pragma unroll
        for (int d = 0; d < 6; ++d) s.ib[d][at] = a.soa[d][id];
    }
    __syncthreads();
    for (int i = tid; i <= m && m > 0; i += kJoinThreads) {
        const int x = i == 0 ? s.il[0] - 1 : s.ir[i - 1]; // the pair between items i - 1 and i
        s.delta[i]  = (x < 0 || x >= n - 1) ? 0 : (uint8_t)treelet_delta<T, KIND>(a, key, x);
        if (i < m) s.slot[i] = -1;
    }
    __syncthreads();
    // ---- climbs ----
    for (int j = tid; j < m; j += kJoinThreads) {
        int l = j, r = j, sp = 0, h = s.ih[j];
        T   box[6];
#pragma unroll
        for (int d = 0; d < 6; ++d) box[d] = s.ib[d][j];
        for (;;) {
            const int  dl = s.delta[l], dr = s.delta[r + 1];
            const bool root     = s.il[l] == 0 && s.ir[r] == n - 1;
            const bool up_right = dr > dl;
            const int  ci       = root ? 0 : (up_right ? r : l);
            if (l < r) {
#pragma unroll
                for (int d = 0; d < 6; ++d) s.bx[d][ci] = box[d];
                s.nl[ci] = (uint16_t)l;
                s.nr[ci] = (uint16_t)r;
                s.ns[ci] = (uint16_t)sp;
                s.nh[ci] = (uint8_t)min(h, 255);
            }
            if (root) break;
            const int split = up_right ? r : l - 1;
            if (split < 0 || split + 1 >= m) {
                s.out[atomicAdd(&s.outs, 1)] = (uint32_t)ci | (l == r ? 0x80000000u : 0u) | (up_right ? 0x40000000u : 0u);
                break;
            }
            __threadfence_block();
            const int prev = atomicExch(&s.slot[split], up_right ? l : r);
            if (prev < 0) break; // first arrival
            s.slot[split] = -2;
            __threadfence_block();
            const int sl = up_right ? split + 1 : prev, sr = up_right ? prev : split;
            const int si = up_right ? sl : sr;
            T         sb[6];
            const volatile T *q = sl == sr ? &s.ib[0][si] : &s.bx[0][si];
#pragma unroll
            for (int d = 0; d < 6; ++d) sb[d] = q[d * kJoinItems];
            const int sh = sl == sr ? s.ih[si] : *(const volatile uint8_t *)&s.nh[si];
#pragma unroll
            for (int d = 0; d < 3; ++d) { // (left, right) order
                box[2 * d]     = up_right ? box_min(box[2 * d], sb[2 * d]) : box_min(sb[2 * d], box[2 * d]);
                box[2 * d + 1] = up_right ? box_max(box[2 * d + 1], sb[2 * d + 1]) : box_max(sb[2 * d + 1], box[2 * d + 1]);
            }
            h  = 1 + max(h, sh);
            sp = split;
            l  = min(l, sl);
            r  = max(r, sr);
        }
    }
    __syncthreads();
    for (int j = tid; j < m - 1; j += kJoinThreads) { // splits where only one side arrived
        const int far = s.slot[j];
        if (far < 0) continue;
        const bool up = far <= j;
        const int  at = up ? j : j + 1;
        s.out[atomicAdd(&s.outs, 1)] = (uint32_t)at | (far == at ? 0x80000000u : 0u) | (up ? 0x40000000u : 0u);
    }
    // ---- the nodes formed here ----
    for (int j = tid; j < m; j += kJoinThreads) {
        const int h = s.nh[j];
        if (h == 0) continue;
        const int  x = s.nl[j], y = s.nr[j], sp = s.ns[j];
        const int  l = s.il[x], r = s.ir[y], sl = s.ir[sp]; // the split's last leaf
        const bool root = l == 0 && r == n - 1;
        const int  v    = root ? 0 : (j == y ? r : l);
        const int  lc = l == sl ? l + n - 1 : sl, rc = sl + 1 == r ? r + n - 1 : sl + 1;
        T          lb[6], rb[6];
#pragma unroll
        for (int d = 0; d < 6; ++d) {
            lb[d] = x == sp ? s.ib[d][x] : s.bx[d][sp];
            rb[d] = sp + 1 == y ? s.ib[d][y] : s.bx[d][sp + 1];
            a.soa[d][v] = s.bx[d][j];
        }
        a.left[v]    = lc;
        a.right[v]   = rc;
        a.parent[lc] = v;
        a.parent[rc] = v;
        a.leaves[v]  = r - l + 1;
        a.height[v]  = (uint8_t)h;
        if (root) {
            const T rb0[6] = {s.bx[0][j], s.bx[1][j], s.bx[2][j], s.bx[3][j], s.bx[4][j], s.bx[5][j]};
            treelet_root<T>(a, rb0);
        }
        treelet_noderec<T>(a.recs + v, lb, rb, lc, rc, sl - l + 1, r - sl, x == sp ? s.ih[x] : s.nh[sp],
                           sp + 1 == y ? s.ih[y] : s.nh[sp + 1]);
        if (root || r - l + 1 > kBucket) a.list[atomicAdd(a.qflag + 1, 1u)] = v;
    }
    __syncthreads();
    // ---- climbs that leave this block too ----
    const int outs = s.outs;
    uint32_t *to   = place(outs);
    for (int o = tid; o < outs; o += kJoinThreads) {
        const uint32_t w  = s.out[o];
        const int      at = (int)(w & 0xffffu);
        const bool     up = (w & 0x40000000u) != 0u;
        const int      x = (w & 0x80000000u) ? at : (int)s.nl[at], y = (w & 0x80000000u) ? at : (int)s.nr[at];
        const int      l = s.il[x], r = s.ir[y];
        to[o] = l == r ? ((uint32_t)l << 2) | 2u : up ? ((uint32_t)r << 2) | 1u : (uint32_t)l << 2;
    }
}

// The climbs that are left (a.left_over).  Warps take entries from a device counter (qflag[2]) and a lane whose climb ended
// takes the next one: one step a lane and round, as many lanes as possible.
template <class T, int KIND, int SRC>
__global__ void __launch_bounds__(128) treelet_climb_kernel(const TreeletArgs<T> a) {
    if (SRC == LEAVES_PACKED && a.stop && *a.stop) return;
    TreeletKeys<T> key = {a.klo, a.khi, nullptr};
    if constexpr (SRC == LEAVES_PACKED) {
        const int par = sort_parity(a.skip, a.passes);
        if (KIND == 2) key.hi = a.key[par]; // (the low words are written out by now)
        else key.lo = a.key[par];
        if (KIND == 2) key.lo = a.klo_out;
    }
    const unsigned FULL = 0xffffffffu;
    const int      lane = threadIdx.x & 31, n = a.n, total = (int)a.qflag[3];
    constexpr int  kChunk = 32;
    int            next = 0, end = 0; // the warp's chunk of entries (warp-uniform)
    bool           more = true, on = false;
    int            l = 0, r = 0, h = 0, dl = 0, dr = 0;
    T              box[6];
    for (;;) {
        unsigned idle = __ballot_sync(FULL, !on);
        while (idle && more) {
            if (next >= end) {
                int b = 0;
                if (lane == 0) b = (int)atomicAdd(a.qflag + 2, (uint32_t)kChunk);
                b = __shfl_sync(FULL, b, 0);
                if (b >= total) {
                    more = false;
                    break;
                }
                next = b;
                end  = min(b + kChunk, total);
            }
            const int take = min(__popc(idle), end - next);
            const int rank = __popc(idle & ((1u << lane) - 1u));
            if (!on && rank < take) {
                const uint32_t w = a.left_over[next + rank];
                treelet_range<T>(a, w, l, r);
                const int id = l == r ? l + n - 1 : (int)(w >> 2);
                h = l == r ? 0 : (int)a.height[id];
#pragma unroll
                for (int d = 0; d < 6; ++d) box[d] = a.soa[d][id];
                dl = l > 0 ? treelet_delta<T, KIND>(a, key, l - 1) : 0;
                dr = r < n - 1 ? treelet_delta<T, KIND>(a, key, r) : 0;
                on = true;
            }
            next += take;
            idle = __ballot_sync(FULL, !on);
        }
        if (!__any_sync(FULL, on)) break;
        if (on) {
            // the node [l, r] -- box, height and everything below it -- is in global memory
            const bool up_right = dr > dl;
            const int  ci       = l == r ? l + n - 1 : (up_right ? r : l);
            const int  split    = up_right ? r : l - 1;
            int        prev;
            asm volatile("atom.acq_rel.gpu.global.exch.b32 %0, [%1], %2;"
                         : "=r"(prev)
                         : "l"(a.slot + split), "r"(up_right ? l : r)
                         : "memory");
            if (prev < 0) {
                on = false; // first arrival
            } else {
                const int sl = up_right ? split + 1 : prev, sr = up_right ? prev : split;
                const int si = sl == sr ? sl + n - 1 : (up_right ? sl : sr);
                const int L  = min(l, sl), R = max(r, sr);
                T         sb[6], lb[6], rb[6];
#pragma unroll
                for (int d = 0; d < 6; ++d) sb[d] = __ldcg(a.soa[d] + si);
                const int sh = sl == sr ? 0 : (int)__ldcg(a.height + si);
                // only the far end's delta is new
                if (up_right) dr = R < n - 1 ? treelet_delta<T, KIND>(a, key, R) : 0;
                else dl = L > 0 ? treelet_delta<T, KIND>(a, key, L - 1) : 0;
                const bool root = L == 0 && R == n - 1;
                const int  v    = root ? 0 : (dr > dl ? R : L);
                const int  lc = up_right ? ci : si, rc = up_right ? si : ci;
                const int  hl = up_right ? h : sh, hr = up_right ? sh : h;
#pragma unroll
                for (int d = 0; d < 6; ++d) {
                    lb[d] = up_right ? box[d] : sb[d];
                    rb[d] = up_right ? sb[d] : box[d];
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    box[2 * d]     = box_min(lb[2 * d], rb[2 * d]);
                    box[2 * d + 1] = box_max(lb[2 * d + 1], rb[2 * d + 1]);
                }
                h = min(255, 1 + max(hl, hr));
#pragma unroll
                for (int d = 0; d < 6; ++d) __stcg(a.soa[d] + v, box[d]);
                __stcg(a.height + v, (uint8_t)h);
                a.left[v]    = lc;
                a.right[v]   = rc;
                a.parent[lc] = v;
                a.parent[rc] = v;
                a.leaves[v]  = R - L + 1;
                if (root) treelet_root<T>(a, box);
                treelet_noderec<T>(a.recs + v, lb, rb, lc, rc, split - L + 1, R - split, hl, hr);
                if (root || R - L + 1 > kBucket) a.list[atomicAdd(a.qflag + 1, 1u)] = v;
                l  = L;
                r  = R;
                on = !root;
            }
        }
    }
}

// The walk records of the nodes formed outside a block (the list), from the finished arrays.
template <class T>
__global__ void __launch_bounds__(128) treelet_qrec_kernel(const TreeletArgs<T> a) {
    if (a.stop && *a.stop) return;
    const int n = a.n, cnt = (int)a.qflag[1];
    QFrame<T> f;
    f.make(a.box, n, a.periodic != 0);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        const int v = a.list[i];
        // the node's leaves follow from its side: a left child's last leaf is its number
        const int  c  = a.leaves[v];
        const int  p  = v == 0 ? -1 : a.parent[v];
        const bool lf = p >= 0 && a.left[p] == v;
        const int  l  = v == 0 ? 0 : lf ? v - c + 1 : v, r = l + c - 1;
        auto       split_of = [&](int node) {
            const int x = a.left[node];
            return x >= n - 1 ? x - (n - 1) : x;
        };
        T own[6];
#pragma unroll
        for (int d = 0; d < 6; ++d) own[d] = a.soa[d][v];
        treelet_qrec<T>(l, r, split_of(v), qdense<T>(c, own, f), f, a.qrec + v,
                        [&](const TreeletChild &ch) { return split_of(ch.node()); },
                        [&](const TreeletChild &ch, T b[6]) {
                            const int id = ch.l == ch.r ? ch.l + n - 1 : ch.node();
#pragma unroll
                            for (int d = 0; d < 6; ++d) b[d] = a.soa[d][id];
                        });
    }
}

} // namespace ft
