// ft_walk.cuh -- the fast walk: one warp answers 32 neighbouring kNN queries (ft_fast.cu describes
// the steps).  Shared by the walk's own kernel and the persistent batched launch.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ft_common.cuh"
#include "ft_fast.h"
#include "ft_internal.h"
#include "ft_qtree.cuh"

namespace ft {

// Resident two-warp blocks the walk is compiled for (90 registers, no spills; 9 / 10 / 11 blocks
// 5.80 / 5.81 / 5.89 ms on 2M clustered uint64 points, k = 32).
#ifndef FT_FAST_MINB
#define FT_FAST_MINB 10
#endif
// The walk's schedule, measured on the same points (with it 2.2 times the lanes of a walk that
// lets each lane branch on its own run together, 14.4 -> 6.1 ms; the walk with exact 64-bit boxes
// down to single leaves took 9.4 ms):
//  * a warp expands while as many lanes want to as wait with a bucket (half / a quarter as many:
//    5.77 / 5.95 against 5.69 ms; every lane waiting at its first bucket: 5.82 ms);
//  * queues of 16 candidates a lane (12 / 24: 6.97 / 7.28 ms, the longer ones cost a block), offered
//    while kOfferLanes lanes have one (6 / 12 / 18 lanes: 6.91 / 6.82 / 6.82 ms).
static constexpr int kQueue = 16, kOfferLanes = 12;
static constexpr int kFastStack = 64; // binary walk
static constexpr int kWalkStack = 96; // 4-wide walk; a full stack hands the query to the replay
struct alignas(8) HeapEntry {
    float   key;
    int32_t leaf; // rank
};
// A block's shared memory: the heaps and the candidate queues (leaf ranks).
constexpr size_t fast_smem(int k, int threads) {
    return (size_t)threads * ((size_t)(k > 1 ? k : 1) * sizeof(HeapEntry) + kQueue * sizeof(int32_t));
}
// Warps per block: k <= 32 heaps take 8 KB a warp (two-warp blocks), 64-entry heaps 16 KB
// (one-warp blocks).
template <int KC> constexpr int fast_warps() { return KC > 32 ? 1 : 2; }
// The fast walk's heap entries are 8 bytes: a float key of the distance and the leaf rank.
// Float coordinates' distances are float sums widened to double (node_distance_sq), so their
// key is the distance itself, exactly.  Other types key a distance by rounding it toward zero
// to a float, which keeps the order (a < b implies key(a) <= key(b)): every decision the
// heap takes on two different keys is the one the exact distances would take, and a decision
// on equal keys (a candidate at the k-th key, an eviction leaving an equal maximum, equal keys
// in the sorted result) compares the exact distances, recomputed from the leaves.  The
// output distances are recomputed exactly from the leaves.  8 bytes instead of 12 (16 with
// alignment) an entry keep more warps resident and make the sifts 32-bit.
template <class T> constexpr bool heap_keyed() { return !std::is_same<T, float>::value; }
template <class T> FT_D float heap_key(typename Coord<T>::dist_t d) {
    if constexpr (!heap_keyed<T>()) return (float)d;
    else if constexpr (Coord<T>::is_float) return __double2float_rz(d);
    else return __ull2float_rz(d);
}
// The largest distance whose key is `key` (so a distance above it has a larger key).
template <class T> FT_D typename Coord<T>::dist_t heap_key_ub(float key) {
    if constexpr (!heap_keyed<T>()) {
        return (double)key;
    } else if constexpr (Coord<T>::is_float) {
        // distances are not negative; FLT_MAX keys every double from FLT_MAX up, infinity and
        // NaN key only themselves
        if (!(key < FLT_MAX)) return key == FLT_MAX ? DBL_MAX : (double)key;
        const float up = __uint_as_float(__float_as_uint(key) + 1u); // the next float
        return __longlong_as_double(__double_as_longlong((double)up) - 1ll); // the double below it
    } else {
        if (key < 16777216.0f) return (unsigned long long)key; // below 2^24 the key is exact
        const float up = __uint_as_float(__float_as_uint(key) + 1u); // an integer from 2^24 up
        return up >= 18446744073709551616.0f ? ~0ull : (unsigned long long)up - 1ull;
    }
}

// Four 8-byte values to a 32-byte aligned address, streaming.
template <class V> FT_D void st_sector(V *p, const V v[4]) {
    static_assert(sizeof(V) == 8, "one sector");
    unsigned long long w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if constexpr (std::is_floating_point<V>::value) w[i] = (unsigned long long)__double_as_longlong(v[i]);
        else w[i] = v[i];
    }
    asm volatile("st.global.cs.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(w[0]), "l"(w[1]), "l"(w[2]), "l"(w[3])
                 : "memory");
}

// A distance rounded up to a float (non-negative values): the key threshold of a bound for
// float coordinates, whose keys are the distances themselves.
template <class D> FT_D float key_up(D d) {
    if constexpr (std::is_floating_point<D>::value) return __double2float_ru((double)d);
    else return __ull2float_ru((unsigned long long)d);
}

// The reference's traversal stack (MAX_STACK_DEPTH 64) pushes the children of a popped
// internal node only while fewer than 62 entries are in use (src/hlbvh.hpp:1152, 1359, 1618,
// 1788); on taller trees it drops them.  It pushes the farther child first and the nearer
// one on top, so the entries below a popped node never change: after popping node v the
// stack holds exactly the number of nearer-child turns (ld2 <= rd2 takes the left child) on
// the root-to-v path, whatever the heap did.  The guard therefore fires only at an internal
// node whose path has 62 such turns, and it can change the query's rows only when that node
// lies within the query's k-th distance dk: a subtree beyond dk holds no neighbour, and no
// point under a node is nearer than the node's box.  Returns true when some internal node
// with 62 nearer-child turns lies within dk (then the reference traversal reruns the query).
// The search follows a child only while its subtree is tall enough to still reach 62 turns
// at an internal node (height >= 63 - turns); that slack never grows along a path and a far
// turn spends one, so trees of height <= 62 need no search and taller ones are searched near
// their tallest paths only.  Bounded: a search that runs long answers true.
// stk: scratch of kGuardStack entries (the walk's own stack, free by then).
static constexpr int kGuardStack = 80;
template <class T, int PER, bool COH = false>
FT_D bool stack_guard_reaches(const TreeDev<T> &t, T px, T py, T pz, typename Coord<T>::dist_t dk,
                              unsigned long long *stk) {
    using D = typename Coord<T>::dist_t;
    const int n = t.n;
    if (n < 2 || (int)t.height[0] < 63) return false;
    constexpr int kCap = kGuardStack; // entries: (node << 8) | nearer-child turns from the root
    int                sp     = 1;
    int                budget = 4096;
    stk[0]                    = 0ull;
    while (sp > 0) {
        if (--budget < 0) return true;
        const unsigned long long e = stk[--sp];
        const int                u = (int)(e >> 8), s = (int)(e & 255ull);
        T                        lb[6], rb[6];
        int                      l, r;
        load_rec<T, COH>(t.recs, u, lb, rb, l, r);
        const D    ld2 = Metric<T>::template dist<(PER != 0), (PER == 2)>(px, py, pz, lb[0], lb[1], lb[2], lb[3],
                                                                         lb[4], lb[5]);
        const D    rd2 = Metric<T>::template dist<(PER != 0), (PER == 2)>(px, py, pz, rb[0], rb[1], rb[2], rb[3],
                                                                         rb[4], rb[5]);
        const bool left_near = ld2 <= rd2;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const int c  = side == 0 ? l : r;
            const D   dc = side == 0 ? ld2 : rd2;
            const int sc = s + (((side == 0) == left_near) ? 1 : 0);
            if (c >= n - 1 || dc > dk) continue; // a leaf, or no neighbour below it
            if (sc >= 62) return true;            // popped with 62 entries below it: dropped
            if ((int)t.height[c] + sc < 63) continue;
            if (sp >= kCap) return true;
            stk[sp++] = ((unsigned long long)c << 8) | (unsigned long long)sc;
        }
    }
    return false;
}

// Slot of this lane's entry in a list whose length is *count, for the lanes with `take`: one
// atomic per warp, and a warp's entries stay together in lane order (so a later launch over
// the list takes neighbouring queries in one warp).  Every lane of the warp must call it.
FT_D uint32_t warp_append(uint32_t *count, bool take, int lane) {
    const unsigned m    = __ballot_sync(0xffffffffu, take);
    uint32_t       base = 0;
    if (m) {
        const int leader = __ffs(m) - 1;
        if (lane == leader) base = atomicAdd(count, (uint32_t)__popc(m));
        base = __shfl_sync(0xffffffffu, base, leader);
    }
    return base + (uint32_t)__popc(m & ((1u << lane) - 1u));
}

// One warp's queries, one a lane: entries [qbase, qbase + lanes) of [0, num), lanes <= 32 -- query
// rows, or entries of the list `lst` when it is given.  NW: warps of the calling block (the heaps are laid out
// per thread of the block); COH: tree records read with ordinary loads (the persistent batch
// kernel, whose blocks read trees that other blocks built earlier in the same launch).
// binary: every lane takes the exact binary walk.
template <class T, int PER, int KC, int NW = fast_warps<KC>(), bool COH = false>
FT_D void fast_warp(const int qbase, const int lanes, const QueryList &lst, const MissList &miss, unsigned char *smem,
                    const TreeDev<T> &t_all, const BatchDev &bt, const T *__restrict__ qx, const T *__restrict__ qy,
                    const T *__restrict__ qz, const uint32_t *__restrict__ order,
                    const int32_t *__restrict__ leaf_ids, int num, int k, int half_window, int exclude_self,
                    int ret_orig, bool binary, const typename Coord<T>::dist_t *__restrict__ bound,
                    unsigned long long *__restrict__ out_idx, typename Coord<T>::dist_t *__restrict__ out_dist,
                    int32_t *__restrict__ replay_ranks, int32_t *__restrict__ replay_rows, uint32_t *replay_count,
                    uint32_t *status, unsigned long long *visit_count) {
    using D = typename Coord<T>::dist_t;
    constexpr int kThreads = 32 * NW; // the block's shape
    // heaps of k entries (<= KC), then the candidate queues; each thread's words are kThreads
    // entries apart, so a lane keeps to its own banks whatever slot it takes
    HeapEntry *heap = reinterpret_cast<HeapEntry *>(smem) + threadIdx.x;
    int32_t   *queue = reinterpret_cast<int32_t *>(reinterpret_cast<HeapEntry *>(smem) + k * kThreads) + threadIdx.x;
    // the walk's per-lane stack, then the stack-guard test's scratch
    unsigned long long lane_stack[kWalkStack];
    static_assert(kWalkStack >= kGuardStack, "guard scratch");

    const int      lane = threadIdx.x & 31;
    const unsigned FULL = 0xffffffffu;
    if (qbase >= num) return; // warp-uniform
    // External query points are walked in the order `order` (sorted by SFC rank, so a warp
    // takes neighbouring queries); q is the output row.  A listed launch takes rows from the
    // list (inactive lanes borrow the first lane's row, which is valid).
    const bool listed = lst.count != nullptr;
    bool       active = lane < lanes && qbase + lane < num;
    const int  q      = listed ? lst.rows[active ? qbase + lane : qbase]
                               : ((qx && order && active) ? (int)order[qbase + lane] : (active ? qbase + lane : qbase));
    // Batched sets: each lane walks the tree of the set its query belongs to (rank local to
    // the set, output row global).
    TreeDev<T> t            = t_all;
    int        rank         = 0;
    bool       force_replay = false;
    if (bt.off) {
        const int qs = q;
        const int s  = find_set(bt.off, bt.S, qs);
        t            = set_view(t_all, bt, s);
        rank         = qs - (int)bt.off[s];
        bool outside = false;
        if constexpr (PER != 0 && !Coord<T>::is_float) {
            // periodic integer set with a coordinate at or above the period (root box maxima):
            // the box distance is not monotone there, so only the reference traversal applies
            constexpr unsigned long long P = 1ull << Coord<T>::bits;
            outside = outside || (unsigned long long)t.max_x[0] >= P || (unsigned long long)t.max_y[0] >= P ||
                      (unsigned long long)t.max_z[0] >= P;
        }
        outside = outside || (*t.qflag & kQFlagPlain) != 0u;
        if (active && outside) {
            force_replay = true;
            active       = false;
        }
    } else if (listed && !qx) {
        rank = active ? lst.ranks[qbase + lane] : 0;
    } else {
        rank = active ? (leaf_ids ? leaf_ids[q] : q) : 0;
    }
    const int n = t.n;
#define HE(s) heap[(s) * kThreads]
#define HD(s) heap[(s) * kThreads].key
#define HI(s) heap[(s) * kThreads].leaf

    // External query points (knn_query): leaf_ids holds each point's SFC rank, the centre of
    // its seeding window (-1: no window); there is no self leaf.
    const bool ext = qx != nullptr;
    if (!ext && active && (rank < 0 || rank >= n)) {
        atomicOr(status, STATUS_BAD_INPUT);
        for (int i = 0; i < k; ++i) {
            out_idx[(size_t)q * k + i]  = ~0ull;
            out_dist[(size_t)q * k + i] = dist_missing<D>();
        }
        active = false;
        rank   = 0;
    }
    const bool seeded   = !ext || rank >= 0;
    if (ext) rank = min(max(rank, 0), n - 1);
    const T *const lx = t.min_x + (n - 1), *const ly = t.min_y + (n - 1), *const lz = t.min_z + (n - 1); // by rank
    const T    px        = ext ? qx[active ? q : 0] : lx[rank];
    const T    py        = ext ? qy[active ? q : 0] : ly[rank];
    const T    pz        = ext ? qz[active ? q : 0] : lz[rank];
    const int  self      = (exclude_self && !ext) ? rank : -1;
    const D    B         = (bound && active) ? bound[q] : dist_heap_max<D>();

    // The tree's 32-bit frame and the query's place in it.  Lanes whose tree or query the
    // frame does not serve walk the binary records with exact distances instead.
    QFrame<T> fr;
    int32_t   u[3] = {0, 0, 0};
    bool      framed;
    if constexpr (PER == 2 && sizeof(T) == 8) { // (the exact distances need it, framed or not)
        u[0] = (int32_t)(uint32_t)((unsigned long long)px >> 10);
        u[1] = (int32_t)(uint32_t)((unsigned long long)py >> 10);
        u[2] = (int32_t)(uint32_t)((unsigned long long)pz >> 10);
    }
    {
        const T rb[6] = {t.min_x[0], t.max_x[0], t.min_y[0], t.max_y[0], t.min_z[0], t.max_z[0]};
        fr.make(rb, n, PER != 0);
        if constexpr (PER == 0 && !Coord<T>::is_float) {
            if (ext && active && open_gaps_wrap<T>(px, py, pz, rb)) { // only the reference traversal applies
                force_replay = true;
                active       = false;
            }
        }
        framed = !binary && fr.ok && *t.qflag == 0u;
        if (framed) {
            const bool a = fr.template query<(PER != 0)>(px, 0, u[0]), b = fr.template query<(PER != 0)>(py, 1, u[1]),
                       c = fr.template query<(PER != 0)>(pz, 2, u[2]);
            framed = a && b && c;
        }
    }

    int   count = 0;
    float hk    = 0.0f; // key of the k-th entry (the heap's root) once the heap is full
    bool  flag  = false;
    // Pruning thresholds: B's until the heap is full, then the smaller of B's and the heap's.
    // kthr: on keys (a distance within the exact threshold has a key within kthr); qlim: on
    // the frame's bounds.
    const bool  noB  = B == dist_heap_max<D>();
    const float kB   = noB ? __int_as_float(0x7f800000) : heap_keyed<T>() ? heap_key<T>(B) : key_up<D>(B);
    float       kthr = kB, qlim = noB ? kB : fr.limit(kB);
    auto        full = [&]() {
        hk   = HD(0);
        kthr = hk < kB ? hk : kB;
        qlim = fr.limit(kthr);
    };

    // exact distance of the query to a leaf (by rank), as node_distance_sq gives it for the
    // leaf's box; from the leaf's QPoint where that holds the whole position
    constexpr bool WHOLE = qpoint_whole<T, PER>();
    uint32_t       ul[3] = {0, 0, 0};
    if constexpr (WHOLE && sizeof(T) == 8) {
        ul[0] = (uint32_t)px << 22;
        ul[1] = (uint32_t)py << 22;
        ul[2] = (uint32_t)pz << 22;
    }
    auto exact_of = [&](const uint4 &v) -> D {
        if constexpr (sizeof(T) == 8 && WHOLE) return qexact42(v, u, ul);
        else if constexpr (WHOLE)
            return Metric<T>::template point<false>(px, py, pz, __uint_as_float(v.x), __uint_as_float(v.y),
                                                    __uint_as_float(v.z));
        else return D(0);
    };
    const uint4 *const pts = reinterpret_cast<const uint4 *>(t.qpts);
    auto exact = [&](int32_t leaf) -> D {
        if constexpr (WHOLE) return exact_of(ld_rec16<COH>(pts + leaf));
        else return Metric<T>::template point<(PER != 0), (PER == 2)>(px, py, pz, lx[leaf], ly[leaf], lz[leaf]);
    };
    // Keyed heaps: the entries sharing the k-th key sit at the top of the max-heap, and
    // exchanging leaves between equal keys keeps the heap valid.  Finds the slot of the
    // exactly largest of them (the root's slot first), its distance, and whether another
    // entry ties it exactly.
    auto kth_exact = [&](int &slot, D &dmax, bool &tie) {
        slot = 0;
        dmax = exact(HI(0));
        tie  = false;
        for (int s2 = 1; s2 < k; ++s2)
            if (HD(s2) == hk) {
                const D e = exact(HI(s2));
                if (e > dmax) {
                    dmax = e;
                    slot = s2;
                    tie  = false;
                } else if (!(e < dmax)) {
                    tie = true; // equal (or not comparable)
                }
            }
    };
    // entry e takes slot i of a heap of `size` entries and sifts down
    auto sift_down = [&](int i, int size, HeapEntry e) {
        for (;;) {
            const int l = 2 * i + 1;
            if (l >= size) break;
            const int r  = min(l + 1, size - 1); // (a lone left child twice)
            HeapEntry c  = HE(l);
            const HeapEntry d = HE(r);
            int       ci = l;
            if (d.key > c.key) {
                c  = d;
                ci = r;
            }
            if (!(c.key > e.key)) break;
            HE(i) = c;
            i     = ci;
        }
        HE(i) = e;
    };
    // id: the leaf's rank (original indices are looked up when the rows are written); kd: the
    // distance's key, heap_key(d2)
    auto insert_k = [&](D d2, float kd, int32_t id) {
        if (count < k) {
            int i = count;
            while (i > 0) {
                const int       p = (i - 1) >> 1;
                const HeapEntry e = HE(p);
                if (kd <= e.key) break;
                HE(i) = e;
                i     = p;
            }
            HE(i) = HeapEntry{kd, id};
            if (++count == k) full();
        } else if (kd < hk) {
            if constexpr (heap_keyed<T>()) {
                // another entry shares the k-th key: evict the exactly largest of them
                if ((k > 1 && HD(1) == hk) || (k > 2 && HD(2) == hk)) {
                    int  slot;
                    D    dmax;
                    bool tie;
                    kth_exact(slot, dmax, tie);
                    if (tie) flag = true; // which of the tied leaves stays is the reference's order
                    if (slot != 0) {
                        const int32_t tmp = HI(0);
                        HI(0)             = HI(slot);
                        HI(slot)          = tmp;
                    }
                }
            }
            const float old = hk;
            sift_down(0, k, HeapEntry{kd, id});
            full();
            // an equal distance stays at the boundary (keyed: the entries left on the old key
            // are exactly nearer than the one evicted, unless tied, flagged above)
            if (!heap_keyed<T>() && hk == old) flag = true;
        } else if (kd == hk) {
            if constexpr (heap_keyed<T>()) {
                // the candidate's key is the k-th key: compare it exactly with the largest entry
                // on that key, and take that entry's place (same key: the heap stays valid)
                int  slot;
                D    dmax;
                bool tie;
                kth_exact(slot, dmax, tie);
                if (d2 < dmax) {
                    HI(slot) = id;
                    if (tie) flag = true;
                } else if (!(d2 > dmax)) {
                    flag = true; // a candidate at exactly the k-th distance was left out
                }
            } else {
                flag = true; // a candidate at exactly the k-th distance was left out
            }
        }
    };
    // whether a leaf may lie within the k-th distance (or the bound)
    auto near_leaf = [&](const uint4 &v) -> bool {
        if constexpr (std::is_same<T, float>::value) return !((float)exact_of(v) > kthr);
        else return !(qdist(u, (int32_t)v.x, (int32_t)v.y, (int32_t)v.z, fr.m, fr.m, fr.m) > qlim);
    };
    auto offer = [&](int32_t leaf) {
        const D     d  = exact(leaf);
        const float kd = heap_key<T>(d);
        if (!(kd > kthr)) insert_k(d, kd, leaf);
    };

    // ---- 1. seed from the SFC window [w0, w1] ----
    // The window's middle fills the heap, which is then put in order at once (one pass of
    // sift-downs from the last parent: about half the steps of as many insertions); the rest is
    // offered from the middle outwards, nearest on the curve first, so most of it fails the
    // k-th key at once.
    const int W  = seeded ? min(n, 2 * half_window + 1) : 0;
    int       w0 = active ? max(0, min(rank - half_window, n - W)) : 0;
    int       w1 = active ? w0 + W - 1 : -1;
    {
        const int m  = min(W, k + (self >= 0 ? 1 : 0));
        const int m0 = active ? max(w0, min(rank - (m >> 1), w0 + W - m)) : 0;
        for (int j = 0; j < m; ++j) {
            const int leaf = m0 + j;
            if (active && leaf != self) {
                HE(count) = HeapEntry{heap_key<T>(exact(leaf)), leaf};
                ++count;
            }
        }
        for (int i = (count >> 1) - 1; i >= 0; --i) sift_down(i, count, HE(i));
        if (count == k) full();
        __syncwarp();
        // (the query's own leaf lies in [m0, m0 + m))
        const int a = active ? m0 - w0 : 0, b = active ? w0 + W - (m0 + m) : 0; // leaves left on either side
        const int c = 2 * min(a, b); // alternating, then the longer side alone
        for (int j = 0; j < a + b; ++j)
            offer(j < c ? ((j & 1) ? m0 + m + (j >> 1) : m0 - 1 - (j >> 1))
                        : (a > b ? m0 - 1 - (j - b) : m0 + m + (j - a)));
        __syncwarp();
    }

    long long budget = 2ll * n + 64;
    int       visits = 0;
    // ---- 2. walk ----
    // A subtree is skipped only when its bound exceeds the limit, so it holds no leaf within
    // the k-th distance; leaves at exactly that distance reach insert_k and raise the tie flag.
    {
        // Warp-synchronous: lanes whose next node is an internal one expand it; a lane that meets a
        // bucket puts it aside and goes on, and waits at its second one, until more lanes wait
        // than expand.  Then every lane with a bucket aside tests it.  Leaves within reach are
        // queued and offered to the heaps when several lanes have some (one a lane and round: the
        // exact distances and the heaps' sifts run with most lanes).
        uint32_t cur  = 0; // next: a node or a bucket
        uint32_t pb   = kQEmpty; // a bucket put aside
        int      sp   = 0;
        bool     have = framed && active && n > 1;
        int      qc   = 0; // queued candidates
        bool     room = true; // every lane's queue has room for a bucket (warp-uniform)
        // a bucket whose leaves all lie in the seeding window: first leaf in [w0, w1 - kBucket + 1]
        const uint32_t wref = kQBucket + (uint32_t)w0, wlen = (uint32_t)max(0, w1 - w0 + 2 - kBucket);
        for (;;) {
            const bool     inner = have && !(cur & kQBucket);
            const unsigned mi    = __ballot_sync(FULL, inner);
            const unsigned mb    = __ballot_sync(FULL, !inner && pb != kQEmpty);
            if (!(mi | mb) || !room) {
                // rounds go on while many lanes have candidates or one has no room for a bucket
                const int keep = (mi | mb) ? kOfferLanes : 1;
                while (__popc(__ballot_sync(FULL, qc > 0)) >= keep || __any_sync(FULL, qc > kQueue - kBucket)) {
                    if (qc > 0) offer(queue[--qc * kThreads]);
                }
                if (!(mi | mb)) break;
                room = true;
            }
            bool pop = false;
            if (mb == 0u || __popc(mi) >= __popc(mb)) {
                if (inner) {
                    --budget;
                    ++visits;
                    const uint4 *p = reinterpret_cast<const uint4 *>(t.qrec + cur);
                    uint4        v[7];
#pragma unroll
                    for (int i = 0; i < 7; ++i) v[i] = ld_rec16<COH>(p + i);
                    const uint32_t *w = reinterpret_cast<const uint32_t *>(v);
                    uint32_t        oc[4];
                    float           od[4];
                    int             nv = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float d = qdist(u, (int32_t)w[6 * i], (int32_t)w[6 * i + 1], (int32_t)w[6 * i + 2],
                                              w[6 * i + 3], w[6 * i + 4], w[6 * i + 5]);
                        oc[i]         = w[24 + i];
                        const bool in = oc[i] != kQEmpty && !(d > qlim) &&
                                        !((oc[i] & 0x8fffffffu) - wref < wlen); // not a bucket of the window
                        od[i]         = in ? d : -1.0f; // sorted behind the needed ones
                        nv += in ? 1 : 0;
                    }
                    // the nearest needed child is walked next, the others are stacked farthest
                    // first (key: the bound)
                    auto cx = [&](int a, int b) {
                        const bool     sw = od[a] < od[b];
                        const uint32_t ca = oc[a], cb = oc[b];
                        const float    da = od[a], db = od[b];
                        oc[a]             = sw ? cb : ca;
                        od[a]             = sw ? db : da;
                        oc[b]             = sw ? ca : cb;
                        od[b]             = sw ? da : db;
                    };
                    cx(0, 1);
                    cx(2, 3);
                    cx(0, 2);
                    cx(1, 3);
                    cx(1, 2);
                    if (sp + 3 > kWalkStack || budget < 0) {
                        // cannot stack them all: the reference traversal reruns the query
                        if (budget < 0) atomicOr(status, STATUS_TRAVERSAL_LIMIT);
                        flag = true;
                        have = false;
                        pb   = kQEmpty;
                    } else {
#pragma unroll
                        for (int i = 0; i < 3; ++i)
                            if (i < nv - 1) lane_stack[sp + i] = ((unsigned long long)__float_as_uint(od[i]) << 32) | oc[i];
                        sp += max(nv - 1, 0);
                        cur = nv == 1 ? oc[0] : nv == 2 ? oc[1] : nv == 3 ? oc[2] : oc[3];
                        pop = nv == 0;
                        if (pop) {
                            if (oc[0] == kQEmpty) { // (unsorted) a dense node: the exact walk takes the query
                                count = -1;
                                have = pop = false;
                                pb         = kQEmpty;
                                qc         = 0;
                            }
                        } else if ((cur & kQBucket) && pb == kQEmpty) {
                            pb  = cur;
                            pop = true;
                        }
                    }
                }
            } else {
                // buckets: leaves whose bound is within reach join the lane's queue
                if (pb != kQEmpty) {
                    ++visits;
                    const int    first = qref_first(pb), cnt = qref_count(pb);
                    const uint4 *p     = pts + first;
#pragma unroll
                    for (int j = 0; j < kBucket; ++j) {
                        const uint4 v    = ld_rec16<COH>(p + min(j, cnt - 1));
                        const int   leaf = first + j; // (the query's own leaf lies in the window)
                        const bool  near = near_leaf(v); // (before the test: all loads in flight at once)
                        if (j < cnt && near && (leaf < w0 || leaf > w1)) queue[qc++ * kThreads] = leaf;
                    }
                    pb  = (have && !inner) ? cur : kQEmpty;
                    pop = have && !inner;
                }
                room = !__any_sync(FULL, qc > kQueue - kBucket);
            }
            __syncwarp();
            if (pop) {
                have = false;
                while (sp > 0) {
                    const unsigned long long e = lane_stack[--sp];
                    if (!(__uint_as_float((uint32_t)(e >> 32)) > qlim)) {
                        cur = (uint32_t)e;
                        if ((cur & kQBucket) && pb == kQEmpty) {
                            pb = cur;
                            continue;
                        }
                        have = true;
                        break;
                    }
                }
            }
            __syncwarp();
        }
    }
    const bool exact_walk = active && n > 1 && (!framed || count < 0);
    if (count < 0) { // from an empty heap: the leaves in it are offered again
        count  = 0;
        flag   = false;
        kthr   = kB;
        budget = 2ll * n + 64;
        w0     = 0;
        w1     = -1;
    }
    if (__any_sync(FULL, exact_walk)) {
        // exact walk over the binary records, the lanes together as above: leaf children within reach
        // are queued, the nearer internal child is walked next, the farther one is stacked
        int  cur = 0, sp = 0, qc = 0;
        bool have  = exact_walk;
        auto needs = [&](D d2) { return !(heap_key<T>(d2) > kthr); };
        for (;;) {
            const bool any = __any_sync(FULL, have);
            if (!any || __any_sync(FULL, qc > kQueue - 2)) {
                const int keep = any ? kOfferLanes : 1;
                while (__popc(__ballot_sync(FULL, qc > 0)) >= keep || __any_sync(FULL, qc > kQueue - 2)) {
                    if (qc > 0) offer(queue[--qc * kThreads]);
                }
                if (!any) break;
            }
            if (have && --budget < 0) {
                atomicOr(status, STATUS_TRAVERSAL_LIMIT);
                have = false;
            }
            if (have) {
                ++visits;
                T   lb[6], rb[6];
                int l, r;
                load_rec<T, COH>(t.recs, cur, lb, rb, l, r);
                const D    ld2 = Metric<T>::template dist<(PER != 0), (PER == 2)>(px, py, pz, lb[0], lb[1], lb[2], lb[3], lb[4], lb[5]);
                const D    rd2 = Metric<T>::template dist<(PER != 0), (PER == 2)>(px, py, pz, rb[0], rb[1], rb[2], rb[3], rb[4], rb[5]);
                const bool ln = needs(ld2), rn = needs(rd2);
                const int  lr = l - (n - 1), rr = r - (n - 1); // ranks of leaves
                if (ln && lr >= 0 && (lr < w0 || lr > w1) && lr != self) queue[qc++ * kThreads] = lr;
                if (rn && rr >= 0 && (rr < w0 || rr > w1) && rr != self) queue[qc++ * kThreads] = rr;
                const bool li = ln && lr < 0, ri = rn && rr < 0;
                if (li && ri) {
                    const bool left = ld2 <= rd2;
                    if (sp >= kWalkStack) {
                        flag = true; // cannot stack it: the reference traversal reruns the query
                        have = false;
                    } else {
                        lane_stack[sp++] = ((unsigned long long)__float_as_uint(heap_key<T>(left ? rd2 : ld2)) << 32) |
                                           (uint32_t)(left ? r : l);
                        cur = left ? l : r;
                    }
                } else if (li) {
                    cur = l;
                } else if (ri) {
                    cur = r;
                } else {
                    have = false;
                    while (sp > 0) {
                        const unsigned long long e = lane_stack[--sp];
                        if (!(__uint_as_float((uint32_t)(e >> 32)) > kthr)) {
                            cur  = (int)(uint32_t)e;
                            have = true;
                            break;
                        }
                    }
                }
            }
            __syncwarp();
        }
    }
    __syncwarp();

    // visit statistics: expansions and buckets, summed per warp
    if (visit_count) {
        const unsigned sum = __reduce_add_sync(FULL, (unsigned)visits);
        if (lane == 0) atomicAdd(visit_count, (unsigned long long)sum);
    }

    // ---- 3. sort, check, write ----
    // a bound that proved too small: the bound may have cut a neighbour, or fewer than k
    // points lie inside it.  With a miss list the query goes to the next launch (the walk
    // without a bound); otherwise the reference traversal reruns it.
    // (k-th key not below the bound's key: the k-th distance may exceed the bound)
    const bool bound_miss =
        active && B != dist_heap_max<D>() && (count < k || !(hk < heap_key<T>(B)));
    if (miss.rows) {
        const uint32_t at = warp_append(miss.count, bound_miss, lane);
        if (bound_miss) {
            if (!ext && !bt.off) miss.ranks[at] = rank;
            miss.rows[at] = q;
            active        = false;
        }
    }
    if (active) {
        if (bound_miss) flag = true;
        // trees of height >= 63: the reference's stack guard may drop part of this query's
        // neighbourhood (fewer than k points found: conservatively so)
        if (!flag && n >= 2 && (int)t.height[0] >= 63 &&
            (count < k ||
             stack_guard_reaches<T, PER, COH>(t, px, py, pz, heap_key_ub<T>(hk), lane_stack)))
            flag = true;
        for (int hs = count; hs > 1; --hs) {
            const HeapEntry last = HE(hs - 1);
            HE(hs - 1)           = HE(0);
            sift_down(0, hs - 1, last);
        }
        if constexpr (heap_keyed<T>()) {
            // runs of equal keys inside the top k: the exact distances order them (the exact
            // order refines the key order); only an exact tie can differ from the reference
            for (int i = 1; i < count; ++i) {
                for (int j = i; j > 0 && HD(j) == HD(j - 1); --j) {
                    const D a = exact(HI(j - 1)), b = exact(HI(j));
                    if (!(b < a)) { // in order, or equal (or not comparable): a tie
                        if (!(a < b)) flag = true;
                        break;
                    }
                    const int32_t tmp = HI(j);
                    HI(j)             = HI(j - 1);
                    HI(j - 1)         = tmp;
                }
            }
        } else {
            // equal distances: their order may differ from the reference's
            for (int i = 1; i < count; ++i)
                if (HD(i) == HD(i - 1)) flag = true;
        }
        const size_t off = (size_t)q * (size_t)k;
        auto         row = [&](int i, unsigned long long &id, D &dd) {
            if (i < count) {
                const HeapEntry e = HE(i);
                if constexpr (heap_keyed<T>()) dd = exact(e.leaf);
                else dd = (D)e.key;
                id = (unsigned long long)(long long)(ret_orig ? t.orig_idx[e.leaf + n - 1] : e.leaf);
            } else {
                id = ~0ull;
                dd = dist_missing<D>();
            }
        };
        // four entries a store where the rows allow it: whole 32-byte sectors
        const bool vec = (k & 3) == 0 && (((uintptr_t)out_idx | (uintptr_t)out_dist) & 31) == 0;
        int        i   = 0;
        if (vec) {
            for (; i < k; i += 4) {
                unsigned long long id[4];
                D                  dd[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) row(i + j, id[j], dd[j]);
                st_sector(out_idx + off + i, id);
                st_sector(out_dist + off + i, dd);
            }
        }
        for (; i < k; ++i) {
            unsigned long long id;
            D                  dd;
            row(i, id, dd);
            __stcs(out_idx + off + i, id);
            __stcs(out_dist + off + i, dd);
        }
    }
    const bool to_replay = (active && flag) || force_replay;
    const uint32_t at    = warp_append(replay_count, to_replay, lane);
    if (to_replay) {
        if (!ext) replay_ranks[at] = rank;
        replay_rows[at] = q;
    }
#undef HE
#undef HD
#undef HI
}

} // namespace ft
