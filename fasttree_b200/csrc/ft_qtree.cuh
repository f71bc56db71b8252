// ft_qtree.cuh -- the fast walks' view of a built tree: positions and boxes in a 32-bit frame.
//
// The walks only need bounds to prune with; the distances that decide a result are computed
// from the tree's own coordinates.  So the walks read
//  * QPoint: a leaf's position in 32-bit units of the tree's frame (16 bytes), in leaf order;
//  * QRec: a 4-wide node, centre and half extent of each child's box in the same units (one
//    128-byte line).  Subtrees of at most kBucket leaves are not opened: a child either is an
//    internal node with a record of its own or a bucket, a run of consecutive leaves.
// The distance from a query to either, one subtraction, absolute value, saturating subtraction,
// conversion and multiply-add per axis, is never above the distance node_distance_sq gives
// (src/hlbvh.hpp:998-1055), in any coordinate type; 42-bit periodic positions wrap with the
// 32-bit subtraction.
//
// The frame (QFrame) follows from the tree's root box alone, so builds and queries derive it
// where they need it:
//  * periodic integers (every coordinate below the period 2^B): the top 32 bits of the B-bit
//    position (B = 42: >> 10, B = 21: << 11), so a wrapped difference wraps in 32 bits too;
//  * open integers: offset from the root box's corner, shifted so that the longest side takes
//    30 bits;
//  * floating point: floor((x - lo) 2^e), e such that the longest side takes at most 30 bits.
// Bound.  Let u = floor of a position in units.  For a query position q and a box [lo, hi] on
// an axis, the real gap is at least max(u(q) - u(hi), u(lo) - u(q), 0) - 1 units, and with
// c = the middle of [u(lo), u(hi)] and h = u(hi) - c at least |u(q) - c| - h - 1 (on the circle
// the same with the wrapped difference).  Integer metrics floor the shifted gap, which takes up
// to 2^dist_shift coordinate units more.  The margin `m` of both is stored with the half
// extents.  Squared and summed in float (relative error below 2^-21) the bound is compared with
// a threshold in units^2 that is rounded up by 2^-17 (QFrame::limit), which also covers the
// rounding of floating-point distances (a few 2^-24 each) and the heap key's rounding.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ft_common.cuh"

namespace ft {

#ifndef FT_BUCKET
#define FT_BUCKET 8
#endif
static constexpr int      kBucket     = FT_BUCKET; // most leaves of a bucket (a 3-bit count)
// References: a node, a bucket, or no child.  A record without any child is a dense node's (below).
static constexpr uint32_t kQBucket = 0x80000000u, kQEmpty = 0xffffffffu;
static constexpr int      kQMaxLeaves = (1 << 28) - 64; // a bucket's first leaf takes 28 bits
static_assert(kBucket >= 1 && kBucket <= 8, "a bucket reference has three bits for its size");

FT_HD uint32_t qref_bucket(int first, int count) {
    return kQBucket | ((uint32_t)(count - 1) << 28) | (uint32_t)first;
}
FT_HD int qref_first(uint32_t r) { return (int)(r & 0x0fffffffu); }
FT_HD int qref_count(uint32_t r) { return (int)((r >> 28) & 7u) + 1; }

// Bits of the per-tree flag (0: the frame serves the walks).  FRAME (no frame for the root box): the
// exact binary walk serves the tree.  NONFINITE (a coordinate is not finite), OVERFLOW
// (integer gaps whose squares may leave 64 bits): box distances are not monotone, so only the
// reference traversal gives its rows.  BOXES (a leaf slot of the caller's whose minimum is not its
// maximum): the walks take leaves for points, the reference traversal measures to their boxes.
enum : uint32_t { QFLAG_NONFINITE = 1u, QFLAG_FRAME = 4u, QFLAG_OVERFLOW = 8u, QFLAG_BOXES = 16u };
static constexpr uint32_t kQFlagPlain = QFLAG_NONFINITE | QFLAG_OVERFLOW | QFLAG_BOXES;
// A node of more than kDenseLeaves leaves whose box spans at most 2 kDenseUnits units on every
// axis: the frame no longer tells its leaves apart.  Its record has no children, and a query that
// reaches it starts again with the exact walk; the others never see it.  (More than 256 /
// 1024 leaves, a clump of 600 in 1M points, 1M self and 200K external queries, k = 16: float64 3.25 /
// 3.63 and 2.19 / 1.89 ms, 42-bit periodic 2.47 / 2.36 and 1.63 / 1.55 ms.)
static constexpr int      kDenseLeaves = 1024;
static constexpr uint32_t kDenseUnits  = 8;

template <class T> struct QFrame {
    using C = Coord<T>;
    T        o[3];  // origin (open frames)
    double   s;     // units per coordinate (floating point)
    int      shift; // integers: right shift, negative: left
    uint32_t m;     // margin in units
    float    ka, kb, slack; // distance -> units^2: limit(d) = d * ka * kb + slack
    bool     ok, overflow;

    // box: the root box (minx, maxx, miny, maxy, minz, maxz); n: leaves
    FT_D void make(const T box[6], int n, bool periodic) {
        ok       = n <= kQMaxLeaves;
        overflow = false;
        s  = 1.0;
        shift = 0;
        m     = 1u;
        slack = 0.0f;
        ka = kb = 1.0f;
#pragma unroll
        for (int a = 0; a < 3; ++a) o[a] = box[2 * a];
        if constexpr (C::is_float) {
            double span = 0.0;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const double e = (double)box[2 * a + 1] - (double)box[2 * a];
                if (!(e >= 0.0) || !(fabs((double)box[2 * a]) <= 1e300)) ok = false; // NaN or an empty box
                span = fmax(span, e);
            }
            // span < 2^(x + 1): span * 2^(29 - x) < 2^30, and 2^(29 - x) is exact, a normal float for
            // -97 <= x <= 126 (spans of 1e-29 to 1e38: distances beyond have no float keys)
            const int x = (int)((__double_as_longlong(span) >> 52) & 2047) - 1023;
            if (x < -97 || x > 126) ok = false;
            if (!ok) return;
            s     = __longlong_as_double((long long)(1023 + 29 - x) << 52);
            ka    = (float)s; // (in two steps: s^2 may be no float, and d * s is one where d * s^2 is)
            kb    = (float)s * (1.0f + 0x1p-17f);
            slack = __double2float_ru(s * s * 0x1p-140); // distances that underflow
        } else {
            int sh; // right shift from coordinate units to frame units
            if (periodic) {
                sh = C::bits - 32;
                constexpr unsigned long long P = 1ull << C::bits;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    o[a] = T(0);
                    if ((unsigned long long)box[2 * a + 1] >= P) ok = false;
                }
            } else {
                unsigned long long span = 0;
#pragma unroll
                for (int a = 0; a < 3; ++a) span = max(span, (unsigned long long)(T)(box[2 * a + 1] - box[2 * a]));
                const int bl = 64 - __clzll((long long)span); // span < 2^bl
                sh           = bl - 30;
                sh           = max(sh, -20);
                // shifted gaps below 2^31 keep the sum of three squares in 64 bits
                overflow = bl > 31 + C::dist_shift;
                if (overflow) ok = false;
            }
            shift = sh;
            // floor of the shifted gap: up to 2^dist_shift coordinate units
            const int du = C::dist_shift - sh;
            m            = 1u + (C::dist_shift > 0 ? (du > 0 ? 1u << min(du, 31) : 1u) : 0u); // du <= 31
            // distance units are 2^dist_shift coordinate units: factor 4^(dist_shift - sh)
            kb = __int_as_float((127 + 2 * du) << 23) * (1.0f + 0x1p-17f);
        }
    }
    // the flag's part that follows from the root box
    FT_D uint32_t flag() const { return (ok ? 0u : QFLAG_FRAME) | (overflow ? QFLAG_OVERFLOW : 0u); }
    FT_D float limit(float key) const {
        const float l = fmaf(key * ka, kb, slack);
        // (FLT_MAX keys every finite distance from there up)
        return C::is_float && key >= FLT_MAX ? __int_as_float(0x7f800000) : l;
    }

    // position in units; in the tree (or a periodic query): always representable
    FT_D int32_t pos(T v, int a) const {
        if constexpr (C::is_float) {
            return __double2int_rd(((double)v - (double)o[a]) * s);
        } else {
            const T d = v - o[a];
            if constexpr (sizeof(T) == 8)
                return shift >= 0 ? (int32_t)(uint32_t)((unsigned long long)d >> shift)
                                  : (int32_t)((uint32_t)d << -shift);
            else return shift >= 0 ? (int32_t)((uint32_t)d >> shift) : (int32_t)((uint32_t)d << -shift);
        }
    }
    // position of any query point; false when the frame cannot hold it (open frames: more
    // than about one box length outside the root box; not a number)
    template <bool PERIODIC> FT_D bool query(T v, int a, int32_t &u) const {
        if constexpr (C::is_float) {
            const double f = floor(((double)v - (double)o[a]) * s);
            u              = 0;
            if (!(f > -1073741824.0 && f < 2147483000.0)) return false;
            u = __double2int_rd(f);
            return true;
        } else if constexpr (PERIODIC) {
            if constexpr (sizeof(T) == 4) {
                u = (int32_t)((uint32_t)v << 11);
                return v < (T(1) << C::bits); // (the metric does not mask a 32-bit query)
            } else {
                u = (int32_t)(uint32_t)(((unsigned long long)v & ((1ull << C::bits) - 1ull)) >> (C::bits - 32));
                return true;
            }
        } else {
            // signed offset in units, floored
            const bool               neg = v < o[a];
            const unsigned long long d   = neg ? (unsigned long long)(T)(o[a] - v) : (unsigned long long)(T)(v - o[a]);
            const unsigned long long lim = shift >= 0 ? (1ull << 30) << shift : (1ull << 30) >> -shift;
            u                            = 0;
            if (d >= (neg ? lim : lim + (lim - 1))) return false;
            unsigned long long e = shift >= 0 ? (neg ? (d + ((1ull << shift) - 1)) >> shift : d >> shift) : d << -shift;
            u = neg ? -(int32_t)e : (int32_t)e;
            return true;
        }
    }
};

// Open integers: whether the squares of a point's gaps to the root box `rb` may leave 64 bits.  Its
// box distances are not monotone then (a tree of that span is flagged, QFLAG_OVERFLOW).
template <class T> FT_D bool open_gaps_wrap(T px, T py, T pz, const T rb[6]) {
    const T            p[3] = {px, py, pz};
    unsigned long long g    = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const T lo = rb[2 * a], hi = rb[2 * a + 1];
        g          = max(g, max((unsigned long long)(p[a] > lo ? p[a] - lo : lo - p[a]),
                                (unsigned long long)(p[a] > hi ? p[a] - hi : hi - p[a])));
    }
    return ((g >> Coord<T>::dist_shift) >> 31) != 0;
}

// Whether a node of n leaves and the box b is dense.
template <class T> FT_D bool qdense(int n, const T b[6], const QFrame<T> &f) {
    if (n <= kDenseLeaves || !(Coord<T>::is_float || f.shift > 0)) return false; // exact frames lose nothing
    uint32_t hm   = 0;
    bool     flat = true; // copies of one point: no frame tells them apart
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        hm   = max(hm, (uint32_t)f.pos(b[2 * a + 1], a) - (uint32_t)f.pos(b[2 * a], a));
        flat = flat && !(b[2 * a] < b[2 * a + 1]);
    }
    return !flat && hm <= 2 * kDenseUnits;
}

// Bound of one axis: |u - c| - h, not below zero.
FT_D float qgap(int32_t u, int32_t c, uint32_t h) {
    const uint32_t a = (uint32_t)abs((int32_t)((uint32_t)u - (uint32_t)c));
    return (float)(a - min(a, h));
}
FT_D float qdist(const int32_t u[3], int32_t cx, int32_t cy, int32_t cz, uint32_t hx, uint32_t hy, uint32_t hz) {
    const float x = qgap(u[0], cx, hx), y = qgap(u[1], cy, hy), z = qgap(u[2], cz, hz);
    return fmaf(z, z, fmaf(y, y, x * x));
}

// The record of internal node v: v's two children, then twice the child with the most leaves
// (more than kBucket) replaced by its own two.
template <class T>
FT_D void qrec_node(int v, int n, const NodeRec<T> *recs, const int32_t *leaves, const QFrame<T> &f, QRec *out) {
    int      id[4];
    uint32_t cn[4];
    bool     rt[4]; // a right child (its first leaf is its index; a left child's last leaf is)
    T        bx[4][6];
    int      c = 2;
    auto     count_of = [&](int ch, uint32_t info) -> uint32_t {
        const uint32_t w = info_leaves(info);
        return (w == kInfoCountMax && ch < n - 1) ? (uint32_t)leaves[ch] : w;
    };
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        id[i] = -1;
        cn[i] = 0;
        rt[i] = false;
#pragma unroll
        for (int d = 0; d < 6; ++d) bx[i][d] = T(0);
    }
    {
        uint32_t il, ir;
        load_rec_info<T, true>(recs, v, bx[0], bx[1], id[0], id[1], il, ir);
        cn[0] = count_of(id[0], il);
        cn[1] = count_of(id[1], ir);
        rt[1] = true;
    }
    T own[6];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        own[2 * a]     = box_min(bx[0][2 * a], bx[1][2 * a]);
        own[2 * a + 1] = box_max(bx[0][2 * a + 1], bx[1][2 * a + 1]);
    }
    const bool dense = qdense<T>((int)(cn[0] + cn[1]), own, f);
#pragma unroll
    for (int step = 0; step < 2; ++step) {
        int      b  = -1, bid = 0;
        uint32_t bc = kBucket;
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (i < c && cn[i] > bc) {
                b   = i;
                bc  = cn[i];
                bid = id[i];
            }
        if (b < 0) break;
        T        lb[6], rb[6];
        int      l, r;
        uint32_t il, ir;
        load_rec_info<T, true>(recs, bid, lb, rb, l, r, il, ir);
#pragma unroll
        for (int i = 3; i > 0; --i)
            if (i > b + 1) { // make room behind the opened child
                id[i] = id[i - 1];
                cn[i] = cn[i - 1];
                rt[i] = rt[i - 1];
#pragma unroll
                for (int d = 0; d < 6; ++d) bx[i][d] = bx[i - 1][d];
            }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i == b) {
                id[i] = l;
                cn[i] = count_of(l, il);
                rt[i] = false;
#pragma unroll
                for (int d = 0; d < 6; ++d) bx[i][d] = lb[d];
            } else if (i == b + 1) {
                id[i] = r;
                cn[i] = count_of(r, ir);
                rt[i] = true;
#pragma unroll
                for (int d = 0; d < 6; ++d) bx[i][d] = rb[d];
            }
        }
        ++c;
    }
    QRec q;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const uint32_t lo = (uint32_t)f.pos(bx[i][2 * a], a), hi = (uint32_t)f.pos(bx[i][2 * a + 1], a);
            const uint32_t ce = lo + ((hi - lo) >> 1);
            q.c[i][a]         = (int32_t)ce;
            q.c[i][3 + a]     = (int32_t)((hi - ce) + f.m);
        }
        const bool leaf = id[i] >= n - 1;
        q.cnt[i]        = i < c ? cn[i] : 0u;
        if (i >= c) q.ref[i] = kQEmpty;
        else if (leaf) q.ref[i] = qref_bucket(id[i] - (n - 1), 1);
        else if (cn[i] <= (uint32_t)kBucket)
            q.ref[i] = qref_bucket(rt[i] ? id[i] : id[i] - (int)cn[i] + 1, (int)cn[i]);
        else q.ref[i] = (uint32_t)id[i];
        if (dense) q.ref[i] = kQEmpty;
    }
    const uint4 *src = reinterpret_cast<const uint4 *>(&q);
    uint4       *dst = reinterpret_cast<uint4 *>(out + v);
#pragma unroll
    for (int i = 0; i < 8; ++i) dst[i] = src[i];
}

// The walk's copy of a leaf's position.  float: the coordinates themselves (x, y, z hold their
// bits; the exact distance is as cheap as a bound).  42-bit periodic positions: the frame
// position and, in w, the 10 low bits of each axis (z y x from the top), so the whole position
// is there.  Other types: the frame position.  A coordinate that is not finite sets the flag.
template <class T>
FT_D QPoint qpoint(T x, T y, T z, const QFrame<T> &f, bool periodic, uint32_t *flag) {
    if constexpr (Coord<T>::is_float)
        if (!(isfinite((double)x) && isfinite((double)y) && isfinite((double)z))) atomicOr(flag, QFLAG_NONFINITE);
    QPoint p;
    if constexpr (std::is_same<T, float>::value) {
        p.x = __float_as_int(x);
        p.y = __float_as_int(y);
        p.z = __float_as_int(z);
        p.w = 0;
    } else {
        p.x = f.pos(x, 0);
        p.y = f.pos(y, 1);
        p.z = f.pos(z, 2);
        p.w = 0;
        if constexpr (!Coord<T>::is_float && sizeof(T) == 8) {
            if (periodic)
                p.w = (int32_t)(((uint32_t)x & 1023u) | (((uint32_t)y & 1023u) << 10) | (((uint32_t)z & 1023u) << 20));
        }
    }
    return p;
}

// Exact distance of a query to a leaf from its QPoint, the value node_distance_sq gives
// (Metric::point), for the types whose QPoint holds the whole position.  u, ul: the query's
// frame position and its low bits at the top of a word (42-bit periodic).
template <class T, int PER> constexpr bool qpoint_whole() {
    return std::is_same<T, float>::value || (PER == 2 && sizeof(T) == 8);
}
// |sext42(x - v)| >> dist_shift of one axis: x << 22 and v << 22 as (high, low) words.
FT_D uint32_t qaxis42(uint32_t xh, uint32_t xl, uint32_t vh, uint32_t vl) {
    const uint32_t l = xl - vl, h = xh - vh - (xl < vl ? 1u : 0u);
    const uint32_t g = (int32_t)h < 0 ? ~h + (l == 0u ? 1u : 0u) : h; // |y| >> 32
    return g >> 1;
}
FT_D unsigned long long qexact42(const uint4 &v, const int32_t u[3], const uint32_t ul[3]) {
    const uint32_t x = qaxis42(v.x, v.w << 22, (uint32_t)u[0], ul[0]);
    const uint32_t y = qaxis42(v.y, (v.w << 12) & 0xffc00000u, (uint32_t)u[1], ul[1]);
    const uint32_t z = qaxis42(v.z, (v.w << 2) & 0xffc00000u, (uint32_t)u[2], ul[2]);
    return (unsigned long long)x * x + (unsigned long long)y * y + (unsigned long long)z * z;
}

} // namespace ft
