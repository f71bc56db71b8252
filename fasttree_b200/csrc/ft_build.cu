// ft_build.cu -- HLBVH build on sm_100a: bounding box, SFC keys, onesweep radix sort of
// (key, original index), leaf gather, Karras radix-tree topology and the bottom-up box refit
// that also writes the traversal's node records.
//
// Reference pipeline: build_bvh (src/hlbvh.hpp:2165-2290) -> compute_bbox (462-572) ->
// sfc_encode (357-423) -> oneDPL sort (2202-2232) -> gather (2266-2279) -> build_tree
// (773-982: Karras 861-903, refit 925-969).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <mutex>
#include <vector>

#include "ft_build_dev.cuh"
#include "ft_common.cuh"
#include "ft_internal.h"
#include "ft_qtree.cuh"
#include "ft_treelet.cuh"

namespace ft {

static constexpr int kSpinLimit = 1 << 24;

size_t coord_bytes(int coord) { return (coord == F32 || coord == U32) ? 4 : 8; }

static int key_words(const ft_options &o) { return (o.coord_type == U64) ? 2 : 1; }

// Karras tie-break / prefix flavour: 0 Morton (clz64), 1 63-bit PH (clz64 - 1), 2 126-bit PH.
static int delta_kind(const ft_options &o) {
    if (o.sfc_type == MORTON) return 0;
    return (o.coord_type == U64) ? 2 : 1;
}

size_t ref_key_bytes(const ft_options &o) {
    if (o.sfc_type == MORTON) return 8;       // uint64 (src/sfc.morton.hpp:17)
    return (o.coord_type == U64) ? 24 : 12;   // {hs,is,ls} of 64- or 32-bit words
}

// =========================================================================================
// Bounding box: per-block partials, then one block folds them (two passes keep the result
// independent of scheduling); the fold is bb_fold.
// =========================================================================================
static constexpr int kBboxBlocks = 1184; // 8 x 148 SMs

template <class T>
__global__ void __launch_bounds__(kBboxThreads) bbox_partial_kernel(const T *__restrict__ x, const T *__restrict__ y,
                                                                    const T *__restrict__ z, size_t n, T *partial) {
    T m[6];
    bb_identity(m);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        T v[6] = {x[i], x[i], y[i], y[i], z[i], z[i]};
        bb_fold(m, v);
    }
    bb_block_reduce(m);
    if (threadIdx.x == 0)
        for (int d = 0; d < 6; ++d) partial[blockIdx.x * 6 + d] = m[d];
}

template <class T> __global__ void __launch_bounds__(kBboxThreads) bbox_final_kernel(const T *partial, int nparts, T *out) {
    T m[6];
    bb_identity(m);
    for (int b = threadIdx.x; b < nparts; b += blockDim.x) bb_fold(m, partial + 6 * b);
    bb_block_reduce(m);
    if (threadIdx.x == 0)
        for (int d = 0; d < 6; ++d) out[d] = m[d];
}

__global__ void keys_to_ref_kernel(const unsigned long long *klo, const unsigned long long *khi, size_t n, int mode,
                                   void *ref) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (mode == 0) {
            ((unsigned long long *)ref)[i] = klo[i];
        } else if (mode == 1) {
            uint32_t *w = (uint32_t *)ref + 3 * i;
            w[0]        = 0;
            w[1]        = (uint32_t)(klo[i] >> 32);
            w[2]        = (uint32_t)klo[i];
        } else {
            unsigned long long *w = (unsigned long long *)ref + 3 * i;
            w[0]                  = 0;
            w[1]                  = khi[i];
            w[2]                  = klo[i];
        }
    }
}

// =========================================================================================
// LSD radix sort of (64-bit key, 32-bit value) pairs: 8-bit digits, one upfront histogram of all
// digit positions, then one onesweep pass per non-constant digit.  Each pass: a tile of 256
// threads x ITEMS keys ranks its keys per warp (the lanes that share a digit are found with eight
// ballots), publishes its digit counts, resolves its global offsets by decoupled look-back
// over preceding tiles (tiles are numbered by an atomic ticket so every predecessor is running
// or done), stages the tile in shared memory in digit order and writes each digit run
// contiguously.  Stable, so equal keys keep their incoming order.
//
// A pass moves 24 bytes a key; what bounds it is the chain of steps of a tile.  Two-word keys and
// the hardware's match instruction took 176 us a pass over 10M keys, the sort word alone (126-bit
// keys: the high word; the low one rides with the packed points) and ballots 120 us: the match
// costs an SM about 57 cycles a warp, the ballots some 10 in issue slots.  The encode kernel adds
// its counts to the histograms with plain shared-memory atomics (a launch of its own with
// match-aggregated counts took 495 us for 10M keys), and a constant digit's pass moves nothing
// (83 us as a copy).
// =========================================================================================
static constexpr int kSortThreads = 256;
static constexpr int kSortWarps   = kSortThreads / 32;
static constexpr int kSortDigits  = 8;
// Words of TreeImpl::tile_counter: [0, 8) one tile ticket per pass; [32] build_bvh of 126-bit keys
// met a run of equal high words too long to order in place.
static constexpr int kTicketWords = 64, kLongRunWord = 32;
static constexpr uint32_t kFlagAgg = 1u << 30, kFlagInc = 2u << 30, kFlagMask = 3u << 30,
                          kCountMask = (1u << 30) - 1u;

// A onesweep tile: 256 threads x ITEMS keys (8 by default; the autotuner's choice for a shape
// otherwise; every tile size gives the same order).
template <int ITEMS> struct SortCfg {
    static constexpr int    tile = kSortThreads * ITEMS;
    static constexpr size_t smem = (size_t)tile * 12 + (size_t)kSortWarps * 256 * 4;
};
static constexpr int kSortItems = 8; // the smallest tile: it sizes the look-back scratch

// The pairs' two buffers.  A constant digit's pass moves nothing, so the buffer that holds them
// follows from the passes that ran (sort_parity, ft_treelet.cuh).
struct SortPairs {
    unsigned long long *k[2];
    uint32_t           *v[2];
};
FT_D void hist_add(uint32_t *s, unsigned long long key) {
#pragma unroll
    for (int d = 0; d < kSortDigits; ++d) atomicAdd(&s[d * 256 + ((unsigned)(key >> (8 * d)) & 255u)], 1u);
}

// Digit histograms of every digit position (hist zero at launch).
__global__ void __launch_bounds__(256) radix_hist_kernel(const unsigned long long *__restrict__ keys, size_t n,
                                                         uint32_t *hist) {
    __shared__ uint32_t s[kSortDigits * 256];
    for (int i = threadIdx.x; i < kSortDigits * 256; i += blockDim.x) s[i] = 0;
    __syncthreads();
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        hist_add(s, keys[i]);
    __syncthreads();
    for (int i = threadIdx.x; i < kSortDigits * 256; i += blockDim.x)
        if (s[i]) atomicAdd(&hist[i], s[i]);
}

// Exclusive offsets per digit position; skip[d] = 1 when one digit value holds every key.
__global__ void radix_scan_kernel(uint32_t *hist, size_t n, uint32_t *skip) {
    __shared__ uint32_t s[256];
    __shared__ int      s_full;
    const int d = blockIdx.x, t = threadIdx.x;
    uint32_t  c = hist[d * 256 + t];
    if (t == 0) s_full = 0;
    __syncthreads();
    if ((size_t)c == n) s_full = 1;
    s[t] = c;
    __syncthreads();
    for (int off = 1; off < 256; off <<= 1) {
        uint32_t v = (t >= off) ? s[t - off] : 0u;
        __syncthreads();
        s[t] += v;
        __syncthreads();
    }
    hist[d * 256 + t] = s[t] - c;
    if (t == 0) skip[d] = (uint32_t)s_full;
}

FT_D uint32_t ld_volatile(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.volatile.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
FT_D void st_volatile(uint32_t *p, uint32_t v) { asm volatile("st.volatile.global.u32 [%0], %1;" ::"l"(p), "r"(v)); }

// The lanes of the warp whose digit equals this lane's, among the lanes with `valid`.
FT_D unsigned digit_peers(uint32_t digit, bool valid) {
    unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool     bit = (digit >> b) & 1u;
        const unsigned has = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? has : ~has;
    }
    return peers;
}

// One onesweep pass.  The grid is persistent (at most the CTAs resident at once): each CTA takes
// tiles by ticket until none are left.  skip: null, or the passes' skip words (then a pass of
// a constant digit returns at once).
template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads, (ITEMS <= 8 ? 4 : ITEMS <= 12 ? 3 : 2))
    onesweep_kernel(const SortPairs pairs, size_t n, size_t num_tiles, int pass, int shift,
                    const uint32_t *__restrict__ offsets, uint32_t *lookback, uint32_t *tile_counter,
                    const uint32_t *__restrict__ skip, uint32_t *status) {
    constexpr int TILE = SortCfg<ITEMS>::tile;
    if (skip && skip[pass]) return; // grid-uniform
    const int from = sort_parity(skip, pass);
    const unsigned long long *__restrict__ in_k = pairs.k[from];
    const uint32_t *__restrict__ in_v           = pairs.v[from];
    unsigned long long *__restrict__ out_k      = pairs.k[from ^ 1];
    uint32_t *__restrict__ out_v                = pairs.v[from ^ 1];
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned long long *s_k  = reinterpret_cast<unsigned long long *>(smem);
    uint32_t           *s_v  = reinterpret_cast<uint32_t *>(s_k + TILE);
    uint32_t           *s_wh = s_v + TILE; // [warp][256]
    __shared__ uint32_t s_tile_excl[256];
    __shared__ uint32_t s_base[256];
    __shared__ uint32_t s_ticket;
    __shared__ uint32_t s_wsum[kSortWarps];

    const int      tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    for (;;) {
        if (tid == 0) s_ticket = atomicAdd(tile_counter, 1u);
        for (int i = tid; i < kSortWarps * 256; i += kSortThreads) s_wh[i] = 0;
        __syncthreads();
        const size_t tile = s_ticket;
        if (tile >= num_tiles) break; // grid-uniform per CTA
        const size_t base = tile * (size_t)TILE;

        unsigned long long key[ITEMS];
        uint32_t           val[ITEMS], rank[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const size_t pos = base + (size_t)warp * 32 * ITEMS + (size_t)i * 32 + lane;
            key[i]           = pos < n ? in_k[pos] : 0ull;
            val[i]           = pos < n ? in_v[pos] : 0u;
        }
        uint32_t *wh = s_wh + warp * 256;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const bool     valid  = base + (size_t)warp * 32 * ITEMS + (size_t)i * 32 + lane < n;
            const uint32_t d      = (uint32_t)(key[i] >> shift) & 255u;
            const unsigned peers  = digit_peers(d, valid);
            const uint32_t before = valid ? wh[d] : 0u;
            __syncwarp();
            if (valid && (peers & lt_mask) == 0u) wh[d] = before + __popc(peers);
            __syncwarp();
            rank[i] = before + __popc(peers & lt_mask);
        }
        __syncthreads();

        // per-digit: warp exclusive prefixes and the tile count
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c    = s_wh[w * 256 + tid];
            s_wh[w * 256 + tid] = run;
            run += c;
        }
        const uint32_t tile_count = run;
        // (published at once: the next tiles' look-back may be waiting for it)
        uint32_t *lb = lookback + tile * 256;
        st_volatile(lb + tid, (tile == 0 ? kFlagInc : kFlagAgg) | tile_count);

        // exclusive scan of tile counts over digits (block scan, 256 threads)
        uint32_t incl = tile_count;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += v;
        }
        if (lane == 31) s_wsum[warp] = incl;
        __syncthreads();
        uint32_t wpre = 0;
        for (int w = 0; w < warp; ++w) wpre += s_wsum[w];
        s_tile_excl[tid] = wpre + incl - tile_count;
        __syncthreads();

        // stage the tile in digit order
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (base + (size_t)warp * 32 * ITEMS + (size_t)i * 32 + lane < n) {
                const uint32_t d  = (uint32_t)(key[i] >> shift) & 255u;
                const uint32_t lp = s_tile_excl[d] + s_wh[warp * 256 + d] + rank[i];
                s_k[lp]           = key[i];
                s_v[lp]           = val[i];
            }
        }

        // decoupled look-back for digit tid (every earlier tile is held by a running CTA or
        // done, since tickets are taken in order and a CTA finishes its tile first)
        uint32_t prefix = 0;
        if (tile > 0) {
            for (long long j = (long long)tile - 1; j >= 0; --j) {
                uint32_t sv;
                int      spins = 0;
                for (;;) {
                    sv = ld_volatile(lookback + (size_t)j * 256 + tid);
                    if (sv & kFlagMask) break;
                    if (++spins > 64) __nanosleep(32);
                    if (spins > kSpinLimit) break;
                }
                if (!(sv & kFlagMask)) {
                    atomicOr(status, STATUS_SPIN_LIMIT);
                    break;
                }
                prefix += sv & kCountMask;
                if (sv & kFlagInc) break;
            }
            st_volatile(lb + tid, kFlagInc | (prefix + tile_count));
        }
        s_base[tid] = offsets[tid] + prefix - s_tile_excl[tid];
        __syncthreads();
        const int tile_n = (int)min((size_t)TILE, n - base);
        for (int j = tid; j < tile_n; j += kSortThreads) {
            const unsigned long long k  = s_k[j];
            const uint32_t           d  = (uint32_t)(k >> shift) & 255u;
            const uint32_t           gp = s_base[d] + (uint32_t)j;
            if (gp >= n) { // only reachable after a failed look-back; never write out of bounds
                atomicOr(status, STATUS_SPIN_LIMIT);
                continue;
            }
            out_k[gp] = k;
            out_v[gp] = s_v[j];
        }
        __syncthreads(); // the tile's shared memory is free for the next ticket
    }
}

// =========================================================================================
// SFC keys (sfc_encode, src/hlbvh.hpp:357-423).
// =========================================================================================
// Peano-Hilbert state tables of two levels at once: state and six bits of the position (the two
// bits of x, then of y, then of z) -> next state << 6 | the two levels' key digits.  Half the
// chain of dependent look-ups of the one-level tables.
static constexpr int kPh2Entries = 48 * 64;
FT_D void ph2_fill(uint16_t *t) { // (every thread of the block; a barrier follows)
    for (int i = threadIdx.x; i < kPh2Entries; i += blockDim.x) {
        const int st = i >> 6, x = (i >> 4) & 3, y = (i >> 2) & 3, z = i & 3;
        const int p1 = ((x >> 1) << 2) | ((y >> 1) << 1) | (z >> 1), p0 = ((x & 1) << 2) | ((y & 1) << 1) | (z & 1);
        const int r  = c_rot[st * 8 + p1];
        t[i]         = (uint16_t)(((int)c_rot[r * 8 + p0] << 6) | (c_sub[st * 8 + p1] << 3) | c_sub[r * 8 + p0]);
    }
}
// ph_key (ft_build_dev.cuh) by pairs of levels, after one plain level when their number is odd.
template <int B>
FT_D void ph2_key(unsigned long long px, unsigned long long py, unsigned long long pz, const uint16_t *t,
                  unsigned long long &hi, unsigned long long &lo) {
    unsigned long long h = 0, l = 0;
    unsigned           st = 0;
    if constexpr (B & 1) {
        const unsigned p = (unsigned)((((px >> (B - 1)) & 1ull) << 2) | (((py >> (B - 1)) & 1ull) << 1) |
                                      ((pz >> (B - 1)) & 1ull));
        l  = c_sub[p];
        st = c_rot[p];
    }
#pragma unroll 7
    for (int b = (B & ~1) - 2; b >= 0; b -= 2) {
        const unsigned p = ((unsigned)(px >> b) & 3u) << 4 | ((unsigned)(py >> b) & 3u) << 2 | ((unsigned)(pz >> b) & 3u);
        const unsigned e = t[st * 64u + p];
        h                = (h << 6) | (l >> 58);
        l                = (l << 6) | (e & 63u);
        st               = e >> 6;
    }
    hi = h;
    lo = l;
}
template <class T, int SFC>
FT_D void encode_point2(T x, T y, T z, const T *par, const uint16_t *t, unsigned long long &hi, unsigned long long &lo) {
    using C = Coord<T>;
    if constexpr (!C::is_float) {
        const unsigned long long mask = (1ull << C::bits) - 1ull;
        ph2_key<C::bits>((unsigned long long)x & mask, (unsigned long long)y & mask, (unsigned long long)z & mask, t, hi,
                         lo);
    } else if constexpr (SFC == MORTON) {
        encode_point<T, SFC>(x, y, z, par, nullptr, nullptr, hi, lo);
    } else {
        unsigned long long c[3];
        sfc_cells<T, SFC>(x, y, z, par, c);
        ph2_key<21>(c[0], c[1], c[2], t, hi, lo);
    }
}
// The sort word of a key: the high word of 126-bit keys (their low word rides in the packed point).
template <class T> FT_D unsigned long long sort_word(unsigned long long hi, unsigned long long lo) {
    return Coord<T>::key_words == 2 ? hi : lo;
}

// Keys of n points.  klo / khi: null, or the key words; with `pack`, the build's form: the sort
// word in key, the input index in perm, the points packed, and the sort word's digit
// histograms added to hist (zero at launch).
template <class T, int SFC>
__global__ void __launch_bounds__(256) encode_kernel(const T *__restrict__ x, const T *__restrict__ y,
                                                     const T *__restrict__ z, size_t n, const T *__restrict__ bbox,
                                                     unsigned long long *klo, unsigned long long *khi,
                                                     unsigned long long *key, uint32_t *perm, PackedPoint<T> *pack,
                                                     uint32_t *hist) {
    using C = Coord<T>;
    __shared__ uint16_t s_ph[SFC == PEANO_HILBERT ? kPh2Entries : 1];
    __shared__ uint32_t s_hist[kSortDigits * 256];
    __shared__ T        s_par[6]; // lo, inv per axis
    if constexpr (SFC == PEANO_HILBERT) ph2_fill(s_ph);
    for (int i = threadIdx.x; i < kSortDigits * 256; i += blockDim.x) s_hist[i] = 0;
    if constexpr (C::is_float)
        if (threadIdx.x < 3) sfc_axis_params(bbox[2 * threadIdx.x], bbox[2 * threadIdx.x + 1], s_par[2 * threadIdx.x],
                                             s_par[2 * threadIdx.x + 1]);
    __syncthreads();
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const T            a = x[i], b = y[i], c = z[i];
        unsigned long long hi, lo;
        encode_point2<T, SFC>(a, b, c, s_par, s_ph, hi, lo);
        if (pack) {
            const unsigned long long w = sort_word<T>(hi, lo);
            key[i]                     = w;
            perm[i]                    = (uint32_t)i;
            PackedPoint<T> p{a, b, c, T(0)};
            if constexpr (C::key_words == 2) p.pad = lo;
            pack[i] = p;
            hist_add(s_hist, w);
        } else {
            klo[i] = lo;
            if (C::key_words == 2) khi[i] = hi;
        }
    }
    if (!pack) return;
    __syncthreads();
    for (int i = threadIdx.x; i < kSortDigits * 256; i += blockDim.x)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// Key layout conversions between the reference's sfc_key and the internal (hi, lo) pair.
// mode 0: Morton uint64; 1: {hs,is,ls} uint32; 2: {hs,is,ls} uint64.
FT_D void key_from_ref(const void *ref, size_t i, int mode, unsigned long long &hi, unsigned long long &lo) {
    hi = 0;
    if (mode == 0) {
        lo = ((const unsigned long long *)ref)[i];
    } else if (mode == 1) {
        const uint32_t *w = (const uint32_t *)ref + 3 * i;
        lo                = ((unsigned long long)w[1] << 32) | w[2];
    } else {
        const unsigned long long *w = (const unsigned long long *)ref + 3 * i;
        hi                          = w[1];
        lo                          = w[2];
    }
}
__global__ void keys_from_ref_kernel(const void *ref, size_t n, int mode, unsigned long long *klo,
                                     unsigned long long *khi) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        unsigned long long hi, lo;
        key_from_ref(ref, i, mode, hi, lo);
        klo[i] = lo;
        if (mode == 2) khi[i] = hi;
    }
}

// The build's form of caller keys (see encode_kernel).
template <class T>
__global__ void __launch_bounds__(256) pack_ref_kernel(const T *__restrict__ x, const T *__restrict__ y,
                                                       const T *__restrict__ z, size_t n, const void *ref, int mode,
                                                       unsigned long long *key, uint32_t *perm, PackedPoint<T> *pack,
                                                       uint32_t *hist) {
    __shared__ uint32_t s_hist[kSortDigits * 256];
    for (int i = threadIdx.x; i < kSortDigits * 256; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        unsigned long long hi, lo;
        key_from_ref(ref, i, mode, hi, lo);
        const unsigned long long w = sort_word<T>(hi, lo);
        key[i]                     = w;
        perm[i]                    = (uint32_t)i;
        PackedPoint<T> p{x[i], y[i], z[i], T(0)};
        if constexpr (Coord<T>::key_words == 2) p.pad = lo;
        pack[i] = p;
        hist_add(s_hist, w);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kSortDigits * 256; i += blockDim.x)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// =========================================================================================
// Box, keys and sort of a small set in one block: for at most kFrontMax points the launches of
// the steps above (two for the box, keys, histogram scan, eight passes) are all latency.  Keys and
// values stay in registers between the passes, which rank per warp like onesweep_kernel and
// scatter in shared memory.  4K float points: some 95 us of kernels in 13 launches become 41 us
// (67 us with all eight passes).
// =========================================================================================
static constexpr int kFrontThreads = 1024, kFrontItems = 8, kFrontMax = kFrontThreads * kFrontItems;
static constexpr int kFrontRun     = 16;
template <class T> struct alignas(16) FrontShared {
    unsigned long long k[kFrontMax];
    uint32_t           v[kFrontMax];
    uint32_t           wh[256 * 33]; // [digit][warp], a word of padding per digit
    uint32_t           tot[256];
    uint16_t           ph[kPh2Entries];
    T                  red[32][6], par[6];
    int                same;
};

// box: the points' box goes to bbox (6), or behind it (6 .. 11) when bbox holds the caller's.
template <class T, int SFC>
__global__ void __launch_bounds__(kFrontThreads, 1)
    front_kernel(const T *__restrict__ x, const T *__restrict__ y, const T *__restrict__ z, int n, int caller_box,
                 T *bbox, unsigned long long *key_out, uint32_t *perm, PackedPoint<T> *pack) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FrontShared<T> &s   = *reinterpret_cast<FrontShared<T> *>(smem_raw);
    const int       tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned  lt  = (1u << lane) - 1u, FULL = 0xffffffffu;
    const int       items = (n + kFrontThreads - 1) / kFrontThreads;
    if constexpr (SFC == PEANO_HILBERT) ph2_fill(s.ph);
    {
        T m[6];
        bb_identity(m);
        for (int i = tid; i < n; i += kFrontThreads) {
            T v[6] = {x[i], x[i], y[i], y[i], z[i], z[i]};
            bb_fold(m, v);
        }
        auto fold_warp = [&]() {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                T o[6];
#pragma unroll
                for (int d = 0; d < 6; ++d) o[d] = __shfl_down_sync(FULL, m[d], off);
                bb_fold(m, o);
            }
        };
        fold_warp();
        if (lane == 0)
#pragma unroll
            for (int d = 0; d < 6; ++d) s.red[warp][d] = m[d];
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int d = 0; d < 6; ++d) m[d] = s.red[lane][d];
            fold_warp();
            if (lane == 0) {
#pragma unroll
                for (int d = 0; d < 6; ++d) bbox[(caller_box ? 6 : 0) + d] = m[d];
                if constexpr (Coord<T>::is_float) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const T lo = caller_box ? bbox[2 * d] : m[2 * d], hi = caller_box ? bbox[2 * d + 1] : m[2 * d + 1];
                        sfc_axis_params(lo, hi, s.par[2 * d], s.par[2 * d + 1]);
                    }
                }
            }
        }
        __syncthreads();
    }
    unsigned long long key[kFrontItems];
    uint32_t           val[kFrontItems], rank[kFrontItems];
    const int          first = warp * 32 * items + lane; // this thread's pairs: first + 32 i
#pragma unroll
    for (int i = 0; i < kFrontItems; ++i) {
        const int e = first + 32 * i;
        key[i]      = 0ull;
        val[i]      = (uint32_t)e;
        if (i < items && e < n) {
            const T            a = x[e], b = y[e], c = z[e];
            unsigned long long hi, lo;
            encode_point2<T, SFC>(a, b, c, s.par, s.ph, hi, lo);
            key[i] = sort_word<T>(hi, lo);
            PackedPoint<T> p{a, b, c, T(0)};
            if constexpr (Coord<T>::key_words == 2) p.pad = lo;
            pack[e] = p;
        }
    }
    // The upper half of the word first: few points share it, and a thread orders such a run of at
    // most kFrontRun pairs in place.  A longer run takes the passes over the whole word from the
    // current order (stable, so equal words keep their input order either way).
    bool whole = false; // block-uniform
    for (int d = kSortDigits / 2;; ++d) {
        if (d == kSortDigits) {
            if (whole) break;
            if (tid == 0) s.same = 0;
            __syncthreads();
#pragma unroll
            for (int i = 0; i < kFrontItems; ++i) {
                const int e = first + 32 * i;
                if (i < items && e < n) {
                    s.k[e] = key[i];
                    s.v[e] = val[i];
                }
            }
            __syncthreads();
            for (int e = tid; e + 1 < n; e += kFrontThreads) { // run starts
                const uint32_t up = (uint32_t)(s.k[e] >> 32);
                if ((uint32_t)(s.k[e + 1] >> 32) != up || (e > 0 && (uint32_t)(s.k[e - 1] >> 32) == up)) continue;
                int f = e + 2;
                while (f < n && f - e <= kFrontRun && (uint32_t)(s.k[f] >> 32) == up) ++f;
                if (f - e > kFrontRun) {
                    s.same = 1;
                    continue;
                }
                for (int j = e + 1; j < f; ++j) {
                    const unsigned long long kj = s.k[j];
                    const uint32_t           vj = s.v[j];
                    int                      m  = j;
                    for (; m > e && s.k[m - 1] > kj; --m) {
                        s.k[m] = s.k[m - 1];
                        s.v[m] = s.v[m - 1];
                    }
                    s.k[m] = kj;
                    s.v[m] = vj;
                }
            }
            __syncthreads();
            whole = s.same != 0;
#pragma unroll
            for (int i = 0; i < kFrontItems; ++i) {
                const int e = first + 32 * i;
                if (i < items && e < n) {
                    key[i] = s.k[e];
                    val[i] = s.v[e];
                }
            }
            __syncthreads();
            if (!whole) break;
            d = 0;
        }
        const int shift = 8 * d;
        for (int i = tid; i < 256 * 33; i += kFrontThreads) s.wh[i] = 0;
        if (tid == 0) s.same = 0;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kFrontItems; ++i) {
            if (i < items) { // block-uniform
                const bool     valid  = first + 32 * i < n;
                const uint32_t g      = (uint32_t)(key[i] >> shift) & 255u;
                const unsigned peers  = digit_peers(g, valid);
                const uint32_t before = valid ? s.wh[g * 33 + warp] : 0u;
                __syncwarp();
                if (valid && (peers & lt) == 0u) s.wh[g * 33 + warp] = before + __popc(peers);
                __syncwarp();
                rank[i] = before + __popc(peers & lt);
            }
        }
        __syncthreads();
        // per digit: exclusive prefixes over the warps (a lane each) and the total
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int      g    = warp * 8 + j;
            const uint32_t c    = s.wh[g * 33 + lane];
            uint32_t       incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += u;
            }
            s.wh[g * 33 + lane] = incl - c;
            if (lane == 31) {
                s.tot[g] = incl;
                if (incl == (uint32_t)n) s.same = 1;
            }
        }
        __syncthreads();
        if (s.same) { // one digit value holds every key (block-uniform)
            __syncthreads();
            continue;
        }
        if (warp == 0) { // exclusive prefixes of the totals
            uint32_t v[8], sum = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[i] = s.tot[lane * 8 + i];
                sum += v[i];
            }
            uint32_t incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += u;
            }
            uint32_t run = incl - sum;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                s.tot[lane * 8 + i] = run;
                run += v[i];
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kFrontItems; ++i) {
            if (i < items && first + 32 * i < n) {
                const uint32_t g  = (uint32_t)(key[i] >> shift) & 255u;
                const uint32_t at = s.tot[g] + s.wh[g * 33 + warp] + rank[i];
                s.k[at]           = key[i];
                s.v[at]           = val[i];
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kFrontItems; ++i) {
            const int e = first + 32 * i;
            if (i < items && e < n) {
                key[i] = s.k[e];
                val[i] = s.v[e];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < kFrontItems; ++i) {
        const int e = first + 32 * i;
        if (i < items && e < n) {
            key_out[e] = key[i];
            perm[e]    = val[i];
        }
    }
}

// Leaf init of build_tree with caller arrays (src/hlbvh.hpp:906-923).
template <class T>
__global__ void leaf_init_kernel(const T *sx, const T *sy, const T *sz, size_t n, const uint32_t *sid,
                                 const int8_t *sghost, const int32_t *sorig, T *mnx, T *mxx, T *mny, T *mxy,
                                 T *mnz, T *mxz, uint32_t *tid_out, int8_t *ghost_out, int32_t *orig_out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        size_t leaf = i + n - 1;
        mnx[leaf] = mxx[leaf] = sx[i];
        mny[leaf] = mxy[leaf] = sy[i];
        mnz[leaf] = mxz[leaf] = sz[i];
        if (sid) tid_out[leaf] = sid[i];
        if (sghost) ghost_out[leaf] = sghost[i];
        if (sorig) orig_out[leaf] = sorig[i];
    }
}

// =========================================================================================
// Host orchestration
// =========================================================================================
static int grid_for(size_t n, int threads, int max_blocks = 148 * 16) {
    size_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    return (int)std::min<size_t>(b, (size_t)max_blocks);
}

void free_scratch(TreeImpl &s) {
    if (s.arena && s.pool) {
        // (freeing memory of a pool does not wait for the work on it, as cudaFree does elsewhere)
        const int dev = s.pool->device;
        int       cur = dev;
        cudaGetDevice(&cur);
        if (cur != dev) cudaSetDevice(dev);
        if (cudaDeviceSynchronize() == cudaSuccess) { // (refused under a capture, as cudaFree is: the piece stays)
            cudaFreeAsync(s.arena, cudaStreamLegacy);
            if (s.pool.use_count() == 1) cudaStreamSynchronize(cudaStreamLegacy); // (the pool goes with it)
        }
        cudaGetLastError();
        if (cur != dev) cudaSetDevice(cur);
    } else if (s.arena) {
        cudaFree(s.arena); // a single tree's: everything below lies in it
    } else {
        void *ptrs[] = {s.recs, s.height, s.counters, s.leafcount, s.pack, s.pend, s.qrec, s.qpts, s.qflag, s.key_lo, s.key_hi, s.tmp_lo, s.tmp_hi,
                        s.perm, s.tmp_perm, s.bbox, s.bbox_partial, s.hist, s.lookback, s.tile_counter, s.status};
        for (void *p : ptrs)
            if (p) cudaFree(p);
    }
    int coord = s.coord;
    s         = TreeImpl{};
    s.coord   = coord;
}

static size_t sort_tiles(size_t n) { // the most tiles any tile size makes
    const size_t tile = (size_t)kSortThreads * kSortItems;
    return (n + tile - 1) / tile;
}

// A tree's scratch in one allocation: the driver maps device memory in blocks of 2 MB and more, some
// 320 us an allocation above 1 MB whatever its size, and as much again to give it back.  Trees
// whose scratch is at most kPooled take it from the device's pool instead, which maps 32 MB at a time
// (210 us, and 140 to make the pool) and hands out pieces in 2 us; it keeps at most kPoolKept unused
// and goes with the last context and tree that have used it.  Host time of the first build on a new
// tree, earlier trees kept / destroyed: 4K float points 606 / 250 us with an allocation per array,
// 800 / 458 with one of its own, 121 / 118 from the pool; 1K 242 / 237 with an allocation per array,
// 104 / 104 from the pool; 100K double (one of its own) 2160 -> 566 us.  No room to grow is taken
// beyond what the tree's node arrays hold.
static constexpr size_t kPooled = size_t(8) << 20, kPoolKept = size_t(32) << 20;

// The current driver context's number (a cudaDeviceReset makes another one); 0: it cannot be read.
static unsigned long long driver_context_id() {
    using GetId  = CUresult (*)(CUcontext, unsigned long long *);
    static GetId fn = [] {
        void                           *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<GetId>(p);
    }();
    unsigned long long id = 0;
    return fn && fn(nullptr, &id) == CUDA_SUCCESS ? id : 0ull;
}

ScratchPool::~ScratchPool() {
    int cur = device;
    cudaGetDevice(&cur);
    if (cur != device) cudaSetDevice(device);
    if (pool && driver_context_id() == context) cudaMemPoolDestroy(pool); // (else it went with its context)
    if (cur != device) cudaSetDevice(cur);
}

static void *pool_alloc(Context &ctx, size_t bytes, cudaStream_t st) {
    constexpr int                     kDevices = 64;
    static std::mutex                 making; // (any thread's contexts and trees)
    static std::weak_ptr<ScratchPool> pools[kDevices];
    std::lock_guard<std::mutex>       lock(making);
    const unsigned long long          context = driver_context_id();
    if (context == 0 || ctx.device < 0 || ctx.device >= kDevices) return nullptr;
    if (!ctx.pool) ctx.pool = pools[ctx.device].lock();
    if (!ctx.pool || ctx.pool->context != context) {
        auto             pool = std::make_shared<ScratchPool>();
        cudaMemPoolProps props{};
        props.allocType         = cudaMemAllocationTypePinned;
        props.location.type     = cudaMemLocationTypeDevice;
        props.location.id       = ctx.device;
        pool->device            = ctx.device;
        pool->context           = context;
        unsigned long long kept = kPoolKept;
        if (cudaMemPoolCreate(&pool->pool, &props) != cudaSuccess ||
            cudaMemPoolSetAttribute(pool->pool, cudaMemPoolAttrReleaseThreshold, &kept) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        ctx.pool          = pool;
        pools[ctx.device] = pool;
    }
    void *p = nullptr;
    if (cudaMallocFromPoolAsync(&p, bytes, ctx.pool->pool, st) == cudaSuccess) return p;
    cudaGetLastError();
    return nullptr;
}

void ensure_scratch(Context &ctx, TreeImpl &s, size_t n, size_t most, cudaStream_t st) {
    if (n <= s.cap && s.key_lo) return;
    free_scratch(s);
    const ft_options &o   = ctx.opts;
    const size_t      cap = std::max(std::max<size_t>(n, 64), std::min(n + n / 2 + 1024, most)), ni = cap - 1;
    const int         W   = key_words(o);
    const size_t      cb  = coord_bytes(o.coord_type);
    s.coord          = o.coord_type;
    s.lookback_words = kSortDigits * sort_tiles(cap) * 256;
    size_t bytes     = 0;
    auto   place     = [&](auto *&p, size_t size) { // nothing to place it in yet: only counted
        if (s.arena) p = reinterpret_cast<std::remove_reference_t<decltype(p)>>((unsigned char *)s.arena + bytes);
        bytes += (size + 255) / 256 * 256;
    };
    auto place_all = [&] {
        bytes = 0;
        place(s.recs, ni * 16 * cb);
        place(s.qrec, ni * sizeof(QRec));
        place(s.qpts, cap * sizeof(QPoint));
        place(s.pack, cap * 4 * cb);
        place(s.key_lo, cap * 8);
        place(s.tmp_lo, cap * 8);
        if (W == 2) {
            place(s.key_hi, cap * 8);
            place(s.tmp_hi, cap * 8);
        }
        place(s.perm, cap * 4);
        place(s.tmp_perm, cap * 4);
        place(s.counters, cap * 4);
        place(s.leafcount, cap * 4);
        place(s.height, cap);
        place(s.pend, (2 * cap + 2 * (cap / kTreeletLeaves + 1)) * 4);
        place(s.lookback, s.lookback_words * 4);
        place(s.bbox, 12 * 8); // the keys' box, then the points' box
        place(s.bbox_partial, (size_t)kBboxBlocks * 6 * 8);
        place(s.hist, (16 * 256 + 16) * 4);
        place(s.qflag, 16);
        place(s.tile_counter, kTicketWords * 4);
        place(s.status, 16 + sizeof(TreeSummary));
    };
    place_all();
    void *p = bytes <= kPooled ? pool_alloc(ctx, bytes, st) : nullptr;
    if (p) {
        s.pool = ctx.pool;
    } else if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        fail(FT_ERR_OUT_OF_MEMORY, "cudaMalloc of build scratch failed");
    }
    s.arena = p;
    place_all();
    s.cap = cap;
    FT_CUDA(cudaMemsetAsync(s.status, 0, 16, st));
}

template <class T>
static void bbox_typed(const void *x, const void *y, const void *z, size_t n, void *partial, void *out,
                       cudaStream_t st) {
    int blocks = grid_for(n, kBboxThreads, kBboxBlocks);
    bbox_partial_kernel<T><<<blocks, kBboxThreads, 0, st>>>((const T *)x, (const T *)y, (const T *)z, n, (T *)partial);
    bbox_final_kernel<T><<<1, kBboxThreads, 0, st>>>((const T *)partial, blocks, (T *)out);
    FT_CUDA(cudaGetLastError());
}

void compute_bbox(Context &ctx, TreeImpl *scratch, const void *x, const void *y, const void *z, size_t n,
                  void *bbox_dev, cudaStream_t st) {
    void *partial = scratch->bbox_partial;
    switch (ctx.opts.coord_type) {
    case F32: bbox_typed<float>(x, y, z, n, partial, bbox_dev, st); break;
    case F64: bbox_typed<double>(x, y, z, n, partial, bbox_dev, st); break;
    case U32: bbox_typed<uint32_t>(x, y, z, n, partial, bbox_dev, st); break;
    case U64: bbox_typed<unsigned long long>(x, y, z, n, partial, bbox_dev, st); break;
    }
}

// fn(value of the coordinate type's, std::integral_constant of the SFC) for the context's options.
template <class F> static void for_type(const ft_options &o, F &&f) {
    auto sfc = [&](auto zero) {
        using T = decltype(zero);
        if constexpr (Coord<T>::is_float) {
            if (o.sfc_type == MORTON) {
                f(zero, std::integral_constant<int, MORTON>{});
                return;
            }
        }
        f(zero, std::integral_constant<int, PEANO_HILBERT>{});
    };
    switch (o.coord_type) {
    case F32: sfc(0.0f); break;
    case F64: sfc(0.0); break;
    case U32: sfc((uint32_t)0); break;
    case U64: sfc((unsigned long long)0); break;
    }
}

static int ref_key_mode(const ft_options &o) {
    if (o.sfc_type == MORTON) return 0;
    return (o.coord_type == U64) ? 2 : 1;
}

void sfc_encode_ref_layout(Context &ctx, TreeImpl &s, const void *x, const void *y, const void *z, size_t n,
                           const void *bbox_dev, void *keys_ref_dev, cudaStream_t st) {
    for_type(ctx.opts, [&](auto zero, auto sfc) {
        using T = decltype(zero);
        encode_kernel<T, decltype(sfc)::value><<<grid_for(n, 256), 256, 0, st>>>(
            (const T *)x, (const T *)y, (const T *)z, n, (const T *)bbox_dev, (unsigned long long *)s.key_lo,
            (unsigned long long *)s.key_hi, nullptr, nullptr, nullptr, nullptr);
    });
    FT_CUDA(cudaGetLastError());
    keys_to_ref_kernel<<<grid_for(n, 256), 256, 0, st>>>((const unsigned long long *)s.key_lo,
                                                          (const unsigned long long *)s.key_hi, n,
                                                          ref_key_mode(ctx.opts), keys_ref_dev);
    FT_CUDA(cudaGetLastError());
}

// 126-bit keys, second stage: after the sort by the high word, runs of equal high words are put
// in (low word, input index) order.  The thread at the start of each run insertion-sorts its
// values in place when it holds at most kRunCap keys (stable, so equal keys keep the index
// order of the sort); a longer run sets flag[0], and the host sorts by both words instead.
static constexpr int kRunCap = 32;

template <class T>
__global__ void __launch_bounds__(256) hi_run_fixup_kernel(const SortPairs pairs, const uint32_t *__restrict__ skip,
                                                           int passes, const PackedPoint<T> *__restrict__ pack,
                                                           size_t n, uint32_t *flag) {
    const int par = sort_parity(skip, passes);
    const unsigned long long *__restrict__ khi = pairs.k[par];
    uint32_t *__restrict__ perm                = pairs.v[par];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i + 1 < n; i += (size_t)gridDim.x * blockDim.x) {
        const unsigned long long h = khi[i];
        if (khi[i + 1] != h || (i > 0 && khi[i - 1] == h)) continue; // not the start of a run
        size_t e = i + 2;
        while (e < n && e - i <= (size_t)kRunCap && khi[e] == h) ++e;
        if (e - i > (size_t)kRunCap) {
            atomicOr(flag, 1u);
            continue;
        }
        for (size_t j = i + 1; j < e; ++j) {
            const uint32_t pv = perm[j];
            const T        kl = pack[pv].pad; // the low key word
            size_t         m  = j;
            while (m > i && pack[perm[m - 1]].pad > kl) {
                perm[m] = perm[m - 1];
                --m;
            }
            perm[m] = pv;
        }
    }
}

// Full sort of 126-bit keys (a long run of equal high words): keys for the passes over the low
// word, and, in the order those leave, for the passes over the high word (from the points, or
// from the caller's keys).
__global__ void __launch_bounds__(256) low_keys_kernel(const PackedPoint<unsigned long long> *__restrict__ pack, size_t n,
                                                       unsigned long long *key, uint32_t *perm) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        key[i]  = pack[i].pad;
        perm[i] = (uint32_t)i;
    }
}
__global__ void __launch_bounds__(256) high_keys_kernel(const PackedPoint<unsigned long long> *__restrict__ pack,
                                                        const unsigned long long *__restrict__ ref,
                                                        const SortPairs pairs, const uint32_t *__restrict__ skip,
                                                        size_t n) {
    __shared__ uint8_t s_rot[48 * 8], s_sub[48 * 8];
    for (int i = threadIdx.x; i < 48 * 8; i += blockDim.x) {
        s_rot[i] = c_rot[i];
        s_sub[i] = c_sub[i];
    }
    __syncthreads();
    const int       par  = sort_parity(skip, kSortDigits);
    const uint32_t *perm = pairs.v[par];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t     src = perm[i];
        unsigned long long hi, lo;
        if (ref) {
            hi = ref[3 * (size_t)src + 1];
        } else {
            const PackedPoint<unsigned long long> p = pack[src];
            encode_point<unsigned long long, PEANO_HILBERT>(p.x, p.y, p.z, nullptr, s_rot, s_sub, hi, lo);
        }
        pairs.k[0][i] = hi;
        pairs.v[0][i] = src; // (par 0: in place)
    }
}

// Persistent grid of a onesweep pass: the CTAs resident at once, never more than the tiles.
template <int ITEMS> static unsigned sort_grid(size_t tiles) {
    static int per_sm = 0, sms = 0;
    static std::once_flag once;
    std::call_once(once, [] {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaFuncSetAttribute(onesweep_kernel<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SortCfg<ITEMS>::smem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, onesweep_kernel<ITEMS>, kSortThreads,
                                                          SortCfg<ITEMS>::smem) != cudaSuccess) {
            cudaGetLastError();
            per_sm = 1;
            sms    = 148;
        }
        per_sm = std::max(per_sm, 1);
    });
    return (unsigned)std::max<size_t>(1, std::min<size_t>(tiles, (size_t)per_sm * (size_t)sms));
}

// The passes of `ndig` digit positions over pairs whose histograms (of all eight positions) are in
// s.hist.  skip: null (every listed pass runs) or the skip words, indexed by position (then the
// positions are 0 .. ndig - 1).
template <int ITEMS>
static void sort_passes(TreeImpl &s, const SortPairs &pairs, size_t n, int ndig, const int *digits,
                        const uint32_t *skip, cudaStream_t st) {
    const size_t   tiles = (n + SortCfg<ITEMS>::tile - 1) / SortCfg<ITEMS>::tile;
    const unsigned grid  = sort_grid<ITEMS>(tiles);
    FT_CUDA(cudaFuncSetAttribute(onesweep_kernel<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SortCfg<ITEMS>::smem));
    for (int i = 0; i < ndig; ++i) {
        const int d = digits[i];
        onesweep_kernel<ITEMS><<<grid, kSortThreads, SortCfg<ITEMS>::smem, st>>>(
            pairs, n, tiles, i, 8 * d, s.hist + d * 256, s.lookback + (size_t)i * tiles * 256, s.tile_counter + i, skip,
            s.status);
        FT_CUDA(cudaGetLastError());
    }
}
static const int kAllDigits[kSortDigits] = {0, 1, 2, 3, 4, 5, 6, 7};

// Scratch words a sort of n pairs starts from: histograms, look-back words and tickets.
static void sort_clear(TreeImpl &s, size_t n, int ndig, int items, cudaStream_t st) {
    const size_t tile  = (size_t)kSortThreads * items;
    const size_t tiles = (n + tile - 1) / tile;
    FT_CUDA(cudaMemsetAsync(s.hist, 0, (kSortDigits * 256 + 16) * sizeof(uint32_t), st));
    FT_CUDA(cudaMemsetAsync(s.tile_counter, 0, kSortDigits * sizeof(uint32_t), st));
    FT_CUDA(cudaMemsetAsync(s.lookback, 0, (size_t)ndig * tiles * 256 * sizeof(uint32_t), st));
}

// Sort of build_bvh's pairs after their histograms (constant digits are skipped on the device).
static void sort_run(TreeImpl &s, const SortPairs &pairs, size_t n, int items, cudaStream_t st) {
    uint32_t *skip = s.hist + kSortDigits * 256;
    radix_scan_kernel<<<kSortDigits, 256, 0, st>>>(s.hist, n, skip);
    FT_CUDA(cudaGetLastError());
    switch (items) {
    case 12: sort_passes<12>(s, pairs, n, kSortDigits, kAllDigits, skip, st); break;
    case 16: sort_passes<16>(s, pairs, n, kSortDigits, kAllDigits, skip, st); break;
    case 20: sort_passes<20>(s, pairs, n, kSortDigits, kAllDigits, skip, st); break;
    default: sort_passes<kSortItems>(s, pairs, n, kSortDigits, kAllDigits, skip, st); break;
    }
}
static int sort_tile_items(int items) { return items == 12 || items == 16 || items == 20 ? items : kSortItems; }

// The same sort over a fixed list of digit positions of (key_lo, perm) (every listed pass runs),
// used by the batched build and the query order.
void sort_pairs_fixed(TreeImpl &s, size_t n, int ndigits, const int *digits, cudaStream_t st) {
    if (n < 2 || ndigits <= 0) return;
    sort_clear(s, n, ndigits, kSortItems, st);
    radix_hist_kernel<<<grid_for(n, 256, 148 * 4), 256, 0, st>>>((const unsigned long long *)s.key_lo, n, s.hist);
    radix_scan_kernel<<<kSortDigits, 256, 0, st>>>(s.hist, n, s.hist + kSortDigits * 256);
    FT_CUDA(cudaGetLastError());
    const SortPairs pairs = {{(unsigned long long *)s.key_lo, (unsigned long long *)s.tmp_lo}, {s.perm, s.tmp_perm}};
    sort_passes<kSortItems>(s, pairs, n, ndigits, digits, nullptr, st);
    if (ndigits & 1) {
        std::swap(s.key_lo, s.tmp_lo);
        std::swap(s.perm, s.tmp_perm);
    }
}

size_t sort_lookback_words(size_t n) {
    return kSortDigits * sort_tiles(n) * 256;
}

const int *sort_item_choices(int *count) {
    static const int items[4] = {8, 12, 16, 20}; // the default first
    *count = 4;
    return items;
}

template <class T> struct SoA {
    T *mnx, *mxx, *mny, *mxy, *mnz, *mxz;
    explicit SoA(const ft_tree &t)
        : mnx((T *)t.min_x), mxx((T *)t.max_x), mny((T *)t.min_y), mxy((T *)t.max_y), mnz((T *)t.min_z),
          mxz((T *)t.max_z) {}
};

// Topology, boxes and records from sorted keys (ft_treelet.cuh): the treelets, then the walk
// records of the nodes formed outside a block.
template <class T, int SRC>
static void build_treelets(const ft_options &o, ft_tree &t, TreeImpl &s, size_t n, const void *box, TreeletArgs<T> a,
                           cudaStream_t st, Context *prof = nullptr) {
    a.n        = (int)n;
    a.periodic = o.periodic;
    a.klo      = (const unsigned long long *)s.key_lo;
    a.khi      = (const unsigned long long *)s.key_hi;
    if (SRC != LEAVES_PACKED) s.sort_passes = 0;
    a.box      = (const T *)box;
    void *soa[6] = {t.min_x, t.max_x, t.min_y, t.max_y, t.min_z, t.max_z};
    for (int d = 0; d < 6; ++d) a.soa[d] = (T *)soa[d];
    a.left      = t.left_child;
    a.right     = t.right_child;
    a.parent    = t.parent;
    a.orig      = t.orig_idx;
    a.id_out    = t.id;
    a.ghost_out = t.is_ghost;
    a.recs      = (NodeRec<T> *)s.recs;
    a.height    = s.height;
    a.leaves    = s.leafcount;
    a.qrec      = (QRec *)s.qrec;
    a.qpts      = (QPoint *)s.qpts;
    a.qflag     = s.qflag;
    a.slot      = s.counters;
    uint32_t *list[2]  = {s.pend, s.pend + s.cap}; // (the four lie in one allocation)
    uint32_t *count[2] = {s.pend + 2 * s.cap, s.pend + 2 * s.cap + s.cap / kTreeletLeaves + 1};
    a.pend             = list[0];
    a.pend_count       = count[0];
    a.list      = (int32_t *)s.lookback; // (at least n words; the sort is done with them)
    a.status    = s.status;
    const bool many = n > (size_t)kTreeletLeaves;
    FT_CUDA(cudaMemsetAsync(s.qflag, 0, 4 * sizeof(uint32_t), st));
    if (many) FT_CUDA(cudaMemsetAsync(s.counters, 0xFF, n * sizeof(int32_t), st));
    if (n == 1) FT_CUDA(cudaMemsetAsync(t.parent, 0xFF, sizeof(int32_t), st));
    const unsigned blocks = (unsigned)((n + kTreeletLeaves - 1) / kTreeletLeaves);
    auto           run    = [&](auto kind) {
        auto fn = treelet_kernel<T, decltype(kind)::value, SRC>;
        FT_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TreeletShared<T>)));
        fn<<<blocks, kTreeletThreads, sizeof(TreeletShared<T>), st>>>(a);
        if (!many) return;
        auto join = treelet_join_kernel<T, decltype(kind)::value, SRC>;
        FT_CUDA(cudaFuncSetAttribute(join, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(JoinShared<T>)));
        JoinLevel lv{list[0], count[0], (int)blocks, (size_t)kTreeletLeaves, list[1], count[1]};
        for (;;) {
            const int groups = (lv.segs + kJoinBlocks - 1) / kJoinBlocks;
            if (groups == 1) lv.out_count = nullptr;
            join<<<groups, kJoinThreads, sizeof(JoinShared<T>), st>>>(a, lv);
            if (groups == 1) break;
            uint32_t *const from = const_cast<uint32_t *>(lv.in), *const from_count = const_cast<uint32_t *>(lv.in_count);
            lv = JoinLevel{lv.out, lv.out_count, groups, lv.stride * kJoinBlocks, from, from_count};
        }
        a.left_over = lv.out;
        treelet_climb_kernel<T, decltype(kind)::value, SRC><<<grid_for(n / 64, 128, 148 * 4), 128, 0, st>>>(a);
    };
    if constexpr (Coord<T>::key_words == 2) run(std::integral_constant<int, 2>{});
    else if (delta_kind(o) == 0) run(std::integral_constant<int, 0>{});
    else run(std::integral_constant<int, 1>{});
    FT_CUDA(cudaGetLastError());
    stage_mark(prof, BS_REFIT, st);
    if (many) treelet_qrec_kernel<T><<<grid_for(n / 64 + 1, 128, 148 * 8), 128, 0, st>>>(a);
    FT_CUDA(cudaGetLastError());
    stage_mark(prof, BS_RECORDS, st);
    if (n < 2) s.height_root = 0;
}

// The same from leaf slots that hold their points (caller arrays, an imported tree).
template <class T> static void build_in_place(Context &ctx, ft_tree &t, TreeImpl &s, size_t n, cudaStream_t st) {
    const size_t leaf = n - 1;
    void        *box  = (T *)s.bbox + 6;
    compute_bbox(ctx, &s, (const T *)t.min_x + leaf, (const T *)t.min_y + leaf, (const T *)t.min_z + leaf, n, box, st);
    build_treelets<T, LEAVES_IN_PLACE>(ctx.opts, t, s, n, box, TreeletArgs<T>{}, st);
}

// The pairs build_bvh sorts: the sort word of each key and its input index.
static SortPairs build_pairs(const ft_options &o, const TreeImpl &s) {
    const bool two = key_words(o) == 2;
    return SortPairs{{(unsigned long long *)(two ? s.key_hi : s.key_lo), (unsigned long long *)(two ? s.tmp_hi : s.tmp_lo)},
                     {s.perm, s.tmp_perm}};
}

// full_sort: 126-bit keys by both words (the last build met a long run of equal high words).
template <class T, int SFC>
static void build_bvh_typed(Context &ctx, ft_tree &t, const void *x, const void *y, const void *z, size_t n,
                            const uint32_t *id, const int8_t *ghost, const void *bbox_host, const void *caller_keys,
                            cudaStream_t st, int sort_items, bool full_sort) {
    constexpr bool TWO = Coord<T>::key_words == 2;
    TreeImpl      &s   = *(TreeImpl *)t.impl;
    ensure_scratch(ctx, s, n, t.capacity, st);
    if (sort_items <= 0) { // the tile the autotuner chose for this shape
        auto it = ctx.tuned.find(tune_key(TUNE_BUILD, key_words(ctx.opts), n));
        if (it != ctx.tuned.end()) sort_items = it->second.items;
    }
    sort_items = sort_tile_items(sort_items);
    stage_mark(&ctx, BS_START, st);
    const T *px = (const T *)x, *py = (const T *)y, *pz = (const T *)z;
    // 1. bounding box.  Only the float encode reads a caller's; integer encoding ignores it, so an
    // integer tree always keeps its true box (the query distance mode depends on it).  The
    // walks' frame follows from the points' own box.
    const bool caller_box = bbox_host && Coord<T>::is_float;
    T         *box        = (T *)s.bbox + (caller_box ? 6 : 0);
    if (caller_box) FT_CUDA(cudaMemcpyAsync(s.bbox, bbox_host, 6 * sizeof(T), cudaMemcpyHostToDevice, st));
    PackedPoint<T> *pack  = (PackedPoint<T> *)s.pack;
    const SortPairs pairs = build_pairs(ctx.opts, s);
    uint32_t       *skip  = s.hist + kSortDigits * 256;
    uint32_t       *runs  = s.tile_counter + kLongRunWord;
    const bool      front = n <= (size_t)kFrontMax && !caller_keys && !full_sort;
    if (front) { // box, keys and sort in one block
        auto fn = front_kernel<T, SFC>;
        FT_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FrontShared<T>)));
        fn<<<1, kFrontThreads, sizeof(FrontShared<T>), st>>>(px, py, pz, (int)n, caller_box ? 1 : 0, (T *)s.bbox,
                                                             pairs.k[0], pairs.v[0], pack);
        FT_CUDA(cudaGetLastError());
        s.sort_passes = 0;
        stage_mark(&ctx, BS_BBOX, st);
        stage_mark(&ctx, BS_ENCODE, st);
    } else {
        compute_bbox(ctx, &s, x, y, z, n, box, st);
        stage_mark(&ctx, BS_BBOX, st);
        // 2. keys, input indices, packed points, digit histograms
        sort_clear(s, n, kSortDigits, sort_items, st);
        const int grid = grid_for(n, 256, 148 * 8);
        if (caller_keys)
            pack_ref_kernel<T><<<grid, 256, 0, st>>>(px, py, pz, n, caller_keys, ref_key_mode(ctx.opts), pairs.k[0],
                                                     pairs.v[0], pack, s.hist);
        else
            encode_kernel<T, SFC><<<grid, 256, 0, st>>>(px, py, pz, n, (const T *)s.bbox, nullptr, nullptr, pairs.k[0],
                                                        pairs.v[0], pack, s.hist);
        FT_CUDA(cudaGetLastError());
        stage_mark(&ctx, BS_ENCODE, st);
        // 3. sort
        if constexpr (TWO) {
            if (full_sort) { // by the low word first
                low_keys_kernel<<<grid_for(n, 256), 256, 0, st>>>(pack, n, pairs.k[0], pairs.v[0]);
                FT_CUDA(cudaMemsetAsync(s.hist, 0, kSortDigits * 256 * sizeof(uint32_t), st));
                radix_hist_kernel<<<grid_for(n, 256, 148 * 4), 256, 0, st>>>(pairs.k[0], n, s.hist);
                sort_run(s, pairs, n, sort_items, st);
                high_keys_kernel<<<grid_for(n, 256), 256, 0, st>>>(pack, (const unsigned long long *)caller_keys, pairs,
                                                                   skip, n);
                sort_clear(s, n, kSortDigits, sort_items, st);
                radix_hist_kernel<<<grid_for(n, 256, 148 * 4), 256, 0, st>>>(pairs.k[0], n, s.hist);
                FT_CUDA(cudaGetLastError());
            }
        }
        sort_run(s, pairs, n, sort_items, st);
        s.sort_passes = kSortDigits;
    }
    if constexpr (TWO) {
        FT_CUDA(cudaMemsetAsync(runs, 0, sizeof(uint32_t), st));
        if (!full_sort)
            hi_run_fixup_kernel<T><<<grid_for(n, 256), 256, 0, st>>>(pairs, skip, s.sort_passes, pack, n, runs);
        FT_CUDA(cudaGetLastError());
    }
    stage_mark(&ctx, BS_SORT, st);
    // 4. leaves, topology, boxes and records
    stage_mark(&ctx, BS_GATHER, st);
    stage_mark(&ctx, BS_TOPOLOGY, st);
    TreeletArgs<T> a{};
    for (int b = 0; b < 2; ++b) {
        a.key[b]  = pairs.k[b];
        a.perm[b] = pairs.v[b];
    }
    a.skip    = skip;
    a.passes  = s.sort_passes;
    a.stop    = TWO ? runs : nullptr;
    a.klo_out = TWO ? (unsigned long long *)s.key_lo : nullptr;
    a.pack    = pack;
    a.id      = id;
    a.ghost   = ghost;
    build_treelets<T, LEAVES_PACKED>(ctx.opts, t, s, n, box, a, st, &ctx);
    ctx.bprof.recorded = ctx.bprof.on;
}

void build_bvh(Context &ctx, ft_tree &t, const void *x, const void *y, const void *z, size_t n, const uint32_t *id,
               const int8_t *ghost, const void *bbox_host, const void *caller_keys, cudaStream_t st, int sort_items,
               bool full_sort) {
    for_type(ctx.opts, [&](auto zero, auto sfc) {
        build_bvh_typed<decltype(zero), decltype(sfc)::value>(ctx, t, x, y, z, n, id, ghost, bbox_host, caller_keys, st,
                                                              sort_items, full_sort);
    });
}

// The sorted keys of a finished build in the reference's layout.
void sorted_keys_to_ref(const ft_options &o, const TreeImpl &s, size_t n, void *keys_ref, cudaStream_t st) {
    keys_to_ref_kernel<<<grid_for(n, 256), 256, 0, st>>>((const unsigned long long *)s.key_lo,
                                                          (const unsigned long long *)s.key_hi, n, ref_key_mode(o),
                                                          keys_ref);
    FT_CUDA(cudaGetLastError());
}

int key_words_of(const ft_options &o) { return key_words(o); }

template <class T>
static void build_tree_typed(Context &ctx, ft_tree &t, const void *keys_ref, const void *sx, const void *sy,
                             const void *sz, const uint32_t *sid, const int8_t *sghost, const int32_t *sorig,
                             cudaStream_t st) {
    TreeImpl &s = *(TreeImpl *)t.impl;
    size_t    n = t.num_leaves;
    ensure_scratch(ctx, s, n, t.capacity, st);
    keys_from_ref_kernel<<<grid_for(n, 256), 256, 0, st>>>(keys_ref, n, ref_key_mode(ctx.opts),
                                                           (unsigned long long *)s.key_lo,
                                                           (unsigned long long *)s.key_hi);
    FT_CUDA(cudaGetLastError());
    SoA<T> a(t);
    if (sx && sy && sz)
        leaf_init_kernel<T><<<grid_for(n, 256), 256, 0, st>>>((const T *)sx, (const T *)sy, (const T *)sz, n, sid,
                                                              sghost, sorig, a.mnx, a.mxx, a.mny, a.mxy, a.mnz,
                                                              a.mxz, t.id, t.is_ghost, t.orig_idx);
    FT_CUDA(cudaGetLastError());
    build_in_place<T>(ctx, t, s, n, st);
}

// Refit-only update of a built tree (no reference counterpart: the reference rebuilds).  The
// keys, leaf order and topology stay; the leaves take the new positions and the bottom-up
// treelets recompute every internal box, the node records, heights and walk records.  The
// result is the tree build_tree (src/hlbvh.hpp:773-982) makes from the same sorted keys with
// the new positions as its leaf arrays.
template <class T>
static void refit_typed(Context &ctx, ft_tree &t, const void *x, const void *y, const void *z, size_t n,
                        bool leaf_order, cudaStream_t st) {
    TreeImpl &s   = *(TreeImpl *)t.impl;
    void     *box = (T *)s.bbox + 6; // (the build's box stays: it encoded the keys)
    compute_bbox(ctx, &s, x, y, z, n, box, st);
    TreeletArgs<T> a{};
    a.x          = (const T *)x;
    a.y          = (const T *)y;
    a.z          = (const T *)z;
    a.leaf_order = leaf_order ? 1 : 0;
    build_treelets<T, LEAVES_MOVED>(ctx.opts, t, s, n, box, a, st);
}

void refit_bvh(Context &ctx, ft_tree &t, const void *x, const void *y, const void *z, size_t n, bool leaf_order,
               cudaStream_t st) {
    switch (ctx.opts.coord_type) {
    case F32: refit_typed<float>(ctx, t, x, y, z, n, leaf_order, st); break;
    case F64: refit_typed<double>(ctx, t, x, y, z, n, leaf_order, st); break;
    case U32: refit_typed<uint32_t>(ctx, t, x, y, z, n, leaf_order, st); break;
    case U64: refit_typed<unsigned long long>(ctx, t, x, y, z, n, leaf_order, st); break;
    }
}

// Topology, internal boxes, node records, heights and walk records recomputed from the
// tree's sorted keys and leaf slots (an imported tree).
void recompute_from_keys(Context &ctx, ft_tree &t, cudaStream_t st) {
    TreeImpl &s = *(TreeImpl *)t.impl;
    size_t    n = t.num_leaves;
    switch (ctx.opts.coord_type) {
    case F32: build_in_place<float>(ctx, t, s, n, st); break;
    case F64: build_in_place<double>(ctx, t, s, n, st); break;
    case U32: build_in_place<uint32_t>(ctx, t, s, n, st); break;
    case U64: build_in_place<unsigned long long>(ctx, t, s, n, st); break;
    }
}

template <class T>
__global__ void tree_summary_kernel(int n, const T *mxx, const T *mxy, const T *mxz, const uint8_t *height,
                                    const uint32_t *status, const uint32_t *qflag, const uint32_t *skip, int passes,
                                    const uint32_t *runs, TreeSummary *out) {
    TreeSummary m;
    m.mx[0]  = Coord<T>::is_float ? 0ull : (unsigned long long)mxx[0];
    m.mx[1]  = Coord<T>::is_float ? 0ull : (unsigned long long)mxy[0];
    m.mx[2]  = Coord<T>::is_float ? 0ull : (unsigned long long)mxz[0];
    m.status = *status;
    m.height = n > 1 ? height[0] : 0u;
    m.qflag  = n > 1 ? *qflag : 0u;
    m.parity    = (uint32_t)sort_parity(skip, passes);
    m.long_runs = runs ? *runs : 0u;
    *out        = m;
}

void tree_summary(const ft_options &o, ft_tree &t, bool sorted, TreeSummary &out, cudaStream_t st) {
    TreeImpl       &s   = *(TreeImpl *)t.impl;
    const uint32_t *runs = sorted && key_words(o) == 2 ? s.tile_counter + kLongRunWord : nullptr;
    TreeSummary    *dev = reinterpret_cast<TreeSummary *>(s.status + 4);
    auto            run = [&](auto *p) {
        using T = std::remove_pointer_t<decltype(p)>;
        tree_summary_kernel<T><<<1, 1, 0, st>>>((int)t.num_leaves, (const T *)t.max_x, (const T *)t.max_y,
                                                (const T *)t.max_z, s.height, s.status, s.qflag,
                                                s.hist + kSortDigits * 256, sorted ? s.sort_passes : 0, runs, dev);
    };
    switch (o.coord_type) {
    case F32: run((float *)nullptr); break;
    case F64: run((double *)nullptr); break;
    case U32: run((uint32_t *)nullptr); break;
    case U64: run((unsigned long long *)nullptr); break;
    }
    FT_CUDA(cudaGetLastError());
    FT_CUDA(cudaMemcpyAsync(&out, dev, sizeof(out), cudaMemcpyDeviceToHost, st));
    FT_CUDA(cudaStreamSynchronize(st));
    if (out.parity) { // the sort left its pairs in the second buffers
        if (key_words(o) == 2) std::swap(s.key_hi, s.tmp_hi);
        else std::swap(s.key_lo, s.tmp_lo);
        std::swap(s.perm, s.tmp_perm);
    }
    s.sort_passes = 0;
}

void build_tree_from_keys(Context &ctx, ft_tree &t, const void *keys_ref, const void *sx, const void *sy,
                          const void *sz, const uint32_t *sid, const int8_t *sghost, const int32_t *sorig,
                          cudaStream_t st) {
    switch (ctx.opts.coord_type) {
    case F32: build_tree_typed<float>(ctx, t, keys_ref, sx, sy, sz, sid, sghost, sorig, st); break;
    case F64: build_tree_typed<double>(ctx, t, keys_ref, sx, sy, sz, sid, sghost, sorig, st); break;
    case U32: build_tree_typed<uint32_t>(ctx, t, keys_ref, sx, sy, sz, sid, sghost, sorig, st); break;
    case U64: build_tree_typed<unsigned long long>(ctx, t, keys_ref, sx, sy, sz, sid, sghost, sorig, st); break;
    }
}

} // namespace ft
