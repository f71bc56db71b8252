// ft_fast_type.cuh -- the fast walk's kernels and their launches, templates over the coordinate
// type; ft_fast_f32.cu, ft_fast_f64.cu, ft_fast_u32.cu and ft_fast_u64.cu each instantiate one
// type, so the types compile in parallel.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ft_build_dev.cuh"
#include "ft_common.cuh"
#include "ft_cta_build.cuh"
#include "ft_fast.h"
#include "ft_internal.h"
#include "ft_walk.cuh"

namespace ft {

// Resident blocks the walk is compiled for (a register budget).
template <class T, int KC> constexpr int fast_min_blocks() { return KC <= 32 ? FT_FAST_MINB : 2 * FT_FAST_MINB; }
// The fast walk over queries [0, num), `lanes` queries a warp; or, with a list, a grid-stride loop
// over the list's entries (the count lives on the device: no host synchronisation).
template <class T, int PER, int KC>
__global__ void __launch_bounds__(32 * fast_warps<KC>(), fast_min_blocks<T, KC>())
    fast_self_knn_kernel(int lanes, QueryList lst, MissList miss, TreeDev<T> t_all, BatchDev bt, const T *__restrict__ qx,
                         const T *__restrict__ qy, const T *__restrict__ qz, const uint32_t *__restrict__ order,
                         const int32_t *__restrict__ leaf_ids, int num, int k, int half_window, int exclude_self,
                         int ret_orig, int binary, const typename Coord<T>::dist_t *__restrict__ bound,
                         unsigned long long *__restrict__ out_idx, typename Coord<T>::dist_t *__restrict__ out_dist,
                         int32_t *__restrict__ replay_ranks, int32_t *__restrict__ replay_rows,
                         uint32_t *replay_count, uint32_t *status, unsigned long long *visit_count) {
    constexpr int W = fast_warps<KC>();
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5;
    const int first = (blockIdx.x * W + warp) * lanes;
    const int cnt  = lst.count ? (int)*lst.count : num;
    const int step = lst.count ? (int)gridDim.x * W * lanes : cnt; // without a list: one round
    for (int base = first; base < cnt; base += step)
        fast_warp<T, PER, KC>(base, lanes, lst, miss, smem, t_all, bt, qx, qy, qz, order, leaf_ids, cnt, k, half_window,
                              exclude_self, ret_orig, binary != 0, bound, out_idx, out_dist, replay_ranks,
                              replay_rows, replay_count, status, visit_count);
}

// Queries a warp takes.  A call whose full warps would leave most of the SMs' warp slots empty
// spreads its queries over more warps with fewer lanes each: a warp lasts as long as its slowest
// lane's chain and alternates between its lanes' steps, so fewer lanes end sooner.  Measured with
// 4 / 8 / 16 / 32 lanes (k = 8 and 16, float): 3K queries 108 / 115 / 113 / 116 us, 12K 118 / 122 /
// 120 / 124 us, 30K 344 / 269 / 261 / 257 us, so 12 warps per SM are kept.
static int fast_lanes(int num) {
    int lanes = 32;
    while (lanes > 4 && num / (lanes / 2) <= 148 * 12) lanes /= 2;
    return lanes;
}

template <class T, int PER, int KC>
static void launch_fast_t(const TreeDev<T> &tv, const BatchDev &bt, const FastLaunch &f, cudaStream_t st) {
    using D               = typename Coord<T>::dist_t;
    constexpr int threads = 32 * fast_warps<KC>();
    const size_t  smem    = fast_smem(f.k, threads);
    auto          fn      = fast_self_knn_kernel<T, PER, KC>;
    FT_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // a listed launch (num: the list's capacity) loops over its entries with a grid of a few
    // blocks per SM; otherwise one warp per 32 queries
    const int lanes  = fast_lanes(f.num);
    const int per    = fast_warps<KC>() * lanes;
    int       blocks = (f.num + per - 1) / per;
    if (f.lst.count) blocks = std::max(1, std::min(blocks, 148 * 8));
    fn<<<blocks, threads, smem, st>>>(lanes, f.lst, f.miss, tv, bt, (const T *)f.eq.x, (const T *)f.eq.y, (const T *)f.eq.z,
                                      f.eq.order, f.leaf_ids, f.num, f.k, f.half, f.excl ? 1 : 0, f.ret_orig ? 1 : 0,
                                      f.variant == 2 ? 1 : 0, (const D *)f.bound, (unsigned long long *)f.idx,
                                      (D *)f.dist, f.rr, f.rw, f.rc, f.status, f.visits);
    FT_CUDA(cudaGetLastError());
}

// Launches the fast walk over `tv` (one tree, or every set of a batch when bt.off is set).
template <class T>
void launch_fast_view(const ft_tree &tr, const BatchDev &bt, int met, const FastLaunch &f, cudaStream_t st) {
    const TreeDev<T> tv = tree_view<T>(tr);
    met_dispatch<T>(met, [&](auto M) {
        constexpr int PER = decltype(M)::value;
        // heap template: 32 (two-warp blocks) for k <= 32 unless one-warp blocks were chosen
        if (f.k <= 32 && f.kc != 64) launch_fast_t<T, PER, 32>(tv, bt, f, st);
        else launch_fast_t<T, PER, 64>(tv, bt, f, st);
    });
}

// SFC rank of external query points: the point's key (the tree's own encoding and box) and
// its lower bound among the sorted keys; -1 without usable keys.
template <class T, int SFC>
__global__ void __launch_bounds__(256)
    seed_rank_kernel(const T *__restrict__ qx, const T *__restrict__ qy, const T *__restrict__ qz, int nq,
                     const T *__restrict__ bbox, const unsigned long long *__restrict__ klo,
                     const unsigned long long *__restrict__ khi, int n, int32_t *out) {
    __shared__ uint8_t s_rot[48 * 8], s_sub[48 * 8];
    __shared__ T       s_par[6];
    for (int i = threadIdx.x; i < 48 * 8; i += blockDim.x) {
        s_rot[i] = c_rot[i];
        s_sub[i] = c_sub[i];
    }
    if constexpr (Coord<T>::is_float)
        if (threadIdx.x < 3)
            sfc_axis_params(bbox[2 * threadIdx.x], bbox[2 * threadIdx.x + 1], s_par[2 * threadIdx.x],
                            s_par[2 * threadIdx.x + 1]);
    __syncthreads();
    const bool wide = Coord<T>::key_words == 2;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
        unsigned long long hi, lo;
        encode_point<T, SFC>(qx[q], qy[q], qz[q], s_par, s_rot, s_sub, hi, lo);
        int a = 0, b = n; // first j with key[j] >= key
        while (a < b) {
            const int  m    = (a + b) >> 1;
            const bool less = wide ? (khi[m] < hi || (khi[m] == hi && klo[m] < lo)) : (klo[m] < lo);
            if (less) a = m + 1;
            else b = m;
        }
        out[q] = a;
    }
}

template <class T>
void seed_ranks(const ft_options &o, const TreeImpl &impl, const void *qx, const void *qy, const void *qz,
                       int nq, int n, int32_t *out, cudaStream_t st) {
    const int grid = std::max(1, std::min((nq + 255) / 256, 148 * 16));
    if (o.sfc_type == MORTON)
        seed_rank_kernel<T, MORTON><<<grid, 256, 0, st>>>((const T *)qx, (const T *)qy, (const T *)qz, nq,
                                                          (const T *)impl.bbox, (const unsigned long long *)impl.key_lo,
                                                          (const unsigned long long *)impl.key_hi, n, out);
    else
        seed_rank_kernel<T, PEANO_HILBERT><<<grid, 256, 0, st>>>(
            (const T *)qx, (const T *)qy, (const T *)qz, nq, (const T *)impl.bbox,
            (const unsigned long long *)impl.key_lo, (const unsigned long long *)impl.key_hi, n, out);
    FT_CUDA(cudaGetLastError());
}

// =========================================================================================
// Persistent batched launch: build every set and answer its self-kNN queries in one kernel.
//
// Phase 1 -- builds.  Blocks take sets by ticket in the order `order` (largest first, so the
// longest builds start first) and build each whole set (cta_build_set).  A finished set is
// published: after a fence, its id goes to the next slot of `ready` with a release store.
// Phase 2 -- queries.  Each warp takes 32 queries of the set at the cursor of `ready` (one
// atomic per chunk on the set's chunk counter); when that set has no chunk left the cursor
// moves on.  The warp runs the fast walk on its 32 queries, reading the set's
// tree through L2 (the records were written by another block of this launch, so the
// read-only path cannot be used for them); tied queries go to the replay list as in every
// other fast walk.
// A block waits only for a set whose build another running block has claimed (every build is
// claimed before any block queries), so the waits end; they are bounded all the same (30 s of
// global time), after which the block sets STATUS_SPIN_LIMIT and stops.
// =========================================================================================
// Block shape: blocks as large as the SM's room for them allows, because a block builds a
// whole set and the largest sets' builds (latency-bound climbs and searches) set the launch's
// tail: for float coordinates 4 warps a block, 7 blocks (28 warps) with k <= 32 heaps; other
// types take more registers a thread (the exact 64-bit distances), 8 warps a block, 2 blocks.
template <class T> constexpr int persist_warps() { return std::is_same<T, float>::value ? 4 : 8; }
template <class T, int KC> constexpr int persist_blocks_per_sm() {
    return std::is_same<T, float>::value ? (KC > 32 ? 3 : 7) : (KC > 32 ? 1 : 2);
}
static constexpr int kPersistItems = 4; // keys per thread of a sort tile

template <class T> struct PersistDev {
    const long long *off, *node_off, *rec_off;
    int              S;
    const T         *x, *y, *z;
    const uint32_t  *id;
    const int8_t    *ghost;
    T               *mnx, *mxx, *mny, *mxy, *mnz, *mxz;
    int32_t         *left, *right, *parent;
    uint32_t        *tid_out;
    int8_t          *ghost_out;
    int32_t         *orig;
    NodeRec<T>      *recs;
    QRec            *qrec;
    QPoint          *qpts;
    uint32_t        *qflag;
    int              periodic;
    uint8_t         *height;
    int32_t         *counters, *leaves;
    unsigned long long *klo, *khi, *tlo, *thi;
    uint32_t        *perm, *tperm;
    T               *bbox;
    uint8_t         *set_height;
    const int32_t   *order;
    int32_t         *ready, *chunk_next;
    uint32_t        *ctl;
    int              query;
};

FT_D unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
FT_D int ld_acquire_gpu(const int32_t *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
FT_D void st_release_gpu(int32_t *p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
FT_D int ld_relaxed_gpu_i(const int32_t *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
FT_D uint32_t ld_relaxed_gpu(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

template <class T, int PER, int KC, int SFC, int KIND>
__global__ void __launch_bounds__(32 * persist_warps<T>(), persist_blocks_per_sm<T, KC>())
    batch_persistent_kernel(PersistDev<T> a, TreeDev<T> t_all, BatchDev bt, int k, int half_window,
                            int exclude_self, int ret_orig, unsigned long long *out_idx,
                            typename Coord<T>::dist_t *out_dist, int32_t *replay_ranks, int32_t *replay_rows,
                            uint32_t *replay_count, uint32_t *status, unsigned long long *visit_count) {
    constexpr int NW = persist_warps<T>(), PT = 32 * NW;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_item;
    const int      tid = threadIdx.x;

    // ---- 1. builds ----
    for (;;) {
        if (tid == 0) s_item = (int)atomicAdd(&a.ctl[0], 1u);
        __syncthreads();
        const int i = s_item;
        __syncthreads();
        if (i >= a.S) break; // block-uniform
        const int       s = a.order[i];
        const long long o = a.off[s];
        const int       n = (int)(a.off[s + 1] - o);
        if (n > 0) {
            const long long no = a.node_off[s], ro = a.rec_off[s];
            CtaTreeOut<T>   out;
            out.mnx      = a.mnx + no;
            out.mxx      = a.mxx + no;
            out.mny      = a.mny + no;
            out.mxy      = a.mxy + no;
            out.mnz      = a.mnz + no;
            out.mxz      = a.mxz + no;
            out.left     = a.left + ro;
            out.right    = a.right + ro;
            out.parent   = a.parent + no;
            out.id       = a.tid_out + no;
            out.ghost    = a.ghost_out + no;
            out.orig     = a.orig + no;
            out.recs     = a.recs + ro;
            out.qrec     = a.qrec + ro;
            out.qpts     = a.qpts + o;
            out.qflag    = a.qflag + s;
            out.periodic = a.periodic;
            out.height   = a.height + ro;
            out.counters = a.counters + ro;
            out.leaves   = a.leaves + ro;
            cta_build_set<T, SFC, KIND, PT, kPersistItems>(
                n, a.x + o, a.y + o, a.z + o, a.id ? a.id + o : nullptr, a.ghost ? a.ghost + o : nullptr, a.klo + o,
                a.khi ? a.khi + o : nullptr, a.perm + o, a.tlo + o, a.thi ? a.thi + o : nullptr, a.tperm + o, out,
                a.bbox + 6 * (size_t)s, a.set_height + s, smem);
        } else if (tid == 0) {
            // an empty set: the box the atomic min / max build leaves (no point folded in)
            using O = typename Ord<T>::type;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                a.bbox[6 * (size_t)s + 2 * d]     = Ord<T>::value((O)~(O)0);
                a.bbox[6 * (size_t)s + 2 * d + 1] = Ord<T>::value((O)0);
            }
            a.set_height[s] = 0;
        }
        if (tid == 0) { // publish the set: its tree is complete
            __threadfence();
            const uint32_t p = atomicAdd(&a.ctl[1], 1u);
            st_release_gpu(&a.ready[p], s);
        }
    }
    if (!a.query) return;

    // ---- 2. queries: each warp takes 32 queries at a time ----
    // A warp acquires a set's publication before it first reads the set's tree; the warp
    // barrier after the broadcast orders the other lanes' reads after it.
    const int lane     = tid & 31;
    int       acquired = -1; // the last set this warp acquired (lane 0)
    for (;;) {
        int s = -1, j = 0;
        if (lane == 0) {
            const unsigned long long t0 = global_ns();
            for (;;) {
                const uint32_t c = ld_relaxed_gpu(&a.ctl[2]);
                if (c >= (uint32_t)a.S) break;
                int r = ld_relaxed_gpu_i(&a.ready[c]);
                if (r >= 0 && r != acquired) {
                    r        = ld_acquire_gpu(&a.ready[c]);
                    acquired = r;
                }
                if (r < 0) { // a build another block holds is still running
                    if (global_ns() - t0 > 30000000000ull) {
                        atomicOr(status, STATUS_SPIN_LIMIT);
                        break;
                    }
                    __nanosleep(256);
                    continue;
                }
                const int n   = (int)(a.off[r + 1] - a.off[r]);
                const int nch = (n + 31) >> 5;
                if (nch > 0) {
                    const int jj = (int)atomicAdd(reinterpret_cast<uint32_t *>(&a.chunk_next[r]), 1u);
                    if (jj < nch) {
                        s = r;
                        j = jj;
                        break;
                    }
                }
                atomicCAS(&a.ctl[2], c, c + 1u); // this set has no chunk left
            }
        }
        s = __shfl_sync(0xffffffffu, s, 0);
        j = __shfl_sync(0xffffffffu, j, 0);
        __syncwarp();
        if (s < 0) break; // warp-uniform
        const int qbase = (int)a.off[s] + j * 32;
        const int end   = (int)a.off[s + 1];
        fast_warp<T, PER, KC, NW, true>(qbase, 32, QueryList{}, MissList{}, smem, t_all, bt, nullptr, nullptr, nullptr,
                                        nullptr, nullptr, end, k, half_window, exclude_self, ret_orig, false, nullptr,
                                        out_idx, out_dist, replay_ranks, replay_rows, replay_count, status,
                                           visit_count);
    }
}

template <class T, int PER, int KC, int SFC, int KIND>
static void launch_persistent_t(Context &ctx, const PersistLaunch &p, const PersistDev<T> &a, const TreeDev<T> &tv,
                                const BatchDev &bt, cudaStream_t st) {
    using D               = typename Coord<T>::dist_t;
    constexpr int NW      = persist_warps<T>(), PT = 32 * NW;
    const size_t  heaps   = p.query ? fast_smem(p.k, PT) : 0;
    const size_t  sorting = cta_sort_smem<Coord<T>::key_words, PT, kPersistItems>();
    const size_t  smem    = std::max(heaps, sorting);
    auto          fn      = batch_persistent_kernel<T, PER, KC, SFC, KIND>;
    FT_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    FT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, PT, smem));
    const int blocks = std::max(1, per_sm) * ctx.num_sms;
    const int half   = p.k; // the seeding window of the fast walk's default
    fn<<<blocks, PT, smem, st>>>(a, tv, bt, p.k, half, p.excl ? 1 : 0, ctx.opts.return_orig_indices ? 1 : 0,
                                 (unsigned long long *)p.idx, (D *)p.dist, p.rr, p.rw, p.counters, ctx.status,
                                 (unsigned long long *)(p.counters + 2));
    FT_CUDA(cudaGetLastError());
}

template <class T, int SFC, int KIND>
static void persistent_sfc(Context &ctx, const PersistLaunch &p, cudaStream_t st) {
    PersistDev<T> a;
    a.off = p.off; a.node_off = p.node_off; a.rec_off = p.rec_off; a.S = p.S;
    a.x = (const T *)p.x; a.y = (const T *)p.y; a.z = (const T *)p.z; a.id = p.id; a.ghost = p.ghost;
    a.mnx = (T *)p.all.min_x; a.mxx = (T *)p.all.max_x; a.mny = (T *)p.all.min_y;
    a.mxy = (T *)p.all.max_y; a.mnz = (T *)p.all.min_z; a.mxz = (T *)p.all.max_z;
    a.left = p.all.left_child; a.right = p.all.right_child; a.parent = p.all.parent;
    a.tid_out = p.all.id; a.ghost_out = p.all.is_ghost; a.orig = p.all.orig_idx;
    a.recs = (NodeRec<T> *)p.scr->recs; a.height = p.scr->height;
    a.qrec = (QRec *)p.scr->qrec; a.qpts = (QPoint *)p.scr->qpts; a.qflag = p.scr->qflag;
    a.periodic = ctx.opts.periodic;
    a.counters = p.scr->counters; a.leaves = p.scr->leafcount;
    a.klo = (unsigned long long *)p.scr->key_lo; a.khi = (unsigned long long *)p.scr->key_hi;
    a.tlo = (unsigned long long *)p.scr->tmp_lo; a.thi = (unsigned long long *)p.scr->tmp_hi;
    a.perm = p.scr->perm; a.tperm = p.scr->tmp_perm;
    a.bbox = (T *)p.bbox; a.set_height = p.set_height;
    a.order = p.order; a.ready = p.ready; a.chunk_next = p.chunk_next; a.ctl = p.ctl;
    a.query = p.query ? 1 : 0;
    BatchDev bt;
    bt.off = p.off; bt.node_off = p.node_off; bt.rec_off = p.rec_off; bt.height = p.set_height; bt.S = p.S;
    const TreeDev<T> tv = tree_view<T>(p.all);
    if (!p.query) { // builds only: the smallest block shape's instance
        launch_persistent_t<T, 0, 32, SFC, KIND>(ctx, p, a, tv, bt, st);
        return;
    }
    met_dispatch<T>(metric_mode<T>(ctx.opts, p.all), [&](auto M) {
        constexpr int PER = decltype(M)::value;
        if (p.k <= 32) launch_persistent_t<T, PER, 32, SFC, KIND>(ctx, p, a, tv, bt, st);
        else launch_persistent_t<T, PER, 64, SFC, KIND>(ctx, p, a, tv, bt, st);
    });
}

// integer positions always take Peano-Hilbert keys; the delta follows build_bvh's
template <class T> void persistent_typed(Context &ctx, const PersistLaunch &p, cudaStream_t st) {
    constexpr int KIND = Coord<T>::key_words == 2 ? 2 : 1;
    if (ctx.opts.sfc_type == MORTON) {
        if constexpr (Coord<T>::is_float) persistent_sfc<T, MORTON, 0>(ctx, p, st);
        else fail(FT_ERR_INVALID_ARGUMENT, "Morton keys are defined for floating-point coordinates only");
    } else {
        persistent_sfc<T, PEANO_HILBERT, KIND>(ctx, p, st);
    }
}

#define FT_FAST_INSTANTIATE(T)                                                                                      \
    template void launch_fast_view<T>(const ft_tree &, const BatchDev &, int, const FastLaunch &, cudaStream_t);    \
    template void seed_ranks<T>(const ft_options &, const TreeImpl &, const void *, const void *, const void *, int, \
                                int, int32_t *, cudaStream_t);                                                       \
    template void persistent_typed<T>(Context &, const PersistLaunch &, cudaStream_t);

} // namespace ft
