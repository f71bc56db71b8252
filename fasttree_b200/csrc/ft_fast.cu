// ft_fast.cu -- fast self-kNN and knn_query with exact fallback (FT_METHOD_FAST, the default).
//
// A warp takes 32 consecutive queries (sorted leaves, or external points sorted by their
// SFC rank), so its lanes work on neighbouring parts of the tree (fast_warp, ft_walk.cuh).
//  1. Seeding: each lane fills its heap (a max-heap of k entries in shared memory) from the
//     leaves of its SFC window [r - h, r + h], so pruning is effective before the walk starts.
//  2. Walk: each lane walks its own query over 4-wide records whose boxes are held in 32-bit
//     units of the tree's frame (QRec, ft_qtree.cuh): the bound of a child costs a dozen 32-bit
//     operations in every coordinate type and never exceeds the exact distance, so a child
//     beyond the k-th distance is skipped safely.  Subtrees of at most 8 leaves are buckets:
//     their leaves' 32-bit positions are tested by the same bound, and only those within the
//     k-th distance get the exact distance and the heap.  Queries the frame does not serve (a box
//     without a frame, a point far outside it, a dense node within reach) walk the binary records
//     with exact distances instead; trees whose box distances are not monotone (kQFlagPlain) take
//     the reference traversal alone.
//  3. Exactness: the result set is the exact k nearest; only the order among equal distances
//     can differ from the reference (its visit order and heap history decide it).  A lane
//     flags its query when any tie could matter -- equal distances inside the top k, a
//     candidate at exactly the current k-th distance left out, an eviction that leaves an
//     equal maximum (subtrees whose bound is within the k-th distance are walked, so such
//     candidates are seen) -- or when an optional per-query bound cut off a possible
//     neighbour, or its stack would overflow.  Flagged queries are rerun by the reference
//     traversal (exact_replay_kernel, or knn_query's heap tier for external points).  On trees
//     of height 63 or more the reference's stack guard drops subtrees; a query whose
//     neighbourhood it could reach is replayed too (stack_guard_reaches).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <type_traits>

#include "ft_common.cuh"
#include "ft_fast.h"
#include "ft_internal.h"

namespace ft {

// Walk of the fast path: 0 = default, 2 the exact binary walk over the node records, 4 the
// 4-wide walk.  The numbers 1, 3 and 5 named walks that the 4-wide one replaced; they select
// it (every walk returns the same rows).
static int walk_variant(int v) { return v == 2 ? 2 : 4; }

// One launch of the walk over `tr` (every set of a batch when bt.off is set) for the
// context's coordinate type.
static void launch_fast(const ft_options &o, const ft_tree &tr, const BatchDev &bt, FastLaunch f, cudaStream_t st) {
    f.ret_orig = o.return_orig_indices != 0;
    switch (o.coord_type) {
    case F32: launch_fast_view<float>(tr, bt, metric_mode<float>(o, tr), f, st); break;
    case F64: launch_fast_view<double>(tr, bt, metric_mode<double>(o, tr), f, st); break;
    case U32: launch_fast_view<uint32_t>(tr, bt, metric_mode<uint32_t>(o, tr), f, st); break;
    case U64: launch_fast_view<unsigned long long>(tr, bt, metric_mode<unsigned long long>(o, tr), f, st); break;
    }
}

// Bound-miss list of the context (queries whose bound proved too small in the first launch).
static void ensure_miss(Context &ctx, size_t num) {
    if (num <= ctx.miss_cap && ctx.miss_ranks) return;
    if (ctx.miss_ranks) cudaFree(ctx.miss_ranks);
    if (ctx.miss_rows) cudaFree(ctx.miss_rows);
    ctx.miss_ranks = ctx.miss_rows = nullptr;
    ctx.miss_cap                   = 0;
    const size_t cap = num + num / 4 + 1024;
    FT_CUDA(cudaMalloc(&ctx.miss_ranks, cap * sizeof(int32_t)));
    FT_CUDA(cudaMalloc(&ctx.miss_rows, cap * sizeof(int32_t)));
    ctx.miss_cap = cap;
}

// The fast walk over num queries (self queries, or external points with eq), its replay, and
// with a per-query bound a second launch of the walk without the bound over the queries
// whose bound proved too small (the walk flags its own ties there, so only those reach the
// reference traversal).  Counters in the context's status words: [1] replayed, [2..3]
// visits, [4] bound misses, [6..7] visits of the second launch.
static void fast_walk_and_replay(Context &ctx, const ft_tree &tr, const int32_t *leaf_ids, size_t num, int k,
                                 bool excl, uint64_t *idx, void *dist, const void *bound, int half_window,
                                 int variant, cudaStream_t st, const ExtQueries &eq = {}, int kc = 0) {
    uint32_t           *rc     = ctx.status + 1;
    unsigned long long *visits = (unsigned long long *)(ctx.status + 2);
    uint32_t           *mc     = ctx.status + 4;
    FT_CUDA(cudaMemsetAsync(rc, 0, 7 * sizeof(uint32_t), st));
    FastLaunch f;
    f.eq       = eq;
    f.leaf_ids = leaf_ids;
    f.num      = (int)num;
    f.k        = k;
    f.half     = half_window;
    f.variant  = variant;
    f.kc       = kc;
    f.excl     = excl;
    f.bound    = bound;
    f.idx      = idx;
    f.dist     = dist;
    f.rr       = ctx.replay_ranks;
    f.rw       = ctx.replay_rows;
    f.rc       = rc;
    f.status   = ctx.status;
    f.visits   = visits;
    if (bound) {
        ensure_miss(ctx, num);
        f.miss = MissList{ctx.miss_ranks, ctx.miss_rows, mc};
    }
    launch_fast(ctx.opts, tr, {}, f, st);
    if (bound) {
        f.miss   = MissList{};
        f.lst    = QueryList{ctx.miss_ranks, ctx.miss_rows, mc};
        f.bound  = nullptr;
        f.visits = (unsigned long long *)(ctx.status + 6);
        launch_fast(ctx.opts, tr, {}, f, st);
    }
}

bool fast_self_knn(Context &ctx, const ft_tree &tr, const int32_t *leaf_ids, size_t num, int k, bool excl,
                   uint64_t *idx, void *dist, const void *bound, int half_window, int variant, cudaStream_t st,
                   int kc) {
    TreeImpl *impl = (TreeImpl *)tr.impl;
    if (k > 64 || tr.num_leaves < 2 || !impl || impl->height_root < 0) return false;
    if (!fast_walk_applies(ctx.opts, *impl)) return false;
    // the autotuner's choice for this shape; it was made on every leaf in SFC order, so a
    // subset (whose warps hold unrelated leaves) keeps the defaults
    if (half_window <= 0 && variant <= 0 && kc <= 0 && !leaf_ids) {
        auto it = ctx.tuned.find(tune_key(TUNE_SELF_KNN, k, tr.num_leaves));
        if (it != ctx.tuned.end()) {
            half_window = it->second.half;
            variant     = it->second.variant;
            kc          = it->second.kc;
        }
    }
    if (half_window <= 0) half_window = k;
    variant = walk_variant(variant);
    ensure_replay(ctx, num);
    fast_walk_and_replay(ctx, tr, leaf_ids, num, k, excl, idx, dist, bound, half_window, variant, st, {}, kc);
    replay_exact(ctx, tr, ctx.replay_ranks, ctx.replay_rows, ctx.status + 1, k, excl, idx, dist, st);
    return true;
}

// (seed rank, query index) pairs for the query sort.
__global__ void rank_pairs_kernel(const int32_t *__restrict__ seeds, int nq, unsigned long long *key, uint32_t *perm) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += gridDim.x * blockDim.x) {
        key[i]  = (unsigned long long)(uint32_t)seeds[i];
        perm[i] = (uint32_t)i;
    }
}

// Sort scratch for external queries (one key word, nq pairs); status words go to the context.
static void ensure_query_sort(Context &ctx, size_t nq) {
    TreeImpl &s = ctx.qsort;
    if (nq <= s.cap && s.key_lo) return;
    void *ptrs[] = {s.key_lo, s.tmp_lo, s.perm, s.tmp_perm, s.hist, s.lookback, s.tile_counter};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    s            = TreeImpl{};
    const size_t cap = nq + nq / 4 + 1024;
    auto alloc = [&](size_t bytes) {
        void       *p = nullptr;
        cudaError_t e = cudaMalloc(&p, bytes);
        if (e != cudaSuccess) {
            cudaGetLastError();
            fail(FT_ERR_OUT_OF_MEMORY, "cudaMalloc of the query sort scratch failed");
        }
        return p;
    };
    s.key_lo         = (uint64_t *)alloc(cap * 8);
    s.tmp_lo         = (uint64_t *)alloc(cap * 8);
    s.perm           = (uint32_t *)alloc(cap * 4);
    s.tmp_perm       = (uint32_t *)alloc(cap * 4);
    s.hist           = (uint32_t *)alloc((16 * 256 + 16) * 4);
    s.lookback_words = sort_lookback_words(cap);
    s.lookback       = (uint32_t *)alloc(s.lookback_words * 4);
    s.tile_counter   = (uint32_t *)alloc(16 * 4);
    s.cap            = cap;
}

void free_query_sort(Context &ctx) {
    TreeImpl &s      = ctx.qsort;
    void     *ptrs[] = {s.key_lo, s.tmp_lo, s.perm, s.tmp_perm, s.hist, s.lookback, s.tile_counter};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    s = TreeImpl{};
}

// SFC rank of each external query in ctx.seed_ranks (-1 without usable keys).
static bool compute_seed_ranks(Context &ctx, const ft_tree &tr, const void *qx, const void *qy, const void *qz,
                               size_t nq, cudaStream_t st) {
    TreeImpl *impl = (TreeImpl *)tr.impl;
    ensure_replay(ctx, nq);
    const int n = (int)tr.num_leaves;
    if (!(impl->own_keys && impl->key_lo)) {
        FT_CUDA(cudaMemsetAsync(ctx.seed_ranks, 0xFF, nq * sizeof(int32_t), st)); // -1: no seeding window
        return false;
    }
    switch (ctx.opts.coord_type) {
    case F32: seed_ranks<float>(ctx.opts, *impl, qx, qy, qz, (int)nq, n, ctx.seed_ranks, st); break;
    case F64: seed_ranks<double>(ctx.opts, *impl, qx, qy, qz, (int)nq, n, ctx.seed_ranks, st); break;
    case U32: seed_ranks<uint32_t>(ctx.opts, *impl, qx, qy, qz, (int)nq, n, ctx.seed_ranks, st); break;
    case U64: seed_ranks<unsigned long long>(ctx.opts, *impl, qx, qy, qz, (int)nq, n, ctx.seed_ranks, st); break;
    }
    return true;
}

void query_seed_ranks(Context &ctx, const ft_tree &tr, const void *qx, const void *qy, const void *qz, size_t nq,
                      cudaStream_t st) {
    compute_seed_ranks(ctx, tr, qx, qy, qz, nq, st);
}

// Query order by SFC rank (ctx.seed_ranks must hold the ranks): sorts (rank, index) pairs.
static const uint32_t *order_by_rank(Context &ctx, size_t nq, int n, cudaStream_t st) {
    ensure_query_sort(ctx, nq);
    TreeImpl &qs = ctx.qsort;
    qs.status    = ctx.status;
    rank_pairs_kernel<<<std::max(1, std::min((int)((nq + 255) / 256), 148 * 16)), 256, 0, st>>>(
        ctx.seed_ranks, (int)nq, (unsigned long long *)qs.key_lo, qs.perm);
    FT_CUDA(cudaGetLastError());
    int bytes = 1;
    while (bytes < 4 && ((unsigned long long)n >> (8 * bytes)) != 0) ++bytes;
    static const int digits[4] = {0, 1, 2, 3};
    sort_pairs_fixed(qs, nq, bytes, digits, st);
    return qs.perm;
}

const uint32_t *sfc_query_order(Context &ctx, const ft_tree &tr, const void *qx, const void *qy, const void *qz,
                                size_t nq, cudaStream_t st) {
    if (nq < 2 || tr.num_leaves < 2 || !tr.impl) return nullptr;
    if (!compute_seed_ranks(ctx, tr, qx, qy, qz, nq, st)) return nullptr;
    return order_by_rank(ctx, nq, (int)tr.num_leaves, st);
}

bool fast_knn(Context &ctx, const ft_tree &tr, const void *qx, const void *qy, const void *qz, size_t nq, int k,
              int max_k, uint64_t *idx, void *dist, int half_window, cudaStream_t st, const void *bound,
              int walk) {
    TreeImpl *impl = (TreeImpl *)tr.impl;
    if (k > 64 || tr.num_leaves < 2 || !impl || impl->height_root < 0) return false;
    if (!fast_walk_applies(ctx.opts, *impl)) return false;
    // SortedMergeHeap with k equal to its capacity keeps the first k leaves it meets, not the
    // nearest: only the reference traversal reproduces that
    int cap = 1;
    while (cap < max_k) cap <<= 1;
    if (k > 32 && max_k > 32 && k >= cap) return false;
    if (half_window <= 0) half_window = k;
    const int  n      = (int)tr.num_leaves;
    const bool ranked = compute_seed_ranks(ctx, tr, qx, qy, qz, nq, st);
    ExtQueries eq;
    eq.x = qx;
    eq.y = qy;
    eq.z = qz;
    if (ranked && nq > 1) eq.order = order_by_rank(ctx, nq, n, st); // walk the queries in SFC order
    const int variant = walk_variant(walk);
    fast_walk_and_replay(ctx, tr, ctx.seed_ranks, nq, k, false, idx, dist, bound, half_window, variant, st, eq);
    replay_external(ctx, tr, qx, qy, qz, ctx.replay_rows, ctx.status + 1, k, max_k, idx, dist, st);
    return true;
}

void batch_self_knn(Context &ctx, const ft_tree &all, const BatchDev &bt, size_t num, int k, bool excl, uint64_t *idx,
                    void *dist, bool fast, int half_window, int variant, int32_t *rr, int32_t *rw, uint32_t *counters,
                    cudaStream_t st, const void *bound, int32_t *mw, int kc) {
    if (num == 0 || k <= 0) return;
    if (!fast || k > 64) {
        batch_self_knn_exact(ctx, all, bt, num, k, excl, idx, dist, st);
        return;
    }
    if (half_window <= 0 && variant <= 0 && kc <= 0) { // the autotuner's choice for this shape
        auto it = ctx.tuned.find(tune_key(TUNE_BATCH, k, num));
        if (it != ctx.tuned.end()) {
            half_window = it->second.half;
            variant     = it->second.variant;
            kc          = it->second.kc;
        }
    }
    if (half_window <= 0) half_window = k;
    variant                        = walk_variant(variant);
    FT_CUDA(cudaMemsetAsync(counters, 0, 8 * sizeof(uint32_t), st));
    FastLaunch f;
    f.num     = (int)num;
    f.k       = k;
    f.half    = half_window;
    f.variant = variant;
    f.kc      = kc;
    f.excl    = excl;
    f.bound   = bound;
    f.idx     = idx;
    f.dist    = dist;
    f.rr      = rr;
    f.rw      = rw;
    f.rc      = counters;
    f.status  = ctx.status;
    f.visits  = (unsigned long long *)(counters + 2);
    // bound misses: leaf ranks follow from the rows inside a batch, so rows suffice
    if (bound) f.miss = MissList{nullptr, mw, counters + 4};
    launch_fast(ctx.opts, all, bt, f, st);
    if (bound) {
        f.miss   = MissList{};
        f.lst    = QueryList{nullptr, mw, counters + 4};
        f.bound  = nullptr;
        f.visits = (unsigned long long *)(counters + 6); // the rerun's visits apart
        launch_fast(ctx.opts, all, bt, f, st);
    }
    replay_exact(ctx, all, rr, rw, counters, k, excl, idx, dist, st, bt);
}

// The three lists lie in one allocation.
void ensure_replay(Context &ctx, size_t num) {
    if (num <= ctx.replay_cap && ctx.replay_ranks) return;
    if (ctx.replay_ranks) cudaFree(ctx.replay_ranks);
    ctx.replay_ranks = ctx.replay_rows = ctx.seed_ranks = nullptr;
    ctx.replay_cap                                       = 0;
    const size_t cap = (num + num / 4 + 1024 + 63) / 64 * 64;
    int32_t     *p   = nullptr;
    FT_CUDA(cudaMalloc(&p, 3 * cap * sizeof(int32_t)));
    ctx.replay_ranks = p;
    ctx.replay_rows  = p + cap;
    ctx.seed_ranks   = p + 2 * cap;
    ctx.replay_cap   = cap;
}

// =========================================================================================
// Self-kNN without any device allocation (ft_self_knn_noalloc).
//
// Some callers cannot let a library allocate device memory in the middle of their work: a
// simulation that hands the whole GPU to its own memory pool at start-up (a cudaMalloc then
// fails), or a time step that must not stall every stream (cudaMalloc / cudaFree
// synchronise the device).  This variant runs the fast self-kNN walk with its only scratch
// -- the list of queries handed to the exact replay and its counter -- in the fixed array
// below, instead of the context's growable buffers.
//
// * The array lives in every GPU that loads the library, for the life of the process:
//   kNoAllocMaxQueries (2^20) queries per call, 8 MiB + a small header.  Larger calls are
//   rejected with FT_ERR_INVALID_ARGUMENT.
// * Host code needs the array's device address: the first call on a device looks it up
//   with cudaGetSymbolAddress (with that device current) and keeps it; make that first call
//   before any stream capture.  The symbol itself is only a host-side stand-in, never a
//   device pointer.
// * All calls share the array.  Each call clears the counter it needs on its stream first;
//   calls whose work overlaps on the GPU (different streams, or threads racing on one
//   device) race on the array and must be serialised by the caller.
// =========================================================================================
static constexpr size_t kNoAllocMaxQueries = size_t(1) << 20;
static constexpr size_t kNoAllocHeader     = 64; // words: [0] replay count, [2..3] visit counter
static __device__ __align__(256) uint32_t g_noalloc_scratch[kNoAllocHeader + 2 * kNoAllocMaxQueries];

static constexpr int kNoAllocMaxDevices = 64;
static std::mutex    g_noalloc_mutex;
static uint32_t     *g_noalloc_addr[kNoAllocMaxDevices] = {};
static CUcontext     g_noalloc_owner[kNoAllocMaxDevices] = {}; // the context the address belongs to

// The current driver context, read through the runtime's driver entry point (the library
// links no driver library); null when it cannot be read.
static CUcontext current_context() {
    using GetCurrent = CUresult (*)(CUcontext *);
    static GetCurrent fn = [] {
        void                           *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<GetCurrent>(p);
    }();
    CUcontext c = nullptr;
    if (!fn || fn(&c) != CUDA_SUCCESS) return nullptr;
    return c;
}

// Device address of g_noalloc_scratch on `device` (device must be current).  Looked up on
// the first call on a device and again whenever the device's context has changed since (a
// cudaDeviceReset makes a new primary context, which holds its own copy of the array).
static uint32_t *noalloc_scratch(int device) {
    if (device < 0 || device >= kNoAllocMaxDevices) fail(FT_ERR_INVALID_ARGUMENT, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    const CUcontext cur = current_context();
    if (!g_noalloc_addr[device] || cur == nullptr || cur != g_noalloc_owner[device]) {
        void       *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || p == nullptr) {
            cudaGetLastError();
            fail(FT_ERR_CUDA, std::string("cudaGetSymbolAddress of the no-allocation scratch failed: ") +
                                  cudaGetErrorString(e));
        }
        g_noalloc_addr[device]  = static_cast<uint32_t *>(p);
        g_noalloc_owner[device] = cur;
    }
    return g_noalloc_addr[device];
}

size_t noalloc_max_queries() { return kNoAllocMaxQueries; }

// Returns false when the fast walk does not apply (k > 64); the
// caller then runs the reference traversal, which needs no scratch.
bool fast_self_knn_noalloc(Context &ctx, const ft_tree &tr, const int32_t *leaf_ids, size_t num, int k, bool excl,
                           uint64_t *idx, void *dist, cudaStream_t st) {
    if (num > kNoAllocMaxQueries)
        fail(FT_ERR_INVALID_ARGUMENT, "ft_self_knn_noalloc: more than 1048576 queries in one call (the fixed "
                                      "scratch holds 2^20); split the call");
    TreeImpl *impl = (TreeImpl *)tr.impl;
    if (k > 64 || tr.num_leaves < 2 || !impl || impl->height_root < 0) return false;
    if (!fast_walk_applies(ctx.opts, *impl)) return false;
    uint32_t           *s      = noalloc_scratch(ctx.device);
    uint32_t           *rc     = s;
    unsigned long long *visits = reinterpret_cast<unsigned long long *>(s + 2);
    int32_t            *ranks  = reinterpret_cast<int32_t *>(s + kNoAllocHeader);
    int32_t            *rows   = ranks + kNoAllocMaxQueries;
    FT_CUDA(cudaMemsetAsync(s, 0, 4 * sizeof(uint32_t), st)); // the replay count must start at zero
    FastLaunch f;
    f.leaf_ids = leaf_ids;
    f.num      = (int)num;
    f.k        = k;
    f.half     = k;
    f.excl     = excl;
    f.idx      = idx;
    f.dist     = dist;
    f.rr       = ranks;
    f.rw       = rows;
    f.rc       = rc;
    f.status   = ctx.status;
    f.visits   = visits;
    launch_fast(ctx.opts, tr, {}, f, st);
    replay_exact(ctx, tr, ranks, rows, rc, k, excl, idx, dist, st);
    // query statistics as ft_self_knn keeps them: the replay count and visits move into the
    // context's status words (a device-to-device copy on the stream; nothing is allocated)
    // (scratch words: [0] replay count, [2..3] visits; context words: [1] and [2..3])
    FT_CUDA(cudaMemcpyAsync(ctx.status + 1, rc, sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
    FT_CUDA(cudaMemcpyAsync(ctx.status + 2, visits, sizeof(unsigned long long), cudaMemcpyDeviceToDevice, st));
    FT_CUDA(cudaMemsetAsync(ctx.status + 4, 0, 4 * sizeof(uint32_t), st)); // no bound, no bound misses
    ctx.stats.queries  = (int64_t)num;
    ctx.stats.replayed = 0;
    ctx.last_fast      = true;
    ctx.last_rows      = false; // the replayed rows stay in the fixed array
    return true;
}

void batch_persistent(Context &ctx, const PersistLaunch &p, cudaStream_t st) {
    if (p.query && (p.k < 1 || p.k > 64)) fail(FT_ERR_INVALID_ARGUMENT, "the persistent batched launch serves k <= 64");
    switch (ctx.opts.coord_type) {
    case F32: persistent_typed<float>(ctx, p, st); break;
    case F64: persistent_typed<double>(ctx, p, st); break;
    case U32: persistent_typed<uint32_t>(ctx, p, st); break;
    case U64: persistent_typed<unsigned long long>(ctx, p, st); break;
    }
}

} // namespace ft
