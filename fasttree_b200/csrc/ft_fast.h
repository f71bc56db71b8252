// ft_fast.h -- one launch of the fast walk, as ft_fast.cu hands it to the coordinate types' units.
#pragma once

#include <cuda_runtime.h>

#include "ft_internal.h"

namespace ft {

// Queries handed from one launch of the walk to the next (bound misses): list entry i is
// output row rows[i] and, for self queries on one tree, leaf rank ranks[i]; *count entries.
struct QueryList {
    const int32_t  *ranks = nullptr;
    const int32_t  *rows  = nullptr;
    const uint32_t *count = nullptr; // null: no list, the launch covers queries [0, num)
};
// Where a launch sends the queries whose pruning bound proved too small (null rows: they
// join the replay list like the other flagged queries).
struct MissList {
    int32_t  *ranks = nullptr;
    int32_t  *rows  = nullptr;
    uint32_t *count = nullptr;
};
// External query points: qx / qy / qz (else self queries) with leaf_ids = their seed ranks.
struct ExtQueries {
    const void     *x = nullptr, *y = nullptr, *z = nullptr;
    const uint32_t *order = nullptr; // walk order (null: input order)
};
struct FastLaunch {
    QueryList       lst;
    MissList        miss;
    ExtQueries      eq;
    const int32_t  *leaf_ids = nullptr;
    int             num = 0, k = 0;
    int             half    = 0; // SFC seeding half-window
    int             variant = 4; // 4: the 4-wide walk, 2: the exact binary walk
    int             kc      = 0; // 64: one-warp blocks whatever k
    bool            excl = true, ret_orig = false;
    const void     *bound = nullptr;
    uint64_t       *idx   = nullptr;
    void           *dist  = nullptr;
    int32_t        *rr = nullptr, *rw = nullptr; // replay list and its count
    uint32_t       *rc     = nullptr;
    uint32_t       *status = nullptr;
    unsigned long long *visits = nullptr;
};

template <class T>
void launch_fast_view(const ft_tree &tr, const BatchDev &bt, int met, const FastLaunch &f, cudaStream_t st);
template <class T>
void seed_ranks(const ft_options &o, const TreeImpl &impl, const void *qx, const void *qy, const void *qz, int nq,
                int n, int32_t *out, cudaStream_t st);
template <class T> void persistent_typed(Context &ctx, const PersistLaunch &p, cudaStream_t st);

} // namespace ft
