"""Builds at the edges of their blocks against the oracle, every tree array bit for bit: treelets
of 512 leaves (and climbs that leave them), the one-block front end (at most 8192 points), tiles
of the sort, runs of equal key halves and equal high key words (ordered in place when short,
by a sort over both words when long), duplicates, refits and caller keys."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import fasttree_b200 as ft  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests.gpu_util import CONFIG_IDS, CONFIGS, NAMES, assert_tree_equal, gen  # noqa: E402

PICK = [0, 3, 5, 7]
CFGS, IDS = [CONFIGS[i] for i in PICK], [CONFIG_IDS[i] for i in PICK]


def make(cfg):
    coord, sfc, per = cfg
    return (ft.Context(NAMES[coord], "morton" if sfc == O.MORTON else "ph", periodic=per),
            O.Options(coord, sfc, per))


def check(cfg, x, y, z):
    ctx, opts = make(cfg)
    tree = ft.TreeSoA(ctx, len(x))
    ft.build_bvh(ctx, ft.particles(x, y, z), tree)
    ot = O.build_bvh(opts, x, y, z)
    assert_tree_equal(tree.to_numpy(), ot, len(x))
    return ctx, opts, tree, ot


@pytest.mark.parametrize("cfg", CFGS, ids=IDS)
@pytest.mark.parametrize("n", [511, 512, 513, 1024, 1025, 2047, 8191, 8192, 8193, 20_481])
def test_block_edges(cfg, n):
    ctx, _, tree, ot = check(cfg, *gen("clustered", n, cfg[0], seed=n))
    a = ft.self_knn_query(ctx, tree, 9, method="plain")
    a = (a[0].clone(), a[1].clone())
    b = ft.self_knn_query(ctx, tree, 9)
    torch.cuda.synchronize()
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.parametrize("cfg", CFGS, ids=IDS)
@pytest.mark.parametrize("n", [700, 8000, 12_000])
@pytest.mark.parametrize("run", [5, 16, 17, 33, 400])
def test_runs_of_equal_keys(cfg, n, run):
    """`run` copies of each point: equal keys and equal halves of keys in runs of that length."""
    x, y, z = gen("uniform", n, cfg[0], seed=run)
    pick = np.random.default_rng(n).permutation(n) // run
    check(cfg, *[np.ascontiguousarray(a[pick]) for a in (x, y, z)])


@pytest.mark.parametrize("spread", [3, 40, 900])
def test_runs_of_equal_high_words(spread):
    """126-bit keys that differ in their low word only: points of one small cell, `spread` apart."""
    rng = np.random.default_rng(spread)
    n = 9000
    base = rng.integers(0, 1 << 41, (3, n // 45 + 1), dtype=np.uint64)
    p = base[:, np.arange(n) // 45] + rng.integers(0, spread, (3, n), dtype=np.uint64)
    p = p[:, rng.permutation(n)]
    for m in (n, 4000):
        check(CONFIGS[7], *[np.ascontiguousarray(a[:m]) for a in p])


def test_caller_keys_with_long_runs():
    """The caller's 126-bit keys come back sorted by both words, input order among equals."""
    rng = np.random.default_rng(1)
    n = 10_000
    ctx, opts = make(CONFIGS[7])
    x, y, z = gen("uniform", n, O.U64, seed=3)
    hi = rng.integers(0, 60, n, dtype=np.uint64) << np.uint64(40)
    lo = rng.integers(0, 50, n, dtype=np.uint64) << np.uint64(20)
    ref = np.zeros((n, 3), np.uint64)
    ref[:, 1], ref[:, 2] = hi, lo
    order = np.lexsort((np.arange(n), lo, hi))
    want = ref[order].copy()
    tree = ft.TreeSoA(ctx, n)
    ft.build_bvh(ctx, ft.particles(x, y, z), tree, key=ref)
    assert np.array_equal(ref, want)
    assert np.array_equal(tree.orig_idx[n - 1:].cpu().numpy(), order)


@pytest.mark.parametrize("cfg", CFGS, ids=IDS)
@pytest.mark.parametrize("n", [512, 700, 9001])
def test_refit_equals_build_tree_of_the_moved_points(cfg, n):
    """Moved positions in input and in leaf order give the same tree; back again, the built one."""
    ctx, opts, tree, ot = check(cfg, *gen("uniform", n, cfg[0], seed=n))
    moved = gen("clustered", n, cfg[0], seed=n + 1)
    ft.refit_bvh(ctx, ft.particles(*moved), tree)
    a = tree.to_numpy()
    order = a["orig_idx"][n - 1:]
    ft.refit_bvh(ctx, ft.particles(*[np.ascontiguousarray(m[order]) for m in moved]), tree, leaf_order=True)
    b = tree.to_numpy()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    for axis, m in zip("xyz", moved):
        assert a["min_" + axis][0] == m.min() and a["max_" + axis][0] == m.max()
        assert np.array_equal(a["min_" + axis][n - 1:], m[order])
    for k in ("left_child", "right_child"):
        assert np.array_equal(a[k], getattr(ot, k)[:n - 1])
    ft.refit_bvh(ctx, ft.particles(*gen("uniform", n, cfg[0], seed=n)), tree)
    assert_tree_equal(tree.to_numpy(), ot, n)


@pytest.mark.parametrize("n", [2, 9, 300, 1500, 9001])
@pytest.mark.parametrize("coord", ["f64", "u64"])
def test_build_tree_of_boxes_in_the_leaf_slots(coord, n):
    """build_tree without coordinate arrays takes what the leaf slots hold, boxes too: internal boxes
    cover them and queries measure the distance to them (src/hlbvh.hpp:941-969, 998-1055)."""
    rng = np.random.default_rng(n)
    ctx = ft.Context(coord, "morton" if coord == "f64" else "ph")
    dt = np.float64 if coord == "f64" else np.uint64
    scale = 1.0 if coord == "f64" else 2.0**40
    order = np.argsort(rng.random(n))
    base = np.sort(rng.random(n))  # along x, so that keys and places agree
    lo = [(base if a == 0 else rng.random(n)) * scale for a in range(3)]
    hi = [v + rng.random(n) * 0.01 * scale for v in lo]
    lo, hi = [v.astype(dt) for v in lo], [v.astype(dt) for v in hi]
    kv = (base * 2.0**60).astype(np.uint64)
    keys = kv if coord == "f64" else np.stack([np.zeros(n, np.uint64), kv, order.astype(np.uint64)], axis=1)
    tree = ft.TreeSoA(ctx, n)
    for a, v, w in zip("xyz", lo, hi):
        getattr(tree, "min_" + a)[n - 1:] = torch.from_numpy(v).cuda()
        getattr(tree, "max_" + a)[n - 1:] = torch.from_numpy(w).cuda()
    ft.build_tree(ctx, tree, keys)
    t = tree.to_numpy()
    for a, v, w in zip("xyz", lo, hi):
        assert np.array_equal(t["min_" + a][n - 1:], v) and np.array_equal(t["max_" + a][n - 1:], w)
        for v2, f, nm in ((v, np.minimum, "min_"), (w, np.maximum, "max_")):
            b = t[nm + a]
            assert np.array_equal(b[:n - 1], f(b[t["left_child"]], b[t["right_child"]])) and b[0] == f.reduce(v2)
    t2 = ft.import_tree(ctx, tree.export())
    for k, v in t2.to_numpy().items():
        assert k in ("id", "is_ghost", "orig_idx") or np.array_equal(v, t[k]), k
    # every query kind against distances to the boxes
    q = [(rng.random(200) * scale).astype(dt) for _ in range(3)]
    k = min(n, 6)

    def gap(p, v, w):
        if coord == "f64":
            return np.maximum(np.maximum(v - p, p - w), 0.0)
        return np.where(p < v, (v - p) >> np.uint64(11), np.where(p > w, (p - w) >> np.uint64(11), np.uint64(0)))

    g = [gap(p[:, None], v[None], w[None]) for p, v, w in zip(q, lo, hi)]
    d = g[0] * g[0] + g[1] * g[1] + g[2] * g[2]
    want = np.sort(d, axis=1)[:, :k]
    for method in ("plain", "fast"):
        _, gd = ft.knn_query(ctx, tree, *q, k, method=method)
        torch.cuda.synchronize()
        assert np.array_equal(gd.cpu().numpy(), want), method
    r = 0.2 * scale
    r2 = np.float64(r) * np.float64(r) if coord == "f64" else np.uint64(int(r) >> 11) ** 2
    cnt = torch.zeros(200, dtype=torch.int32, device="cuda")
    res = torch.zeros(200 * 4, dtype=torch.int32, device="cuda")
    one = np.ones(200)
    ft.range_query(ctx, tree, *q, (0 * one).astype(dt), (r * one).astype(dt), 4, res, cnt)
    torch.cuda.synchronize()
    assert np.array_equal(cnt.cpu().numpy(), (d <= r2).sum(axis=1))


def test_scratch_of_small_trees_from_a_shared_pool():
    """Small trees take their scratch from a pool of their context: it is handed on only when the
    queries of the tree before have ended, it outlives the context with its trees, and several
    threads may build at once."""
    import threading

    n = 3000
    sets = [[torch.from_numpy(a).cuda() for a in gen("uniform", n, O.F32, seed=s)] for s in range(8)]
    want = []
    for s in sets:
        c = ft.Context("f32", "morton")
        t = ft.TreeSoA(c, n)
        ft.build_bvh(c, ft.particles(*s), t)
        want.append([a.clone() for a in ft.self_knn_query(c, t, 16)])
    torch.cuda.synchronize()
    # a tree goes while its query runs on another stream; the next is built at once
    ctx, streams, got = ft.Context("f32", "morton"), [torch.cuda.Stream() for _ in range(2)], []
    for i, s in enumerate(sets * 3):
        st = streams[i % 2]
        t = ft.TreeSoA(ctx, n)
        ft.build_bvh(ctx, ft.particles(*s), t, stream=st)
        idx = torch.empty(n * 16, dtype=torch.uint64, device="cuda")
        dist = torch.empty(n * 16, dtype=torch.float64, device="cuda")
        ft.self_knn_query(ctx, t, 16, idx, dist, stream=st)
        t.free()
        got.append((idx, dist))
    torch.cuda.synchronize()
    for i, (idx, dist) in enumerate(got):
        assert torch.equal(idx, want[i % 8][0].reshape(-1)) and torch.equal(dist, want[i % 8][1].reshape(-1)), i
    # the context goes before its tree
    t = ft.TreeSoA(ctx, n)
    ft.build_bvh(ctx, ft.particles(*sets[0]), t)
    other = ft.Context("f32", "morton")
    t.ctx = other
    del ctx
    t2 = ft.TreeSoA(other, n)
    ft.build_bvh(other, ft.particles(*sets[1]), t2)
    for tree, w in ((t, want[0]), (t2, want[1])):
        r = ft.self_knn_query(other, tree, 16)
        torch.cuda.synchronize()
        assert torch.equal(r[0], w[0]) and torch.equal(r[1], w[1])
    t.free()
    # four threads build trees of one context
    trees = [[None] * 6 for _ in range(4)]

    def work(k):
        st = torch.cuda.Stream()
        for j in range(6):
            tr = ft.TreeSoA(other, n)
            ft.build_bvh(other, ft.particles(*sets[(k + j) % 8]), tr, stream=st)
            if j % 2:
                trees[k][j] = tr
            else:
                tr.free()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for k in range(4):
        for j in (1, 3, 5):
            r = ft.self_knn_query(other, trees[k][j], 16)
            torch.cuda.synchronize()
            w = want[(k + j) % 8]
            assert torch.equal(r[0], w[0]) and torch.equal(r[1], w[1])


def spine_keys(blocks, bits):
    """Sorted keys whose common prefixes fall from the edges of each block of 512 leaves towards its
    middle, about bits / 4 leaves deep on either side: each of those leaves' parents reaches beyond the
    block's edge."""
    low = bits - 6  # a slot of keys for each block
    c = int("01" * (low // 2 + 1), 2) & ((1 << low) - 1)
    below = sorted(((c >> j) ^ 1) << j for j in range(low) if c >> j & 1)
    above = sorted(((c >> j) | 1) << j for j in range(low) if not c >> j & 1)
    keys = []
    for b in range(blocks):
        lo, hi = b << low, (b + 1) << low
        left, right = [lo + a for a in above], [hi + v for v in below] + [hi + c]
        fill = 512 - len(left) - len(right)
        step = (right[0] - left[-1]) // (fill + 1)
        keys += left + [left[-1] + step * (i + 1) for i in range(fill)] + right
    return keys


def leaving(ot, n):
    """Subtrees of each block of 512 leaves whose parent reaches beyond it."""
    node = {}  # first and last leaf
    for v in np.argsort(-depths(ot, n)):
        if v >= n - 1:
            node[v] = (v - (n - 1), v - (n - 1))
        else:
            node[v] = (node[ot.left_child[v]][0], node[ot.right_child[v]][1])
    out = np.zeros((n + 511) // 512, np.int64)
    for v, (a, b) in node.items():
        if a // 512 != b // 512 or ot.parent[v] < 0:
            continue
        pa, pb = node[ot.parent[v]]
        out[a // 512] += pa // 512 != pb // 512
    return out


def depths(ot, n):
    d = np.zeros(2 * n - 1, np.int64)
    p = ot.parent[:2 * n - 1].astype(np.int64)
    while (p >= 0).any():
        d += p >= 0
        p = np.where(p >= 0, ot.parent[np.maximum(p, 0)], -1)
    return d


@pytest.mark.parametrize("coord", ["f32", "f64", "u64"])
@pytest.mark.parametrize("blocks", [16, 33])
def test_climbs_past_the_joins(coord, blocks):
    """More climbs leave 16 blocks than a join takes: they are passed on, past both levels of joins
    with 33 blocks, and end in global memory.  Every array and the rows of queries as the oracle's."""
    cfg = {"f32": (O.F32, O.MORTON, False), "f64": (O.F64, O.PEANO_HILBERT, False),
           "u64": (O.U64, O.PEANO_HILBERT, True)}[coord]
    ctx, opts = make(cfg)
    keys = spine_keys(blocks, 126 if coord == "u64" else 63)
    n = len(keys)
    hi = np.array([v >> 64 for v in keys], np.uint64)
    lo = np.array([v & (2**64 - 1) for v in keys], np.uint64)
    if cfg[1] == O.MORTON:
        ref = lo
    elif coord == "u64":
        ref = np.stack([np.zeros(n, np.uint64), hi, lo], axis=1)
    else:
        ref = np.stack([np.zeros(n, np.uint64), lo >> np.uint64(32), lo & np.uint64(2**32 - 1)], axis=1).astype(np.uint32)
    rng = np.random.default_rng(blocks)
    unit = 2.0**42 if coord == "u64" else 1.0
    xyz = [(p * unit).astype(O.NP_COORD[cfg[0]]) for p in
           ((np.arange(n) + rng.random(n)) / n, rng.random(n) * 0.05, rng.random(n) * 0.05)]
    orig = rng.permutation(n).astype(np.int32)
    ids = rng.integers(0, 1 << 32, n).astype(np.uint32)
    ghost = rng.integers(0, 2, n).astype(np.int8)
    ot = O.build_tree(opts, hi if coord == "u64" else None, lo, *xyz, ids, ghost, orig)
    out = leaving(ot, n)
    assert out[:16].sum() > 512 and (blocks == 16 or (out[16:32].sum() > 512 and out.sum() > 512))
    tree = ft.TreeSoA(ctx, n)
    for a in ("id", "is_ghost", "orig_idx"):  # (build_tree leaves their internal slots alone)
        getattr(tree, a).view(torch.int8).zero_()
    ft.build_tree(ctx, tree, ref, *xyz, ids, ghost, orig)
    assert_tree_equal(tree.to_numpy(), ot, n)
    oi, od = O.self_knn(opts, ot, 8, True)
    for method in ("plain", "fast"):
        gi, gd = ft.self_knn_query(ctx, tree, 8, method=method)
        torch.cuda.synchronize()
        assert np.array_equal(gi.cpu().numpy(), oi) and np.array_equal(gd.cpu().numpy(), od), method
    # the same tree from a refit whose leaves keep their places
    ft.refit_bvh(ctx, ft.particles(*xyz), tree, leaf_order=True)
    assert_tree_equal(tree.to_numpy(), ot, n)
