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
