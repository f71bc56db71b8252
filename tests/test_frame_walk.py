"""The walks over the 32-bit records (knn, self-kNN, range) against the walks that use exact
distances throughout: the reference traversal for kNN, the binary walk for range queries.

The inputs sit where the frame's bounds or its rules could go wrong: fewer leaves than a
bucket or a node holds, coordinates on a coarse lattice (ties), planes and lines, boxes far
from the origin, spans at the frame's limits, tight clusters in a long box, the periodic wrap,
and query points on, beyond and far outside the box.  Rows and counts must be equal bit for
bit: both sides return the same neighbours by contract."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import fasttree_b200 as ft  # noqa: E402

NP = {"f32": np.float32, "f64": np.float64, "u32": np.uint32, "u64": np.uint64}
CFGS = [("f32", "morton", False), ("f64", "ph", False), ("u32", "ph", True), ("u32", "ph", False),
        ("u64", "ph", True), ("u64", "ph", False)]
IDS = [f"{c}-{s}{'-per' if p else ''}" for c, s, p in CFGS]


def box(coord):
    """Side of the usual box in coordinate units."""
    return {"f32": 1.0, "f64": 1.0, "u32": float(1 << 21), "u64": float(1 << 42)}[coord]


def points(kind, n, coord, seed):
    """(3, n) float64 in units of the usual box."""
    rng = np.random.default_rng(seed)
    p = rng.random((3, n))
    if kind == "lattice":
        p = np.floor(p * 8) / 8
    elif kind == "plane":
        p[2] = 0.25
    elif kind == "line":
        p[1:] = 0.5
    elif kind == "clusters":  # two tight clusters at opposite corners of a long box
        p = np.where(np.arange(n) % 2 == 0, 0.001 + 1e-5 * p, 0.999 - 1e-5 * p)
    elif kind == "edges":  # around the periodic wrap
        p = np.where(rng.random((3, n)) < 0.5, 1e-4 * p, 1.0 - 1e-4 * (1 - p))
    return p


def to_coord(p, coord):
    if coord[0] == "u":
        return [np.clip(np.floor(a * box(coord)), 0, box(coord) - 1).astype(NP[coord]) for a in p]
    return [a.astype(NP[coord]) for a in p]


def build(coord, sfc, per, xyz):
    ctx = ft.Context(coord, sfc, periodic=per)
    tree = ft.TreeSoA(ctx, len(xyz[0]))
    ft.build_bvh(ctx, ft.particles(*xyz), tree)
    return ctx, tree


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def same(a, b):
    torch.cuda.synchronize()
    return torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


def check_self(ctx, tree, ks):
    for k in ks:
        for excl in (True, False):
            a = ft.self_knn_query(ctx, tree, k, exclude_self=excl, max_k=64, method="plain")
            a = (a[0].clone(), a[1].clone())
            assert same(a, ft.self_knn_query(ctx, tree, k, exclude_self=excl, max_k=64)), (k, excl)


def check_points(ctx, tree, q, ks):
    for k in ks:
        a = ft.knn_query(ctx, tree, *q, k, max_k=256, method="plain")
        a = (a[0].clone(), a[1].clone())
        assert same(a, ft.knn_query(ctx, tree, *q, k, max_k=256)), k


def check_range(ctx, tree, q, r0, r1, rows):
    """The default walk, the one per query and the forced group counts against the binary walk."""
    n = len(q[0])
    lo, hi = (dev(np.full(n, r, NP[{0: "f32", 1: "f64", 2: "u32", 3: "u64"}[ctx.coord]])) for r in (r0, r1))
    want = None
    for walk in (1, 0, 3, 4):
        ctx.set_range_walk(walk)
        res = torch.full((n * max(rows, 1),), -1, dtype=torch.int32, device="cuda")
        cnt = torch.zeros(n, dtype=torch.int32, device="cuda")
        ft.range_query(ctx, tree, *q, lo, hi, rows, res, cnt)
        torch.cuda.synchronize()
        if want is None:
            want = (res, cnt)
        else:
            assert torch.equal(cnt, want[1]) and torch.equal(res, want[0]), (walk, r0, r1, rows)
    ctx.set_range_walk(0)


@pytest.mark.parametrize("coord,sfc,per", CFGS, ids=IDS)
def test_small_trees(coord, sfc, per):
    """Around one bucket, one node and two levels of nodes."""
    for n in (2, 3, 4, 7, 8, 9, 10, 16, 17, 31, 33, 65, 130):
        xyz = to_coord(points("uniform", n, coord, n), coord)
        ctx, tree = build(coord, sfc, per, xyz)
        check_self(ctx, tree, (1, 8, 20))
        q = [dev(a) for a in to_coord(points("uniform", 40, coord, 99), coord)]
        check_points(ctx, tree, q, (1, 9))
        for r in (0.0, 0.1 * box(coord), 2.0 * box(coord)):
            check_range(ctx, tree, q, 0, min(r, 2.0**31 if coord == "u32" else 2.0**60), 5)


@pytest.mark.parametrize("kind", ["uniform", "lattice", "plane", "line", "clusters", "edges"])
@pytest.mark.parametrize("coord,sfc,per", CFGS, ids=IDS)
def test_shapes_of_the_box(coord, sfc, per, kind):
    n = 6007
    xyz = to_coord(points(kind, n, coord, 5), coord)
    ctx, tree = build(coord, sfc, per, xyz)
    check_self(ctx, tree, (1, 16, 33))
    q = [dev(a) for a in to_coord(points("uniform", 700, coord, 6), coord)]
    near = [dev(a[::7]) for a in xyz]
    check_points(ctx, tree, q, (4, 40))
    check_points(ctx, tree, near, (4,))
    b = box(coord)
    for r0, r1, rows in ((0, 1e-3 * b, 16), (0, 0.06 * b, 8), (0.03 * b, 0.08 * b, 8), (0, 0.4 * b, 0)):
        check_range(ctx, tree, near, r0, r1, rows)
    check_range(ctx, tree, q, 0, 0.1 * b, 30)


@pytest.mark.parametrize("coord,span,lo", [("f64", 1e-10, 0.0), ("f64", 3e-9, 1.0), ("f64", 1e-3, 1e6), ("f64", 1e20, 0.0),
                                           ("f64", 1e26, -5e25), ("f64", 1e-28, 0.0),
                                           ("f64", 1e-31, 0.0), ("f64", 1e37, 0.0), ("f64", 1e40, 1e39),
                                           ("f32", 1e-28, 0.0), ("f32", 1e-32, 0.0), ("f32", 1e37, -5e36),
                                           ("f32", 1e-12, 0.0), ("f32", 1e-4, 0.0),
                                           ("f32", 4.0, 1000.0), ("f32", 1e18, 0.0), ("u64", 100.0, 5.0),
                                           ("u64", 2.0**13, 2.0**50), ("u64", 2.0**42, 0.0), ("u64", 2.0**45, 7.0),
                                           ("u32", 50.0, 3.0), ("u32", 2.0**31, 9.0)])
def test_spans_of_open_boxes(coord, span, lo):
    """Spans inside, at and beyond what the frame serves; integers over few and many cells."""
    rng = np.random.default_rng(8)
    xyz = [(lo + span * rng.random(5000)).astype(NP[coord]) for _ in range(3)]
    ctx, tree = build(coord, "ph", False, xyz)
    check_self(ctx, tree, (1, 24))
    out = [(lo + span * (a * 1.2 - 0.1)).clip(0 if coord[0] == "u" else None, None).astype(NP[coord])
           for a in rng.random((3, 500))]
    check_points(ctx, tree, [dev(a) for a in out], (3, 40))
    for r in (0.02 * span, 0.3 * span):
        check_range(ctx, tree, [dev(a) for a in out], 0, r, 12)


@pytest.mark.parametrize("coord", ["f32", "f64", "u32", "u64"])
def test_points_outside_the_box(coord):
    """Query points beyond the frame walk the binary records; the others of their warp do not."""
    rng = np.random.default_rng(3)
    side = 1000.0
    xyz = [(2000 + side * rng.random(4000)).astype(NP[coord]) for _ in range(3)]
    ctx, tree = build(coord, "ph", False, xyz)
    q = 2000 + side * rng.random((3, 640))
    far = rng.random(640)
    scale = np.select([far < 0.3, far < 0.4, far < 0.5, far < 0.6], [0.9, 1.1, 3.0, 1e5], 0.0)
    q = q + np.sign(rng.random((3, 640)) - 0.3) * scale * side
    q = [dev(a.clip(0 if coord[0] == "u" else None, None).astype(NP[coord])) for a in q]
    check_points(ctx, tree, q, (1, 8, 40))
    for r in (0.1 * side, 2.5 * side):
        check_range(ctx, tree, q, 0, r, 20)


def test_dense_parts_of_a_long_box():
    """A cluster the frame cannot resolve (a cell of it holds hundreds of leaves): the exact walk
    serves the tree, and rows stay equal."""
    rng = np.random.default_rng(4)
    p = rng.random((3, 3000)) * 1e-11 + 0.5
    p = np.concatenate([p, rng.random((3, 50))], axis=1)
    ctx, tree = build("f64", "morton", False, [a.copy() for a in p])
    check_self(ctx, tree, (8, 33))
    q = [dev(a[:400]) for a in p]
    check_points(ctx, tree, q, (8,))
    check_range(ctx, tree, q, 0, 3e-12, 10)


@pytest.mark.parametrize("n", [1, 3, 33, 300, 3000, 25_000, 60_000])
def test_query_counts_spread_over_warps(n):
    """Small calls give a warp fewer queries: every split returns the rows of the full walk."""
    xyz = to_coord(points("uniform", 70_000, "f32", 2), "f32")
    ctx, tree = build("f32", "morton", False, xyz)
    ids = torch.from_numpy(np.sort(np.random.default_rng(n).choice(70_000, n, replace=False)).astype(np.int32)).cuda()
    a = ft.self_knn_query_subset(ctx, tree, ids, 12, method="plain")
    a = (a[0].clone(), a[1].clone())
    assert same(a, ft.self_knn_query_subset(ctx, tree, ids, 12))


@pytest.mark.parametrize("coord", ["f32", "f64"])
def test_radii_that_are_not_numbers(coord):
    """A shell with a NaN on either side holds nothing; the other queries of the warp are not
    touched."""
    rng = np.random.default_rng(12)
    n = 6000
    xyz = [rng.random(n).astype(NP[coord]) for _ in range(3)]
    ctx, tree = build(coord, "ph", False, xyz)
    q = [dev(a[:640]) for a in xyz]
    lo = np.where(rng.random(640) < 0.3, 0.05, 0.0)
    hi = np.full(640, 0.3)
    lo[rng.random(640) < 0.2] = np.nan
    hi[rng.random(640) < 0.2] = np.nan
    bad = np.isnan(lo) | np.isnan(hi)
    lo, hi = dev(lo.astype(NP[coord])), dev(hi.astype(NP[coord]))
    for rows in (0, 1, 8):
        want = None
        for walk in (1, 0, 3, 4):
            ctx.set_range_walk(walk)
            res = torch.full((640 * max(rows, 1),), -1, dtype=torch.int32, device="cuda")
            cnt = torch.zeros(640, dtype=torch.int32, device="cuda")
            ft.range_query(ctx, tree, *q, lo, hi, rows, res, cnt)
            torch.cuda.synchronize()
            want = want or (res, cnt)
            assert (cnt.cpu().numpy()[bad] == 0).all(), (walk, rows)
            assert torch.equal(cnt, want[1]) and torch.equal(res, want[0]), (walk, rows)


@pytest.mark.parametrize("coord,powers", [("f64", (-40, -90, 40, 61)), ("f32", (-20, -40, 40, 58))], ids=["f64", "f32"])
def test_walks_do_not_depend_on_the_unit(coord, powers):
    """Points scaled by a power of two: the same rows, and after the same walk (visits counted) as long
    as squared distances are normal floats: whether positions are given in metres or in megaparsecs."""
    p = np.random.default_rng(6).random((3, 20_000))
    want = None
    for e in (0,) + powers:
        xyz = [(a.astype(NP[coord]) * NP[coord](2.0**e)) for a in p]
        ctx, tree = build(coord, "morton", False, xyz)
        i, d = ft.self_knn_query(ctx, tree, 16)
        torch.cuda.synchronize()
        got = (i.cpu().numpy(), d.cpu().numpy() * 2.0 ** (-2 * e), ctx.query_stats()["visits"])
        want = want or got
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), e
        assert got[2] == want[2] or got[1].min() * 2.0 ** (2 * e) < 2.0**-126, e


@pytest.mark.parametrize("size", [257, 3000])
@pytest.mark.parametrize("coord,sfc,per", [("f32", "ph", False), ("f64", "morton", False), ("u64", "ph", True),
                                           ("u64", "ph", False)], ids=["f32", "f64", "u64-per", "u64"])
def test_dense_nodes_among_others(coord, sfc, per, size):
    """A clump the frame does not resolve in a box of ordinary points: queries that reach it start
    again with exact distances, the others do not; single trees, batches of both build methods."""
    rng = np.random.default_rng(size)
    b = box(coord)
    p = rng.random((3, 5000 + size)) * b
    tight = {"f32": 1e-9, "f64": 1e-11, "u64": 6000.0}[coord]  # (float positions near 0 are that fine)
    p[:, :size] = (0.0 if coord == "f32" else 0.5 * b) + rng.random((3, size)) * tight
    xyz = [a.astype(NP[coord]) for a in (np.floor(p) if coord[0] == "u" else p)]
    ctx, tree = build(coord, sfc, per, xyz)
    check_self(ctx, tree, (1, 8, 33))
    q = p[:, rng.permutation(p.shape[1])[:600]] + rng.normal(0, 1e-4 * b, (3, 600)) * (rng.random(600) < 0.5)
    q = [dev(a.clip(0, b * (1 - 1e-6)).astype(NP[coord])) for a in q]
    check_points(ctx, tree, q, (8, 40))
    for r0, r1, rows in ((0, 0.3 * tight, 10), (0, 2e-4 * b, 100), (0.01 * b, 0.1 * b, 8), (0, 0.05 * b, 0)):
        check_range(ctx, tree, q, r0, r1, rows)
    if coord == "u64" and not per:
        return
    other = [np.concatenate([a[:40], a, a[size:]]) for a in xyz]
    off = np.array([0, 40, 40 + len(xyz[0]), len(other[0])])
    bt = ft.BatchedSets(ctx, len(other[0]), 3)
    for method in ("default", "persistent"):
        bt.set_build_method(method)
        bt.build(off, *other)
        want = bt.self_knn(16, method="plain")
        want = (want[0].clone(), want[1].clone())
        assert same(want, bt.self_knn(16)), method


@pytest.mark.parametrize("coord,per", [("f32", False), ("f64", False), ("u32", True), ("u32", False), ("u64", True),
                                       ("u64", False)], ids=["f32", "f64", "u32-per", "u32", "u64-per", "u64"])
def test_shells_that_pass_through_leaves(coord, per):
    """Points on a lattice and radii at, one step below and one step above its distances: the bounds
    that decide most leaves must leave those at the shell's edges to the exact distance."""
    rng = np.random.default_rng(3)
    n, step = 8000, {"f32": 1 / 16, "f64": 1 / 16, "u32": 1 << 16, "u64": 1 << 37}[coord]
    xyz = [(rng.integers(0, 16, n) * step).astype(NP[coord]) for _ in range(3)]
    ctx, tree = build(coord, "ph", per, xyz)
    q = [dev(a[:500]) for a in xyz]
    for m in (1, 2, 5):
        r = NP[coord](m * step)
        unit = NP[coord]({"u32": 1, "u64": 1 << 11}.get(coord, 0))
        below, above = (r - unit, r + unit) if coord[0] == "u" else (np.nextafter(r, NP[coord](0)),
                                                                     np.nextafter(r, NP[coord](9)))
        for r0, r1 in ((0, r), (0, below), (0, above), (r, r), (below, r), (above, r + r), (below, above)):
            check_range(ctx, tree, q, r0, r1, 0)
            check_range(ctx, tree, q, r0, r1, 40)


@pytest.mark.parametrize("coord,bits", [("u64", 42), ("u32", 31)], ids=["u64", "u32"])
def test_query_points_whose_squared_gaps_wrap(coord, bits):
    """External points so far off that the squares of their gaps leave 64 bits: such distances wrap,
    and rows are the reference traversal's."""
    rng = np.random.default_rng(1)
    xyz = [(rng.random(6000) * 2.0**bits).astype(NP[coord]) for _ in range(3)]
    ctx, tree = build(coord, "ph", False, xyz)
    top = 2.0 ** (32 - bits) if coord == "u32" else 1e5
    for lo, hi in ((1.0, 1.3), (1.0, 1.9), (0.5, 3.0), (3.0, 30.0), (1e3, 1e5)):
        q = [(lo + (min(hi, top * 0.999) - lo) * rng.random(500)) * 2.0**bits for _ in range(3)]
        if lo < top:
            q = [dev(a.astype(NP[coord])) for a in q]
            check_points(ctx, tree, q, (1, 8, 40))
            for r in (0.1, 0.9):
                check_range(ctx, tree, q, 0, r * 2.0**bits, 20)


@pytest.mark.parametrize("coord", ["f32", "f64"])
@pytest.mark.parametrize("n", [40, 3000, 9000])
def test_coordinates_that_are_not_finite(coord, n):
    """NaN and infinite coordinates in a build, a refit, one set of a batch and query points: the
    default method's rows are the reference traversal's."""
    rng = np.random.default_rng(n)
    ok = [rng.random(n).astype(NP[coord]) for _ in range(3)]
    bad = [a.copy() for a in ok]
    bad[0][3], bad[1][n // 2], bad[2][n - 2] = np.nan, np.inf, -np.inf
    ctx, tree = build(coord, "morton", False, bad)
    check_self(ctx, tree, (1, 8, 33))
    q = [dev(a[:40]) for a in ok]
    check_points(ctx, tree, q, (4, 40))
    ft.refit_bvh(ctx, ft.particles(*ok), tree)
    check_self(ctx, tree, (8,))
    ft.refit_bvh(ctx, ft.particles(*bad), tree)
    check_self(ctx, tree, (8,))
    ctx, tree = build(coord, "morton", False, ok)
    odd = rng.random((3, 64)).astype(NP[coord])
    odd[0, ::7], odd[1, ::11], odd[2, ::13] = np.nan, np.inf, -np.inf
    check_points(ctx, tree, [dev(a) for a in odd], (1, 9, 40))
    off = np.array([0, n, 2 * n, 2 * n + 1, 3 * n + 1])
    one = np.full(1, np.nan, NP[coord])
    xyz = [np.concatenate([a, b, one, a]) for a, b in zip(ok, bad)]
    b = ft.BatchedSets(ctx, len(xyz[0]), 4)
    for method in ("default", "persistent"):
        b.set_build_method(method)
        b.build(off, *xyz)
        want = b.self_knn(8, method="plain")
        want = (want[0].clone(), want[1].clone())
        got = b.self_knn(8)
        assert same(want, got), method


@pytest.mark.parametrize("k", [4, 8, 40])
@pytest.mark.parametrize("shift", [0, 1, 2, 4])
def test_rows_that_start_off_a_sector(k, shift):
    """Output arrays 8, 16 and 32 bytes into an allocation: the same rows as aligned ones."""
    xyz = to_coord(points("uniform", 5000, "u64", 3), "u64")
    ctx, tree = build("u64", "ph", True, xyz)
    want = ft.self_knn_query(ctx, tree, k, max_k=64, method="plain")
    idx = torch.zeros(5000 * k + 8, dtype=want[0].dtype, device="cuda")
    dist = torch.zeros(5000 * k + 8, dtype=want[1].dtype, device="cuda")
    for a, b in ((shift, shift), (0, shift), (shift, 0)):
        i, d = idx[a:a + 5000 * k], dist[b:b + 5000 * k]
        ft.self_knn_query(ctx, tree, k, i, d, max_k=64)
        assert same((want[0].reshape(-1), want[1].reshape(-1)), (i, d)), (a, b)
