"""Measured cases: the build, refit and neighbour queries of fasttree_b200 over the sizes its
users run, from a few thousand points to ten million.

A case is one call a simulation step makes on arrays that are already on the GPU.  The point
sets are those of the repository's benchmark, made on the GPU: "uniform" in the unit box, or
"clustered" (70% in Plummer spheres with power-law member counts, 30% uniform).  "fixed"
positions are 2^40 cells per side in uint64 (2^20 in uint32).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fasttree_b200 as ft

DEV = "cuda"
TORCH = {"f32": torch.float32, "f64": torch.float64, "u32": torch.uint32, "u64": torch.uint64}
SIZE = {"f32": 4, "f64": 8, "u32": 4, "u64": 8}
FIXED_BITS = {"u32": 20, "u64": 40}


def listed():
    return [
        # One halo or one small box rebuilt on its own: launches and latency decide.
        dict(name="build_4k_f32", op="build", coord="f32", sfc="ph", periodic=False, dist="uniform", n=4099),
        # The repository's small configuration: 100K float64 points, Morton keys.
        dict(name="build_100k_f64", op="build", coord="f64", sfc="morton", periodic=False, dist="uniform", n=100_000),
        # The production shape: 10M clustered fixed-point positions in a periodic box, rebuilt each step.
        dict(name="build_10m_u64", op="build", coord="u64", sfc="ph", periodic=True, dist="clustered",
             n=10_000_000),
        # The same points moved a little: the tree kept, its boxes and records refreshed.
        dict(name="refit_3m_f64", op="refit", coord="f64", sfc="ph", periodic=False, dist="clustered", n=3_000_001),
        # Neighbours of a small open box in single precision: latency of one query call.
        dict(name="self_3k_f32_k8", op="self", coord="f32", sfc="morton", periodic=False, dist="uniform", n=3001, k=8),
        # The small configuration's query.
        dict(name="self_100k_f64_k16", op="self", coord="f64", sfc="morton", periodic=False, dist="uniform",
             n=100_000, k=16),
        # Every particle's 32 neighbours (a density estimate), the headline workload.
        dict(name="self_10m_u64_k32", op="self", coord="u64", sfc="ph", periodic=True, dist="clustered",
             n=10_000_000, k=32),
        # The active tenth of a time-step hierarchy, many neighbours each.
        dict(name="subset_200k_u64_k64", op="subset", coord="u64", sfc="ph", periodic=True, dist="clustered",
             n=2_000_003, q=200_000, k=64),
        # Points that are not in the tree (grid samples and jittered particles), the merge-heap tier.
        dict(name="ext_1m_f64_k64", op="ext", coord="f64", sfc="morton", periodic=False, dist="uniform", n=100_000,
             q=1_000_000, k=64, max_k=256),
        # Fixed radius of 2e-3 of a clustered box: rows overflow in the dense spheres, full counts come back.
        dict(name="range_1m_u64", op="range", coord="u64", sfc="ph", periodic=True, dist="clustered", n=1_000_000,
             q=1_000_000, r=2e-3, rows=256),
        # Fixed radius holding about 50 neighbours, as a smoothing kernel's support; rows never overflow.
        dict(name="range_500k_f32", op="range", coord="f32", sfc="ph", periodic=False, dist="uniform", n=500_009,
             q=500_009, r=2.88e-2, rows=192),
        # Many independent halos of uneven size, built and queried together as one graph.
        dict(name="batch_512_f32_k32", op="batch", coord="f32", sfc="morton", periodic=False, sets=512, median=8000.0,
             k=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["build", "build", "refit", "self", "self", "self", "subset", "ext", "range", "batch"])
    coord = rng.choice(["f32", "f64", "u32", "u64", "u64"])
    integer = coord[0] == "u"
    c = dict(op=op, coord=coord, sfc="ph" if integer else rng.choice(["morton", "ph"]),
             periodic=integer and rng.random() < 0.7, dist=rng.choice(["uniform", "clustered"]))
    k = rng.choice([1, 2, 5, 8, 16, 20, 32, 32, 48, 64])
    if op in ("build", "refit"):
        c["n"] = _log(rng, 2_000, 8_000_000)
    elif op == "self":
        c.update(n=_log(rng, 2_000, min(8_000_000, 160_000_000 // k)), k=k)
    elif op == "subset":
        n = _log(rng, 20_000, 3_000_000)
        c.update(n=n, q=max(1, int(n * rng.uniform(0.02, 0.2))), k=k)
    elif op == "ext":
        c.update(n=_log(rng, 5_000, 2_000_000), q=_log(rng, 2_000, 800_000), k=k, max_k=rng.choice([64, 256]))
        c["max_k"] = max(c["max_k"], 2 * k)
    elif op == "range":
        n = _log(rng, 5_000, 800_000)
        # a radius that holds 10 to 100 points of a uniform box
        c.update(n=n, q=n, r=(rng.uniform(10, 100) * 3 / (4 * math.pi * n)) ** (1 / 3), rows=rng.choice([64, 128, 256]))
    else:
        if coord in ("u32", "u64"):
            c.update(coord="f32", sfc="morton", periodic=False)
        c.update(sets=_log(rng, 16, 400), median=float(_log(rng, 1_000, 8_000)), k=min(k, 32))
        c.pop("dist")
    return c


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _plummer(g, scale):
    u = _rand(g, scale.numel()).clamp(1e-12, 1 - 1e-12)
    r = scale / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    ct = 2.0 * _rand(g, scale.numel()) - 1.0
    st = torch.sqrt((1.0 - ct * ct).clamp_min(0.0))
    ph = 2.0 * math.pi * _rand(g, scale.numel())
    return torch.stack([r * st * torch.cos(ph), r * st * torch.sin(ph), r * ct])


def _unit(g, n, dist):
    """(3, n) float64 positions in [0, 1)."""
    if dist == "uniform":
        return _rand(g, 3, n)
    n_cl = int(0.7 * n)
    spheres = max(10, n // 500)
    centre = _rand(g, 3, spheres)
    scale = 10.0 ** (-4.0 + 2.0 * _rand(g, spheres))
    weight = _rand(g, spheres).clamp_min(1e-12) ** (-1.0 / 0.9)
    edge = torch.cumsum(weight, 0)
    which = torch.searchsorted(edge, _rand(g, n_cl) * edge[-1]).clamp_max(spheres - 1)
    p = torch.cat([centre[:, which] + _plummer(g, scale[which]), _rand(g, 3, n - n_cl)], dim=1)
    p = p - torch.floor(p)
    p = torch.where(p >= 1.0, torch.zeros_like(p), p)
    return p[:, torch.randperm(n, generator=g, device=DEV)]


def _coords(p, coord):
    """Unit-box positions as three contiguous arrays of the coordinate type."""
    if coord in FIXED_BITS:
        cells = float(1 << FIXED_BITS[coord])
        v = torch.floor(p * cells).clamp(0.0, cells - 1.0).to(torch.int64)
        v = v.view(torch.uint64) if coord == "u64" else v.to(torch.int32).view(torch.uint32)
    else:
        v = p.to(TORCH[coord])
        if coord == "f32":
            v = v.clamp_max(1.0 - 2.0 ** -24)
    return [a.clone() for a in v]


def _set_sizes(case):
    """Log-normal set sizes: the case's own, the same for every seed."""
    rng = np.random.default_rng(4)
    s = np.exp(math.log(case["median"]) + 1.2 * rng.standard_normal(case["sets"]))
    return np.clip(np.round(s), 256, 500_000).astype(np.int64)


def _set_points(case, seed):
    total = int(_set_sizes(case).sum())
    g = _gen(seed)
    p = 0.5 + _plummer(g, torch.full((total,), 0.05, device=DEV, dtype=torch.float64))
    out = ((p < 0.0) | (p >= 1.0)).any(0)  # the few far members spread over the box
    p = torch.where(out, _rand(g, 3, total), p)
    return _coords(p, case["coord"])


def _points(case, seed):
    g = _gen(seed)
    return _unit(g, case["n"], case["dist"]), g


def _queries(case, p, g):
    """Half uniform points, half particles jittered by a little."""
    q = case["q"]
    pick = torch.randint(case["n"], (q - q // 2,), generator=g, device=DEV)
    j = p[:, pick] + 1e-4 * torch.randn(3, q - q // 2, generator=g, device=DEV, dtype=torch.float64)
    return _coords(torch.cat([_rand(g, 3, q // 2), j.clamp(0.0, 1.0 - 1e-9)], dim=1), case["coord"])


def _out(rows, k, coord):
    """Neighbour buffers as a torch program holds them (64-bit indices, distances)."""
    d = torch.int64 if coord[0] == "u" else torch.float64
    return torch.zeros(rows * k, dtype=torch.int64, device=DEV), torch.zeros(rows * k, dtype=d, device=DEV)


_SIGNED = {torch.uint64: torch.int64, torch.uint32: torch.int32}
_ARRAYS = ("min_x", "max_x", "min_y", "max_y", "min_z", "max_z", "left_child", "right_child", "parent", "id",
           "is_ghost", "orig_idx")


def _tree_arrays(tree):
    """The tree's arrays without a copy; each keeps the tree, which owns the memory, alive."""
    out = {}
    for name in _ARRAYS:
        a = tree.array(name)
        out[name] = a.view(_SIGNED[a.dtype]) if a.dtype in _SIGNED else a
        out[name].owner = tree
    return out


def prepare(case, seed):
    ctx = ft.Context(case["coord"], case["sfc"], periodic=case["periodic"])
    s = dict(case=case, ctx=ctx)
    op, coord = case["op"], case["coord"]
    if op == "batch":
        sizes = _set_sizes(case)
        off = np.zeros(len(sizes) + 1, np.int64)
        off[1:] = np.cumsum(sizes)
        s["pos"] = _set_points(case, seed)
        s["off"] = torch.from_numpy(off).to(DEV)
        s["sets"] = ft.BatchedSets(ctx, int(off[-1]), len(sizes))
        s["out"] = _out(int(off[-1]), case["k"], coord)
        return s
    p, g = _points(case, seed)
    n = case["n"]
    s["pos"] = ft.particles(*_coords(p, coord))
    s["tree"] = ft.TreeSoA(ctx, n)
    if op == "build":
        s["arrays"] = _tree_arrays(s["tree"])
        return s
    ft.build_bvh(ctx, s["pos"], s["tree"])
    if op == "refit":
        step = 1e-6 * torch.randn(3, n, generator=g, device=DEV, dtype=torch.float64)
        s["moved"] = ft.particles(*_coords((p + step).clamp(0.0, 1.0 - 1e-9), coord))
        s["arrays"] = _tree_arrays(s["tree"])
    elif op == "self":
        s["out"] = _out(n, case["k"], coord)
    elif op == "subset":
        ids = torch.randperm(n, generator=g, device=DEV)[:case["q"]]
        s["ids"] = torch.sort(ids).values.to(torch.int32)
        s["out"] = _out(case["q"], case["k"], coord)
    elif op == "ext":
        s["q"] = _queries(case, p, g)
        s["out"] = _out(case["q"], case["k"], coord)
    elif op == "range":
        s["q"] = _coords(p, coord)
        r = torch.full((1,), case["r"], dtype=torch.float64, device=DEV)
        if coord in FIXED_BITS:
            r = torch.floor(r * float(1 << FIXED_BITS[coord])).to(torch.int64)
            r = r.view(torch.uint64) if coord == "u64" else r.to(torch.int32).view(torch.uint32)
            zero = torch.zeros(n, dtype=torch.int64, device=DEV)
            zero = zero.view(torch.uint64) if coord == "u64" else zero.to(torch.int32).view(torch.uint32)
            signed = _SIGNED[r.dtype]
            s["r"] = (zero, r.view(signed).expand(n).contiguous().view(r.dtype))
        else:
            s["r"] = (torch.zeros(n, dtype=TORCH[coord], device=DEV), r.to(TORCH[coord]).expand(n).contiguous())
        s["out"] = (torch.full((n * case["rows"],), -1, dtype=torch.int32, device=DEV),
                    torch.zeros(n, dtype=torch.int32, device=DEV))
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    op = case["op"]
    if op == "batch":
        return s["sets"].build_knn(s["off"], *s["pos"], case["k"], *s["out"])
    if op == "build":
        ft.build_bvh(ctx, s["pos"], s["tree"])
        return s["arrays"]
    if op == "refit":
        ft.refit_bvh(ctx, s["moved"], s["tree"])
        return s["arrays"]
    if op == "self":
        return ft.self_knn_query(ctx, s["tree"], case["k"], *s["out"], max_k=64)
    if op == "subset":
        return ft.self_knn_query_subset(ctx, s["tree"], s["ids"], case["k"], *s["out"])
    if op == "ext":
        return ft.knn_query(ctx, s["tree"], *s["q"], case["k"], *s["out"], max_k=case["max_k"])
    return ft.range_query(ctx, s["tree"], *s["q"], *s["r"], case["rows"], *s["out"])


# ---------------------------------------------------------------------------------------------
# Work: the inputs read once and the outputs written once, and for a query the distances of the
# neighbours it returns (8 operations each).
# ---------------------------------------------------------------------------------------------
def _tree_bytes(n, c):
    return (2 * n - 1) * (6 * c + 13) + (n - 1) * 8


def work(case):
    c, op = SIZE[case["coord"]], case["op"]
    if op == "batch":
        n, k = int(_set_sizes(case).sum()), case["k"]
        return dict(bytes=n * (3 * c + 16 * k) + 8 * case["sets"], flops=8 * n * k)
    n = case["n"]
    if op == "build":
        return dict(bytes=3 * c * n + _tree_bytes(n, c), flops=0)
    if op == "refit":
        return dict(bytes=3 * c * n + (2 * n - 1) * 6 * c + (n - 1) * 8 + 4 * n, flops=0)
    tree = n * 3 * c  # the leaves' positions: every method has to read them
    if op == "range":
        per_row = min(case["rows"], 4 / 3 * math.pi * case["r"] ** 3 * n)
        return dict(bytes=tree + case["q"] * (5 * c + 4 + 4 * per_row), flops=8 * case["q"] * per_row)
    q, k = case.get("q", n), case["k"]
    read = {"self": 0, "subset": 4, "ext": 3 * c}[op]
    return dict(bytes=tree + q * (read + 16 * k), flops=8 * q * k)


# ---------------------------------------------------------------------------------------------
# The distances by brute force in 64 bits.  Rows of a self query are in the order of the tree's
# leaves, which for Morton keys is a stable sort by the interleaved cells.
# ---------------------------------------------------------------------------------------------
def _cells(a):
    lo = a.min()
    span = a.max() - lo
    top = 1.0 - 2.0 ** (-24 if a.dtype == torch.float32 else -53)
    one = 1.0 + ((a - lo) * (1.0 / span)).clamp(0.0, top)
    if a.dtype == torch.float32:
        return ((one.view(torch.int32) & 0x7FFFFF) >> 2).to(torch.int64)
    return (one.view(torch.int64) & 0xFFFFFFFFFFFFF) >> 31


def _spread(x):
    for shift, mask in ((32, 0x1F00000000FFFF), (16, 0x1F0000FF0000FF), (8, 0x100F00F00F00F00F),
                        (4, 0x10C30C30C30C30C3), (2, 0x1249249249249249)):
        x = (x | (x << shift)) & mask
    return x


def _brute(points, queries, k, skip):
    """k smallest squared distances of each query; skip: the query's own point left out."""
    n, q = points.shape[1], queries.shape[1]
    out = torch.empty(q, k, dtype=torch.float64, device=DEV)
    step = max(1, min(q, 200_000_000 // n))
    for a in range(0, q, step):
        b = min(q, a + step)
        d = torch.zeros(b - a, n, dtype=torch.float64, device=DEV)
        for axis in range(3):
            d.add_((queries[axis, a:b, None] - points[axis][None, :]).square_())
        if skip:
            d[torch.arange(b - a, device=DEV), torch.arange(a, b, device=DEV)] = float("inf")
        out[a:b] = torch.topk(d, k, dim=1, largest=False, sorted=True).values
    return out


def exact(case, seed):
    op, coord = case["op"], case["coord"]
    if op not in ("self", "ext") or coord[0] == "u" or case.get("q", case["n"]) * case["n"] > 12e10:
        return None
    p, g = _points(case, seed)
    xyz = _coords(p, coord)
    points = torch.stack(xyz).to(torch.float64)
    if op == "ext":
        queries = torch.stack(_queries(case, p, g)).to(torch.float64)
        return None, _brute(points, queries, case["k"], False)
    if case["sfc"] != "morton":
        return None
    key = sum(_spread(_cells(a)) << i for i, a in enumerate(xyz))
    points = points[:, torch.sort(key, stable=True).indices].contiguous()
    return None, _brute(points, points, case["k"], True)
