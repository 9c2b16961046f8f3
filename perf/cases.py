"""Timing cases of pptk_b200: what a user's program asks of it, call by call.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a program holds before the call (clouds, resident
trees, query arrays, all on the GPU), ``run`` makes the call once, ``work``
counts the bytes and operations the answer cannot do without, and ``exact``
evaluates the floating-point results in 64 bits without this package.

Clouds follow the distributions of ``pptk_b200.synth`` (uniform cube, street
scene, translated planar patches, ragged batches of blobs and planes), drawn
on the GPU so that a fresh cloud costs milliseconds.
"""
import math

import numpy as np
import torch

import pptk_b200 as pptk
from pptk_b200 import ragged, serving

_DTYPES = {"float32": torch.float32, "float64": torch.float64, "int16": torch.int16, "int32": torch.int32}
_SIZE = {"float32": 4, "float64": 8, "int16": 2, "int32": 4}


# ---------------------------------------------------------------- cases ----
def listed():
    return [
        # a handful of lookups on a resident tree: one click, one robot pose;
        # launch latency is all of it
        {"name": "knn_10_of_200k", "do": "knn", "cloud": "uniform", "n": 200_000, "dtype": "float32", "dim": 3,
         "queries": "points", "m": 10, "k": 16},
        # normals of one small object scan, tree build included as in the
        # reference's call
        {"name": "normals_3001", "do": "normals", "cloud": "uniform", "n": 3_001, "dtype": "float32", "k": 16},
        # load a cloud, index it, look up a few points
        {"name": "build_200k", "do": "build", "cloud": "uniform", "n": 200_000, "dtype": "float32", "dim": 3,
         "m": 1_000, "k": 16},
        # survey coordinates (large offsets) need float64 throughout
        {"name": "normals_patches_f64", "do": "normals", "cloud": "patches", "n": 1_000_003, "dtype": "float64",
         "k": 16},
        # normals of a whole street scene in one call
        {"name": "normals_scene_20M", "do": "normals", "cloud": "scene", "n": 20_000_000, "dtype": "float32", "k": 16},
        # neighbour lists of every point of a scene (feature extraction,
        # graph construction)
        {"name": "knn32_scene_20M", "do": "knn", "cloud": "scene", "n": 20_000_000, "dtype": "float32", "dim": 3,
         "queries": "points", "m": 20_000_000, "k": 32},
        # a large batch of coordinate lookups in no particular order
        {"name": "knn_1M_scene_20M", "do": "knn", "cloud": "scene", "n": 20_000_000, "dtype": "float32", "dim": 3,
         "queries": "points", "m": 1_000_003, "k": 16},
        # wide-radius neighbourhoods of sampled key points
        {"name": "rnear_20k_scene_20M", "do": "rnear", "cloud": "scene", "n": 20_000_000, "dtype": "float32", "dim": 3,
         "queries": "points", "m": 20_000, "r": 0.5, "hits": 44_900},
        # small-radius neighbourhoods of every point (Points.nbhds(r=...))
        {"name": "rnear_all_300k", "do": "rnear", "cloud": "uniform", "n": 300_001, "dtype": "float32", "dim": 3,
         "queries": "rows", "m": 300_001, "r": 0.0288, "hits": 29},
        # a training batch of small object clouds
        {"name": "ragged_512_small", "do": "ragged", "clouds": 512, "lo": 500, "hi": 5_000, "dtype": "float32", "k": 16},
        # a batch of scans of very different sizes
        {"name": "ragged_256_large", "do": "ragged", "clouds": 256, "lo": 1_000, "hi": 200_000, "dtype": "float32",
         "k": 16},
        # a resident scene serving a burst of kNN and normal requests of 1k to
        # 1M queries
        {"name": "serve_scene_20M", "do": "serve", "cloud": "scene", "n": 20_000_000, "dtype": "float32",
         "requests": 12, "lo": 1_000, "hi": 1_000_000, "k": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes spread over the logarithm of the listed range, all
    point types, 2 to 4 dimensions, k from 1 to beyond the register lists,
    radius neighbourhoods and rows with missing (NaN) coordinates."""
    do = rng.choice(["knn", "knn", "normals", "normals", "build", "rnear", "ragged"])
    if do == "ragged":
        clouds = _log_int(rng, 2, 1_000)
        lo = _log_int(rng, 50, 2_000)
        return {"do": do, "clouds": clouds, "lo": lo, "hi": min(lo * _log_int(rng, 2, 100), 10_000_000 // clouds + lo),
                "dtype": rng.choice(["float32", "float32", "float64"]), "k": rng.choice([4, 8, 10, 16, 24])}
    if do == "normals":
        dtype = rng.choice(["float32", "float32", "float64"])
        cloud = rng.choice(["uniform", "patches"] if dtype == "float64" else ["uniform", "scene"])
        case = {"do": do, "cloud": cloud, "n": _log_int(rng, 300, 10_000_000 if dtype == "float32" else 1_000_000),
                "dtype": dtype, "k": rng.choice([6, 8, 12, 16, 20, 30])}
        form = rng.choice(["plain", "all", "nan", "radius", "large_k"])
        if form == "all":
            case["all"] = True
        elif form == "nan":
            case["nan"] = 0.01
        elif form == "radius":
            case.update(cloud="uniform", n=min(case["n"], 500_000), k=-1)
            case["r"] = round(_radius(case["n"], 3, rng.uniform(10.0, 60.0)), 5)
        elif form == "large_k":
            case.update(n=min(case["n"], 100_000), k=rng.choice([70, 100]))
        return case
    dtype = rng.choice(["float32", "float32", "float32", "float64", "int16", "int32"])
    dim = rng.choice([2, 3, 3, 3, 4])
    wide = dtype == "float32" and dim == 3
    cloud = rng.choice(["uniform", "scene"]) if wide else "uniform"
    n = _log_int(rng, 1_000, 10_000_000 if wide else 1_000_000)
    if do == "build":
        return {"do": do, "cloud": cloud, "n": n, "dtype": dtype, "dim": dim, "m": _log_int(rng, 1, 1_000),
                "k": rng.choice([1, 8, 16])}
    queries = rng.choice(["points", "rows", "all"])
    m = n if queries == "all" else _log_int(rng, 1, min(n, 2_000_000))
    case = {"do": do, "cloud": cloud, "n": n, "dtype": dtype, "dim": dim, "queries": "points" if queries == "points" else "rows",
            "m": m}
    if do == "rnear":
        case.update(cloud="uniform", n=min(n, 2_000_000), m=min(m, min(n, 2_000_000), 500_000))
        hits = rng.uniform(5.0, 100.0) if case["m"] > 20_000 else rng.uniform(5.0, 1_000.0)
        hits = min(hits, case["n"] / 20)
        case.update(r=round(_radius(case["n"], dim, hits), 5), hits=round(hits))
        if case["dtype"] != "float64":
            case["dtype"] = "float32"
        return case
    case["k"] = rng.choice([1, 3, 5, 8, 10, 16, 20, 32, 50, 64, 100])
    if case["k"] > 32:
        case["m"] = min(case["m"], 100_000)
    return case


def _radius(n, dim, hits):
    """Radius of a ball that holds `hits` of n uniform points of the unit cube."""
    ball = {2: math.pi, 3: 4.0 / 3.0 * math.pi, 4: math.pi ** 2 / 2.0}[dim]
    return (hits / (n * ball)) ** (1.0 / dim)


# --------------------------------------------------------------- clouds ----
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _ground(g, n, half=100.0, sigma=0.01):
    """Ground returns: density falls with the squared distance from the sensor
    at the origin (constant within 1 m), on a square of +-half metres."""
    th = (_rand(g, int(1.12 * n) + 64) * 2.0 - 1.0) * math.pi
    edge = half / torch.maximum(th.cos().abs(), th.sin().abs())
    keep = _rand(g, th.shape[0]) * (0.5 + math.log(half * math.sqrt(2.0))) < 0.5 + edge.log()
    th, edge = th[keep][:n], edge[keep][:n]
    n = th.shape[0]
    inner = _rand(g, n) * (0.5 + edge.log()) < 0.5
    rad = torch.where(inner, _rand(g, n).sqrt(), (_rand(g, n) * edge.log()).exp())
    return torch.stack([rad * th.cos(), rad * th.sin(), _randn(g, n) * sigma], 1)


def _pick(g, weights, n):
    edges = torch.cumsum(weights / weights.sum(), 0)
    return torch.searchsorted(edges, _rand(g, n)).clamp_(max=weights.shape[0] - 1)


def _boxes(g, n, count=500, half=100.0):
    c = (_rand(g, count, 2) * 2.0 - 1.0) * half
    s = 1.0 + 9.0 * _rand(g, count, 3)
    top, ends, sides = s[:, 0] * s[:, 1], s[:, 0] * s[:, 2], s[:, 1] * s[:, 2]
    area = top + 2.0 * ends + 2.0 * sides
    obj = _pick(g, area / c.norm(dim=1).clamp(min=1.0) ** 2, n)
    pick = _rand(g, n) * area[obj]
    u, v, flip = _rand(g, n), _rand(g, n), torch.where(_rand(g, n) < 0.5, -0.5, 0.5)
    sx, sy, sz = s[obj, 0], s[obj, 1], s[obj, 2]
    on_top, on_end = pick < top[obj], pick < (top + 2.0 * ends)[obj]
    x = torch.where(on_end, (u - 0.5) * sx, flip * sx)
    y = torch.where(on_top, (v - 0.5) * sy, torch.where(on_end, flip * sy, (u - 0.5) * sy))
    z = torch.where(on_top, sz, v * sz)
    return torch.stack([x + c[obj, 0], y + c[obj, 1], z], 1)


def _cylinders(g, n, count=300, half=100.0):
    c = (_rand(g, count, 2) * 2.0 - 1.0) * half
    rad, h = 0.2 + 0.8 * _rand(g, count), 2.0 + 6.0 * _rand(g, count)
    side = 2.0 * math.pi * rad * h
    area = side + math.pi * rad ** 2
    obj = _pick(g, area / c.norm(dim=1).clamp(min=1.0) ** 2, n)
    on_side = _rand(g, n) * area[obj] < side[obj]
    th = 2.0 * math.pi * _rand(g, n)
    r = torch.where(on_side, rad[obj], rad[obj] * _rand(g, n).sqrt())
    z = torch.where(on_side, _rand(g, n) * h[obj], h[obj])
    return torch.stack([c[obj, 0] + r * th.cos(), c[obj, 1] + r * th.sin(), z], 1)


def _scene(g, n):
    ng, nb = int(round(0.7 * n)), int(round(0.2 * n))
    parts = [_ground(g, ng), _boxes(g, nb)]
    parts.append(_cylinders(g, n - sum(p.shape[0] for p in parts)))
    pts = torch.cat(parts)
    return pts[torch.randperm(n, generator=g, device="cuda")]


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _plane_axes(nrm):
    e = torch.zeros_like(nrm)
    e[:, 0] = (nrm[:, 0].abs() < 0.9).to(nrm.dtype)
    e[:, 1] = 1.0 - e[:, 0]
    a = _unit(torch.linalg.cross(nrm, e))
    return a, torch.linalg.cross(nrm, a)


def _patches(g, n, count=200, size=10.0, sigma=1e-4, offset=1e5, outliers=0.05):
    n_out = int(round(outliers * n))
    nrm = _unit(_randn(g, count, 3))
    a, b = _plane_axes(nrm)
    cen = _rand(g, count, 3) * torch.tensor([400.0, 400.0, 50.0], device="cuda", dtype=torch.float64)
    obj = torch.randint(count, (n - n_out,), generator=g, device="cuda")
    uv = (_rand(g, n - n_out, 2) - 0.5) * size
    p = cen[obj] + uv[:, :1] * a[obj] + uv[:, 1:] * b[obj] + _randn(g, n - n_out, 1) * sigma * nrm[obj]
    lo, hi = p.min(0).values, p.max(0).values
    pts = torch.cat([p, lo + _rand(g, n_out, 3) * (hi - lo)])[torch.randperm(n, generator=g, device="cuda")]
    pts[:, :2] += offset
    return pts


def _cloud(g, case):
    n, dim = case["n"], case.get("dim", 3)
    dt = _DTYPES[case["dtype"]]
    if case["cloud"] == "scene":
        pts = _scene(g, n).to(dt)
    elif case["cloud"] == "patches":
        pts = _patches(g, n).to(dt)
    elif dt.is_floating_point:
        pts = torch.rand(n, dim, generator=g, device="cuda", dtype=dt)
    else:  # scans stored on an integer grid
        pts = torch.randint(-30_000, 30_000, (n, dim), generator=g, device="cuda").to(dt)
    if case.get("nan"):
        pts[torch.rand(n, generator=g, device="cuda") < case["nan"], 1] = math.nan
    return pts.contiguous()


def _ragged_sizes(case, seed):
    """Sizes spread evenly over their logarithm (a batch costs the same under
    every seed), in an order drawn from the seed."""
    c = case["clouds"]
    q = (np.arange(c) + 0.5) / c
    sizes = np.exp(math.log(case["lo"]) + q * math.log(case["hi"] / case["lo"])).astype(np.int64)
    return np.random.default_rng(seed).permutation(sizes)


def _ragged(g, sizes, dt):
    """Clouds of Gaussian blobs and one noisy plane, concatenated."""
    c, n = len(sizes), int(sizes.sum())
    sz = torch.from_numpy(sizes).cuda()
    cloud = torch.repeat_interleave(torch.arange(c, device="cuda"), sz)
    row = torch.arange(n, device="cuda") - (torch.cumsum(sz, 0) - sz)[cloud]
    cen = _rand(g, c, 5, 3) * 10.0 - 5.0
    sig = 0.05 + 0.45 * _rand(g, c, 5)
    blobs = torch.randint(1, 6, (c,), generator=g, device="cuda")
    which = (_rand(g, n) * blobs[cloud]).long()
    blob = cen[cloud, which] + _randn(g, n, 3) * sig[cloud, which][:, None]
    nrm = _unit(_randn(g, c, 3))
    a, b = _plane_axes(nrm)
    uv = _rand(g, n, 2) * 10.0 - 5.0
    plane = uv[:, :1] * a[cloud] + uv[:, 1:] * b[cloud] + 0.01 * _randn(g, n, 1) * nrm[cloud]
    return torch.where((row < sz[cloud] // 3)[:, None], plane, blob).to(dt).contiguous()


# -------------------------------------------------------------- prepare ----
class _Service:
    """A server with one resident tree, closed when the program lets it go."""

    def __init__(self, points):
        self.server = serving.Server()
        torch.cuda.synchronize()  # the server works on streams of its own
        self.tree = self.server.build(points).result()

    def __del__(self):
        self.server.close()


def _request_sizes(case):
    """kNN and normal requests alternate; sizes spread evenly over their
    logarithm, large and small ones mixed."""
    c = case["requests"]
    q = (np.random.default_rng(0).permutation(c) + 0.5) / c
    return np.exp(math.log(case["lo"]) + q * math.log(case["hi"] / case["lo"])).astype(np.int64)


def prepare(case, seed):
    g = _generator(seed)
    state = {"case": case}
    if case["do"] == "ragged":
        sizes = _ragged_sizes(case, seed)
        state["offsets"] = np.concatenate([[0], np.cumsum(sizes)])
        state["points"] = _ragged(g, sizes, _DTYPES[case["dtype"]])
        return state
    if case["do"] == "rnear":
        # the seed orders the rows of one cloud and one set of queries, so
        # that the lists of every seed hold as many hits in all
        base = _generator(17)
        points = _cloud(base, case)
        pick = torch.randperm(case["n"], generator=base, device="cuda")[:case["m"]]
        order = torch.randperm(case["n"], generator=g, device="cuda")
        points = points[order]
        rows = torch.empty_like(order).scatter_(0, order, torch.arange(case["n"], device="cuda"))[pick]
        rows = rows[torch.randperm(case["m"], generator=g, device="cuda")]
        state["queries"] = points[rows] if case["queries"] == "points" else rows.to(torch.int32)
        state["tree"] = pptk.kdtree._build(points)
        return state
    points = _cloud(g, case)
    if case["do"] == "normals":
        state["points"] = points
        return state
    if case["do"] == "serve":
        state["service"] = _Service(points)
        state["requests"] = []
        for i, m in enumerate(_request_sizes(case)):
            rows = torch.randint(case["n"], (int(m),), generator=g, device="cuda", dtype=torch.int32)
            state["requests"].append(("normals", rows) if i % 2 else ("knn", points[rows.long()]))
        return state
    n, m = case["n"], case["m"]
    rows = torch.randint(n, (m,), generator=g, device="cuda") if m < n else torch.arange(n, device="cuda")
    by_point = case["do"] == "build" or case["queries"] == "points"
    state["queries"] = points[rows] if by_point else rows.to(torch.int32)
    if case["do"] == "build":
        state["points"] = points
    else:
        state["tree"] = pptk.kdtree._build(points)
    return state


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "knn":
        return pptk.kdtree.knn(state["tree"], state["queries"], case["k"])
    if do == "rnear":
        return pptk.kdtree.rnear(state["tree"], state["queries"], case["r"])
    if do == "build":
        tree = pptk.kdtree._build(state["points"])
        return pptk.kdtree.knn(tree, state["queries"], case["k"])
    if do == "normals":
        wide = bool(case.get("all"))
        return pptk.estimate_normals(state["points"], case["k"], case.get("r", math.inf), output_eigenvalues=wide,
                                     output_all_eigenvectors=wide, output_neighborhood_sizes=wide, verbose=False)
    if do == "ragged":
        return ragged.Forest(state["points"], state["offsets"]).knn_normals(case["k"])
    service = state["service"]
    futures = [service.server.knn(service.tree, q, case["k"]) if kind == "knn" else
               service.server.normals(service.tree, q, case["k"]) for kind, q in state["requests"]]
    return [f.result() for f in futures]


# ----------------------------------------------------- work and answers ----
def _knn_flops(m, k, dim):
    return m * k * (3.0 * dim - 1.0)  # one squared distance per neighbour


def _pca_flops(m, k):
    # shift, mean, centred second moments of k neighbours; a 3 x 3 eigensolve
    return m * (24.0 * k + 300.0)


def work(case):
    """Every input read once and every output written once; one distance per
    neighbour kept.  A query of a resident tree reads the neighbours it
    returns, and no point of the tree more than once."""
    do, s = case["do"], _SIZE[case["dtype"]]
    if do == "ragged":
        n, k = int(_ragged_sizes(case, 0).sum()), case["k"]
        return {"bytes": n * (3 * s + 4 * k + 4 + 3 * s), "flops": _knn_flops(n, k, 3) + _pca_flops(n, k)}
    n = case["n"]
    if do == "normals":
        k = case["k"] if case["k"] > 0 else 4.0 / 3.0 * math.pi * case["r"] ** 3 * n
        return {"bytes": n * (3 * s + (12 * s + 4 if case.get("all") else 3 * s)),
                "flops": _knn_flops(n, k, 3) + _pca_flops(n, k)}
    if do == "serve":
        sizes, k = _request_sizes(case), case["k"]
        near, flat = int(sizes[0::2].sum()), int(sizes[1::2].sum())
        read = min(n, (near + flat) * k) * (3 * s + 4)
        return {"bytes": near * (3 * s + 4 * k + 4) + flat * (4 + 3 * s) + read,
                "flops": _knn_flops(near + flat, k, 3) + _pca_flops(flat, k)}
    m, dim = case["m"], case["dim"]
    row = dim * s if do == "build" or case["queries"] == "points" else 4
    if do == "rnear":
        hits = m * case["hits"]
        return {"bytes": m * (row + 8) + min(n, hits) * (dim * s + 4) + 4 * hits,
                "flops": _knn_flops(m, case["hits"], dim)}
    k = case["k"]
    answer = m * (row + 4 * k + 4)
    if do == "build":
        return {"bytes": n * dim * s + answer, "flops": _knn_flops(m, k, dim) + 2.0 * n * dim}
    return {"bytes": answer + min(n, m * k) * (dim * s + 4), "flops": _knn_flops(m, k, dim)}


def _neighbourhoods(points, k, r):
    """(rows x w neighbour indices, rows x w mask, chunk by chunk) of every
    valid point, the point itself included.  Neighbours are chosen by the
    distance the package documents (squared differences summed in axis order
    in the points' own type); everything computed from them is in 64 bits."""
    n = points.shape[0]
    step = max(1, min(n, 200_000_000 // n))
    for lo in range(0, n, step):
        d2 = None
        for d in range(3):
            e = points[None, :, d] - points[lo:lo + step, d, None]
            d2 = e.mul_(e) if d2 is None else d2.add_(e.mul_(e))
        if k > 0:
            near = d2.topk(min(k, n), dim=1, largest=False, sorted=False)
            yield near.indices, near.values < math.inf
        else:
            inside = d2 < torch.tensor(r, dtype=points.dtype, device=points.device).square()
            w = int(inside.sum(1).max())
            near = inside.to(torch.uint8).topk(w, dim=1, sorted=False)
            yield near.indices, near.values > 0


def _pca64(points, k, r):
    """Eigenvalues (ascending) and eigenvectors (rows, largest component
    positive) of every valid point's neighbourhood, NaN elsewhere."""
    n = points.shape[0]
    rows = points.isfinite().all(1).nonzero()[:, 0]
    valid = points[rows]
    w = torch.full((n, 3), math.nan, dtype=torch.float64)
    v = torch.full((n, 3, 3), math.nan, dtype=torch.float64)
    lo = 0
    for idx, mask in _neighbourhoods(valid, k, r):
        y = valid[idx].double()
        f = mask.double()[:, :, None]
        y = y - valid[lo:lo + idx.shape[0], None].double()
        y = (y - (y * f).sum(1, keepdim=True) / f.sum(1, keepdim=True)) * f
        cov = (y.transpose(1, 2) @ y / f.sum(1, keepdim=True)).cpu().numpy()
        ew, ev = np.linalg.eigh(cov)
        ev = np.swapaxes(ev, 1, 2)
        top = np.take_along_axis(ev, np.abs(ev).argmax(2)[:, :, None], 2)
        at = rows[lo:lo + idx.shape[0]].cpu()
        w[at], v[at] = torch.from_numpy(ew), torch.from_numpy(ev * np.where(top < 0, -1.0, 1.0))
        lo += idx.shape[0]
    return w, v


def exact(case, seed):
    """Normals (and eigenvalues) in 64 bits where comparing every pair of
    points is a matter of seconds; neighbour lists are whole numbers and have
    no such value."""
    g = _generator(seed)
    if case["do"] == "ragged":
        sizes = _ragged_sizes(case, seed)
        if float((sizes.astype(np.float64) ** 2).sum()) > 2e10:
            return None
        points = _ragged(g, sizes, _DTYPES[case["dtype"]])
        v = [_pca64(p, case["k"], math.inf)[1][:, 0] for p in points.split(sizes.tolist())]
        return (None, None, torch.cat(v))
    if case["do"] != "normals" or case["n"] > 150_000:
        return None
    w, v = _pca64(_cloud(g, case), case["k"], case.get("r", math.inf))
    return (v, w, None) if case.get("all") else v[:, 0]
