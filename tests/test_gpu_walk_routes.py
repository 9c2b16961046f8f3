"""The routes that batches take between packets and one warp per query:
multi-tree batches on both, batches large enough to be sorted before a warp
answers each query, warps that answer several queries, lists of more than 64,
and builds of more than four million points with ties."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def spans(gpu):
    """Runs a callable with packets only (lane_span -1) and with warps (0)."""
    from pptk_b200 import _native as N
    before = N.tune_get("lane_span")

    def both(f):
        out = []
        for s in (-1, 0):
            N.tune_set("lane_span", s)
            out.append(f())
        return out

    yield both
    N.tune_set("lane_span", before)


def _surface(rng, n, dtype=np.float32):
    p = rng.random((n, 3)) * (40, 40, 1)
    p[:, 2] = np.sin(p[:, 0]) + 0.01 * rng.normal(size=n)
    return p.astype(dtype)


def _trees(gpu, rng, dtype, sizes, queries):
    clouds = [_surface(rng, n, dtype) for n in sizes]
    trees = [gpu.kdtree._build(c) for c in clouds]
    rows = np.concatenate([[0], np.cumsum(queries)]).astype(np.int64)
    return clouds, trees, rows, (ctypes.c_void_p * len(trees))(*[t._h.value for t in trees])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("queries", [(4_000, 0, 33, 2_047), (1_060_001, 0, 2_500, 31)], ids=["small", "sorted"])
def test_multi_tree_knn_on_both_routes(gpu, port, spans, dtype, queries):
    from pptk_b200 import _native as N
    rng = np.random.default_rng(len(str(queries)))
    clouds, trees, rows, handles = _trees(gpu, rng, dtype, (150_000, 3, 9_000, 700), queries)
    Q = np.concatenate([c[rng.integers(0, len(c), m)] + dtype(1e-3) for c, m in zip(clouds, queries)])
    for k in (3, 16, 64) if len(Q) < 10_000 else (3,):
        def run():
            idx, cnt = np.empty((len(Q), k), np.int32), np.empty(len(Q), np.int32)
            N.call("pptkg_multi_knn", handles, len(trees), N.ptr(Q), N.ptr(rows), 0 if dtype == np.float32 else 1,
                   N.MEM_HOST, k, float("inf"), N.ptr(idx), N.ptr(cnt), None)
            return idx, cnt
        (ip, cp), (iw, cw) = spans(run)
        assert np.array_equal(ip, iw) and np.array_equal(cp, cw), k
        for g, c in enumerate(clouds):
            at = slice(rows[g], min(rows[g + 1], rows[g] + 3_000))
            want = port.PortTree(c).knn(Q[at], k)
            assert np.array_equal(ip[at], want[0]) and np.array_equal(cp[at], want[1]), (k, g)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("queries", [(4_000, 0, 33, 700), (270_001, 0, 2_500, 31)], ids=["small", "sorted"])
def test_multi_tree_normals_on_both_routes(gpu, spans, dtype, queries):
    from pptk_b200 import _native as N
    rng = np.random.default_rng(len(str(queries)) + 1)
    clouds, trees, rows, handles = _trees(gpu, rng, dtype, (150_000, 3, 9_000, 700), queries)
    ids = np.concatenate([rng.integers(0, len(c), m) for c, m in zip(clouds, queries)]).astype(np.int32)
    for k in (8, 20):
        def run():
            ev = np.empty((len(ids), 3), dtype)
            N.call("pptkg_multi_normals", handles, len(trees), N.ptr(ids), N.ptr(rows), N.MEM_HOST, k,
                   ctypes.c_float(np.inf), 1, 0, N.ptr(ev), None, None, None)
            for g, t in enumerate(trees):
                part = np.ascontiguousarray(ids[rows[g]:rows[g + 1]])
                if len(part) == 0:
                    continue
                alone = np.empty((len(part), 3), dtype)
                N.call("pptkg_tree_normals", t._h, N.ptr(part), len(part), N.MEM_HOST, k, ctypes.c_float(np.inf), 1, 0,
                       N.ptr(alone), None, None, None)
                assert np.array_equal(ev[rows[g]:rows[g + 1]], alone, equal_nan=True), (k, g)
            return ev
        packets, warps = spans(run)
        assert np.array_equal(packets, warps, equal_nan=True), k


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_large_batches_on_both_routes(gpu, port, spans, dtype):
    # more queries than a warp batch takes as they come (2^20 points, 2^18
    # rows), all points in tree order, and normals with several queries to a
    # warp
    rng = np.random.default_rng(7)
    P = _surface(rng, 150_000, dtype)
    t, o = gpu.kdtree._build(P), port.PortTree(P)
    Q = P[rng.integers(0, len(P), 1_060_001)] + dtype(2e-3)
    rows = rng.integers(0, len(P), 270_001).astype(np.int32)
    for k in (5, 32):
        for queries, oracle in ((Q if k == 5 else Q[:140_001], o.knn), (rows, o.knn_self), (None, None)):
            (ip, cp), (iw, cw) = spans(lambda: gpu.kdtree.knn(t, queries, k))
            assert np.array_equal(ip, iw) and np.array_equal(cp, cw), k
            if oracle:
                want = oracle(queries[:2_000], k)
                assert np.array_equal(ip[:2_000], want[0]) and np.array_equal(cp[:2_000], want[1]), k
    for sub in (None, rows, np.arange(1, 40_000, 2)):
        packets, warps = spans(lambda: gpu.estimate_normals(P, 16, np.inf, subsample=sub, output_eigenvalues=True,
                                                            output_all_eigenvectors=True, verbose=False))
        assert np.array_equal(packets[0], warps[0]) and np.array_equal(packets[1], warps[1])


@pytest.mark.parametrize("n", [9_000, 30_000, 64_000])
def test_whole_clouds_on_both_routes(gpu, port, spans, n):
    # every point of a cloud, in tree order: alone, as a forest, with the
    # normals, and without allocations
    import torch
    from pptk_b200 import _native as N, ragged
    rng = np.random.default_rng(n)
    P = _surface(rng, n)
    d = torch.from_numpy(P).cuda()
    t = gpu.kdtree._build(d)
    f = ragged.Forest(d, [0, n // 3, n])
    want = port.PortTree(P).knn_self(np.arange(n, dtype=np.int32), 16)

    def run():
        ev = torch.empty((n, 3), device="cuda")
        N.call("pptkg_tree_normals_noalloc", t._h, None, 0, 16, ctypes.c_float(np.inf), 1, 0, N.ptr(ev), None, None,
               N.torch_stream(ev.device))
        out = [ev, gpu.estimate_normals(d, 16, np.inf, verbose=False), *gpu.kdtree.knn(t, None, 16), *f.knn(8),
               *f.knn_normals(16), f.normals(30)]
        return [x.cpu().numpy() if hasattr(x, "cpu") else x for x in out]

    packets, warps = spans(run)
    assert all(np.array_equal(a, b) for a, b in zip(packets, warps))
    assert np.array_equal(packets[0], packets[1])
    assert np.array_equal(packets[2], want[0]) and np.array_equal(packets[3], want[1])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("k", [64, 65, 128, 200, 256])
def test_normals_of_long_lists(gpu, port, spans, dtype, k):
    # against the FP64 oracle, dropped rows and copies of points included;
    # 64 on both routes
    rng = np.random.default_rng(k)
    P = np.concatenate([_surface(rng, 3_000, dtype), rng.random((5, 3))[rng.integers(0, 5, 1_500)].astype(dtype)])
    P = P[rng.permutation(len(P))]
    P[::97] = np.nan
    packets, warps = spans(lambda: gpu.estimate_normals(P, k, np.inf, output_eigenvalues=True,
                                                        output_all_eigenvectors=True, output_neighborhood_sizes=True,
                                                        verbose=False))
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(packets, warps))
    ev, ew, sz = warps
    _, _, osz, nb = port.port_estimate_normals(P, k, np.inf, num_eigen=3, want_nbrs=True)
    assert np.array_equal(sz, osz)
    has = sz > 0
    assert np.isnan(ev[~has]).all() and has.sum() == np.isfinite(P).all(1).sum()
    # (shifted to the query point, which is exact: copies of it stay at zero)
    nb = nb[has]
    near = np.where((nb >= 0)[..., None], P[nb].astype(np.float64) - P[has].astype(np.float64)[:, None, :], 0.0)
    own = np.where(nb >= 0, np.arange(nb.size).reshape(nb.shape), -1)
    w, V, _ = port.normals_fp64(near.reshape(-1, 3), own)
    # as for shorter lists: eigenvalues to 1e-5 of the largest, normals to
    # |dot| >= 1 - 1e-6 where the two smallest eigenvalues differ
    scale = np.abs(w[:, 2:3])
    assert (np.abs(ew[has] - w) <= 1e-5 * scale + 1e-30).all()
    ok = (w[:, 1] - w[:, 0]) >= 1e-4 * np.maximum(scale[:, 0], 1e-300)
    dots = np.abs((ev[has][:, 0, :].astype(np.float64) * V[:, 0, :]).sum(1))
    assert (dots[ok] >= 1 - 1e-6).all()


@pytest.mark.parametrize("kind", ["lattice", "plane", "late"])
def test_large_tied_trees_are_the_reference_trees(gpu, port, kind):
    # tiles of 4,096 points, a look at every fourth level
    rng = np.random.default_rng(3)
    n = 4_300_000
    p = rng.random((n, 3), dtype=np.float32)
    if kind == "lattice":
        p = np.floor(p * 200)
    elif kind == "plane":
        p[rng.random(n) < 0.35, 0] = 0.5
        p[0], p[1] = 0.0, 1.0
    else:
        c = (p < 0.2).all(1)
        p[c] = np.round(p[c] * 1024) / 1024
    t, o = gpu.kdtree._build(p), port.PortTree(p)
    assert np.array_equal(t.reverse_indices(), o.reverse_indices())
    assert np.array_equal(t.ref_nodes(), o.nodes())
