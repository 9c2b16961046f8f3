"""The wide hierarchy under the kNN walks: node counts at the edges of a
level, far more siblings than a warp has lanes, leaf ranges that no split
divides, queries without neighbours; each as 32-query packets (lane_span -1)
and with one warp per query (0).  Every answer must equal the CPU oracle's,
which breaks distance ties by point index as the GPU does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(kind, n, dtype, dim=3):
    rng = np.random.default_rng(n + dim)
    if kind == "uniform":
        p = rng.random((n, dim))
    elif kind == "skewed":  # midpoint splits peel off a few points at a time
        p = np.exp(-rng.random((n, dim)) * 30.0)
    elif kind == "chain":  # one point per power of two: as deep as a tree gets
        p = np.ldexp(1.0, -(np.arange(n) % 100))[:, None] * np.ones(dim) + rng.random((n, dim)) * 1e-9
    else:  # "copies": leaf ranges of hundreds of equal points
        p = rng.random((max(n // 300, 1), dim))[rng.integers(0, max(n // 300, 1), n)]
    return p.astype(dtype)


@pytest.fixture(params=[-1, 0], ids=["packets", "warps"])
def span(request, gpu):
    from pptk_b200 import _native as N
    before = N.tune_get("lane_span")
    N.tune_set("lane_span", request.param)
    yield request.param
    N.tune_set("lane_span", before)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 65, 511, 513, 8191, 8193, 40_000])
@pytest.mark.parametrize("kind", ["uniform", "skewed", "chain", "copies"])
def test_walk_equals_the_oracle(gpu, port, span, kind, n):
    P = _cloud(kind, n, np.float32)
    rng = np.random.default_rng(5)
    t, o = gpu.kdtree._build(P), port.PortTree(P)
    Q = np.concatenate([P[rng.integers(0, n, 200)] + rng.normal(0, 0.01, (200, 3)), rng.random((50, 3)) * 40 - 20])
    Q = Q.astype(np.float32)
    rows = np.arange(min(n, 9_000), dtype=np.int32)
    deep = kind == "chain"  # (k > 64 is refused on trees deeper than 128 levels)
    for k in (1, 5, 16, 32, 64) if span or deep else (1, 32, 33, 64, 65, 128, 129, 256, 257):
        for got, want in ((gpu.kdtree.knn(t, Q, k), o.knn(Q, k)),
                          (gpu.kdtree.knn(t, rows, k), o.knn_self(rows, k))):
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), k
    # a query without a number, and one beyond every float distance, meet
    # ordinary ones in their warp
    Q[::7, 1] = np.nan
    Q[3::11, 0] = np.inf
    idx, cnt = gpu.kdtree.knn(t, Q, 8)
    fine = np.isfinite(Q).all(1)
    want = o.knn(Q[fine], 8)
    assert np.array_equal(idx[fine], want[0]) and (cnt[~fine] == 0).all() and (idx[~fine] == -1).all()


@pytest.mark.parametrize("dtype,dim", [(np.float64, 3), (np.float32, 2), (np.float64, 4), (np.int16, 3), (np.int64, 2)])
@pytest.mark.parametrize("bucket", [1, 16, 200])
def test_walk_over_types_and_buckets(gpu, port, span, dtype, dim, bucket):
    P = _cloud("skewed", 3_001, np.float64, dim)
    P = (P * 30_000).astype(dtype) if np.dtype(dtype).kind == "i" else P.astype(dtype)
    t, o = gpu.kdtree._build(P), port.PortTree(P)
    t.set_bucket(bucket)
    got, want = gpu.kdtree.knn(t, None, 10), o.knn_self(np.arange(len(P), dtype=np.int32), 10)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def test_walk_in_a_forest_and_a_loaded_tree(gpu, port, span, tmp_path):
    from pptk_b200 import ragged
    clouds = [_cloud(k, n, np.float32) for k, n in
              (("uniform", 33), ("chain", 700), ("copies", 2_000), ("uniform", 1), ("skewed", 9_000), ("uniform", 513))]
    off = np.concatenate([[0], np.cumsum([len(c) for c in clouds])])
    f = ragged.Forest(np.concatenate(clouds), off)
    f.save(tmp_path / "forest")
    for forest in (f, ragged.Forest.load(tmp_path / "forest", off)):
        idx, cnt = forest.knn(9)
        for c, cl in enumerate(clouds):
            oi, oc = port.PortTree(cl).knn_self(np.arange(len(cl), dtype=np.int32), 9)
            rows = slice(off[c], off[c + 1])
            assert np.array_equal(cnt[rows], oc) and np.array_equal(idx[rows], np.where(oi < 0, -1, oi + off[c])), c


@pytest.mark.parametrize("n", [1, 33, 513, 8193, 40_000])
@pytest.mark.parametrize("kind", ["uniform", "skewed", "chain", "copies"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_rnear_walk_equals_the_oracle(gpu, port, dtype, kind, n):
    # hits in ascending tree position: nodes inside the ball as runs of ids
    # (around the query's own point), runs of cut leaf ranges, more siblings
    # than lanes; from no hit to every point
    P = _cloud(kind, n, dtype)
    rng = np.random.default_rng(6)
    t, o = gpu.kdtree._build(P), port.PortTree(P)
    rows = rng.integers(0, n, min(n, 120)).astype(np.int32)
    Q = np.concatenate([P[rows], rng.random((30, 3)).astype(dtype)])
    for r in (0.0, 1e-6, 0.02, 0.3, 1.1, 5.0):
        r = float(np.float32(r))
        for got, want in ((gpu.kdtree.rnear(t, Q, r), o.rnear(Q, r)),
                          (gpu.kdtree.rnear(t, rows, r), o.rnear_self(rows, r))):
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), r
    Q[::5, 2] = np.nan
    off, _ = gpu.kdtree.rnear(t, Q, 0.3)
    assert (np.diff(off)[::5] == 0).all()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("k", [3, 16, 40, 100])
def test_normals_by_warp_equal_those_of_packets(gpu, dtype, k):
    # the same neighbours in the same order, solved by the same arithmetic:
    # equal bits, alone and in a forest with the self kNN, ties and dropped
    # rows included
    from pptk_b200 import _native as N, ragged
    P = np.concatenate([_cloud("uniform", 3_000, dtype), _cloud("copies", 1_000, dtype)])
    P[::97] = np.nan
    off = np.array([0, 50, 50, 3_100, 4_000])
    got, before = [], N.tune_get("lane_span")
    try:
        for s in (-1, 0):
            N.tune_set("lane_span", s)
            out = list(gpu.estimate_normals(P, k, np.inf, output_eigenvalues=True, output_all_eigenvectors=True,
                                            output_neighborhood_sizes=True, verbose=False))
            out.append(gpu.estimate_normals(P, k, 0.05, subsample=list(range(1, 700)), verbose=False))
            if k <= 64:
                out += ragged.Forest(P, off).knn_normals(k)
            got.append(out)
    finally:
        N.tune_set("lane_span", before)
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(*got))
