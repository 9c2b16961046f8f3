"""Trees of clouds with many points at split values: the build's tie pass in
segments of one block and of the whole grid, splits that ties move off the
first pass's boundary, and levels that wait for a pass launched late.  Every
tree must be the reference's (permutation and node list, from the CPU
oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(kind, n, dtype=np.float64):
    rng = np.random.default_rng(n)
    p = rng.random((n, 3))
    if kind == "lattice":  # ties at every level
        p = rng.integers(0, 17, (n, 3)) * 0.0625
    elif kind == "plane":  # a third of the points at the root's split value
        p[rng.random(n) < 0.35, 0] = 0.5
        p[0], p[1] = 0.0, 1.0
    elif kind == "late":  # ties only deep in the tree, in one corner
        c = (p < 0.25).all(1)
        p[c] = np.round(p[c] * 64) / 64
    elif kind == "two":  # two values on the widest axis, most points at one
        p[:, 1] = np.where(rng.random(n) < 0.9, -3.0, 5.0)
    elif kind == "heavy":  # more points at one place than a block takes
        p[rng.random(n) < 0.6] = (0.25, 0.5, 0.75)
    return (p * 4096 if np.dtype(dtype).kind == "i" else p).astype(dtype)


@pytest.mark.parametrize("n", [700, 9_000, 70_000])
@pytest.mark.parametrize("kind", ["lattice", "plane", "late", "two", "heavy"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int16])
def test_tied_trees_are_the_reference_trees(gpu, port, dtype, kind, n):
    P = _cloud(kind, n, dtype)
    t, o = gpu.kdtree._build(P), port.PortTree(P)
    assert np.array_equal(t.reverse_indices(), o.reverse_indices())
    assert np.array_equal(t.ref_nodes(), o.nodes())


def test_rebuilds_take_ties_as_they_come(gpu, port):
    # a capture-ready forest rebuilt from clouds without ties, then with them
    import torch
    from pptk_b200 import ragged
    kinds = ["lattice", "uniform", "plane", "heavy", "late"]
    sizes = [30_000, 500, 20_000, 12_000, 40_000]
    off = np.concatenate([[0], np.cumsum(sizes)])
    f = ragged.Forest(torch.from_numpy(np.concatenate([_cloud("lattice", n, np.float32) for n in sizes])).cuda(), off)
    f.capture_ready()
    for ks in (["uniform"] * 5, kinds, kinds[::-1]):
        clouds = [_cloud(k, n, np.float32) for k, n in zip(ks, sizes)]
        f.rebuild(torch.from_numpy(np.concatenate(clouds)).cuda())
        rev = f.reverse_indices()
        for c, cl in enumerate(clouds):
            o = port.PortTree(cl)
            assert np.array_equal(rev[off[c]:off[c + 1]] - off[c], o.reverse_indices()), (ks, c)
            assert np.array_equal(f.ref_nodes(c), o.nodes()), (ks, c)
