"""Builds and in-place rebuilds at the edges of their capacities: chains of
thousands of levels, the second attempt of a build whose list of small
segments overflowed, and rebuilds that need other shapes of tree than the
first build's.  Every accepted tree must be the reference's (from the CPU
oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _is_reference_tree(t, o):
    assert np.array_equal(t.reverse_indices(), o.reverse_indices())
    assert np.array_equal(t.ref_nodes(), o.nodes())


def _axis_chains(per_axis, lowest=1e-300):
    """Points on the axes from 1e300 down by factors of 2.05 (float64): every midpoint split
    takes one point off."""
    v = 10.0 ** (300 - np.log10(2.05) * np.arange(per_axis))
    assert v[-1] > lowest
    p = np.zeros((3 * per_axis, 3))
    for d in range(3):
        p[d * per_axis:(d + 1) * per_axis, d] = v
    return p


def test_more_than_4096_levels_of_large_segments(gpu, port):
    # 4,800 levels, 4,544 of them with a segment above the subtree kernel's 256
    # float64 points
    P = _axis_chains(1600)[np.random.default_rng(0).permutation(4800)]
    _is_reference_tree(gpu.kdtree._build(P), port.PortTree(P))


def test_second_attempt_builds_from_the_input_order(gpu, port):
    # 2,850 levels give more small segments than the first attempt's list
    # holds; the lattice below them has splits inside runs of equal values,
    # whose order depends on that of the points the attempt starts from
    rng = np.random.default_rng(1)
    P = np.concatenate([_axis_chains(950, 20.0), rng.integers(0, 9, (1500, 3)) * 1.0])
    P = P[rng.permutation(len(P))]
    _is_reference_tree(gpu.kdtree._build(P), port.PortTree(P))


def _rebuilt(first, second, off, maxleafsize=10):
    import torch
    from pptk_b200 import ragged
    f = ragged.Forest(torch.from_numpy(first).cuda(), off, maxleafsize=maxleafsize)
    f.capture_ready()
    f.rebuild(torch.from_numpy(second).cuda())
    return f


def _are_reference_trees(f, P, off, port, maxleafsize=10):
    rev = f.reverse_indices()
    for c in range(0, len(off) - 1, max(1, (len(off) - 1) // 50)):
        o = port.PortTree(P[off[c]:off[c + 1]], maxleafsize=maxleafsize)
        assert np.array_equal(rev[off[c]:off[c + 1]] - off[c], o.reverse_indices()), c
        assert np.array_equal(f.ref_nodes(c), o.nodes()), c


def _chain_to_copies(rng, n, chain, copies):
    """Half a box of points, and in the other half powers of two along an axis
    down to copies of one point."""
    p = rng.random((n, 3))
    p[:, 0] = 0.5 + 0.5 * p[:, 0]
    p[:chain + copies] = (0.0, 0.25, 0.25)
    p[:chain, 0] = 0.25 * 2.0 ** -np.arange(chain)
    return p


@pytest.mark.parametrize("dtype,copies", [(np.float32, 700), (np.float64, 400)])
def test_rebuild_with_segments_below_the_planned_levels(gpu, port, dtype, copies):
    # a tree of 14 levels where 19 are planned for, but with 700 (400) points
    # in one segment three levels below the last grid-wide one
    rng = np.random.default_rng(0)
    off = np.array([0, 3000, 6000])
    A = rng.random((6000, 3)).astype(dtype)
    B = np.concatenate([_chain_to_copies(rng, 3000, 24, copies) for _ in range(2)]).astype(dtype)
    _are_reference_trees(_rebuilt(A, B, off), B, off, port)


def test_rebuild_with_more_wide_nodes_than_the_first_build(gpu, port):
    # clouds of 40 points: two leaf ranges each in the first build, nine of a
    # chain in the second, with as many records as before
    rng = np.random.default_rng(0)
    clouds = 3000
    off = 40 * np.arange(clouds + 1)
    one = rng.random((40, 3)) * 2.0 ** -9
    one[:8] = 0.0
    one[:8, 0] = 2.0 ** -np.arange(8)
    A = rng.random((40 * clouds, 3)).astype(np.float32)
    B = np.tile(one, (clouds, 1)).astype(np.float32)
    f = _rebuilt(A, B, off, maxleafsize=1)
    _are_reference_trees(f, B, off, port, maxleafsize=1)
    idx, cnt = f.knn(5)
    oi, oc = port.PortTree(B[:40]).knn_self(np.arange(40, dtype=np.int32), 5)
    assert np.array_equal(cnt.cpu().numpy(), np.tile(oc, clouds))
    assert np.array_equal(idx.cpu().numpy(), np.tile(oi, (clouds, 1)) + np.repeat(off[:-1], 40)[:, None])


def test_refused_rebuild_leaves_every_record_readable(gpu):
    # ties move every split of a chain of segments above 8,192 points, past the
    # last planned level: the segment left over has a record but no decision
    import torch
    from pptk_b200 import ragged
    n = 20_000
    rng = np.random.default_rng(2)
    A = rng.random((n, 3)).astype(np.float32)
    B = np.zeros((n, 3))
    B[:, 1:] = rng.random((n, 2)) * 1e-30
    B[:90, 0] = -2.0 ** -np.arange(90)
    B = B.astype(np.float32)
    f = ragged.Forest(torch.from_numpy(A).cuda(), [0, n])
    f.capture_ready()
    for _ in range(2):
        with pytest.raises(NotImplementedError, match="more tree levels"):
            f.rebuild(torch.from_numpy(B).cuda())
        f.refresh()
        assert f.n_valid == n
    f.rebuild(torch.from_numpy(A).cuda())
    idx, cnt = f.knn(4)
    want, _ = ragged.Forest(torch.from_numpy(A).cuda(), [0, n]).knn(4)
    assert torch.equal(idx, want)


@pytest.mark.parametrize("dim", [2, 3, 4])
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int8, np.int16, np.int32, np.int64, np.uint8, np.uint16,
                                   np.uint32, np.uint64])
def test_segments_at_the_edges_of_block_and_warp(gpu, port, dtype, dim):
    # the largest segments of a warp and of a block and one point beyond, of
    # words of 32 points, with and without ties, leaves of one point included
    rng = np.random.default_rng(dim)
    top = 1.0 if np.dtype(dtype).kind == "f" else float(min(np.iinfo(dtype).max, 10**6))
    for n in (255, 257, 511, 513, 1023, 1025, 1056, 2047, 2048, 2049, 5000):
        for steps in (5, 10**6):  # lattice positions per axis
            P = (np.floor(rng.random((n, dim)) * steps) / steps * top).astype(dtype)
            for leaf in (1, 10):
                _is_reference_tree(gpu.kdtree._build(P, maxleafsize=leaf), port.PortTree(P, maxleafsize=leaf))
    # every split takes a few points off, or divides a run of equal values
    P = (np.exp(-rng.random((1500, dim)) * 12.0) * top).astype(dtype)
    _is_reference_tree(gpu.kdtree._build(P), port.PortTree(P))
    P[rng.random(1500) < 0.6, 0] = dtype(top / 2)
    _is_reference_tree(gpu.kdtree._build(P), port.PortTree(P))
