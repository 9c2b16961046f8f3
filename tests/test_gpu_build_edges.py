"""Builds and in-place rebuilds at the edges of their capacities.  Every
accepted tree must be the reference's (from the CPU oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
