"""Row numbers and masks held in CUDA tensors give what the same numpy
arrays give: every integer type, negative rows, empty and 0-d forms, strided
views, and the same errors for what is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forms(n):
    import torch
    rng = np.random.default_rng(3)
    rows = rng.integers(-n, n, 500)
    yield torch.from_numpy(rows)
    yield torch.from_numpy(rows.astype(np.int32))
    yield torch.from_numpy(rng.integers(-128, 128, 64).astype(np.int8))
    yield torch.from_numpy(rng.integers(-n, n, 64).astype(np.int16))
    yield torch.from_numpy(rng.integers(0, 256, 64).astype(np.uint8))
    yield torch.from_numpy(rng.random(n) < 0.1)
    yield torch.zeros(0, dtype=torch.int64)
    yield torch.tensor(-1)
    yield torch.from_numpy(rows)[::3]


def test_device_rows_equal_host_rows(gpu):
    import torch
    P = np.random.default_rng(1).random((3_000, 3), dtype=np.float32)
    t, tg = gpu.kdtree._build(P), gpu.kdtree._build(torch.from_numpy(P).cuda())
    for rows in _forms(len(P)):
        want, got = gpu.kdtree.knn(t, rows.numpy(), 5), gpu.kdtree.knn(tg, rows.cuda(), 5)
        assert all(g.is_cuda and np.array_equal(g.cpu().numpy(), w) for g, w in zip(got, want)), rows.dtype
        want, got = gpu.kdtree.rnear(t, rows.numpy(), 0.1), gpu.kdtree.rnear(tg, rows.cuda(), 0.1)
        assert all(np.array_equal(g.cpu().numpy(), w) for g, w in zip(got, want)), rows.dtype
        want = gpu.estimate_normals(P, 6, np.inf, subsample=rows.numpy(), verbose=False)
        got = gpu.estimate_normals(torch.from_numpy(P).cuda(), 6, np.inf, subsample=rows.cuda(), verbose=False)
        assert np.array_equal(got.cpu().numpy(), want), rows.dtype


@pytest.mark.parametrize("rows", [[0, 3_000], [-3_001], [0.5], [True, False]])
def test_refused_rows_raise_as_host_rows_do(gpu, rows):
    import torch
    P = np.random.default_rng(1).random((3_000, 3), dtype=np.float32)
    t = gpu.kdtree._build(P)
    with pytest.raises(Exception) as host:
        gpu.kdtree.knn(t, np.asarray(rows), 5)
    with pytest.raises(type(host.value)) as device:
        gpu.kdtree.knn(t, torch.from_numpy(np.asarray(rows)).cuda(), 5)
    assert str(device.value) == str(host.value)
