"""A tree whose hierarchies could not be made for want of memory refuses
queries until they are made again."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# a process of its own: nothing freed earlier for the library to use again
CHILD = """
import sys
import numpy as np, torch
from pptk_b200 import kdtree
t = kdtree.load(sys.argv[1], 0)
Q = np.load(sys.argv[2])
hold = []
for step in (1 << 30, 1 << 26, 1 << 22):
    while torch.cuda.mem_get_info()[0] > step + (24 << 20):
        try:
            hold.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            break
def raises(f, kind=Exception, words=""):
    try:
        f()
    except kind as e:
        assert words in str(e), e
    else:
        raise AssertionError("no error")
# buckets of one point: a million traversal nodes, 64 MB
raises(lambda: t.set_bucket(1))
for call in (lambda: kdtree.knn(t, Q[:10], 5), lambda: kdtree.rnear(t, Q[:10], 0.1), lambda: kdtree.knn(t, Q[:10], 300)):
    raises(call)
hold.clear()
torch.cuda.empty_cache()
raises(lambda: kdtree.knn(t, Q[:10], 5), ValueError, "incomplete")
t.set_bucket(64)
np.save(sys.argv[3], kdtree.knn(t, Q, 5)[0])
"""


def test_failed_set_bucket_leaves_a_tree_that_refuses_queries(gpu, tmp_path):
    P = np.random.default_rng(0).random((1_000_000, 3), dtype=np.float32)
    t = gpu.kdtree._build(P, maxleafsize=1)
    t.save(tmp_path / "tree")
    np.save(tmp_path / "q.npy", P[:1000])
    subprocess.run([sys.executable, "-c", CHILD, str(tmp_path / "tree"), str(tmp_path / "q.npy"),
                    str(tmp_path / "out.npy")], check=True, timeout=300, cwd=ROOT)
    assert np.array_equal(np.load(tmp_path / "out.npy"), gpu.kdtree.knn(t, P[:1000], 5)[0])
