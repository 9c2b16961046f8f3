"""The choices that the walks make by sizes and settings (csrc/rules.cuh),
compiled for the host."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    """evaluate(expressions): their integer values."""
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    tmp = tmp_path_factory.mktemp("rules")

    def run(expressions):
        body = "".join(f'  printf("%lld\\n", (long long)({e}));\n' for e in expressions)
        (tmp / "t.cpp").write_text('#include <cstdio>\n#include "rules.cuh"\nusing namespace pptkg;\n'
                                   f"int main() {{\n{body}}}\n")
        subprocess.check_call([cxx, "-std=c++17", "-I", os.path.join(ROOT, "pptk_b200", "csrc"), str(tmp / "t.cpp"),
                               "-o", str(tmp / "t")])
        return [int(v) for v in subprocess.check_output([str(tmp / "t")]).split()]

    return run


def test_warm_window(evaluate):
    # a setting of 1 is the k-position start for every batch; others are one
    # wider for short lists of scattered queries
    M = 1_000_000
    assert evaluate([f"warm_window(1, {nv}, {m}, {k})" for nv, m in ((M, M), (20 * M, 10), (20 * M, M))
                     for k in (4, 16, 32)]) == [1] * 9
    assert evaluate([f"warm_window({w}, {20 * M}, {M}, {k})" for w in (2, 3, 8) for k in (4, 16, 32)]) == \
        [3, 3, 2, 4, 4, 3, 9, 9, 8]
    assert evaluate([f"warm_window({w}, {M}, {M}, 16)" for w in (1, 2, 8)]) == [1, 2, 8]


def _by_warp(nv, m, k, f64=False, a="normals", order="tree", span=1024):
    return f"by_warp({nv}, {m}, {k}, {int(f64)}, Answer::{a}, BatchOrder::{order}, {span})"


def test_by_warp_takes_the_faster_walk(evaluate):
    # sizes at which one walk was measured clearly faster (packets, warps in us)
    M = 1_000_000
    measured = [
        (_by_warp(50, 65_000, 32), 0), (_by_warp(50, 65_000, 64, a="both"), 0), (_by_warp(200, 67_200, 16, a="knn"), 0),
        (_by_warp(200, 67_200, 32, a="both"), 0), (_by_warp(200, 67_200, 64, a="both"), 1),
        (_by_warp(60_000, 60_000, 16, a="knn"), 1), (_by_warp(60_000, 60_000, 32, a="both"), 1),
        (_by_warp(5_000, 60_000, 32, a="both"), 1), (_by_warp(5_000, 300_000, 16, a="both"), 0),
        (_by_warp(1_000, 60_000, 16, f64=True, a="knn"), 1), (_by_warp(1_000, 60_000, 16, f64=True, a="both"), 0),
        (_by_warp(3_000, 3_000, 16), 1), (_by_warp(20_000, 20_000, 4), 0), (_by_warp(40_000, 40_000, 4), 0),
        (_by_warp(40_000, 40_000, 16), 0), (_by_warp(65_000, 65_000, 8), 0), (_by_warp(65_000, 65_000, 16), 0),
        (_by_warp(10_000, 10_000, 32), 1), (_by_warp(65_000, 65_000, 32), 0), (_by_warp(65_000, 65_000, 64), 1),
        (_by_warp(65_000, 65_000, 8, a="knn"), 0), (_by_warp(65_000, 65_000, 32, a="knn"), 1),
        (_by_warp(20 * M, 20 * M, 32, a="knn"), 0), (_by_warp(20 * M, 20 * M, 16), 0),
        (_by_warp(65_000, 65_000, 4, f64=True), 0), (_by_warp(10_000, 10_000, 16, f64=True), 1),
        (_by_warp(300_000, 300_000, 32, f64=True), 1),
        (_by_warp(20 * M, 10, 16, a="knn", order="points"), 1), (_by_warp(65_000, 40_000, 4, a="knn", order="points"), 1),
        (_by_warp(20 * M, 500_000, 1, a="knn", order="points"), 0),
        (_by_warp(20 * M, 500_000, 8, a="knn", order="points"), 0),
        (_by_warp(20 * M, 140_000, 1, a="knn", order="points"), 1),
        (_by_warp(2 * M, 200_000, 8, a="knn", order="points"), 0),
        (_by_warp(20 * M, M, 32, a="knn", order="points"), 1), (_by_warp(20 * M, M, 16, a="knn", order="points"), 0),
        (_by_warp(2 * M, 140_000, 8, f64=True, a="knn", order="points"), 1),
        (_by_warp(2 * M, 500_000, 8, f64=True, a="knn", order="points"), 0),
        (_by_warp(2 * M, 40_000, 8, order="rows"), 1), (_by_warp(2 * M, 100_000, 8, order="rows"), 0),
        (_by_warp(20 * M, 140_000, 8, order="rows"), 1), (_by_warp(20 * M, 200_000, 8, order="rows"), 0),
        (_by_warp(2 * M, 500_000, 16, f64=True, order="rows"), 0),
    ]
    assert evaluate([e for e, _ in measured]) == [w for _, w in measured]


def test_by_warp_settings(evaluate):
    batches = [(nv, m, k, f64, a, order) for nv in (100, 60_000, 20_000_000) for m in (1, 3_000, 70_000, 3_000_000)
               for k in (1, 16, 32, 64) for f64 in (False, True) for a in ("knn", "both", "normals")
               for order in ("tree", "rows", "points")]
    assert not any(evaluate([_by_warp(*b, span=-1) for b in batches]))
    assert all(evaluate([_by_warp(*b, span=0) for b in batches]))
    fewer, more = (evaluate([_by_warp(*b, span=s) for b in batches]) for s in (4096, 64))
    line = evaluate([_by_warp(*b) for b in batches])
    assert all(a <= b <= c for a, b, c in zip(fewer, line, more)) and sum(fewer) < sum(line) < sum(more)
    # between the packets' lists and the heaps there is one walk, beyond them none of the two
    assert all(evaluate([_by_warp(nv, m, k, span=s) for nv, m in ((100, 5), (10**7, 10**7)) for k in (65, 256)
                         for s in (-1, 0, 1024)]))
    assert not any(evaluate([_by_warp(100, 5, 257, span=s) for s in (-1, 0, 1024)]))
