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
