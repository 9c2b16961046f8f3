"""The build's intermediate nodes hold the largest record, cloud, level and
position that a build can have (compiled for the host)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <climits>
#include <initializer_list>
#include "build_nodes.cuh"
using namespace pptkg;
template <typename N> bool holds(int parent, int side, int b, int e) {
  N n;
  n.parent = parent;
  n.side = side;
  n.b = b;
  n.e = e;
  return n.parent == parent && n.side == side && n.b == b && n.e == e;
}
int main() {
  // a tree over the most points, 2^30 - 65, has up to 2^31 - 131 records
  const int last = INT_MAX - 131, most = (1 << 30) - 65;
  bool ok = true;
  for (int parent : {0, 1, (1 << 30) - 1, 1 << 30, (1 << 30) + 1, last, -1, -1 - most})
    for (int side = 0; side < 2; side++)
      ok = ok && holds<Small<float, 3>>(parent, side, most - 1, most) &&
           holds<Entry<float, 3>>(parent, side, 1023, 1024) && holds<Entry<double, 4>>(parent, side, 0, 1);
  Small<double, 2> s;
  s.lvl = 16384;
  return ok && s.lvl == 16384 ? 0 : 1;
}
"""


def test_links_hold_every_record(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(SOURCE)
    exe = tmp_path / "t"
    subprocess.check_call([cxx, "-std=c++17", "-I", os.path.join(ROOT, "pptk_b200", "csrc"), str(tmp_path / "t.cpp"),
                           "-o", str(exe)])
    assert subprocess.call([str(exe)]) == 0
