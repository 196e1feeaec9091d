"""The loop kernels' sums of block visits hold what a long solve adds up."""
import os
import subprocess

from conftest import ROOT

SRC = r"""
#include <cstdio>
#include "visit_sum.hpp"
int main() {
  eikgb::VisitSum s, t;
  eikgb::PassSum p;
  s.clear();
  t.clear();
  p.clear();
  for (int i = 0; i < 3000000; ++i) {
    s.add(3300, 2000, 1500);
    p.add(3300, 2000, 1500);
    if (i % 100000 == 99999) eikgb::take(t, p, false);  // passes of 100,000 visits
  }
  p.add(1, 3, 4);
  eikgb::take(t, p, true);
  printf("%llu %llu %llu %llu ", s.visits, s.slots, s.halo, s.owned);
  printf("%llu %llu %llu %llu", t.visits, t.slots, t.halo, t.owned);
}
"""


def test_sums_pass_32_bits(tmp_path):
    (tmp_path / "sum.cc").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "sci-solver_eikonal_gb300", "csrc"),
                    str(tmp_path / "sum.cc"), "-o", str(tmp_path / "sum")], check=True)
    r = subprocess.run([str(tmp_path / "sum")], capture_output=True, text=True, check=True)
    n = 3000000
    assert list(map(int, r.stdout.split())) == [n, 3300 * n, 2000 * n, 1500 * n, n + 1, 3300 * n + 1, 2000 * n + 3,
                                                1500 * n + 4]


def test_the_loop_kernels_keep_them():
    """No 32-bit counter of a whole solve is left beside them."""
    for name in ("loop2d.cuh", "loop3d.cuh"):
        with open(os.path.join(ROOT, "sci-solver_eikonal_gb300", "csrc", name)) as fh:
            text = fh.read()
        assert "__shared__ VisitSum" in text and "unsigned s_cnt" not in text
