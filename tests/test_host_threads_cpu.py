"""The partition's threads: where the system gives none, the halves run one behind the
other and the labels are the same."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r"""
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <pthread.h>
#include "setup.hpp"
#ifdef NO_THREADS
// in place of the system's: every thread is refused
extern "C" int pthread_create(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*) noexcept { return EAGAIN; }
#endif
int main(int, char** argv) {
  const int nv = atoi(argv[1]);
  std::vector<float> x(3 * (size_t)nv);
  unsigned r = 1;
  for (float& v : x) v = (float)((r = r * 1664525u + 1013904223u) >> 20);  // equal coordinates among them
  std::vector<int> labels;
  eikgb::partition_rcb(nv, x.data(), nv / 64 + 1, labels);
  fwrite(labels.data(), sizeof(int), labels.size(), stdout);
}
"""


@pytest.fixture(scope="module")
def programs(tmp_path_factory):
    d, csrc = tmp_path_factory.mktemp("threads"), os.path.join(ROOT, "sci-solver_eikonal_gb300", "csrc")
    (d / "main.cc").write_text(SRC)
    cxx = ["g++", "-std=c++17", "-ffp-contract=off", "-I", csrc]
    subprocess.run([*cxx, "-c", os.path.join(csrc, "setup.cpp"), "-o", str(d / "setup.o")], check=True)
    for name, flag in (("with", []), ("without", ["-DNO_THREADS"])):
        subprocess.run([*cxx, *flag, str(d / "main.cc"), str(d / "setup.o"), "-o", str(d / name), "-lpthread"], check=True)
    return d


@pytest.mark.parametrize("nv", [4095, 4096, 5000, 40000])
def test_partition_without_threads(programs, nv):
    out = []
    for name in ("with", "without"):
        r = subprocess.run([str(programs / name), str(nv)], capture_output=True)
        assert r.returncode == 0, r.stderr
        out.append(np.frombuffer(r.stdout, np.int32))
    assert out[0].size == nv and np.array_equal(out[0], out[1])
    assert set(out[0]) == set(range(nv // 64 + 1))
