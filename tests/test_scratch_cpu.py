"""Working memory of a device build (scratch.hpp), with an allocator on the host: what a
build holds stays near what it asked for, and a build whose arrays fit is not refused."""
import os
import subprocess

from conftest import ROOT

SRC = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include "scratch.hpp"
static std::map<void*, size_t> live;
static size_t held = 0, most = 0, limit = 0;
static uintptr_t next_address = 4096;
struct Fake {  // addresses only: nothing is written
  bool get(void** p, size_t bytes) {
    if (held + bytes > limit) return false;
    *p = (void*)next_address;
    next_address += (bytes + 4096) / 256 * 256;
    live[*p] = bytes;
    held += bytes;
    if (held > most) most = held;
    return true;
  }
  void put(void* p) { held -= live.at(p); live.erase(p); }
};
// argv: the limit, then the arrays' sizes
int main(int argc, char** argv) {
  limit = strtoull(argv[1], 0, 10);
  size_t refused = 0;
  {
    eikgb::ScratchPieces<Fake> s;
    std::map<uintptr_t, size_t> got;
    for (int i = 2; i < argc; ++i) {
      const size_t n = strtoull(argv[i], 0, 10);
      const uintptr_t p = (uintptr_t)s.get(n);
      if (!p) { ++refused; continue; }
      auto next = got.lower_bound(p);
      if (p % 256 || (next != got.end() && p + n > next->first)) return 2;
      if (next != got.begin() && std::prev(next)->first + std::prev(next)->second > p) return 3;
      bool inside = false;
      for (auto& l : live) inside = inside || ((uintptr_t)l.first <= p && p + n <= (uintptr_t)l.first + l.second);
      if (!inside) return 4;
      got[p] = n;
    }
  }
  if (held || !live.empty()) return 5;
  printf("%zu %zu\n", most, refused);
}
"""
MB = 1 << 20


def _program(tmp_path):
    src, exe = tmp_path / "scratch.cc", tmp_path / "scratch"
    src.write_text(SRC)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-I",
                        os.path.join(ROOT, "sci-solver_eikonal_gb300", "csrc"), str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return lambda limit, sizes: tuple(map(int, subprocess.run(
        [str(exe), str(limit), *map(str, sizes)], capture_output=True, text=True, check=True).stdout.split()))


def test_working_memory(tmp_path):
    run = _program(tmp_path)
    small = [1, 255, 256, 257, 4 * 36000, 8 * 36000, 4 * 200000] * 6
    mesh = [4 * MB, 3 * MB, 900 * MB, 1800 * MB, 12, 5 * MB, 1800 * MB, 15 * MB, 900 * MB, 1, 40 * MB, 16 * MB]
    for sizes in (small, mesh, mesh + small, mesh[::-1], [4 * 10 ** 9, 10, 8 * MB, 10]):
        asked = sum((n + 255) // 256 * 256 for n in sizes)
        most, refused = run(1 << 40, sizes)
        assert refused == 0 and most <= asked + 48 * MB, (most / MB, asked / MB)
        # a little more memory than the arrays need
        assert run(asked + 48 * MB, sizes)[1] == 0
        # none to spare for a shared piece: the array alone is asked for
        assert run(sizes[0] + 255, sizes[:1])[1] == 0
    # a 33^3 cube's build takes a few allocations, one that cannot be had is refused
    assert run(1 << 40, small)[0] == 8 * MB
    assert run(100 * MB, [60 * MB, 60 * MB, 30 * MB])[1] == 1
