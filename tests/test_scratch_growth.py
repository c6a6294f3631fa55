"""CPU test of how the backend's device scratch grows, with a counting allocator: a buffer that went into a CUDA graph
is never released, and what is kept stays below what is in use."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "tritium_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include <map>
#include "tb_scratch.h"
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  std::map<void*, size_t> live;
  size_t next = 4096, largest = ~size_t(0);
  const auto alloc = [&](size_t n) -> void* {
    if (n > largest) return nullptr;
    void* p = reinterpret_cast<void*>(next += n);
    live[p] = n;
    return p;
  };
  const auto release = [&](void* p) { live.erase(p); };
  const auto in_use = [&] { size_t sum = 0; for (auto& b : live) sum += b.second; return sum; };
  std::vector<void*> kept;
  tb_scratch s;
  CHECK(tb_scratch_grow(&s, &kept, 10000, alloc, release) && s.cap == 10000);
  void* first = s.ptr;
  CHECK(tb_scratch_grow(&s, &kept, 9999, alloc, release) && s.ptr == first);
  CHECK(tb_scratch_grow(&s, &kept, 20000, alloc, release) && live.size() == 1 && kept.empty());   // no graph: replaced, exact size
  s.recorded = true;
  void* held = s.ptr;
  CHECK(tb_scratch_grow(&s, &kept, 20001, alloc, release));
  CHECK(live.count(held) && kept.size() == 1 && kept[0] == held && s.ptr != held && s.cap == 40000 && !s.recorded);
  s.recorded = true;   // no room: a recorded buffer stays as it is
  void* current = s.ptr;
  largest = 50000;
  CHECK(!tb_scratch_grow(&s, &kept, 60000, alloc, release) && s.ptr == current && s.cap == 40000 && s.recorded);
  CHECK(tb_scratch_grow(&s, &kept, 45000, alloc, release) && s.cap == 45000);   // no room for twice the size
  largest = ~size_t(0);
  for (size_t n = s.cap; n < (size_t(1) << 30); n += n / 16 + 1) {
    s.recorded = true;
    CHECK(tb_scratch_grow(&s, &kept, n, alloc, release));
  }
  CHECK(in_use() < 2 * s.cap + 100000);
  for (void* p : kept) CHECK(live.count(p));
  return 0;
}
"""


def test_scratch_that_a_graph_holds_is_kept(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.check_call([cxx, "-std=c++17", "-Wall", "-I", CSRC, str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")])
    run = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
