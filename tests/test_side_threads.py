"""The host threads that solve several matrices of a plan side by side: an
exception in one of them comes out as a status, and all of them end."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "genericlinearalgebra.jl_gb300", "csrc")

SOURCE = r"""
#include <atomic>
#include <cstdio>
#include <stdexcept>
#include "side_threads.h"
using namespace gla;
// eight threads take 100 items; item `bad` throws; the first status is kept
static int run(int bad, int kind, int* done) {
  std::atomic<int> next{0}, status{0}, n{0};
  auto work = [&](int) {
    int rc = 0;
    for (int c; !rc && !status.load() && (c = next.fetch_add(1)) < 100;)
      rc = guarded([&]() -> int {
        if (c == bad && kind == 0) throw std::bad_alloc();
        if (c == bad && kind == 1) throw std::runtime_error("x");
        if (c == bad && kind == 2) throw 7;
        if (c == bad) return -5;
        n++;
        return 0;
      });
    int none = 0;
    if (rc) status.compare_exchange_strong(none, rc);
  };
  on_threads(8, work);
  *done = n;
  return status;
}
int main() {
  int done = 0;
  for (int bad : {0, 3, 99}) {
    const int want[] = {kStatusNoMemory, kStatusUnknown, kStatusUnknown, -5};
    for (int kind = 0; kind < 4; kind++)
      if (run(bad, kind, &done) != want[kind] || done > 99) return 1;
  }
  if (run(-1, 0, &done) != 0 || done != 100) return 2;
  int one = 0;
  on_threads(1, [&](int t) { one += 1 + t; });
  return one == 1 && kStatusNoMemory == -1002 ? 0 : 3;
}
"""


def test_exceptions_become_statuses(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SOURCE)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", str(exe), str(src)],
                       capture_output=True, text=True)
    if r.returncode == 127:
        pytest.skip("no g++")
    assert r.returncode == 0, r.stderr
    for _ in range(20):
        assert subprocess.run([str(exe)], timeout=60).returncode == 0
