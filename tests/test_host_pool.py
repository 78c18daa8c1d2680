"""Host tasks shared out over threads (csrc/host_pool.h): every task once, and
an exception of one reaches the caller instead of ending the process."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import PKG_DIR

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <new>
#include <vector>
#include "host_pool.h"

int main() {
  for (size_t extra : {0, 1, 7}) {
    for (size_t count : {0, 1, 5, 1000}) {
      std::vector<std::atomic<int>> done(count);
      perm::for_each_shared(count, extra, [&](size_t i) { done[i]++; });
      for (auto& d : done)
        if (d != 1) return 1;
      std::atomic<size_t> begun{0};
      bool caught = false;
      try {
        perm::for_each_shared(count, extra, [&](size_t) {
          begun++;
          throw std::bad_alloc();
        });
      } catch (const std::bad_alloc&) {
        caught = true;
      }
      // each thread ends at its first exception
      if (caught != (count > 0) || begun > extra + 1) return 2;
    }
  }
  puts("ok");
}
"""


def test_exceptions_reach_the_caller(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src = tmp_path / "pool.cpp"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", f"-I{PKG_DIR / 'csrc'}", str(src), "-o", str(tmp_path / "pool")],
                   check=True, timeout=120)
    r = subprocess.run([str(tmp_path / "pool")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stderr)
