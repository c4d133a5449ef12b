"""The host worker pool: every chunk of a pass runs once, and an exception of a
chunk reaches the caller after the pass and leaves the pool usable."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..",
                    "symbolic_regression_gpu_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <new>
#include "sr_parallel.hpp"
int main() {
  sr::WorkerPool pool;
  for (int pass = 0; pass < 300; ++pass) {
    const int chunks = 1 + pass % 9;
    const int bad = pass % 3 == 0 ? pass % chunks : -1;
    std::atomic<int> runs[9] = {};
    bool caught = false;
    try {
      pool.run(chunks, 4, [&](int c) {
        runs[c].fetch_add(1);
        if (c == bad) throw std::bad_alloc();
      });
    } catch (const std::bad_alloc &) {
      caught = true;
    }
    if (caught != (bad >= 0)) return 1;
    for (int c = 0; c < chunks; ++c) {
      if (runs[c].load() != 1) return 2;
    }
  }
  std::puts("ok");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_exceptions_reach_the_caller(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout == "ok\n", out
