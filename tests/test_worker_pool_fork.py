"""A pool inherited through fork(): the child has none of its threads, so
destroying it there may not wait for them (an Evaluator collected, or left to the
interpreter's exit, in a forked process)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..",
                    "symbolic_regression_gpu_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <sys/wait.h>
#include <unistd.h>
#include "sr_parallel.hpp"
int main(int argc, char **argv) {
  auto *pool = new sr::WorkerPool;
  std::atomic<int> runs{0};
  pool->run(8, 4, [&](int) { runs.fetch_add(1); });
  if (argc > 1) usleep(50000);  // the workers are asleep when the process forks
  const pid_t child = fork();
  if (child == 0) {
    alarm(10);
    delete pool;
    _exit(0);
  }
  int status = 0;
  if (waitpid(child, &status, 0) != child || status != 0) return 1;
  pool->run(8, 4, [&](int) { runs.fetch_add(1); });  // the parent's is as before
  delete pool;
  if (runs.load() != 16) return 2;
  std::puts("ok");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
@pytest.mark.parametrize("args", [[], ["asleep"]])
def test_a_forked_process_destroys_its_copy(tmp_path, args):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)] + args, capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout == "ok\n", out
