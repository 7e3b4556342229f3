"""The host thread pool of the setup work: an exception of a task reaches the caller."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <new>
#include "mhd_parallel.h"
int main() {
  std::vector<int> hit(1000, 0);
  mhd::parallel_for(1000, [&](int i) { ++hit[i]; });
  for (int h : hit)
    if (h != 1) return 1;
  for (int at : {0, 7, 999}) {
    bool caught = false;
    try {
      mhd::parallel_for(1000, [&](int i) { if (i == at) throw std::bad_alloc(); });
    } catch (const std::bad_alloc &) {
      caught = true;
    }
    if (!caught) return 2;
  }
  mhd::parallel_for(0, [](int) { throw 1; });
  std::puts("ok");
  return 0;
}
"""


def test_tasks_run_once_and_exceptions_reach_the_caller(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(ROOT, "mpcns_mercury_b200", "csrc"),
                           str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)
