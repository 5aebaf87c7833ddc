"""run_team (csrc/ms_team.h) when threads cannot be started.

A harness compiled here makes every allocation of a thread's state fail in
turn, as an exhausted host does, and checks that each share of the work still
runs exactly once and that nothing is thrown or aborted."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include "ms_team.h"
static std::atomic<int> left{1 << 30};
void* operator new(std::size_t n) {
  if (left-- <= 0) throw std::bad_alloc();
  if (void* p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main() {
  for (int shares = 1; shares <= 8; ++shares)
    for (int allowed = 0; allowed <= 9; ++allowed) {
      std::atomic<int> done[8] = {};
      left = allowed == 9 ? 1 << 30 : allowed;
      ms::run_team<8>(shares, [&](std::size_t t) { ++done[t]; });
      left = 1 << 30;
      for (int t = 0; t < 8; ++t)
        if (done[t] != (t < shares)) return std::printf("%d shares, %d allocations: share %d ran %d times\n", shares, allowed, t, (int)done[t]), 1;
    }
  return 0;
}
"""


def test_every_share_runs_once(tmp_path):
    src, exe = tmp_path / "team.cpp", tmp_path / "team"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(ROOT, "cudamultislice_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
