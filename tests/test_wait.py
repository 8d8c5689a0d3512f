"""Counted arrivals (pg_wait.h) over the wrap of the count: with n CTAs, no one
passes the wait of a step before all n have arrived there, and all pass then."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "process_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "pg_wait.h"
int main() {
  const uint32_t ns[] = {1, 2, 7, 608}, firsts[] = {0u, 0xffffffffu, 0xfffffff0u, 0x7ffffff0u};
  for (uint32_t n : ns)
    for (uint32_t first : firsts)          // the count before the first arrival
      for (uint32_t step = 0; step < 40; ++step) {
        const uint32_t target = first + (step + 1) * n;
        for (uint32_t k = 0; k <= 2 * n; ++k)   // k arrivals at this step and the next
          if (pg::arrived(first + step * n + k, target) != (k >= n)) { std::printf("%u %u %u %u\n", n, first, step, k); return 1; }
      }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_arrivals_over_the_wrap(tmp_path):
    src, exe = tmp_path / "wait.cpp", tmp_path / "wait"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
