"""The engine's device memory (pg_pool.h) against a device of a given size: what
is not in use can be given back up to a bound, and small blocks are found as
long as they fit."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "process_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include <new>
#include <vector>
#include <cuda_runtime.h>

static size_t g_size = 0, g_used = 0;
static std::map<void*, size_t>* g_live;
extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_used + n > g_size) return cudaErrorMemoryAllocation;
  static char* at = reinterpret_cast<char*>(size_t(1) << 40);   // addresses only, never written
  *p = at;
  at += n;
  (*g_live)[*p] = n; g_used += n;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p) {
  auto it = g_live->find(p);
  if (it == g_live->end()) { std::printf("free of an unknown block\n"); std::exit(1); }
  g_used -= it->second; g_live->erase(it);
  return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
static void ck(cudaError_t e, const char*) { if (e != cudaSuccess) throw std::bad_alloc(); }

#include "pg_pool.h"

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
static bool has(Pool& p, size_t n, void** out = nullptr) {
  try { void* q = p.get(n); if (out) *out = q; return true; } catch (const std::bad_alloc&) { return false; }
}

int main() {
  g_live = new std::map<void*, size_t>;
  const size_t MB = size_t(1) << 20;
  {   // scratch of many calls among small tables that stay: all but 64 MB comes back
    g_size = 4096 * MB;
    Pool p;
    std::vector<void*> scratch;
    for (int i = 0; i < 1000; ++i) { scratch.push_back(p.get(19 * MB / 10)); p.get(300); }
    CHECK(g_used > 1800 * MB);
    for (void* q : scratch) p.put(q);
    void* big = nullptr;
    CHECK(has(p, g_size - 66 * MB, &big));
    p.put(big);
    p.release_all();
    CHECK(g_used == 0 && g_live->empty());
  }
  {   // blocks are distinct and inside what was allocated
    g_size = 4096 * MB;
    Pool p;
    std::map<char*, size_t> mine;
    for (int i = 0; i < 3000; ++i) {
      const size_t n = size_t(1) + size_t(i) * 7919 % (3 * MB);
      char* q = static_cast<char*>(p.get(n));
      auto next = mine.lower_bound(q);
      CHECK(next == mine.end() || q + n <= next->first);
      if (next != mine.begin()) { auto before = std::prev(next); CHECK(before->first + before->second <= q); }
      auto whole = g_live->upper_bound(q);
      CHECK(whole != g_live->begin());
      --whole;
      CHECK(q + n <= static_cast<char*>(whole->first) + whole->second);
      mine[q] = n;
      if (i % 3 == 0) { p.put(mine.begin()->first); mine.erase(mine.begin()); }
    }
    p.release_all();
    CHECK(g_used == 0);
  }
  {   // a nearly full device still gives small blocks
    g_size = 1024 * MB;
    Pool p;
    CHECK(has(p, g_size - MB));
    CHECK(has(p, 256) && has(p, 1000));
    CHECK(!has(p, 4 * MB));
    p.release_all();
    CHECK(g_used == 0);
  }
  return 0;
}
"""

CUDA = Path("/usr/local/cuda/include")


@pytest.mark.skipif(shutil.which("g++") is None or not (CUDA / "cuda_runtime.h").exists(), reason="needs g++ and CUDA headers")
def test_pool(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-I", str(CUDA), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
