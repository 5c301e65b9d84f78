"""The engine's device arrays when an allocation fails (CPU: the header compiled
against a runtime whose cudaMalloc fails on demand)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = """
#pragma once
#include <cstddef>
#include <cstdlib>
#include <cstring>
typedef int cudaError_t;
typedef void *cudaStream_t;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaMemcpyHostToDevice = 1 };
inline bool g_fail = false;
inline int g_last = 0, g_live = 0;
inline cudaError_t cudaMalloc(void **p, size_t n) {
  if (g_fail) return g_last = cudaErrorMemoryAllocation;
  ++g_live;
  *p = malloc(n);
  return cudaSuccess;
}
inline cudaError_t cudaFree(void *p) { --g_live; free(p); return cudaSuccess; }
inline cudaError_t cudaGetLastError() { int e = g_last; g_last = 0; return e; }
inline const char *cudaGetErrorString(cudaError_t) { return "out of memory"; }
inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, int, cudaStream_t) { memcpy(d, s, n); return 0; }
inline cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { memset(d, v, n); return 0; }
"""

PROGRAM = """
#include "dev_array.hpp"
#include <cstdio>
#define CHECK(c) if (!(c)) { printf("line %d: %s\\n", __LINE__, #c); return 1; }
int main() {
  {
    scb::DevArray<double> a;
    a.alloc(8);
    CHECK(a.p && a.n == 8 && g_live == 1)
    for (size_t want : {16u, 4u}) {  // larger and smaller than what it held
      g_fail = true;
      int code = 0;
      try { a.alloc(want); } catch (const scb::EngineError &e) { code = e.code; }
      CHECK(code == SC_ERR_CUDA)
      CHECK(!a.p && a.n == 0)  // a test for room must not find any
      CHECK(cudaGetLastError() == cudaSuccess)
      a.zero(nullptr);
      g_fail = false;
      a.alloc(want);
      CHECK(a.p && a.n == want)
    }
    a.upload(std::vector<double>(3, 1.5), nullptr);
    CHECK(a.n == 3 && a.p[2] == 1.5)
    a.alloc(0);
    CHECK(!a.p && a.n == 0)
  }
  CHECK(g_live == 0)
  return 0;
}
"""


def test_a_failed_allocation_leaves_an_empty_array(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-I", str(tmp_path), "-I", os.path.join(ROOT, "superconga_b200", "csrc"),
                    str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
