// Device arrays of the engine and the errors of its CUDA calls.
#pragma once

#include <cuda_runtime.h>

#include <string>
#include <utility>
#include <vector>

#include "../../include/scb200.h"

namespace scb {

struct EngineError {
  int code;
  std::string msg;
  EngineError(int c, std::string m) : code(c), msg(std::move(m)) {}
};

#define CUDA_TRY(expr)                                                          \
  do {                                                                          \
    cudaError_t _e = (expr);                                                    \
    if (_e != cudaSuccess)                                                      \
      throw scb::EngineError(SC_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(_e)); \
  } while (0)

// n counts what p points to: an allocation that fails leaves an empty array
// (a caller that asks whether the array is large enough allocates again) and
// no error behind for the next launch's check to find.
template <typename T>
struct DevArray {
  T *p = nullptr;
  size_t n = 0;
  DevArray() = default;
  DevArray(const DevArray &) = delete;
  DevArray &operator=(const DevArray &) = delete;
  ~DevArray() { free(); }
  void alloc(size_t count) {
    free();
    if (!count) return;
    const cudaError_t e = cudaMalloc((void **)&p, count * sizeof(T));
    if (e != cudaSuccess) {
      p = nullptr;
      (void)cudaGetLastError();
      throw EngineError(SC_ERR_CUDA, std::string("cudaMalloc: ") + cudaGetErrorString(e));
    }
    n = count;
  }
  void upload(const std::vector<T> &v, cudaStream_t s) {
    alloc(v.size());
    if (n) CUDA_TRY(cudaMemcpyAsync(p, v.data(), n * sizeof(T), cudaMemcpyHostToDevice, s));
  }
  void zero(cudaStream_t s) {
    if (n) CUDA_TRY(cudaMemsetAsync(p, 0, n * sizeof(T), s));
  }
  void free() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
};

}  // namespace scb
