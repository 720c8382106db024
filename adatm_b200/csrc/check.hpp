// check.hpp -- the library's exceptions and the check of CUDA calls.
#pragma once

#include <cuda_runtime.h>

#include <cstdio>
#include <stdexcept>
#include <string>

namespace adatm {

struct CudaError : std::runtime_error {
  explicit CudaError(const std::string &s) : std::runtime_error(s) {}
};
struct BadInput : std::runtime_error {
  explicit BadInput(const std::string &s) : std::runtime_error(s) {}
};
struct NoMemory : std::runtime_error {
  explicit NoMemory(const std::string &s) : std::runtime_error(s) {}
};

inline void check_cuda(cudaError_t e, const char *what, const char *file, int line) {
  if (e == cudaSuccess) return;
  char buf[512];
  snprintf(buf, sizeof(buf), "%s failed at %s:%d: %s", what, file, line, cudaGetErrorString(e));
  if (e == cudaErrorMemoryAllocation) throw NoMemory(buf);
  throw CudaError(buf);
}

#define ADATM_CUDA(call) ::adatm::check_cuda((call), #call, __FILE__, __LINE__)
#define ADATM_LAUNCH() ::adatm::check_cuda(cudaGetLastError(), "kernel launch", __FILE__, __LINE__)

}  // namespace adatm
