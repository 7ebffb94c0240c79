// Error types, the CUDA-call check and the graph calls used across the host runtime.
#pragma once
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "step_graph.hpp"

namespace tf {

struct CudaError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
struct UnsupportedError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
struct SolverError : std::runtime_error {
  using std::runtime_error::runtime_error;
};

inline void cuda_check(cudaError_t e, const char* what, const char* file, int line) {
  if (e != cudaSuccess)
    throw CudaError(std::string(what) + " failed at " + file + ":" + std::to_string(line) + ": " +
                    cudaGetErrorString(e));
}

// Graph calls of capture_steps.
struct CudaGraphs {
  using Stream = cudaStream_t;
  using Graph = cudaGraph_t;
  using Exec = cudaGraphExec_t;
  static bool begin(Stream s) { return cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess; }
  static bool end(Stream s, Graph* g) { return cudaStreamEndCapture(s, g) == cudaSuccess; }
  static bool instantiate(Exec* x, Graph g) { return cudaGraphInstantiate(x, g, 0) == cudaSuccess; }
  static void destroy(Graph g) { cudaGraphDestroy(g); }
  static void clear_error() { cudaGetLastError(); }
};

}  // namespace tf

#define CU(call) ::tf::cuda_check((call), #call, __FILE__, __LINE__)

namespace tf {

// Makes a device current for a call that launches and whose caller may have
// another one current, and puts that back.
class DeviceGuard {
 public:
  explicit DeviceGuard(int device) {
    CU(cudaGetDevice(&before_));
    if (before_ != device) CU(cudaSetDevice(device));
    else before_ = -1;
  }
  ~DeviceGuard() {
    if (before_ >= 0) cudaSetDevice(before_);
  }
  DeviceGuard(const DeviceGuard&) = delete;
  DeviceGuard& operator=(const DeviceGuard&) = delete;

 private:
  int before_ = -1;
};

}  // namespace tf
