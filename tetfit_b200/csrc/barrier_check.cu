// tf_barrier_check: self-check of the bounded grid barrier (grid_barrier.cuh)
// that the persistent CG kernels use.  No reference counterpart: it shows, on
// the GPU, that a barrier wait which can never complete ends with the error
// status instead of a hung launch, and it measures the barrier's latency.
// tf_exchange_check does the same for the exchange of the resident CG kernels
// (cg_resident.cuh), whose sums it also compares.
#include <cuda_runtime.h>

#include <string>

#include "../../include/tetfit.h"
#include "cg_resident.cuh"
#include "grid_barrier.cuh"

namespace tf {
void set_thread_error(const std::string& m);
}

namespace {

// Every block passes `rounds` barriers that wait for `expected` arrivals.
__global__ void barrier_check_kernel(unsigned int* bar, int* err, unsigned int expected, int rounds,
                                     uint64_t limit_ns) {
  for (int k = 0; k < rounds; k++) tf::grid_barrier(bar, err, expected, limit_ns);
}

// The first gridDim.x - absent blocks form the exchange's sums from number
// `first` on, every value a whole number, so that the sums are exact.
constexpr int kExchangeThreads = 128;
__global__ void __launch_bounds__(kExchangeThreads) exchange_check_kernel(uint4* box, int* err, int* wrong,
                                                                          uint32_t first, int rounds, int cluster,
                                                                          int absent, uint64_t limit_ns) {
  __shared__ tf::CgShared sh;
  if (blockIdx.x >= gridDim.x - absent) return;
  if (threadIdx.x == 0) sh.dead = 0;
  tf::CgExchange ex{box, (int)gridDim.x, 0, (int)gridDim.x, err, &sh, first, cluster, limit_ns};
  ex.enter();
  const double n = (double)gridDim.x * kExchangeThreads, id = (double)blockIdx.x * kExchangeThreads + threadIdx.x;
  bool alive = true;
  for (int k = 0; k < rounds && alive; k++) {
    double v[3] = {id, id + k, 1099511627776.0 - id};
    alive = ex.sum<3, true>(v);
    const double s = n * (n - 1) / 2;
    bool ok = v[0] == s && v[1] == s + n * k && v[2] == n * 1099511627776.0 - s;
    double w[1] = {id - k};
    alive = alive && ex.sum<1, false>(w);
    ok = ok && w[0] == s - n * k;
    if (alive && !ok) atomicOr(wrong, 1);
  }
}

int fail(int code, const std::string& m, const char* who = "tf_barrier_check") {
  tf::set_thread_error(std::string(who) + ": " + m);
  return code;
}

}  // namespace

extern "C" int tf_barrier_check(int32_t device, uint32_t blocks, uint32_t expected, uint32_t rounds,
                                uint32_t timeout_us, int32_t* status, double* ms) {
  if (!status) return fail(TF_E_ARG, "status is NULL");
  if (blocks < 1 || expected < 1 || expected > 2 * blocks || rounds < 1 || rounds > 100000 || timeout_us < 1 ||
      timeout_us > 1000000)
    return fail(TF_E_ARG, "blocks >= 1, 1 <= expected <= 2 blocks, 1 <= rounds <= 100000, "
                          "1 <= timeout_us <= 1000000");
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return fail(TF_E_CUDA, cudaGetErrorString(e));
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if ((int)blocks > sms) return fail(TF_E_ARG, "blocks exceeds the SM count (" + std::to_string(sms) + ")");
  unsigned int* words = nullptr;  // bar[0], bar[1], err
  e = cudaMalloc(&words, 3 * sizeof(unsigned int));
  if (e != cudaSuccess) return fail(TF_E_CUDA, cudaGetErrorString(e));
  cudaEvent_t ev[2] = {nullptr, nullptr};
  int32_t flag = 0;
  float t = 0.f;
  e = cudaMemset(words, 0, 3 * sizeof(unsigned int));
  if (e == cudaSuccess) e = cudaEventCreate(&ev[0]);
  if (e == cudaSuccess) e = cudaEventCreate(&ev[1]);
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(128);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaEventRecord(ev[0]);
    e = cudaLaunchKernelEx(&cfg, barrier_check_kernel, words, (int*)(words + 2), expected, (int)rounds,
                           (uint64_t)timeout_us * 1000ull);
    cudaEventRecord(ev[1]);
  }
  if (e == cudaSuccess) e = cudaEventSynchronize(ev[1]);
  if (e == cudaSuccess) e = cudaEventElapsedTime(&t, ev[0], ev[1]);
  if (e == cudaSuccess) e = cudaMemcpy(&flag, words + 2, sizeof(flag), cudaMemcpyDeviceToHost);
  for (cudaEvent_t x : ev)
    if (x) cudaEventDestroy(x);
  cudaFree(words);
  if (e != cudaSuccess) return fail(TF_E_CUDA, cudaGetErrorString(e));
  *status = flag;
  if (ms) *ms = t;
  return TF_OK;
}

extern "C" int tf_exchange_check(int32_t device, uint32_t blocks, uint32_t cluster, uint32_t first, uint32_t rounds,
                                 uint32_t absent, uint32_t timeout_us, int32_t* status, double* ms) {
  auto bad = [](int code, const std::string& m) { return fail(code, m, "tf_exchange_check"); };
  if (!status) return bad(TF_E_ARG, "status is NULL");
  const bool pow2 = cluster > 0 && cluster <= tf::kCgCluster && (cluster & (cluster - 1)) == 0;
  if (blocks < 1 || !pow2 || blocks % cluster || (cluster > 1 && blocks / cluster > 32) || first < 1 || rounds < 1 ||
      rounds > 100000 || absent >= blocks || absent % cluster || timeout_us < 1 || timeout_us > 1000000)
    return bad(TF_E_ARG, "cluster 1, 2, 4, 8 or 16, blocks >= 1 a multiple of it and at most 32 clusters, first >= 1, "
                         "1 <= rounds <= 100000, absent < blocks whole clusters, 1 <= timeout_us <= 1000000");
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return bad(TF_E_CUDA, cudaGetErrorString(e));
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if ((int)blocks > sms || blocks > 32 * tf::kCgChunks)
    return bad(TF_E_ARG, "blocks exceeds the SM count (" + std::to_string(sms) + ")");
  const size_t boxes = (size_t)2 * tf::kCgVals * blocks * blocks * sizeof(uint4);
  char* work = nullptr;  // boxes, then the error flag and the wrong-sum flag
  e = cudaMalloc(&work, boxes + 2 * sizeof(int));
  if (e != cudaSuccess) return bad(TF_E_CUDA, cudaGetErrorString(e));
  cudaEvent_t ev[2] = {nullptr, nullptr};
  int32_t flags[2] = {0, 0};
  float t = 0.f;
  e = cudaMemset(work, 0, boxes + 2 * sizeof(int));
  if (e == cudaSuccess) e = cudaEventCreate(&ev[0]);
  if (e == cudaSuccess) e = cudaEventCreate(&ev[1]);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(exchange_check_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kExchangeThreads);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    int* words = (int*)(work + boxes);
    cudaEventRecord(ev[0]);
    e = cudaLaunchKernelEx(&cfg, exchange_check_kernel, (uint4*)work, words, words + 1, first, (int)rounds, (int)cluster,
                           (int)absent, (uint64_t)timeout_us * 1000ull);
    cudaEventRecord(ev[1]);
  }
  if (e == cudaSuccess) e = cudaEventSynchronize(ev[1]);
  if (e == cudaSuccess) e = cudaEventElapsedTime(&t, ev[0], ev[1]);
  if (e == cudaSuccess) e = cudaMemcpy(flags, work + boxes, sizeof(flags), cudaMemcpyDeviceToHost);
  for (cudaEvent_t x : ev)
    if (x) cudaEventDestroy(x);
  cudaFree(work);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return bad(TF_E_CUDA, cudaGetErrorString(e));
  }
  *status = flags[0] | flags[1];
  if (ms) *ms = t;
  return TF_OK;
}
