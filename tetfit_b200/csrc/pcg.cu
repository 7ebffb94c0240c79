// Standalone Jacobi-PCG solve through the C ABI: the persistent cooperative
// kernel of the gfdtd path (tet_cg, tet_kernels.cu) applied to a caller's CSR
// system in device memory (ConjugateGradientSolver.hpp:52-129 semantics:
// Jacobi preconditioner, ||r||/||r0|| <= tol or ||r|| <= tol ||b||, hard
// iteration limit).
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "../../include/tetfit.h"
#include "tet_kernels.cuh"

namespace tf {
cudaError_t pcg_launch_solve(DevPtrs d, int blocks, int device, cudaStream_t st);
size_t pcg_box_bytes(int device);
bool pcg_resident_fits(int64_t n, int device);
template <typename T>
int tet_cg_blocks(int device);
void set_thread_error(const std::string& m);
}  // namespace tf

using tf::DevPtrs;

namespace {

int check_args(const tf_pcg_args* a) {
  if (!a || a->n <= 0 || !a->row_ptr || !a->col || !a->val || !a->b || !a->x || a->maxiter < 0 ||
      !(a->tol >= 0)) {
    tf::set_thread_error("tf_pcg_solve: missing pointer or invalid size / tolerance / iteration limit");
    return TF_E_ARG;
  }
  return TF_OK;
}

// The call's results, in the layout of the work space's head.
struct Head {
  double resid;
  int64_t iters, limit, err;  // int32 values in 8-byte slots
  int64_t step;
  unsigned int gbar[2];
};
constexpr size_t kHeadDoubles = sizeof(Head) / 8;
static_assert(sizeof(Head) == 48, "six 8-byte slots");

// work layout: head, part_a [blocks], part_b [3 blocks], boxes, then pre, r, p,
// q [n each] from a 256-byte boundary (the resident kernel's pairs are pre and r)
size_t vector_offset(int blocks, size_t box_bytes) {
  return (kHeadDoubles + 4 * (size_t)blocks + box_bytes / 8 + 31) / 32 * 32;
}
size_t work_doubles(int64_t n, int blocks, size_t box_bytes) {
  return vector_offset(blocks, box_bytes) + 4 * (size_t)n;
}

DevPtrs make_ptrs(const tf_pcg_args* a, double* work, int blocks, size_t box_bytes) {
  const int64_t n = a->n;
  DevPtrs d;
  Head* h = (Head*)work;
  d.nfree = a->n;
  d.a_ptr = a->row_ptr;
  d.a_col = a->col;
  d.a_val = a->val;
  d.rhs = (void*)a->b;
  d.x = a->x;
  d.cg_resid = &h->resid;
  d.cg_iters = (int32_t*)&h->iters;
  d.cg_limit = (int32_t*)&h->limit;
  d.err = (int*)&h->err;
  d.step = (int*)&h->step;
  d.gbar = h->gbar;
  d.part_a = work + kHeadDoubles;
  d.part_b = d.part_a + blocks;
  double* v = work + vector_offset(blocks, box_bytes);
  d.box = box_bytes ? (uint4*)(v - box_bytes / 8) : nullptr;  // box_bytes is a multiple of 16
  d.jac = v;
  d.r = v + n;
  d.p = v + 2 * n;
  d.q = v + 3 * n;
  d.tol = a->tol;
  d.cg_maxiter = a->maxiter > 0 ? a->maxiter : 100;
  d.cg_criterion = a->criterion;
  return d;
}

int finish(cudaStream_t st, const double* work, int32_t* iters, double* resid) {
  Head h;
  cudaError_t e = cudaMemcpyAsync(&h, work, sizeof(h), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    tf::set_thread_error(std::string("tf_pcg_solve: ") + cudaGetErrorString(e));
    return TF_E_CUDA;
  }
  if ((int32_t)h.err) {
    tf::set_thread_error("tf_pcg_solve: a wait of the CG kernel ran out of time; no valid result");
    return TF_E_CUDA;
  }
  if (iters) *iters = (int32_t)h.iters;
  if (resid) *resid = h.resid;
  if ((int32_t)h.limit) {
    tf::set_thread_error("tf_pcg_solve: iteration limit reached before the tolerance");
    return TF_E_SOLVER;
  }
  return TF_OK;
}

constexpr int kNoAllocMaxN = 1 << 18;    // 262,144 unknowns
constexpr int kNoAllocMaxBlocks = 1024;  // reduction slots for the cooperative grid

// Head, reduction slots, boxes and four vectors of kNoAllocMaxN doubles.  The
// resident kernel, which every size the array takes goes to, uses two of the
// four vectors: its boxes (3.5 MB on 148 SMs) fit the others' room.
__device__ __align__(256) double g_pcg_scratch[4 * (size_t)kNoAllocMaxN + 4 * kNoAllocMaxBlocks + 8];

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
double* g_scratch_addr[kMaxDevices] = {nullptr};
int g_scratch_blocks[kMaxDevices] = {0};
// held by the call that uses a device's array, from its launch to its results
std::mutex g_scratch_use[kMaxDevices];

// Device address of the array on `device` (which must be current), looked
// up once per device: in host code the symbol name is only a host-side handle.
// The address is kept for the life of the process; cudaDeviceReset reloads
// the module and may move the array, so it is not supported while this
// library is loaded.
int scratch_for(int device, double** addr, int* blocks) {
  if (device < 0 || device >= kMaxDevices) {
    tf::set_thread_error("tf_pcg_solve_noalloc: device ordinal out of range");
    return TF_E_ARG;
  }
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  if (!g_scratch_addr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_pcg_scratch);
    if (e != cudaSuccess) {
      tf::set_thread_error(std::string("tf_pcg_solve_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
      return TF_E_CUDA;
    }
    int b = tf::tet_cg_blocks<double>(device);
    if (b < 1) {
      tf::set_thread_error("tf_pcg_solve_noalloc: no co-resident blocks for the cooperative kernel");
      return TF_E_CUDA;
    }
    g_scratch_blocks[device] = b < kNoAllocMaxBlocks ? b : kNoAllocMaxBlocks;
    g_scratch_addr[device] = (double*)p;
  }
  *addr = g_scratch_addr[device];
  *blocks = g_scratch_blocks[device];
  return TF_OK;
}

// boxes of a solve of n unknowns: none where the resident kernel does not take it
size_t boxes_for(int64_t n, int device) { return tf::pcg_resident_fits(n, device) ? tf::pcg_box_bytes(device) : 0; }

// whether the array holds a solve's work space (the resident kernel needs two
// of the four vectors)
bool scratch_holds(int64_t n, int blocks, size_t box_bytes) {
  return n <= kNoAllocMaxN && vector_offset(blocks, box_bytes) + (box_bytes ? 2 : 4) * (size_t)n <=
                                  sizeof(g_pcg_scratch) / sizeof(double);
}

int solve(const tf_pcg_args* a, double* work, int blocks, size_t box_bytes, int32_t* iters, double* rel_resid) {
  cudaStream_t st = (cudaStream_t)a->stream;
  // Every value the kernels read is written earlier in the same call (the
  // head's counters and the boxes are cleared by pcg_launch_solve).
  const cudaError_t e = tf::pcg_launch_solve(make_ptrs(a, work, blocks, box_bytes), blocks, a->device, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    tf::set_thread_error(std::string("tf_pcg_solve: ") + cudaGetErrorString(e));
    return TF_E_CUDA;
  }
  return finish(st, work, iters, rel_resid);
}

}  // namespace

extern "C" int tf_pcg_solve(const tf_pcg_args* a, int32_t* iters, double* rel_resid) {
  int rc = check_args(a);
  if (rc) return rc;
  cudaError_t e = cudaSetDevice(a->device);
  if (e != cudaSuccess) {
    tf::set_thread_error(std::string("tf_pcg_solve: ") + cudaGetErrorString(e));
    return TF_E_CUDA;
  }
  // the file-scope work space below when it is large enough and no other call
  // is using it, else a work space of the call's own (cudaMalloc and cudaFree
  // cost a few hundred microseconds and can synchronize the device)
  double* work = nullptr;
  int blocks = 0;
  const size_t box_bytes = boxes_for(a->n, a->device);
  if (a->device < kMaxDevices && scratch_for(a->device, &work, &blocks) == TF_OK &&
      scratch_holds(a->n, blocks, box_bytes)) {
    std::unique_lock<std::mutex> use(g_scratch_use[a->device], std::try_to_lock);
    if (use.owns_lock()) return solve(a, work, blocks, box_bytes, iters, rel_resid);
  }
  blocks = tf::tet_cg_blocks<double>(a->device);
  e = cudaMalloc(&work, work_doubles(a->n, blocks, box_bytes) * sizeof(double));
  if (e != cudaSuccess) {
    tf::set_thread_error(std::string("tf_pcg_solve: ") + cudaGetErrorString(e));
    return TF_E_CUDA;
  }
  rc = solve(a, work, blocks, box_bytes, iters, rel_resid);
  cudaFree(work);
  return rc;
}

// ---------------------------------------------------------------------------
// tf_pcg_solve_noalloc: the same solve with its work space in a file-scope
// device array instead of cudaMalloc.  For callers that cannot allocate device
// memory while they solve: a host whose own pool allocator already holds the
// GPU's memory (a cudaMalloc there fails or fragments the pool), or a loop
// that must not stall other streams (cudaMalloc and cudaFree can synchronize
// the device).  The array (g_pcg_scratch) holds kNoAllocMaxN unknowns (4 vectors
// of 8 B each, 8 MiB plus reduction slots) and stays resident on every GPU that
// loads the library until the process exits.  A call that finds it in use by
// another host thread waits for that call.
extern "C" int tf_pcg_solve_noalloc(const tf_pcg_args* a, int32_t* iters, double* rel_resid) {
  int rc = check_args(a);
  if (rc) return rc;
  if (a->n > kNoAllocMaxN) {
    tf::set_thread_error("tf_pcg_solve_noalloc: n = " + std::to_string(a->n) +
                         " exceeds the static work space of " + std::to_string(kNoAllocMaxN) + " unknowns");
    return TF_E_ARG;
  }
  cudaError_t e = cudaSetDevice(a->device);
  if (e != cudaSuccess) {
    tf::set_thread_error(std::string("tf_pcg_solve_noalloc: ") + cudaGetErrorString(e));
    return TF_E_CUDA;
  }
  double* work = nullptr;
  int blocks = 0;
  rc = scratch_for(a->device, &work, &blocks);
  if (rc) return rc;
  const size_t box_bytes = boxes_for(a->n, a->device);
  if (!scratch_holds(a->n, blocks, box_bytes)) {
    tf::set_thread_error("tf_pcg_solve_noalloc: the static work space is too small on this device");
    return TF_E_ARG;
  }
  std::lock_guard<std::mutex> use(g_scratch_use[a->device]);
  return solve(a, work, blocks, box_bytes, iters, rel_resid);
}
