// Kernels of the explicit tetrahedral DGA method (dga) for sm_100a, and the
// standalone CG solve of the C ABI.  (gfdtd simulations run on the group
// engine, tet_group_kernels.cu, also when a simulation is alone.)
//
//   tet_curl_f        cf = C^T F + Ctb Fb - I, with the step's source values:
//                     E values to U, boundary dual-edge H sources, currents
//                     (:821-868, :878-879)
//   tet_h_update      U = P U + dt H cf on interior edges (P = 1 when
//                     lossless), boundary flux partials (:887-894)
//   tet_frac_update   U_c = Q U_c_old + dt Mq cf: node-star fractions of the
//                     fractured edges (:891)
//   tet_frac_gather   U = sum of a fractured edge's two fractions (:892), flux
//   tet_curl_u        cu = C U (3 signed edges per face), B -= dt cu
//                     (:902-916); flux sum
//   tet_nmul          F = R F - dt N cu (:917-918; R = 1 without magnetic
//                     losses); Whitney E and face-flux H at the probe points
//                     (:3768-3897); step counter
//   tet_cg            persistent cooperative Jacobi-PCG on a CSR system
//                     (ConjugateGradientSolver.hpp:52-103): SpMV, dots and
//                     axpys fused, FP64 reductions in a fixed order, a hard
//                     iteration limit and three bounded grid barriers per
//                     iteration
//   pcg_resident      the same solve for systems of up to 8 rows a thread with
//                     one block an SM: rows and matrix on chip, two exchanges
//                     of partial sums per iteration (cg_resident.cuh)
#include <cuda_runtime.h>

#include <atomic>

#include "cg_resident.cuh"
#include "grid_barrier.cuh"
#include "tet_kernels.cuh"

namespace tf {

constexpr int kBlock = 256;

template <typename T>
__device__ __forceinline__ T ld(const void* p, int64_t i) {
  return ((const T*)p)[i];
}

// deterministic block sum of one double (all threads get the result)
__device__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) sh[32] = s;
  }
  __syncthreads();
  return sh[32];
}

// A step is four launches (six with fractured edges), each waiting for the one
// before it (programmatic dependent launch) with its matrix row's first loads
// already made.  The matrices are SELL-32 in the device numbering: edges and
// faces ordered by the column offsets of their H and N rows, so that a warp
// reads one entry slot with one 128- or 256-byte load and gathers from
// neighbouring places.  Bound by launch latency up to some 10^5 edges, then by
// the matrices' bytes.  24^3 FP64 (102 k edges): 49 us a step with eight
// launches, one thread walking one CSR row each, 14.4 us now; 36^3 FP32 (0.12 GB a
// step, half of it H) 83 us, 30 us now.
__device__ __forceinline__ int32_t ld_index(const int32_t* p) {
  int32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_value(const float* p) {
  float v;
  asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_value(const double* p) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// Sum over row i's entries in stored order of val * x[col]; ready() runs
// between the first entries' loads and their gathers.
template <typename T, int CH, typename W>
__device__ __forceinline__ T tet_row(const TetSell& m, int i, const T* x, W ready) {
  const int64_t b = m.ptr[i >> 5];
  const int len = (int)((m.ptr[(i >> 5) + 1] - b) >> 5);
  const int32_t* col = m.col + b + (i & 31);
  const T* val = (const T*)m.val + b + (i & 31);
  T s = 0;
  for (int j0 = 0; j0 < len || j0 == 0; j0 += CH) {
    int32_t c[CH];
    T v[CH];
#pragma unroll
    for (int k = 0; k < CH; k++)
      if (j0 + k < len) {
        c[k] = ld_index(col + 32 * (j0 + k));
        v[k] = ld_value(val + 32 * (j0 + k));
      }
    if (j0 == 0) ready();
#pragma unroll
    for (int k = 0; k < CH; k++)
      if (j0 + k < len) s += v[k] * x[c[k]];
  }
  return s;
}

__device__ __forceinline__ double source_value(const DevPtrs& d, int s, int row) {
  double v[3] = {0.0, 0.0, 0.0};
  for (int p = d.se_begin[s]; p < d.se_begin[s + 1]; p++) {
    const int si = d.pair_src[p];
    double ret = d.src_amp[si] * d.carrier[(int64_t)row * d.nsrc + si];
    ret *= d.pair_fac[4 * p + 0];
    ret *= d.pair_fac[4 * p + 1];
    ret *= d.pair_fac[4 * p + 2];
    ret *= d.pair_fac[4 * p + 3];
    const int a = d.pair_dir[p];
    if (a == 0) v[0] += ret;
    else if (a == 1) v[1] += ret;
    else v[2] += ret;
  }
  const double* w = d.se_vec + 3 * (int64_t)s;
  return d.se_post[s] * ((v[0] * w[0] + v[1] * w[1]) + v[2] * w[2]);
}

// kStep: the step's source values first (an H-source edge's cb and a current
// edge's I are rewritten every step; every other edge's stay zero)
template <typename T, bool kStep>
__global__ void __launch_bounds__(kBlock) tet_curl_f(DevPtrs d) {
  constexpr int CH = 6;
  if (kStep) cudaTriggerProgrammaticLaunchCompletion();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const T* F = (const T*)d.F;
  const bool ok = e < d.nE;
  int64_t b = 0;
  int len = 0, src = -1;
  int32_t c[CH];
  if (ok) {
    b = d.Ct.ptr[e >> 5];
    len = (int)((d.Ct.ptr[(e >> 5) + 1] - b) >> 5);
    b += e & 31;
    src = d.edge_src[e];
#pragma unroll
    for (int k = 0; k < CH; k++) c[k] = k < len ? ld_index(d.Ct.col + b + 32 * k) : kNoFace;
  }
  if (kStep) cudaGridDependencySynchronize();
  if (!ok) return;
  T s = 0;
  for (int j0 = 0;;) {
    T f[CH];
#pragma unroll
    for (int k = 0; k < CH; k++) f[k] = c[k] != kNoFace ? F[c[k] & 0x7fffffff] : (T)0;
#pragma unroll
    for (int k = 0; k < CH; k++)
      if (c[k] != kNoFace) s = c[k] < 0 ? s - f[k] : s + f[k];
    j0 += CH;
    if (j0 >= len) break;
#pragma unroll
    for (int k = 0; k < CH; k++) c[k] = j0 + k < len ? ld_index(d.Ct.col + b + 32 * (j0 + k)) : kNoFace;
  }
  T cb = ((const T*)d.cb)[e], cur = ((const T*)d.I)[e];
  if (kStep && src >= 0) {
    const T v = (T)source_value(d, src, d.step[0]);
    const int kind = d.se_kind[src];
    if (kind == 1) {
      ((T*)d.U)[e] = v;
    } else if (kind == 2) {
      ((T*)d.cb)[e] = cb = v;
    } else if (kind == 3) {
      ((T*)d.I)[e] = cur = v;
    }
  }
  ((T*)d.cf)[e] = s + cb - cur;
}

template <typename T>
__global__ void __launch_bounds__(kBlock) tet_h_update(DevPtrs d) {
  __shared__ double sh[33];
  cudaTriggerProgrammaticLaunchCompletion();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  double fl = 0.0;
  const bool ok = e < d.nE && d.edge_upd[e];
  T s = 0;
  if (ok) s = tet_row<T, 9>(d.H, e, (const T*)d.cf, [] { cudaGridDependencySynchronize(); });
  else cudaGridDependencySynchronize();
  if (ok) {
    T* U = (T*)d.U;
    const T uo = U[e];
    const T un = d.h_p ? ((const T*)d.h_p)[e] * uo + (T)d.dt * s : uo + (T)d.dt * s;
    U[e] = un;
    const T cb = ((const T*)d.cb)[e];
    if (cb != (T)0) fl = ((double)uo + (double)un) * (double)cb;
  }
  if (__syncthreads_or(fl != 0.0)) fl = block_sum(fl, sh);
  if (threadIdx.x == 0) d.flux_part[blockIdx.x] = fl;
}

// the last block sums the step's boundary flux
template <typename T>
__global__ void __launch_bounds__(kBlock) tet_curl_u(DevPtrs d) {
  __shared__ double sh[33];
  cudaTriggerProgrammaticLaunchCompletion();
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  int32_t e0 = 0, e1 = 0, e2 = 0;
  if (f < d.nF) {
    e0 = d.fte[f];
    e1 = d.fte[d.nF + f];
    e2 = d.fte[2 * (int64_t)d.nF + f];
  }
  cudaGridDependencySynchronize();
  if (blockIdx.x == gridDim.x - 1) {
    double a = 0.0;
    for (int b = threadIdx.x; b < d.nflux_part; b += blockDim.x) a += d.flux_part[b];
    a = block_sum(a, sh);
    if (threadIdx.x == 0) {
      d.flux[d.step[0]] = 0.5 * a;
      d.step[1] = d.step[0];
    }
    return;
  }
  if (f >= d.nF) return;
  const T* U = (const T*)d.U;
  const T c = U[e0] - U[e1] + U[e2];
  ((T*)d.cu)[f] = c;
  T* B = (T*)d.B;
  B[f] = B[f] - (T)d.dt * c;
}

// Probe export of component c (E x y z, H x y z) of probe p into print slot `slot`.
template <typename T>
__device__ __forceinline__ void tet_probe(const DevPtrs& d, int p, int c, int slot) {
  const int a = c % 3;
  double v = 0.0;
  if (c < 3) {
    const T* U = (const T*)d.U;
    for (int q = 0; q < 6; q++) v += d.p_we[18 * (int64_t)p + 3 * q + a] * (double)U[d.p_edges[6 * (int64_t)p + q]];
  } else {
    const T* B = (const T*)d.B;
    for (int q = 0; q < 4; q++) v += d.p_hf[12 * (int64_t)p + 3 * q + a] * (double)B[d.p_faces[4 * (int64_t)p + q]];
  }
  d.samples[((int64_t)slot * d.np + p) * 6 + c] = v;
}

// F = R F - dt N cu; the first npb blocks sample the probes, one thread per
// probe and component, and advance the step counter
template <typename T>
__global__ void __launch_bounds__(kBlock) tet_nmul(DevPtrs d, int npb) {
  cudaTriggerProgrammaticLaunchCompletion();
  if ((int)blockIdx.x < npb) {
    cudaGridDependencySynchronize();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int step = d.step[1];  // tet_curl_u's copy: step[0] advances below
    if (t == 0) d.step[0] = step + 1;
    if (t >= 6 * d.np) return;
    const int slot = d.slot_of_step[step + 1];
    if (slot >= 0) tet_probe<T>(d, t / 6, t % 6, slot);
    return;
  }
  const int f = (blockIdx.x - npb) * blockDim.x + threadIdx.x;
  if (f >= d.nF) {
    cudaGridDependencySynchronize();
    return;
  }
  const T s = tet_row<T, 7>(d.N, f, (const T*)d.cu, [] { cudaGridDependencySynchronize(); });
  T* F = (T*)d.F;
  F[f] = d.n_r ? ((const T*)d.n_r)[f] * F[f] - (T)d.dt * s : F[f] - (T)d.dt * s;
}

template <typename T>
__global__ void __launch_bounds__(kBlock) tet_frac_update(DevPtrs d) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= d.nq) return;
  const T* uo = (const T*)d.Uc_old;
  const T* cf = (const T*)d.cf;
  T a = 0, b = 0;
  for (int64_t k = d.q_ptr[r]; k < d.q_ptr[r + 1]; k++) a += ld<T>(d.q_val, k) * uo[d.q_col[k]];
  for (int64_t k = d.mq_ptr[r]; k < d.mq_ptr[r + 1]; k++) b += ld<T>(d.mq_val, k) * cf[d.mq_col[k]];
  ((T*)d.Uc)[r] = a + (T)d.dt * b;
}

// flux partials after tet_h_update's, at flux_part[nblk(nE) + block]
template <typename T>
__global__ void __launch_bounds__(kBlock) tet_frac_gather(DevPtrs d, int part0) {
  __shared__ double sh[33];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double fl = 0.0;
  if (i < d.nfe) {
    const T* uc = (const T*)d.Uc;
    const int e = d.fe_edge[i];
    T* U = (T*)d.U;
    const T uo = U[e];
    const T un = uc[d.fe_a[i]] + uc[d.fe_b[i]];
    U[e] = un;
    const T cb = ((const T*)d.cb)[e];
    if (cb != (T)0) fl = ((double)uo + (double)un) * (double)cb;
  }
  fl = block_sum(fl, sh);
  if (threadIdx.x == 0) d.flux_part[part0 + blockIdx.x] = fl;
}

// dga energy (tf_energy).  W^n = 1/2 U^n.H^-1.U^{n+1} + 1/2 B.N.B over the
// class-1 edges, the leapfrog invariant of the lossless scheme; with
// U^{n+1} = U^n + dt H cf it is 1/2 u.x + 1/2 dt u.cf + 1/2 B.N.B, u the
// class-1 values of U^n, x = H^-1 u (a PCG solve), cf from the current F.
template <typename T>
__global__ void __launch_bounds__(kBlock) tet_energy_gather(DevPtrs d, const int32_t* ie, double* u, int ni) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ni) u[i] = (double)((const T*)d.U)[ie[i]];
}

// part[2 b] = sum of u.x, part[2 b + 1] = sum of u.cf over block b's rows
template <typename T>
__global__ void __launch_bounds__(kBlock) tet_energy_e(DevPtrs d, const int32_t* ie, const double* x, int ni,
                                                      double* part) {
  __shared__ double sh[33];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double a = 0.0, b = 0.0;
  if (i < ni) {
    const double u = (double)((const T*)d.U)[ie[i]];
    a = u * x[i];
    b = u * (double)((const T*)d.cf)[ie[i]];
  }
  a = block_sum(a, sh);
  b = block_sum(b, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = a;
    part[2 * blockIdx.x + 1] = b;
  }
}

// part[b] = sum over block b's faces of B_f (N B)_f
template <typename T>
__global__ void __launch_bounds__(kBlock) tet_energy_m(DevPtrs d, double* part) {
  __shared__ double sh[33];
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  double c = 0.0;
  if (f < d.nF) {
    const T* B = (const T*)d.B;
    const int64_t b = d.N.ptr[f >> 5] + (f & 31), e = d.N.ptr[(f >> 5) + 1];
    double s = 0.0;
    for (int64_t k = b; k < e; k += 32) s += (double)((const T*)d.N.val)[k] * (double)B[d.N.col[k]];
    c = (double)B[f] * s;
  }
  c = block_sum(c, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = c;
}

// out = 1/2 (sum u.x) + 1/2 dt (sum u.cf) + 1/2 (sum B.N.B), partials in order
__global__ void tet_energy_sum(const double* pe, int nbe, const double* pm, int nbm, double dt, double* out) {
  double a = 0.0, b = 0.0, c = 0.0;
  for (int q = 0; q < nbe; q++) {
    a += pe[2 * q];
    b += pe[2 * q + 1];
  }
  for (int q = 0; q < nbm; q++) c += pm[q];
  *out = 0.5 * a + 0.5 * dt * b + 0.5 * c;
}

template <typename T>
__device__ __forceinline__ T spmv_row(const int64_t* ptr, const int32_t* col, const void* val, const T* x, int i) {
  T s = 0;
  for (int64_t k = ptr[i]; k < ptr[i + 1]; k++) s += ld<T>(val, k) * x[col[k]];
  return s;
}

// deterministic grid sum of per-block partials (every block computes it)
__device__ double sum_parts(const double* part, int nb, int stride, int off, double* sh) {
  double a = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) a += part[(int64_t)b * stride + off];
  return block_sum(a, sh);
}

// Persistent Jacobi-PCG (ConjugateGradientSolver.hpp:52-103).  Stops when
// ||r||/||r0|| <= tol (criterion 0, the reference) or ||r|| <= tol ||b||
// (criterion 1), or after cg_maxiter iterations.  State in T, every inner
// product and norm accumulated in FP64.
template <typename T>
__global__ void __launch_bounds__(kBlock) tet_cg(DevPtrs d) {
  __shared__ double sh[33];
  const int n = d.nfree;
  const int nb = gridDim.x;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nth = (int64_t)nb * blockDim.x;
  T* x = (T*)d.x;
  T* r = (T*)d.r;
  T* p = (T*)d.p;
  T* q = (T*)d.q;
  const T* b = (const T*)d.rhs;
  const T* pre = (const T*)d.jac;
  // r = b - A x, rz = r.(pre r), rr = r.r, bb = b.b
  double rr = 0, rz = 0, bb = 0;
  for (int64_t i = tid; i < n; i += nth) {
    const T ri = b[i] - spmv_row<T>(d.a_ptr, d.a_col, d.a_val, x, (int)i);
    r[i] = ri;
    const double rd = (double)ri;
    rr += rd * rd;
    rz += rd * (double)(pre[i] * ri);
    bb += (double)b[i] * (double)b[i];
  }
  rr = block_sum(rr, sh);
  rz = block_sum(rz, sh);
  bb = block_sum(bb, sh);
  if (threadIdx.x == 0) {
    d.part_b[3 * blockIdx.x + 0] = rr;
    d.part_b[3 * blockIdx.x + 1] = rz;
    d.part_b[3 * blockIdx.x + 2] = bb;
  }
  grid_barrier(d.gbar, d.err, nb);
  rr = sum_parts(d.part_b, nb, 3, 0, sh);
  rz = sum_parts(d.part_b, nb, 3, 1, sh);
  bb = sum_parts(d.part_b, nb, 3, 2, sh);
  const double res0 = sqrt(rr);
  const double bnorm = sqrt(bb);
  double res = res0;
  int it = 0;
  double rz_prev = 1.0;
  auto go_on = [&](double rs) {
    if (it >= d.cg_maxiter) return false;
    if (d.cg_criterion == 0) return rs / res0 > d.tol;  // NaN (res0 = 0) stops, as the reference
    return rs > d.tol * bnorm;
  };
  while (go_on(res)) {
    const T beta = it == 0 ? (T)0 : (T)(rz / rz_prev);
    for (int64_t i = tid; i < n; i += nth) {
      const T z = pre[i] * r[i];
      p[i] = it == 0 ? z : z + beta * p[i];
    }
    grid_barrier(d.gbar, d.err, nb);
    double pq = 0;
    for (int64_t i = tid; i < n; i += nth) {
      const T qi = spmv_row<T>(d.a_ptr, d.a_col, d.a_val, p, (int)i);
      q[i] = qi;
      pq += (double)p[i] * (double)qi;
    }
    pq = block_sum(pq, sh);
    if (threadIdx.x == 0) d.part_a[blockIdx.x] = pq;
    grid_barrier(d.gbar, d.err, nb);
    pq = sum_parts(d.part_a, nb, 1, 0, sh);
    const T alpha = (T)(rz / pq);
    double rr2 = 0, rz2 = 0;
    for (int64_t i = tid; i < n; i += nth) {
      x[i] = x[i] + alpha * p[i];
      const T ri = r[i] - alpha * q[i];
      r[i] = ri;
      const double rd = (double)ri;
      rr2 += rd * rd;
      rz2 += rd * (double)(pre[i] * ri);
    }
    rr2 = block_sum(rr2, sh);
    rz2 = block_sum(rz2, sh);
    if (threadIdx.x == 0) {
      d.part_b[3 * blockIdx.x + 0] = rr2;
      d.part_b[3 * blockIdx.x + 1] = rz2;
    }
    grid_barrier(d.gbar, d.err, nb);
    rr = sum_parts(d.part_b, nb, 3, 0, sh);
    rz_prev = rz;
    rz = sum_parts(d.part_b, nb, 3, 1, sh);
    res = sqrt(rr);
    it++;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const int step = *d.step;
    d.cg_iters[step] = it;
    d.cg_resid[step] = res / res0;
    if (d.cg_limit) {
      const bool unmet = d.cg_criterion == 0 ? res / res0 > d.tol : res > d.tol * bnorm;
      d.cg_limit[step] = unmet ? 1 : 0;
    }
  }
}

// tet_cg for systems that fit one block an SM, R rows a thread: x, r, p and the
// Jacobi factor in registers, the rows' entries in shared memory as 32-row
// slices (as many slices as fit; the rest is read from the CSR each time), the
// pair (z, p) of a column gathered with one load, where p_j = z + beta p_{j-1}
// is formed with the rounding of the row's owner.  zp (2 n doubles) takes the
// place of jac and r.  Bound by latency: 131 k rows of 7 entries took 22.8 us an
// iteration with tet_cg, the call's other costs included, and take 8.5.
template <int R>
__global__ void __launch_bounds__(kPcgThreads, 1) pcg_resident(DevPtrs d, int rows_per_block, int entries,
                                                              int cluster) {
  constexpr int CH = 7;
  extern __shared__ __align__(16) unsigned char pcg_raw[];
  __shared__ CgShared sh;
  __shared__ int width[R * kPcgThreads / 32 + 1];
  double* sval = reinterpret_cast<double*>(pcg_raw);
  int32_t* scol = reinterpret_cast<int32_t*>(sval + entries);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
  const int n = d.nfree, r0 = min(n, (int)blockIdx.x * rows_per_block), r1 = min(n, r0 + rows_per_block);
  CgExchange ex{d.box, (int)gridDim.x, 0, (int)gridDim.x, d.err, &sh, 1u, cluster};
  const double* val = (const double*)d.a_val;
  const double* b = (const double*)d.rhs;
  double* x = (double*)d.x;
  double2* zp = (double2*)d.jac;
  // slot k of a warp: rows r0 + 32 (k W + warp) + lane
  int64_t at[R];
  int len[R], off[R];
  if (threadIdx.x == 0) sh.dead = 0;
#pragma unroll
  for (int k = 0; k < R; k++) {
    const int i = r0 + 32 * (k * W + warp) + lane;
    at[k] = i < r1 ? d.a_ptr[i] : 0;
    len[k] = i < r1 ? (int)(d.a_ptr[i + 1] - at[k]) : 0;
    const int w = __reduce_max_sync(0xffffffffu, len[k]);
    if (lane == 0) width[k * W + warp] = w;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int q = 0; q < R * W; q++) {
      const int w = width[q];
      width[q] = s + 32 * w <= entries ? s : -1;  // a slice that does not fit is read from the CSR
      if (width[q] >= 0) s += 32 * w;
    }
  }
  ex.enter();
  double xk[R], rk[R], pk[R], dk[R], qk[R];
#pragma unroll
  for (int k = 0; k < R; k++) {
    const int i = r0 + 32 * (k * W + warp) + lane;
    off[k] = width[k * W + warp];
    double dg = 0.0;
    if (off[k] >= 0) off[k] += lane;
    for (int j = 0; j < len[k]; j++) {
      const int32_t c = d.a_col[at[k] + j];
      const double v = val[at[k] + j];
      if (c == i) dg = v;
      if (off[k] >= 0) {
        scol[off[k] + 32 * j] = c;
        sval[off[k] + 32 * j] = v;
      }
    }
    dk[k] = dg != 0.0 ? 1.0 / dg : 1.0;
    xk[k] = i < r1 ? x[i] : 0.0;
    rk[k] = i < r1 ? b[i] : 0.0;
    pk[k] = 0.0;
    qk[k] = 0.0;
  }
  // a thread reads back the entries it wrote itself
  auto row_dot = [&](int k, auto load, auto form) -> double {
    double s = 0.0;
    if (off[k] >= 0) {
      for (int j0 = 0; j0 < len[k]; j0 += CH) {
        decltype(load(0)) g[CH];
#pragma unroll
        for (int q = 0; q < CH; q++)
          if (j0 + q < len[k]) g[q] = load(scol[off[k] + 32 * (j0 + q)]);
#pragma unroll
        for (int q = 0; q < CH; q++)
          if (j0 + q < len[k]) s += sval[off[k] + 32 * (j0 + q)] * form(g[q]);
      }
    } else {
      for (int j = 0; j < len[k]; j++) s += val[at[k] + j] * form(load(d.a_col[at[k] + j]));
    }
    return s;
  };
  double v3[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < R; k++) {
    const int i = r0 + 32 * (k * W + warp) + lane;
    if (i >= r1) continue;
    const double bi = rk[k];
    const double ri = bi - row_dot(k, [&](int32_t c) { return x[c]; }, [](double g) { return g; });
    const double zi = __dmul_rn(dk[k], ri);
    rk[k] = ri;
    zp[i] = make_double2(zi, 0.0);
    v3[0] += ri * ri;
    v3[1] += ri * zi;
    v3[2] += bi * bi;
  }
  bool alive = ex.sum<3, true>(v3);
  const double res0 = sqrt(v3[0]), bnorm = sqrt(v3[2]);
  double res = res0, rz = v3[1], beta = 0.0;
  int it = 0;
  auto unmet = [&]() { return d.cg_criterion == 0 ? res / res0 > d.tol : res > d.tol * bnorm; };  // NaN (res0 = 0) stops
  while (alive && it < d.cg_maxiter && unmet()) {
    const bool first = it == 0;
    auto p_of = [&](double z, double p) { return first ? z : __fma_rn(beta, p, z); };
    double v1[1] = {0.0};
#pragma unroll
    for (int k = 0; k < R; k++) {
      if (r0 + 32 * (k * W + warp) + lane >= r1) continue;
      qk[k] = row_dot(k, [&](int32_t c) { return zp[c]; }, [&](double2 g) { return p_of(g.x, g.y); });
      pk[k] = p_of(__dmul_rn(dk[k], rk[k]), pk[k]);
      v1[0] += pk[k] * qk[k];
    }
    alive = ex.sum<1, false>(v1);
    const double alpha = rz / v1[0];
    double v2[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < R; k++) {
      const int i = r0 + 32 * (k * W + warp) + lane;
      if (i >= r1) continue;
      xk[k] = __fma_rn(alpha, pk[k], xk[k]);
      rk[k] = rk[k] - alpha * qk[k];
      const double zi = __dmul_rn(dk[k], rk[k]);
      zp[i] = make_double2(zi, pk[k]);
      v2[0] += rk[k] * rk[k];
      v2[1] += rk[k] * zi;
    }
    alive = ex.sum<2, true>(v2) && alive;
    res = sqrt(v2[0]);
    beta = v2[1] / rz;
    rz = v2[1];
    it++;
  }
#pragma unroll
  for (int k = 0; k < R; k++) {
    const int i = r0 + 32 * (k * W + warp) + lane;
    if (i < r1) x[i] = xk[k];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    d.cg_iters[0] = it;
    d.cg_resid[0] = res / res0;
    if (d.cg_limit) d.cg_limit[0] = unmet() ? 1 : 0;
  }
}

// export before the first step (t = 0)
template <typename T>
__global__ void __launch_bounds__(kBlock) tet_initial_probes(DevPtrs d) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int slot = d.slot_of_step[0];
  if (t < 6 * d.np && slot >= 0) tet_probe<T>(d, t / 6, t % 6, slot);
}

// ------------------------------------------------------------------ launch
static inline unsigned nblk(int64_t n) { return (unsigned)((n + kBlock - 1) / kBlock > 0 ? (n + kBlock - 1) / kBlock : 1); }

template <typename T>
int tet_cg_blocks(int device) {
  int per_sm = 0, sms = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tet_cg<T>, kBlock, 0);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (per_sm > 2) per_sm = 2;
  return per_sm * sms;
}

// out[i] = v[where[i]]: a field in the reference's numbering, as double
template <typename T>
__global__ void __launch_bounds__(kBlock) tet_export(const T* v, const int32_t* where, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (double)v[where[i]];
}
template <typename T>
cudaError_t tet_launch_export(const void* v, const int32_t* where, double* out, int n, cudaStream_t st) {
  tet_export<T><<<nblk(n), kBlock, 0, st>>>((const T*)v, where, out, n);
  return cudaGetLastError();
}
template cudaError_t tet_launch_export<double>(const void*, const int32_t*, double*, int, cudaStream_t);
template cudaError_t tet_launch_export<float>(const void*, const int32_t*, double*, int, cudaStream_t);

// One leapfrog step of the dga method (Discretization.hpp:810-931).  ev
// (optional, 6 events) brackets: sources (none of their own), H half, flux (in
// the E half), E half, probes (in the E half).
template <typename T>
cudaError_t tet_launch_step(const DevPtrs& d, cudaStream_t st, cudaEvent_t* ev) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kBlock);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (ev) cudaEventRecord(ev[0], st);
  if (ev) cudaEventRecord(ev[1], st);
  cfg.gridDim = dim3(nblk(d.nE));
  cudaError_t e = cudaLaunchKernelEx(&cfg, tet_curl_f<T, true>, d);
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, tet_h_update<T>, d);
  if (e != cudaSuccess) return e;
  if (d.nq > 0) {
    cudaMemcpyAsync(d.Uc_old, d.Uc, sizeof(T) * (size_t)d.nq, cudaMemcpyDeviceToDevice, st);
    tet_frac_update<T><<<nblk(d.nq), kBlock, 0, st>>>(d);
  }
  if (d.nfe > 0) tet_frac_gather<T><<<nblk(d.nfe), kBlock, 0, st>>>(d, (int)nblk(d.nE));
  if (ev) cudaEventRecord(ev[2], st);
  if (ev) cudaEventRecord(ev[3], st);
  cfg.gridDim = dim3(nblk(d.nF) + 1);
  e = cudaLaunchKernelEx(&cfg, tet_curl_u<T>, d);
  const int npb = (int)nblk(6 * (int64_t)d.np);
  cfg.gridDim = dim3(nblk(d.nF) + npb);
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, tet_nmul<T>, d, npb);
  if (ev) cudaEventRecord(ev[4], st);
  if (ev) cudaEventRecord(ev[5], st);
  return e != cudaSuccess ? e : cudaGetLastError();
}

// Jacobi preconditioner from the CSR diagonal (1 where the diagonal is
// missing or zero, ConjugateGradientSolver.hpp:119-127)
__global__ void jacobi_from_csr(const int64_t* ptr, const int32_t* col, const double* val, double* pre, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double dg = 0.0;
  for (int64_t k = ptr[i]; k < ptr[i + 1]; k++)
    if (col[k] == i) dg = val[k];
  pre[i] = dg != 0.0 ? 1.0 / dg : 1.0;
}

// Matrix entries a block's shared memory holds on a device, 0 when the kernel
// cannot be launched; the limit the runtime has to be told is set on the first
// call for the device (the set-up's estimate launches hundreds of solves).
template <int R>
static int pcg_resident_entries(int device) {
  constexpr int kDevices = 64;
  static std::atomic<int> known[kDevices];
  const bool keep = device >= 0 && device < kDevices;
  if (keep && known[device].load() > 0) return known[device].load();
  int most = 0, per_sm = 0;
  cudaFuncAttributes fa{};
  if (cudaFuncGetAttributes(&fa, pcg_resident<R>) != cudaSuccess ||
      cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  const int entries = (most - (int)fa.sharedSizeBytes) / (12 * 32) * 32;
  if (cudaFuncSetAttribute(pcg_resident<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, entries * 12) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pcg_resident<R>, kPcgThreads, entries * 12) != cudaSuccess ||
      per_sm < 1) {
    cudaGetLastError();
    return 0;
  }
  if (keep) known[device].store(entries);
  return entries;
}
static int pcg_sms(int device) {
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms < 32 * kCgChunks ? sms : 32 * kCgChunks;
}
// bytes of DevPtrs::box
size_t pcg_box_bytes(int device) { return cg_box_bytes((size_t)pcg_sms(device)); }

static int pcg_entries(int rows, int device) {
  switch (rows) {
    case 1: return pcg_resident_entries<1>(device);
    case 2: return pcg_resident_entries<2>(device);
    case 3: return pcg_resident_entries<3>(device);
    case 4: return pcg_resident_entries<4>(device);
    default: return pcg_resident_entries<8>(device);
  }
}
static ResidentChoice pcg_flat_choice(int64_t n, int device) {
  return pcg_flat(n, pcg_sms(device), [&](int rows) { return pcg_entries(rows, device); });
}

// whether pcg_launch_solve takes the resident kernel (given boxes)
bool pcg_resident_fits(int64_t n, int device) { return pcg_flat_choice(n, device).rows > 0; }

static cudaError_t pcg_launch_resident(const DevPtrs& d, const ResidentChoice& c, cudaStream_t st) {
  const int slices = (d.nfree + 31) / 32;
  const int rows = (slices + c.blocks - 1) / c.blocks * 32;  // evenly
  const int blocks = c.cluster > 1 ? c.blocks : (d.nfree + rows - 1) / rows;
  cudaMemsetAsync(d.box, 0, cg_box_bytes((size_t)blocks), st);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)c.cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(32 * c.warps);
  cfg.dynamicSmemBytes = (size_t)c.entries * 12;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = c.cluster > 1 ? 2 : 1;
  auto launch = [&](auto kernel) { return cudaLaunchKernelEx(&cfg, kernel, d, rows, c.entries, c.cluster); };
  switch (c.rows) {
    case 1: return launch(pcg_resident<1>);
    case 2: return launch(pcg_resident<2>);
    case 3: return launch(pcg_resident<3>);
    case 4: return launch(pcg_resident<4>);
    default: return launch(pcg_resident<8>);
  }
}

// Clusters of 8 blocks that run at once with the kernels' full shared memory, no
// more than one block an SM (the boxes are laid out for that), looked up once for
// a device.
static int pcg_clusters(int device) {
  constexpr int kDevices = 64;
  static std::atomic<int> known[kDevices];  // one more than the number, 0 not looked up
  const bool keep = device >= 0 && device < kDevices;
  if (keep && known[device].load() > 0) return known[device].load() - 1;
  int n = pcg_sms(device) / 8;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(8);
  cfg.blockDim = dim3(kPcgThreads);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 8;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto look = [&](auto kernel, int entries) {
    int m = 0;
    cfg.dynamicSmemBytes = (size_t)entries * 12;
    if (entries < 1 || cudaOccupancyMaxActiveClusters(&m, kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      m = 0;
    }
    n = m < n ? m : n;
  };
  look(pcg_resident<1>, pcg_resident_entries<1>(device));
  look(pcg_resident<2>, pcg_resident_entries<2>(device));
  look(pcg_resident<3>, pcg_resident_entries<3>(device));
  if (keep) known[device].store(n + 1);
  return n;
}

// Standalone FP64 solve.  With boxes (DevPtrs::box) and at most 8 rows a thread
// the resident kernel, which beat tet_cg at every size it takes (rows of 7
// entries, us an iteration of a call: 1 k rows 5.3 against 21.1, 131 k 8.5
// against 22.8, 594 k 31.8 against 35.8); otherwise, and where the device does
// not give it its shared memory, preconditioner, then the persistent PCG kernel.
cudaError_t pcg_launch_solve(DevPtrs d, int blocks, int device, cudaStream_t st) {
  cudaMemsetAsync(d.err, 0, sizeof(int), st);
  const ResidentChoice flat = d.box ? pcg_flat_choice(d.nfree, device) : ResidentChoice();
  if (flat.rows) {
    const ResidentChoice c = pcg_clustered(
        d.nfree, [&] { return pcg_clusters(device); }, [&](int rows) { return pcg_entries(rows, device); });
    if (c.rows && pcg_launch_resident(d, c, st) == cudaSuccess) return cudaSuccess;
    if (c.rows) cudaGetLastError();  // a cluster launch the device refused
    return pcg_launch_resident(d, flat, st);
  }
  jacobi_from_csr<<<nblk(d.nfree), kBlock, 0, st>>>(d.a_ptr, d.a_col, (const double*)d.a_val, (double*)d.jac,
                                                    d.nfree);
  cudaMemsetAsync(d.step, 0, sizeof(int), st);
  cudaMemsetAsync(d.gbar, 0, 2 * sizeof(unsigned int), st);
  void* args[] = {(void*)&d};
  cudaError_t err = cudaLaunchCooperativeKernel((void*)tet_cg<double>, dim3(blocks), dim3(kBlock), args, 0, st);
  if (err != cudaSuccess) return err;
  return cudaGetLastError();
}

template <typename T>
void tet_launch_initial_probes(const DevPtrs& d, cudaStream_t st) {
  if (d.np) tet_initial_probes<T><<<nblk(6 * (int64_t)d.np), kBlock, 0, st>>>(d);
}

// dga energy: gather u, solve H x = u (d_cg: the class-1 block of H and the
// PCG work), then the three sums; *out receives W (device)
template <typename T>
cudaError_t tet_launch_energy(const DevPtrs& d, DevPtrs d_cg, int cg_blocks, int device, const int32_t* ie, int ni,
                              double* part, double* out, cudaStream_t st) {
  tet_curl_f<T, false><<<nblk(d.nE), kBlock, 0, st>>>(d);
  tet_energy_gather<T><<<nblk(ni), kBlock, 0, st>>>(d, ie, (double*)d_cg.rhs, ni);
  cudaMemsetAsync(d_cg.x, 0, sizeof(double) * (size_t)ni, st);
  cudaError_t e = pcg_launch_solve(d_cg, cg_blocks, device, st);
  if (e != cudaSuccess) return e;
  const int nbe = (int)nblk(ni), nbm = (int)nblk(d.nF);
  tet_energy_e<T><<<nbe, kBlock, 0, st>>>(d, ie, (const double*)d_cg.x, ni, part);
  tet_energy_m<T><<<nbm, kBlock, 0, st>>>(d, part + 2 * nbe);
  tet_energy_sum<<<1, 1, 0, st>>>(part, nbe, part + 2 * nbe, nbm, d.dt, out);
  return cudaGetLastError();
}

template cudaError_t tet_launch_energy<double>(const DevPtrs&, DevPtrs, int, int, const int32_t*, int, double*, double*,
                                               cudaStream_t);
template cudaError_t tet_launch_energy<float>(const DevPtrs&, DevPtrs, int, int, const int32_t*, int, double*, double*,
                                              cudaStream_t);
template cudaError_t tet_launch_step<double>(const DevPtrs&, cudaStream_t, cudaEvent_t*);
template cudaError_t tet_launch_step<float>(const DevPtrs&, cudaStream_t, cudaEvent_t*);
template int tet_cg_blocks<double>(int);
template void tet_launch_initial_probes<double>(const DevPtrs&, cudaStream_t);
template void tet_launch_initial_probes<float>(const DevPtrs&, cudaStream_t);

}  // namespace tf
