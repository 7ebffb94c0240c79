// All-to-all sums and on-chip matrix of the resident CG kernels.
//
// A system whose rows fit one launch with a few rows a thread is bound by
// latency: the two inner products of an iteration each end in an exchange of
// partial sums between every block of the system.  Here a block publishes its
// partial as one 16-byte record, a double in two 8-byte words of 32 data bits
// and the 32-bit number of the exchange, so that a record announces itself (the
// line format of NCCL's low-latency protocol; the vector accesses below are of
// 8-byte elements, each of which the memory model writes and reads whole), and
// every block polls the records of its system and adds them in a fixed order:
// one store and one load through L2 instead of an atomic counter, a generation
// word and a read of the partials.
// Records alternate between two sets: a block overwrites the set of exchange k
// in exchange k + 2, after it has read every record of k + 1, whose writers had
// read theirs of k.  Every block of a system is resident (cooperative launch),
// and a wait is bounded like the grid barrier's (grid_barrier.cuh).
//
// Exchanges are numbered from 1 (cleared boxes hold 0) and go on from solve to
// solve when the boxes are not cleared in between; the number may wrap.  A solve
// of `it` iterations takes 2 it + 1 exchanges, an odd count, so the sets take
// turns at a solve's first exchange and every record in use is written again
// within two solves: a wrapped number meets no record of its last time round.
#pragma once
#include <cstdint>

#include "grid_barrier.cuh"
#include "resident_choice.hpp"

namespace tf {

struct CgShared {
  double warp[kCgVals][32];
  double part[kCgVals][kCgCluster];  // of the cluster's blocks, in its first block
  double total[kCgVals * kCgChunks];
  int dead;
  alignas(8) uint64_t bar;  // the matrix copy's mbarrier
};

__device__ __forceinline__ double cg_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// The blocks [first, first + count) of one system.  Every block has a box per
// value with a record from each block of its system: a record has one reader,
// which keeps the pollers out of one another's way (148 blocks reading one set
// of 148 records wait 3.4 to 5.4 us for one another in L2, with boxes 2.3 to 3.3).
// box[parity][value][block][producer]
//
// With clusters of `cluster` blocks (one system a launch, at most 32 clusters)
// a block hands its sums to the cluster's first block through distributed
// shared memory, those exchange records with one another, and hand the totals
// back: fewer records in flight, and none for a system of one cluster.
struct CgExchange {
  uint4* box;
  int blocks;       // boxes per value, and records of a box
  int first, count;
  int* err;
  CgShared* sh;
  uint32_t round;   // number of the next exchange
  int cluster;      // blocks of a cluster, 1 none
  uint64_t limit_ns = kBarrierLimitNs;

  // Waits for the record of exchange k at p; false when it ran out.
  template <bool kAcquire>
  __device__ __forceinline__ bool read(const uint4* p, uint32_t k, double& a) {
    uint64_t t0 = 0;
    for (uint32_t n = 0;; n++) {
      uint64_t lo, hi;  // data in the lower half, number in the upper
      if (kAcquire)
        asm volatile("ld.acquire.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
      else
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
      if ((uint32_t)(lo >> 32) == k && (uint32_t)(hi >> 32) == k) {
        a = __hiloint2double((int)(uint32_t)hi, (int)(uint32_t)lo);
        return true;
      }
      if ((n & 255) == 255) {  // no clock read in a wait that ends at once
        const uint64_t now = global_ns();
        if (t0 == 0) t0 = now;
        if (*(volatile int*)err != 0 || now - t0 > limit_ns) {
          atomicOr(err, kBarrierTimedOut);
          return false;
        }
      }
    }
  }
  __device__ __forceinline__ void write(uint4* p, uint32_t k, double a) {
    const uint64_t tag = (uint64_t)k << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(tag | (uint32_t)__double2loint(a)),
                 "l"(tag | (uint32_t)__double2hiint(a))
                 : "memory");
  }
  static __device__ __forceinline__ uint32_t peer(const void* p, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(a)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
  }
  static __device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }

  // before the first sum(): the block's set-up of shared memory is visible to its
  // threads, and with clusters every block of the cluster has started
  __device__ __forceinline__ void enter() {
    if (cluster > 1)
      cluster_sync();
    else
      __syncthreads();
  }

  // sum() with clusters, from the warps' sums on
  template <int NV, bool kPublish>
  __device__ __forceinline__ void cluster_sum(uint32_t k) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
    const int rank = blockIdx.x % cluster, me = blockIdx.x / cluster, clusters = count / cluster;
    for (int q = warp; q < NV; q += W) {
      const double t = cg_warp_sum(lane < W ? sh->warp[q][lane] : 0.0);
      if (lane == 0)
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(peer(&sh->part[q][rank], 0)), "d"(t) : "memory");
    }
    cluster_sync();
    if (rank == 0)
      for (int q = warp; q < NV; q += W) {
        double t = __shfl_sync(0xffffffffu, cg_warp_sum(lane < cluster ? sh->part[q][lane] : 0.0), 0);
        if (clusters > 1) {
          uint4* set = box + ((size_t)(k & 1) * kCgVals + q) * blocks * blocks;
          if (kPublish) __threadfence();
          double a = 0.0;
          if (lane < clusters) {
            write(set + (size_t)lane * clusters + me, k, t);
            if (!read<kPublish>(set + (size_t)me * clusters + lane, k, a)) sh->dead = 1;
          }
          t = __shfl_sync(0xffffffffu, cg_warp_sum(a), 0);
          __syncwarp();
        }
        if (lane < cluster) {
          asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(peer(&sh->total[q], lane)), "d"(t) : "memory");
          if (*(volatile int*)&sh->dead)
            asm volatile("st.shared::cluster.u32 [%0], 1;" ::"r"(peer(&sh->dead, lane)) : "memory");
        }
      }
    cluster_sync();
  }

  // v[] becomes the sums over the system's threads.  With kPublish, global
  // stores made before the call by any thread of the system are visible to
  // every thread after it.  False when a wait ran out.
  //
  // Without it (the p.q sum) the records still keep the threads' gathers of the
  // pairs before the owners' next stores of them: every gathered value is a term
  // of the sum, so its load has returned before the thread's part of the record
  // is written, and an owner stores after its loop on the records has ended.
  // That is a chain of data and control dependencies, not a release and an
  // acquire, which the memory model asks for and which cost 336 us a step
  // against 319 at 28^3 FP64 (24^3 264 / 261, 40^3 FP32 564 / 556).
  template <int NV, bool kPublish>
  __device__ __forceinline__ bool sum(double (&v)[NV]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
    const uint32_t k = round++;
    const int me = blockIdx.x - first, chunks = (count + 31) >> 5;
#pragma unroll
    for (int q = 0; q < NV; q++) v[q] = cg_warp_sum(v[q]);
    if (lane == 0)
#pragma unroll
      for (int q = 0; q < NV; q++) sh->warp[q][warp] = v[q];
    __syncthreads();
    if (cluster > 1) {
      cluster_sum<NV, kPublish>(k);
#pragma unroll
      for (int q = 0; q < NV; q++) v[q] = sh->total[q];
      return sh->dead == 0;
    }
    // a warp adds the block's warps, writes to 32 boxes, then reads 32 records
    for (int t = warp; t < NV * chunks; t += W) {
      const int q = t / chunks, i = (t - q * chunks) * 32 + lane;
      uint4* set = box + ((size_t)(k & 1) * kCgVals + q) * blocks * blocks;
      double a = __shfl_sync(0xffffffffu, cg_warp_sum(lane < W ? sh->warp[q][lane] : 0.0), 0);
      if (kPublish) __threadfence();
      if (i < count) {
        write(set + (size_t)(first + i) * blocks + me, k, a);
        if (!read<kPublish>(set + (size_t)(first + me) * blocks + i, k, a)) sh->dead = 1;
      } else {
        a = 0.0;
      }
      a = cg_warp_sum(a);
      if (lane == 0) sh->total[t] = a;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; q++) {
      double a = 0.0;
      for (int c = 0; c < chunks; c++) a += sh->total[q * chunks + c];
      v[q] = a;
    }
    return sh->dead == 0;
  }
};

// Bulk copy of global memory into shared memory (sizes and addresses multiples
// of 16 bytes), one thread; completion is counted on the mbarrier.
__device__ __forceinline__ uint32_t cg_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cg_bar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cg_smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void cg_bar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(cg_smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cg_bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  constexpr uint32_t kPiece = 32768;
  for (uint32_t o = 0; o < bytes; o += kPiece) {
    const uint32_t n = bytes - o < kPiece ? bytes - o : kPiece;
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     cg_smem_u32(dst) + o),
                 "l"((const char*)src + o), "r"(n), "r"(cg_smem_u32(bar))
                 : "memory");
  }
}
// bounded wait for the copies of phase 0
__device__ __forceinline__ bool cg_bar_wait(uint64_t* bar) {
  for (long it = 0; it < (1L << 22); it++) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(cg_smem_u32(bar))
        : "memory");
    if (ok) return true;
  }
  return false;
}

}  // namespace tf
