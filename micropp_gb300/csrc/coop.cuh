// coop.cuh -- groups of blocks that iterate together inside one cooperative launch.
//
// A cooperative launch keeps all its blocks resident, so the blocks of a group may wait for one another between
// the phases of an iteration; every wait is bounded, and a wait that runs out is reported to the host
// (InstOut.stalled) instead of hanging.
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace mgb {

constexpr unsigned int kSpinLimit = 1u << 22;

// A matrix value that is read once per pass: past L1, which the vectors use.
__device__ __forceinline__ double ld_value(const double *p) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Barrier over the G blocks of a group: `ctr` counts arrivals, `target` the count that ends this barrier.  Returns
// false (in every thread of the block) when the wait ran out, after `polls` of them.
__device__ __forceinline__ bool group_barrier(unsigned int *ctr, unsigned int target, int *ok, unsigned int polls) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    unsigned int spin = 0;
    while ((int)(ld_acquire(ctr) - target) < 0 && ++spin < polls) {
    }
    *ok = spin < polls;
  }
  __syncthreads();
  return *ok != 0;
}

// SMs of the current device, 0 where cooperative launches are not to be had.
inline int coop_sms() {
  int dev = 0, sms = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop || sms < 1) {
    cudaGetLastError();
    return 0;
  }
  return sms;
}

}  // namespace mgb
