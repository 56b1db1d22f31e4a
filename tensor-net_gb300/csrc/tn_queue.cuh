// tn_queue.cuh -- the pushed sweep items of the dependency-driven schedule.
#pragma once

#include <cuda_runtime.h>

#include "tn_internal.h"

namespace tn {

__device__ __forceinline__ int load_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void store_release(int *p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Appends the sweep item of listed trajectory i to the pushed queue (one thread).
__device__ inline void push_sweep(Item *dyn, int *tail, const Item *sweeps, int i) {
  const int slot = atomicAdd(tail, 1);
  const Item s = sweeps[i];
  dyn[slot].traj = s.traj;
  dyn[slot].off = s.off;
  dyn[slot].len = s.len;
  store_release(&dyn[slot].aux, 1);
}

}  // namespace tn
