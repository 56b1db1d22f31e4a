// tn_run.cuh -- k_run, the persistent executor: CTAs pull work items (one
// trajectory's instruction list each) from an atomic counter and run them with
// the device routines of tn_device.cuh.  One translation unit per precision
// (tn_run_*.cu) instantiates it, so that they compile in parallel.
#pragma once

#include "tn_device.cuh"
#include "tn_internal.h"
#include "tn_queue.cuh"
#include "tn_tc.cuh"

namespace tn {

__device__ __forceinline__ unsigned long long global_ns() { return tc::global_ns(); }

// Static schedule (la.rem == nullptr): items[0, count) in counter order.
// Dependency-driven schedule: a CTA takes a pushed sweep item when one is
// ready (claimed by compare-and-swap on the sweep head below the push tail),
// else the next gate item; once the gate items are gone it claims the next
// sweep slot and waits (bounded by kQueueWaitNs) for its push.  Every pushed
// item depends only on gate items already taken by running CTAs, so the
// waits end; a wait that runs out sets qerr and the CTA moves on.
template <typename T, int NT, int W>
__global__ void __launch_bounds__(NT, 1) k_run(LaunchArgs la, int sortP, int ws_cap) {
  extern __shared__ __align__(256) unsigned char smem[];
  __shared__ Item s_item;
  __shared__ int s_kind;  // 0 done, 1 gate / static item, 2 pushed sweep item, 3 skip
  __shared__ uint64_t s_bar, s_gbar[2];
  __shared__ uint32_t s_tmem;
  Smem<T, W> sm(smem, sortP);
  Team tm;
  if (la.cluster > 1) {
    tm.size = la.cluster;
    tm.rank = int(blockIdx.x) % la.cluster;  // clusters are consecutive blocks of a one-dimensional grid
  }
  const int team_id = int(blockIdx.x) / tm.size;
  Work<T> wk = make_work<T>(reinterpret_cast<unsigned char *>(la.ws) + size_t(team_id) * la.ws_stride, ws_cap);
  if (la.team) wk.team = reinterpret_cast<unsigned char *>(la.team) + size_t(team_id) * la.team_stride;
  const bool dd = la.rem != nullptr;
  // float: one 128 x 256 FP32 accumulator tile (theta and recovery GEMMs);
  // double-float: eight 128 x 64 level accumulators of the tensor-core update
  constexpr bool kTC = sizeof(T) == 4 || std::is_same<T, ::tn::dd>::value;
  constexpr uint32_t kTmemCols = sizeof(T) == 4 ? 256 : 512;
  if constexpr (kTC) {
    // the executor owns kTmemCols tensor-memory columns for its whole
    // life (one CTA per SM); released below on the kernel's only exit path
    if ((threadIdx.x >> 5) == 0) {
      tc::tmem_alloc(&s_tmem, kTmemCols);
      tc::tmem_relinquish();
    }
    if (threadIdx.x == 0) {
      tc::mbar_init(&s_bar, 1);
      tc::mbar_init(s_gbar, 1);
      tc::mbar_init(s_gbar + 1, 1);
      tc::mbar_fence_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    sm.tmem = s_tmem;
    sm.bar = &s_bar;
    sm.gbar = s_gbar;
    sm.phase = 0;
    sm.tc = la.theta_simt == 0;
  }
  // A team's first member takes the items and passes them on through the team's
  // part (launch_run refuses clusters without one).
  volatile unsigned int *pass = tm.size > 1 ? team_work<T>(wk.team, ws_cap).flag + kTeamFlags : nullptr;
  for (;;) {
    if (threadIdx.x == 0 && tm.rank == 0) {
      const int G = la.nitems_dev ? *la.nitems_dev : la.nitems;
      int kind = 0, slot_i = -1;
      if (dd) {
        // A pushed sweep item that is already there goes first: the sweeps
        // are the serial chains that bound the launch, the gate items are
        // independent filler.
        int h = *reinterpret_cast<volatile int *>(la.dyn_head);
        while (h < *reinterpret_cast<volatile int *>(la.dyn_tail)) {
          const int prev = atomicCAS(la.dyn_head, h, h + 1);
          if (prev == h) {
            slot_i = h;
            break;
          }
          h = prev;
        }
      }
      if (slot_i < 0) {
        const int it = atomicAdd(la.counter, 1);
        if (it < G) {
          s_item = la.items[it];
          kind = 1;
        } else if (dd) {
          // no gate left: claim the next sweep slot and wait for its push
          const int h = atomicAdd(la.dyn_head, 1);
          if (h < la.nsweeps) slot_i = h;
        }
      }
      if (slot_i >= 0) {
        Item *slot = la.dyn + slot_i;
        const unsigned long long t0 = global_ns();
        const unsigned long long limit = la.queue_wait_ns ? la.queue_wait_ns : kQueueWaitNs;
        kind = 2;
        while (load_acquire(&slot->aux) == 0) {
          if (global_ns() - t0 > limit) {
            atomicExch(la.qerr, 1);
            kind = 3;
            break;
          }
          __nanosleep(200);
        }
        if (kind == 2) s_item = Item{slot->traj, slot->off, slot->len, 0};
      }
      s_kind = kind;
      if (tm.size > 1) {
        pass[0] = unsigned(kind);
        if (kind == 1 || kind == 2) {
          pass[1] = unsigned(s_item.traj);
          pass[2] = unsigned(s_item.off);
          pass[3] = unsigned(s_item.len);
          pass[4] = unsigned(s_item.aux);
        }
      }
    }
    int kind;
    Item item;
    if (tm.size > 1) {
      tm.sync();
      kind = int(pass[0]);
      item = Item{int(pass[1]), int(pass[2]), int(pass[3]), int(pass[4])};
      tm.sync();
    } else {
      __syncthreads();
      kind = s_kind;
      item = s_item;
      __syncthreads();
    }
    if (kind == 0) break;
    if (kind == 3) continue;
    if (kind == 2) __threadfence();  // acquire side for every thread of the CTA
    run_program<T, NT, W>(tm, la, (dd && kind == 1) ? la.gprog : la.prog, item, wk, sm);
    if (dd && kind == 1) {
      __threadfence();  // this thread's writes of the gate's result, visible device-wide
      tm.sync();
      if (threadIdx.x == 0 && tm.rank == 0 && atomicSub(la.rem + item.aux, 1) == 1) {
        __threadfence();
        push_sweep(la.dyn, la.dyn_tail, la.sweeps, item.aux);
      }
    }
  }
  if constexpr (kTC) {
    tc::fence_before_sync();
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) {
      tc::fence_after_sync();
      tc::tmem_dealloc(sm.tmem, kTmemCols);
    }
  }
}

// Dynamic shared memory limit configured for k_run<T> on the current
// device (raised on demand; set when a handle or batch is created, so that
// a stream capture of a launch finds it already in place).
template <typename T, int NT, int W>
static cudaError_t ensure_run_smem(size_t smem) {
  static int configured[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  int &have = configured[dev & 63];
  if (int(smem) > have) {
    cudaError_t e = cudaFuncSetAttribute(k_run<T, NT, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
    have = int(smem);
  }
  return cudaSuccess;
}

template <typename T, int NT, int W>
static cudaError_t launch_run_t(const LaunchArgs &la, int grid, int sortP, int ws_cap, cudaStream_t st) {
  const size_t smem = SmemLayout<T, W>::total(sortP);
  cudaError_t e = ensure_run_smem<T, NT, W>(smem);
  if (e != cudaSuccess) return e;
  if (la.cluster <= 1) {
    k_run<T, NT, W><<<grid, NT, smem, st>>>(la, sortP, ws_cap);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(grid) * unsigned(la.cluster));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(la.cluster);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_run<T, NT, W>, la, sortP, ws_cap);
}

// Clusters of `cluster` CTAs of k_run<T> that can be resident at once (0: none).
template <typename T, int NT, int W>
static int run_clusters_t(int sortP, int cluster) {
  const size_t smem = SmemLayout<T, W>::total(sortP);
  if (ensure_run_smem<T, NT, W>(smem) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(cluster));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(cluster);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k_run<T, NT, W>, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

// Blocks of k_run<T> that fit on an SM (at least 1).
template <typename T, int NT, int W>
static int run_blocks_t(int sortP) {
  int nb = 0;
  const size_t smem = SmemLayout<T, W>::total(sortP);
  cudaError_t e = ensure_run_smem<T, NT, W>(smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_run<T, NT, W>, NT, smem);
  return e != cudaSuccess || nb < 1 ? 1 : nb;
}

#define TN_INSTANTIATE_RUN(T, SUFFIX)                                                                       \
  cudaError_t launch_run_##SUFFIX(const LaunchArgs &la, int grid, int sortP, int ws_cap, cudaStream_t st) { \
    return launch_run_t<T, kThreads, kBlockW>(la, grid, sortP, ws_cap, st);                                \
  }                                                                                                         \
  size_t run_smem_##SUFFIX(int sortP) { return SmemLayout<T, kBlockW>::total(sortP); }                      \
  size_t run_work_##SUFFIX(int cap) { return work_bytes<T>(cap); }                                          \
  size_t run_team_##SUFFIX(int cap) { return team_bytes<T>(cap); }                                          \
  int run_blocks_##SUFFIX(int sortP) { return run_blocks_t<T, kThreads, kBlockW>(sortP); }                  \
  int run_clusters_##SUFFIX(int sortP, int cluster) { return run_clusters_t<T, kThreads, kBlockW>(sortP, cluster); }

}  // namespace tn
