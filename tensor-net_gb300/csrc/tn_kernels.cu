// tn_kernels.cu -- kernels of the trajectory engine and their launchers.
//
//  (k_run, the persistent executor, is in tn_run.cuh)
//  k_compile    builds every trajectory's instruction list for one brickwork
//               layer on the device (apply_bilayer, circuit.rs:624-659 ->
//               apply_meas_prob_layer control flow, mps.rs:2206-2252).
//  k_reset      re-initialises trajectory slots to |0...0> (MPS::new,
//               mps.rs:370-391).
#include "tn_device.cuh"
#include "tn_internal.h"
#include "tn_queue.cuh"

namespace tn {

__global__ void k_reset(TrajDev *trajs, const int *list, int count, int prec) {
  const int t = list[blockIdx.x];
  const TrajDev tr = trajs[t];
  const size_t slot = size_t(2) * tr.cap * tr.cap;
  for (int k = threadIdx.x; k < tr.n; k += blockDim.x) {
    if (prec == 0) {
      cpx<double> *g = reinterpret_cast<cpx<double> *>(tr.gamma) + size_t(k) * slot;
      g[0] = mkc<double>(1.0, 0.0);
      g[1] = mkc<double>(0.0, 0.0);
    } else if (prec == 2) {
      cpx<dd> *g = reinterpret_cast<cpx<dd> *>(tr.gamma) + size_t(k) * slot;
      g[0] = mkc<dd>(dd(1.f, 0.f), dd(0.f, 0.f));
      g[1] = mkc<dd>(dd(0.f, 0.f), dd(0.f, 0.f));
    } else {
      cpx<float> *g = reinterpret_cast<cpx<float> *>(tr.gamma) + size_t(k) * slot;
      g[0] = mkc<float>(1.f, 0.f);
      g[1] = mkc<float>(0.f, 0.f);
    }
  }
  for (int s = threadIdx.x; s <= tr.n; s += blockDim.x) {
    tr.lam[size_t(s) * tr.cap] = 1.0;
    tr.chi[s] = 1;
  }
}

// One thread per listed trajectory.  The layer's gates act on disjoint bonds
// (a brickwork layer, circuit.rs:523-563), so each becomes its own work item
// (gprog[g], gitems[g]) of the first launch, spread over all SMs; the
// measurement layer with its refactor sweep and the entropy read form the
// trajectory's program of the second launch, at prog + i * pcap, placed at
// items[order[i]] so that the executor pulls the most expensive trajectories
// first.  A trajectory whose gates overlap keeps them, in order, at the head
// of its second-launch program instead.
__global__ void k_compile(const TrajDev *trajs, const int *list, int nt, const int *order, const int *gate_off,
                          const int *gate_ks, const int *meas_off, const int *meas_ks, const int *posts, int pcap,
                          Instr *prog, Item *items, Instr *gprog, Item *gitems, int gcap, int *gcount) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *gcount = min(gate_off[nt], gcap);
  if (i >= nt) return;
  const int t = list[i];
  const int n = trajs[t].n;
  Instr *p = prog + size_t(i) * pcap;
  int pc = 0;
  auto emit = [&](int op, int k, int a, int b) {
    if (pc < pcap) p[pc] = Instr{op, k, a, b};
    ++pc;
  };
  const int g0 = gate_off[i], g1 = gate_off[i + 1];
  bool disjoint = true;
  for (int g = g0; g < g1 && disjoint; ++g)
    for (int h = g + 1; h < g1; ++h)
      if (abs(gate_ks[g] - gate_ks[h]) < 2) {
        disjoint = false;
        break;
      }
  for (int g = g0; g < g1; ++g) {
    const int k = gate_ks[g];
    const bool valid = n > 1 && k >= 0 && k < n - 1;
    if (g < gcap) {
      gprog[g] = (disjoint && valid) ? Instr{OP_GATE, k, g, 0} : Instr{OP_NOP, 0, 0, 0};
      gitems[g] = Item{t, g, 1, 0};
    } else if (disjoint) {
      atomicOr(trajs[t].status, ST_BAD_INSTR);
    }
    if (!disjoint && valid) emit(OP_GATE, k, g, 0);
  }
  const int m0 = meas_off[i], m1 = meas_off[i + 1];
  int last = -1;
  for (int j = m0; j < m1; ++j) {
    const int k = meas_ks[j];
    if (k < 0 || k >= n || k <= last) continue;  // host guarantees sorted unique
    if (last >= 0)
      for (int b = last; b < k; ++b) emit(OP_REFACTOR, b, 0, 0);
    emit(OP_MEAS, k, j, posts ? (posts[j] == 0 || posts[j] == 1 ? posts[j] : -1) : -1);
    last = k;
  }
  if (last >= 0) {
    for (int b = last; b < n - 1; ++b) emit(OP_REFACTOR, b, 0, 0);
    for (int b = n - 3; b >= 0; --b) emit(OP_REFACTOR, b, 0, 0);
  }
  if (n >= 2) emit(OP_ENTROPY, n / 2 - 1, i, 0);
  if (pc > pcap) {  // program did not fit: run nothing, flag the trajectory
    atomicOr(trajs[t].status, ST_BAD_INSTR);
    pc = 0;
  }
  items[order[i]] = Item{t, int(size_t(i) * pcap), pc, 0};
}

// Execution rank of every listed trajectory, most expensive first (one
// block of 1024 threads).  Cost from the current bond dimensions: the
// trajectory's critical path is its most expensive gate (gates run in
// parallel) plus, when the layer measures, its serial refactor sweep over
// every bond, each bond op ~ chi^3.  Ties keep list order; more than
// kLptMax trajectories keep list order altogether.
constexpr int kLptMax = 4096;

__global__ void __launch_bounds__(1024) k_lpt_order(const TrajDev *trajs, const int *list, int nt,
                                                    const int *meas_off, int *order) {
  extern __shared__ __align__(16) unsigned char lsm[];
  if (nt > kLptMax) {
    for (int i = threadIdx.x; i < nt; i += blockDim.x) order[i] = i;
    return;
  }
  int P = 1;
  while (P < nt) P <<= 1;
  double *key = reinterpret_cast<double *>(lsm);
  int *idx = reinterpret_cast<int *>(key + P);
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    double c = -1.0;
    if (i < nt) {
      const TrajDev tr = trajs[list[i]];
      double sweep = 0.0, gmax = 0.0;
      for (int b = 1; b < tr.n; ++b) {
        const double x = double(tr.chi[b]);
        const double x3 = x * x * x;
        sweep += x3;
        gmax = fmax(gmax, x3);
      }
      c = gmax + (meas_off[i + 1] > meas_off[i] ? sweep : 0.0);
    }
    key[i] = c;
    idx[i] = i;
  }
  __syncthreads();
  bitonic_desc<float, 1024, kBlockW>(key, idx, P);
  for (int r = threadIdx.x; r < nt; r += blockDim.x) order[idx[r]] = r;
}

// First gate-queue slot of every listed trajectory when trajectories are
// taken in `order` rank: an exclusive scan of the gate counts by rank (one
// block; scratch holds the counts by rank).  An `order` that is not a
// permutation of [0, nt) is replaced by the identity.
__global__ void k_gate_slots(int nt, const int *order, const int *gate_off, int *scratch, int *gstart) {
  __shared__ int carry, wsum[32];
  for (int i = threadIdx.x; i < nt; i += blockDim.x) scratch[i] = 0;
  __syncthreads();
  int bad = 0;
  for (int i = threadIdx.x; i < nt; i += blockDim.x) {
    const int r = order[i];
    if (r < 0 || r >= nt)
      bad = 1;
    else
      atomicAdd(scratch + r, 1);
  }
  __syncthreads();
  for (int r = threadIdx.x; r < nt; r += blockDim.x) bad |= scratch[r] != 1;
  bad = __syncthreads_or(bad);
  auto rank = [&](int i) { return bad ? i : order[i]; };
  for (int i = threadIdx.x; i < nt; i += blockDim.x) scratch[rank(i)] = gate_off[i + 1] - gate_off[i];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int base = 0; base < nt; base += blockDim.x) {
    const int r = base + threadIdx.x;
    const int v = r < nt ? scratch[r] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int w = lane < nw ? wsum[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      if (lane < nw) wsum[lane] = w;  // inclusive sums over warps
    }
    __syncthreads();
    const int excl = carry + (warp ? wsum[warp - 1] : 0) + x - v;
    __syncthreads();
    if (r < nt) scratch[r] = excl;
    if (threadIdx.x == blockDim.x - 1) carry = excl + v;
    __syncthreads();
  }
  for (int i = threadIdx.x; i < nt; i += blockDim.x) gstart[i] = scratch[rank(i)];
}

// k_compile for the dependency-driven schedule: the same instruction lists,
// with gate items at gitems[gstart[i] + j] (aux = i), the sweep program as
// sweeps[i], rem[i] = number of gate items of trajectory i; a trajectory
// without gate items has its sweep item pushed here.
__global__ void k_compile_dd(const TrajDev *trajs, const int *list, int nt, const int *gate_off, const int *gate_ks,
                             const int *meas_off, const int *meas_ks, const int *posts, int pcap, Instr *prog,
                             Item *sweeps,
                             Instr *gprog, Item *gitems, int gcap, int *gcount, const int *gstart, int *rem, Item *dyn,
                             int *dyn_tail) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *gcount = min(gate_off[nt], gcap);
  if (i >= nt) return;
  const int t = list[i];
  const int n = trajs[t].n;
  Instr *p = prog + size_t(i) * pcap;
  int pc = 0;
  auto emit = [&](int op, int k, int a, int b) {
    if (pc < pcap) p[pc] = Instr{op, k, a, b};
    ++pc;
  };
  const int g0 = gate_off[i], g1 = gate_off[i + 1];
  bool disjoint = true;
  for (int g = g0; g < g1 && disjoint; ++g)
    for (int h = g + 1; h < g1; ++h)
      if (abs(gate_ks[g] - gate_ks[h]) < 2) {
        disjoint = false;
        break;
      }
  int placed = 0;
  for (int g = g0; g < g1; ++g) {
    const int k = gate_ks[g];
    const bool valid = n > 1 && k >= 0 && k < n - 1;
    const int slot = gstart[i] + (g - g0);
    if (slot < gcap) {
      gprog[g < gcap ? g : slot] = (disjoint && valid) ? Instr{OP_GATE, k, g, 0} : Instr{OP_NOP, 0, 0, 0};
      gitems[slot] = Item{t, g < gcap ? g : slot, 1, i};
      ++placed;
    } else if (disjoint) {
      atomicOr(trajs[t].status, ST_BAD_INSTR);
    }
    if (!disjoint && valid) emit(OP_GATE, k, g, 0);
  }
  const int m0 = meas_off[i], m1 = meas_off[i + 1];
  int last = -1;
  for (int j = m0; j < m1; ++j) {
    const int k = meas_ks[j];
    if (k < 0 || k >= n || k <= last) continue;  // host guarantees sorted unique
    if (last >= 0)
      for (int b = last; b < k; ++b) emit(OP_REFACTOR, b, 0, 0);
    emit(OP_MEAS, k, j, posts ? (posts[j] == 0 || posts[j] == 1 ? posts[j] : -1) : -1);
    last = k;
  }
  if (last >= 0) {
    for (int b = last; b < n - 1; ++b) emit(OP_REFACTOR, b, 0, 0);
    for (int b = n - 3; b >= 0; --b) emit(OP_REFACTOR, b, 0, 0);
  }
  if (n >= 2) emit(OP_ENTROPY, n / 2 - 1, i, 0);
  if (pc > pcap) {  // program did not fit: run nothing, flag the trajectory
    atomicOr(trajs[t].status, ST_BAD_INSTR);
    pc = 0;
  }
  sweeps[i] = Item{t, int(size_t(i) * pcap), pc, 0};
  rem[i] = placed;
  if (placed == 0) {
    __threadfence();
    push_sweep(dyn, dyn_tail, sweeps, i);
  }
}

// ------------------------------------------------------------- launchers
#define TN_DECLARE_RUN(SUFFIX)                                                                              \
  cudaError_t launch_run_##SUFFIX(const LaunchArgs &la, int grid, int sortP, int ws_cap, cudaStream_t st);  \
  size_t run_smem_##SUFFIX(int sortP);                                                                      \
  size_t run_work_##SUFFIX(int cap);                                                                        \
  size_t run_team_##SUFFIX(int cap);                                                                        \
  int run_blocks_##SUFFIX(int sortP);                                                                       \
  int run_clusters_##SUFFIX(int sortP, int cluster);
TN_DECLARE_RUN(f32)
TN_DECLARE_RUN(f64)
TN_DECLARE_RUN(df)

cudaError_t launch_run(int prec, const LaunchArgs &la, int grid, int sortP, int ws_cap, cudaStream_t st) {
  if (la.cluster > 1 && !la.team) return cudaErrorInvalidValue;  // its members meet in the part
  if (prec == 0) return launch_run_f64(la, grid, sortP, ws_cap, st);
  if (prec == 2) return launch_run_df(la, grid, sortP, ws_cap, st);
  return launch_run_f32(la, grid, sortP, ws_cap, st);
}

size_t run_smem_bytes(int prec, int sortP) {
  return prec == 0 ? run_smem_f64(sortP) : (prec == 2 ? run_smem_df(sortP) : run_smem_f32(sortP));
}

size_t run_work_bytes(int prec, int cap) {
  return prec == 0 ? run_work_f64(cap) : (prec == 2 ? run_work_df(cap) : run_work_f32(cap));
}

size_t run_team_bytes(int prec, int cap) {
  return prec == 0 ? run_team_f64(cap) : (prec == 2 ? run_team_df(cap) : run_team_f32(cap));
}

namespace {
struct OutsideCaptures {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  OutsideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~OutsideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
}  // namespace

int DeviceMem::alloc(void **p, size_t bytes) {
  OutsideCaptures relaxed;
  const cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) {
    *p = nullptr;
    (void)cudaGetLastError();
  }
  return int(e);
}

void DeviceMem::free(void *p) {
  OutsideCaptures relaxed;
  (void)cudaFree(p);
}

size_t DeviceMem::available() {
  size_t avail = 0, total = 0;
  if (cudaMemGetInfo(&avail, &total) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return avail;
}

int run_clusters(int prec, int sortP, int cluster) {
  if (prec == 0) return run_clusters_f64(sortP, cluster);
  return prec == 2 ? run_clusters_df(sortP, cluster) : run_clusters_f32(sortP, cluster);
}

int run_blocks_per_sm(int prec, int sortP) {
  return prec == 0 ? run_blocks_f64(sortP) : (prec == 2 ? run_blocks_df(sortP) : run_blocks_f32(sortP));
}

// Observables (and one-site gates) of a single state without the executor:
// its arguments arrive by value, so a read is one launch and one copy back
// instead of four copies in, a launch of the whole executor and a copy back
// (an entropy, a Renyi entropy and the site probabilities of one state: 99 us
// through the executor, 78 us here).  Bound by launch and copy latency; the
// probabilities of a wide site by the loads that one SM has in flight (chi = 1024,
// df: 735 us in the executor, 1160 us on 256 threads, 360 us on 1024), while an
// entropy of a few hundred values takes longer on more threads.
constexpr int kObserveThreads = 256, kProbsThreads = 1024;

template <typename T, int NT>
__global__ void __launch_bounds__(NT) k_observe(const TrajDev *traj, int op, int k, double alpha, double *out) {
  extern __shared__ __align__(256) unsigned char osm[];
  Smem<T, kBlockW> sm(osm, 1);
  const TrajDev tr = *traj;
  if (op == OP_PROBS) {
    double p0, p1, sum;
    site_probs<T, NT, kBlockW>(tr, k, p0, p1, sum, sm);
    if (threadIdx.x == 0) {
      out[0] = p0;
      out[1] = p1;
    }
  } else {
    const double e = bond_entropy<NT>(tr, k, alpha, sm.red);
    if (threadIdx.x == 0) out[0] = e;
  }
}

// apply_unitary1 (mps.rs:1298-1314): Gamma_k[v,:,u] <- op Gamma_k[v,:,u]
struct Op1 {
  double v[8];
};

template <typename T>
__global__ void __launch_bounds__(kObserveThreads) k_unitary1(const TrajDev *traj, int k, Op1 op) {
  const TrajDev tr = *traj;
  const int cL = tr.chi[k], cR = tr.chi[k + 1];
  cpx<T> *g = gamma_slot<T>(tr, k);
  const cpx<T> o00 = mkc<T>(T(op.v[0]), T(op.v[1])), o01 = mkc<T>(T(op.v[2]), T(op.v[3]));
  const cpx<T> o10 = mkc<T>(T(op.v[4]), T(op.v[5])), o11 = mkc<T>(T(op.v[6]), T(op.v[7]));
  for (size_t idx = blockIdx.x * size_t(blockDim.x) + threadIdx.x; idx < size_t(cL) * cR;
       idx += size_t(gridDim.x) * blockDim.x) {
    const size_t v = idx / cR, u = idx % cR;
    const cpx<T> a = g[(v * 2 + 0) * cR + u], b = g[(v * 2 + 1) * cR + u];
    g[(v * 2 + 0) * cR + u] = cfma(o01, b, cmul(o00, a));
    g[(v * 2 + 1) * cR + u] = cfma(o11, b, cmul(o10, a));
  }
}

template <typename T>
static cudaError_t launch_observe_t(const TrajDev *traj, int cap, int op, int k, double alpha, double *out,
                                    cudaStream_t st) {
  // site_probs keeps the squared Lambdas of both bonds in shared memory
  const size_t smem = SmemLayout<T, kBlockW>::head_bytes + 2 * size_t(cap) * sizeof(T);
  if (smem > 48 * 1024) return cudaErrorInvalidValue;
  if (op == OP_PROBS)
    k_observe<T, kProbsThreads><<<1, kProbsThreads, smem, st>>>(traj, op, k, alpha, out);
  else
    k_observe<T, kObserveThreads><<<1, kObserveThreads, smem, st>>>(traj, op, k, alpha, out);
  return cudaGetLastError();
}

bool observe_fits(int prec, int cap) { return 2048 + 2 * size_t(cap) * (prec == 1 ? 4 : 8) <= 48 * 1024; }

cudaError_t launch_observe(int prec, const TrajDev *traj, int cap, int op, int k, double alpha, double *out,
                           cudaStream_t st) {
  if (prec == 0) return launch_observe_t<double>(traj, cap, op, k, alpha, out, st);
  if (prec == 2) return launch_observe_t<dd>(traj, cap, op, k, alpha, out, st);
  return launch_observe_t<float>(traj, cap, op, k, alpha, out, st);
}

cudaError_t launch_unitary1(int prec, const TrajDev *traj, int cap, int k, const double *op, cudaStream_t st) {
  Op1 o;
  for (int i = 0; i < 8; ++i) o.v[i] = op[i];
  const size_t blocks = (size_t(cap) * cap + kObserveThreads - 1) / kObserveThreads;
  const int grid = int(blocks < 64 ? blocks : 64);
  if (prec == 0)
    k_unitary1<double><<<grid, kObserveThreads, 0, st>>>(traj, k, o);
  else if (prec == 2)
    k_unitary1<dd><<<grid, kObserveThreads, 0, st>>>(traj, k, o);
  else
    k_unitary1<float><<<grid, kObserveThreads, 0, st>>>(traj, k, o);
  return cudaGetLastError();
}

cudaError_t launch_reset(TrajDev *trajs, const int *list, int count, int prec, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  k_reset<<<count, 128, 0, st>>>(trajs, list, count, prec);
  return cudaGetLastError();
}

cudaError_t launch_compile(const TrajDev *trajs, const int *list, int nt, const int *order, const int *gate_off,
                           const int *gate_ks, const int *meas_off, const int *meas_ks, const int *posts, int pcap,
                           Instr *prog, Item *items, Instr *gprog, Item *gitems, int gcap, int *gcount,
                           cudaStream_t st) {
  if (nt <= 0) return cudaSuccess;
  k_compile<<<(nt + 127) / 128, 128, 0, st>>>(trajs, list, nt, order, gate_off, gate_ks, meas_off, meas_ks, posts,
                                              pcap, prog, items, gprog, gitems, gcap, gcount);
  return cudaGetLastError();
}

cudaError_t launch_lpt_order(const TrajDev *trajs, const int *list, int nt, const int *meas_off, int *order,
                             cudaStream_t st) {
  if (nt <= 0) return cudaSuccess;
  int P = 1;
  while (P < nt && P < kLptMax) P <<= 1;
  k_lpt_order<<<1, 1024, size_t(P) * (sizeof(double) + sizeof(int)), st>>>(trajs, list, nt, meas_off, order);
  return cudaGetLastError();
}

cudaError_t launch_compile_dd(const TrajDev *trajs, const int *list, int nt, const int *order, const int *gate_off,
                              const int *gate_ks, const int *meas_off, const int *meas_ks, const int *posts, int pcap,
                              Instr *prog, Item *sweeps, Instr *gprog, Item *gitems, int gcap, int *gcount,
                              int *gstart, int *scratch, int *rem, Item *dyn, int *dyn_tail, cudaStream_t st) {
  if (nt <= 0) return cudaSuccess;
  k_gate_slots<<<1, 1024, 0, st>>>(nt, order, gate_off, scratch, gstart);
  k_compile_dd<<<(nt + 127) / 128, 128, 0, st>>>(trajs, list, nt, gate_off, gate_ks, meas_off, meas_ks, posts, pcap,
                                                 prog, sweeps, gprog, gitems, gcap, gcount, gstart, rem, dyn,
                                                 dyn_tail);
  return cudaGetLastError();
}

}  // namespace tn
