// tn_team.cuh -- SVD of large bonds (more vectors than svd_local takes), on one
// CTA or shared by a team: float block Jacobi for the bulk of the sweeps, then
// the transition to the working precision and the refinement of svd_local as
// tensor-core double-float products (tn_oz.cuh).
//
// Why: with the sweeps run on the double-float vectors themselves every block
// step paid a double-float update (66 of 175 us at 512 x 512), rebuilt
// double-float rotations (49 us) and, in the finishing sweeps, a double-float
// Gram matrix (54 us).  A float step costs a quarter of that, and the
// double-float work shrinks to a handful of whole products.
#pragma once

namespace tn {

// Workspace of svd_team beside Work<T> (global memory, per team).
struct TeamWork {
  cpx<float> *A32;   // ell x c float vectors (float: the vectors themselves)
  cpx<float> *V32;   // c x c accumulated rotations, then K; columns contiguous
  cpx<dd> *S;        // c x c: V^H V - I, W, G
  cpx<dd> *B;        // ell x c intermediate product
  void *plP, *plQ;   // digit planes
  int *exP, *exQ;
  float *nrm;        // c squared column norms
  dd *dg;            // c factors of the unitary correction
  float *cs;         // c column scales (powers of two)
  unsigned int *flag;  // cross-CTA flags and maxima
};
constexpr int kTeamFlags = 64;
constexpr int kTeamItem = 8;  // words after the flags: the work item that the first member took

// Bytes of that workspace for bond capacity cap; zero where svd_team does not run.
template <typename T>
size_t __host__ __device__ team_bytes(int cap) {
  if (2 * cap <= 64) return 0;  // bond_local takes every bond
  if (!std::is_same<T, dd>::value) return sizeof(T) == 4 ? size_t(2) * cap * sizeof(float) + 2048 : 0;
  const size_t n4 = size_t(4) * cap * cap, rows = size_t(2) * cap, ld = size_t(4) * cap + 32;
  size_t b = 2 * n4 * sizeof(cpx<float>) + 2 * n4 * sizeof(cpx<dd>) + 2 * (8 * rows * ld * 2) + 2 * rows * sizeof(int) +
             rows * (2 * sizeof(float) + sizeof(dd)) + (kTeamFlags + kTeamItem) * sizeof(int) + 4096;
  return (b + 255) & ~size_t(255);
}

template <typename T>
__device__ inline TeamWork team_work(void *base, int cap) {
  TeamWork w{};
  unsigned char *p = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(base) + 255) & ~uintptr_t(255));
  auto take = [&](size_t bytes) {
    unsigned char *q = p;
    p += (bytes + 255) & ~size_t(255);
    return q;
  };
  const size_t n4 = size_t(4) * cap * cap, rows = size_t(2) * cap, ld = size_t(4) * cap + 32;
  w.flag = reinterpret_cast<unsigned int *>(take((kTeamFlags + kTeamItem) * sizeof(int)));
  w.nrm = reinterpret_cast<float *>(take(rows * sizeof(float)));
  if (std::is_same<T, dd>::value) {
    w.dg = reinterpret_cast<dd *>(take(rows * sizeof(dd)));
    w.cs = reinterpret_cast<float *>(take(rows * sizeof(float)));
    w.exP = reinterpret_cast<int *>(take(rows * sizeof(int)));
    w.exQ = reinterpret_cast<int *>(take(rows * sizeof(int)));
    w.A32 = reinterpret_cast<cpx<float> *>(take(n4 * sizeof(cpx<float>)));
    w.V32 = reinterpret_cast<cpx<float> *>(take(n4 * sizeof(cpx<float>)));
    w.S = reinterpret_cast<cpx<dd> *>(take(n4 * sizeof(cpx<dd>)));
    w.B = reinterpret_cast<cpx<dd> *>(take(n4 * sizeof(cpx<dd>)));
    w.plP = take(8 * rows * ld * 2);
    w.plQ = take(8 * rows * ld * 2);
  }
  return w;
}

// Largest of the team's non-negative values (uniform over the team).  Slots of
// flag rotate so that a slot is cleared long before its next use.
template <int NT>
__device__ float team_max(const Team &tm, float v, TeamWork &tw, int &slot, double *red) {
  v = block_max<NT>(v, red);
  if (tm.size == 1) return v;
  const int s = slot % kTeamFlags;
  slot++;
  if (threadIdx.x == 0) atomicMax(tw.flag + s, __float_as_uint(v));
  tm.sync();
  const unsigned int m = *reinterpret_cast<volatile unsigned int *>(tw.flag + s);
  if (tm.rank == 0 && threadIdx.x == 0) tw.flag[(s + kTeamFlags / 2) % kTeamFlags] = 0u;
  return __uint_as_float(m);
}

// One block-pair step of the float sweeps: the 32 columns cols of A32 (length
// ell) are orthogonalised against each other, V32 (c rows, when set) follows.
// rot / far: some pair was above the threshold / above `done` (kLastWord: by pair_far's rule).
template <int NT, int W>
__device__ void float_step(cpx<float> *A32, int ell, cpx<float> *V32, int c, const int *cols, float tol, float done,
                           float tiny2, int inner, int &rot, int &far, Smem<float, W> &sf) {
  constexpr int B = W / 2, GP = W + 1;
  using L = SmemLayout<float, W>;
  const bool res = ell <= L::RES_ROWS;
  if (res) {
    load_half_res<float, NT, W>(A32, ell, cols, 0, sf);
    load_half_res<float, NT, W>(A32, ell, cols, B, sf);
    __syncthreads();
    gram_res<float, NT, W>(ell, sf);
  } else {
    gram_stream<float, NT, W>(A32, ell, cols, sf);
  }
  int need = 0;  // 1: a pair inside a half, 2: a pair across the halves, 4: far
  for (int idx = threadIdx.x; idx < W * W; idx += NT) {
    const int p = idx / W, q = idx % W;
    if (p < q && cols[p] >= 0 && cols[q] >= 0) {
      const float a = sf.G[p * GP + p].x, b = sf.G[q * GP + q].x;
      const cpx<float> g = sf.G[p * GP + q];
      if (pair_active<float>(a, b, g, tol, tiny2)) need |= (p < B) != (q < B) ? 2 : 1;
      if (done > kLastWord ? pair_active<float>(a, b, g, done, tiny2) : pair_far(a, b, g, tol, tiny2)) need |= 4;
    }
  }
  const int w1 = __syncthreads_or(need & 1), w2 = __syncthreads_or(need & 2), w4 = __syncthreads_or(need & 4);
  far |= w4;
  if (!(w1 || w2)) {
    __syncthreads();
    return;
  }
  rot = 1;
  const int mode = w1 && w2 ? 0 : (w2 ? 1 : 2);
  const cpx<float> *Jm = jacobi_gram<float, NT, W>(sf, cols, tol, tiny2, mode, inner);
  if (res) {
    update_res<float, NT, W>(ell, Jm, sf);
    store_half_res<float, NT, W>(A32, ell, cols, 0, sf);
    store_half_res<float, NT, W>(A32, ell, cols, B, sf);
  } else {
    update_stream<float, NT, W>(A32, ell, ell, cols, Jm, sf);
  }
  if (V32) {
    if (c <= L::RES_ROWS) {
      __syncthreads();
      load_half_res<float, NT, W>(V32, c, cols, 0, sf);
      load_half_res<float, NT, W>(V32, c, cols, B, sf);
      __syncthreads();
      update_res<float, NT, W>(c, Jm, sf);
      store_half_res<float, NT, W>(V32, c, cols, 0, sf);
      store_half_res<float, NT, W>(V32, c, cols, B, sf);
    } else {
      update_stream<float, NT, W>(V32, c, c, cols, Jm, sf);
    }
  }
  __syncthreads();
}

// Float block Jacobi sweeps of the team over half-blocks of 16 columns, renamed
// by decreasing norm each sweep (de Rijk).  The pairs go in the row-cyclic
// order's own parallel schedule: round r holds the disjoint pairs (i, r + 1 - i),
// which the members share, one team barrier a round; every pair still comes
// after the ones that row-cyclic order puts before it.  A round-robin ordering
// has half as many rounds but converges in 9 sweeps where this takes 5 (a
// 256 x 256 theta): the large columns no longer meet all others first.
// Returns the sweeps, -1 at the limit.  Team-uniform.
template <int NT, int W, typename S>
__device__ int float_sweeps(const Team &tm, cpx<float> *A32, int ell, cpx<float> *V32, int c, float floor_, float done,
                            int max_sweeps, TeamWork &tw, int &slot, S &sm, long long *cyc) {
  constexpr int B = W / 2;
  Smem<float, W> sf(as_shared(sm.base), 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nblk = (c + B - 1) / B;
  const float tol = 4.f * sqrtf(float(ell)) * Eps<float>::v;
  int *cols = sf.ired + 128;
  // the order of the columns, at the end of the arena (beyond the float areas)
  int *ord = reinterpret_cast<int *>(sm.r0 + sm.arena) - ((c + 3) & ~3);
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    for (int j = tm.rank * (NT / 32) + warp; j < c; j += tm.size * (NT / 32)) {
      float s = 0.f;
      for (int i = lane; i < ell; i += 32) s += cabs2(A32[size_t(j) * ell + i]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) tw.nrm[j] = s;
    }
    tm.sync();
    int P = 1;
    while (P < c) P <<= 1;
    double *key = reinterpret_cast<double *>(sm.r0);
    int *kidx = reinterpret_cast<int *>(key + P);
    float part = 0.f;
    for (int j = threadIdx.x; j < P; j += NT) {
      const float x = j < c ? tw.nrm[j] : 0.f;
      key[j] = j < c ? double(order_key(x)) : kOrderPad;
      kidx[j] = j;
      if (j < c) part += x;
    }
    double fro = block_sum<NT>(double(part), sm.red);
    __syncthreads();
    bitonic_desc<float, NT, W>(key, kidx, P);
    for (int j = threadIdx.x; j < c; j += NT) ord[j] = kidx[j];
    const float tiny2 = fmaxf(float(fro) * floor_ * floor_, 1e-37f);
    tm.sync();  // every member has read the norms
    int rot = 0, far = 0;
    const int inner = sweep < 3 ? 2 : 1;
    for (int r = 0; r <= 2 * nblk - 4; ++r) {
      for (int I = max(0, r + 2 - nblk) + tm.rank; 2 * I < r + 1; I += tm.size) {
        const int J = r + 1 - I;
        if (threadIdx.x < W) {
          const int q = threadIdx.x, pos = q < B ? I * B + q : J * B + q - B;
          cols[q] = pos < c ? ord[pos] : -1;
        }
        __syncthreads();
        cyc[3] += 1;
        float_step<NT, W>(A32, ell, V32, c, cols, tol, done, tiny2, inner, rot, far, sf);
      }
      tm.sync();
    }
    const float any = team_max<NT>(tm, float((far ? 2 : 0) | (rot ? 1 : 0)), tw, slot, sm.red);
    if (any < 2.f) return sweep + 1;
  }
  return -1;
}

// Largest row sum of |M| (its leading parts), each row by a warp: the same on
// teams of every size.  get(r, k): entry as cpx<float>.
template <int NT, class FG>
__device__ float team_row_sum(const Team &tm, int c, FG get, TeamWork &tw, int &slot, double *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = NT / 32;
  float most = 0.f;
  for (int r = tm.rank * nw + warp; r < c; r += tm.size * nw) {
    float s = 0.f;
    for (int k = lane; k < c; k += 32) {
      const cpx<float> v = get(r, k);
      s += fabsf(v.x) + fabsf(v.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    most = s > most || s != s ? s : most;  // (NaN stays)
  }
  return team_max<NT>(tm, most, tw, slot, red);
}

// W (unit_entry) of S (c x c, Hermitian) in place of S, transposed: S[y][k] =
// W[k][y], the rows that a product with W on the right takes.  The square from
// 3 digits (a relative 2^-21 of its 1e-6 at the most), and where the square's
// norm asks for it the next two terms, S1^2 (-5/16 S1 + 35/128 S1^2), too
// (the matrices commute, so the product is Hermitian).  The norms are row sums
// of S1^2, each by a warp: the same on teams of every size.  Returns false (S
// spoilt) when the series does not reach: the terms left out are below 3/5 of
// the norm of S1 to the third power (1e-15) or the fifth (5e-16).
// Scratch: the planes' memory.
constexpr float kTeamSquare = 1.2e-5f, kTeamMax = 1e-3f;
template <int NT, typename S>
__device__ bool team_correction(const Team &tm, int c, TeamWork &tw, int &slot, S &sm) {
  const OzPlanes p = oz_planes(tw.plP, tw.exP, c, c, 3);
  cpx<dd> *sq = reinterpret_cast<cpx<dd> *>(tw.plQ), *hi = sq;
  float w2 = 0.375f;
  for (int k = tm.rank * NT + threadIdx.x; k < c; k += tm.size * NT) tw.dg[k] = dg_minus1(tw.S[size_t(k) * c + k].x);
  tm.sync();
  oz_split<NT, 3>(tm, p, c, [&](int r, int k) {
    if (r == k) return czero<dd>();
    const cpx<dd> s = tw.S[size_t(r) * c + k];
    const float g = (1.f + tw.dg[r].hi) * (1.f + tw.dg[k].hi);
    return mkc<dd>(dd(s.x.hi * g), dd(s.y.hi * g));
  });
  tm.sync();
  oz_gemm<NT>(tm, p, p, true, 3, kOzHerm, sq, c, nullptr, sm);  // S1 S1^H
  tm.sync();
  const float n2 = team_row_sum<NT>(
      tm, c, [&](int r, int k) { return mkc<float>(sq[size_t(r) * c + k].x.hi, sq[size_t(r) * c + k].y.hi); }, tw, slot,
      sm.red);
  if (!(n2 <= kTeamMax * kTeamMax)) return false;
  if (n2 > kTeamSquare * kTeamSquare) {
    // planes of S1^2 behind it, those of the other factor and the result in the
    // other buffer (each holds 8 planes of c rows; S1's own have served)
    unsigned char *const after = reinterpret_cast<unsigned char *>(tw.plQ) + ((size_t(c) * c * sizeof(cpx<dd>) + 255) & ~size_t(255));
    const OzPlanes a = oz_planes(after, tw.exQ, c, c, 3), b = oz_planes(tw.plP, tw.exP, c, c, 3);
    hi = reinterpret_cast<cpx<dd> *>(reinterpret_cast<unsigned char *>(tw.plP) + ((3 * b.stride * 2 + 255) & ~size_t(255)));
    w2 = 1.f;
    oz_split<NT, 3>(tm, a, c, [&](int r, int k) { return sq[size_t(r) * c + k]; });
    oz_split<NT, 3>(tm, b, c, [&](int r, int k) {
      const cpx<dd> q = sq[size_t(r) * c + k];
      cpx<float> v = mkc<float>(0.2734375f * q.x.hi, 0.2734375f * q.y.hi);
      if (r != k) {
        const cpx<dd> s = tw.S[size_t(r) * c + k];
        const float g = -0.3125f * (1.f + tw.dg[r].hi) * (1.f + tw.dg[k].hi);
        v = mkc<float>(fmaf(s.x.hi, g, v.x), fmaf(s.y.hi, g, v.y));
      }
      return mkc<dd>(dd(v.x), dd(v.y));
    });
    tm.sync();
    oz_gemm<NT>(tm, a, b, true, 3, kOzHerm, hi, c, nullptr, sm);  // A B^H = S1^2 B
    tm.sync();
    for (int e = tm.rank * NT + threadIdx.x; e < c * c; e += tm.size * NT) {
      const cpx<dd> q = sq[e], h = hi[e];
      hi[e] = mkc<dd>(dd(fmaf(0.375f, q.x.hi, h.x.hi)), dd(fmaf(0.375f, q.y.hi, h.y.hi)));
    }
    tm.sync();
  }
  // S[x][y] = conj(S[y][x]): entry (y, x) of W^T is W[x][y] with S[x][y] = conj of what is there
  for (int e = tm.rank * NT + threadIdx.x; e < c * c; e += tm.size * NT) {
    const int y = e / c, x = e - y * c;
    const cpx<dd> s = tw.S[e];
    tw.S[e] = unit_entry(x == y, mkc<dd>(s.x, -s.y), tw.dg[x], tw.dg[y], mkc<float>(w2 * hi[e].x.hi, -w2 * hi[e].y.hi));
  }
  tm.sync();
  return true;
}

// Powers of two near the norms of the columns of M (length ell): a product with
// the columns divided and the other operand's rows multiplied by them keeps
// small columns accurate relative to themselves, although the digits of a row
// are cut relative to its largest entry.
template <int NT>
__device__ void team_scales(const Team &tm, const cpx<dd> *M, int ell, int c, TeamWork &tw) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = NT / 32;
  for (int j = tm.rank * nw + warp; j < c; j += tm.size * nw) {
    float s = 0.f;
    for (int i = lane; i < ell; i += 32) {
      const cpx<dd> v = M[size_t(j) * ell + i];
      s = fmaf(v.x.hi, v.x.hi, fmaf(v.y.hi, v.y.hi, s));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) tw.cs[j] = s > 1e-36f && isfinite(s) ? pow2f(oz_exponent(sqrtf(s))) : 1.f;
  }
  tm.sync();
}
__device__ __forceinline__ cpx<dd> dd_scale(cpx<dd> v, float f) {  // f a power of two
  return mkc<dd>(dd(v.x.hi * f, v.x.lo * f), dd(v.y.hi * f, v.y.lo * f));
}

// A <- A X (1 + W) with X the columns V32 (add = false: V, rounded to 28-bit
// fixed point, whose S = V^H V - I is exact; add = true: I + K, S = K^H K) and
// W from team_correction: a unitary X (1 + W) near X applied in double-float.
// Returns false (A unchanged) when X is too far from unitary for that.
template <int NT, typename S>
__device__ bool team_transform(const Team &tm, cpx<dd> *A, int ell, int c, bool add, TeamWork &tw, int &slot, S &sm) {
  OzPlanes x = oz_planes(tw.plQ, tw.exQ, c, c, add ? 6 : 4);
  auto col = [&](int y, int k) {
    const cpx<float> v = tw.V32[size_t(y) * c + k];
    return mkc<dd>(dd(v.x), dd(v.y));
  };
  if (add)
    oz_split<NT, 6>(tm, x, c, col);
  else
    oz_split<NT, 4>(tm, x, c, col, 1);
  tm.sync();
  // S[p][q] = sum_k conj(X[k][p]) X[k][q]: planes by column serve both operands
  oz_gemm<NT>(tm, x, x, true, add ? 5 : 7, kOzHermT, tw.S, c, nullptr, sm);
  tm.sync();
  float dmax = 0.f;
  for (int k = tm.rank * NT + threadIdx.x; k < c; k += tm.size * NT) {
    dd &v = tw.S[size_t(k) * c + k].x;
    if (!add) v = v - dd(1.f);
    dmax = fabsf(v.hi) > dmax || v.hi != v.hi ? fabsf(v.hi) : dmax;
  }
  dmax = team_max<NT>(tm, dmax, tw, slot, sm.red);
  if (!(dmax <= 0.1f)) return false;
  // B = A X (+ A): rows of A against the columns of X
  const OzPlanes pa = oz_planes(tw.plP, tw.exP, ell, c, add ? 6 : 8);
  if (add) {
    team_scales<NT>(tm, A, ell, c, tw);
    oz_split<NT, 6>(tm, pa, c, [&](int i, int k) { return dd_scale(A[size_t(k) * ell + i], 1.f / tw.cs[k]); });
    oz_split<NT, 6>(tm, x, c, [&](int y, int k) { return dd_scale(col(y, k), tw.cs[k]); });
  } else {
    // (V mixes all columns; theta's are of one size)
    oz_split<NT, 8>(tm, pa, c, [&](int i, int k) { return A[size_t(k) * ell + i]; });
  }
  tm.sync();
  oz_gemm<NT>(tm, pa, x, false, add ? 6 : 8, kOzTrans, tw.B, ell, add ? A : nullptr, sm);
  tm.sync();
  if (!team_correction<NT>(tm, c, tw, slot, sm)) return false;
  // A = B + B W; W below 1e-3, so six digits leave 1e-16 of every column
  team_scales<NT>(tm, tw.B, ell, c, tw);
  const OzPlanes pb = oz_planes(tw.plP, tw.exP, ell, c, 6), w = oz_planes(tw.plQ, tw.exQ, c, c, 6);
  oz_split<NT, 6>(tm, pb, c, [&](int i, int k) { return dd_scale(tw.B[size_t(k) * ell + i], 1.f / tw.cs[k]); });
  oz_split<NT, 6>(tm, w, c, [&](int y, int k) { return dd_scale(tw.S[size_t(y) * c + k], tw.cs[k]); });
  tm.sync();
  oz_gemm<NT>(tm, pb, w, false, 6, kOzTrans, A, ell, tw.B, sm);
  tm.sync();
  return true;
}

// Orthogonalises the c double-float vectors of A (vector-contiguous, length
// ell, global memory).  Same plan and result as svd_local; team-uniform.
template <int NT, int W>
__device__ int svd_team(const Team &tm, cpx<dd> *A, int ell, int c, int max_sweeps, TeamWork &tw, Smem<dd, W> &sm,
                        long long *cyc) {
  const float floor_t = float(sweep_floor<dd>(ell));
  const float tol = float(4.0 * sqrt(double(ell)) * double(Eps<dd>::v));
  constexpr int kMaxStages = 3, kMaxSteps = 10;
  constexpr float kSlight = 1e-7f;
  const int gthreads = tm.size * NT, gid = tm.rank * NT + threadIdx.x;
  int sweeps = 0, stages = 0, slot = 0;
  if (tm.rank == 0)
    for (int i = threadIdx.x; i < kTeamFlags; i += NT) tw.flag[i] = 0u;
  bool bulk = true, fine = false;
  for (int step = 0; step < kMaxSteps; ++step) {
    long long t0 = clock64();
    if (bulk) {
      for (size_t i = gid; i < size_t(c) * ell; i += gthreads) tw.A32[i] = mkc<float>(A[i].x.hi, A[i].y.hi);
      for (int i = gid; i < c * c; i += gthreads) tw.V32[i] = mkc<float>(i % (c + 1) == 0 ? 1.f : 0.f, 0.f);
      tm.sync();
      const int sw = float_sweeps<NT, W>(tm, tw.A32, ell, tw.V32, c, stages == 0 ? Eps<float>::v : floor_t, 1e-4f,
                                         min(max_sweeps, 20), tw, slot, sm, cyc);
      sweeps += sw < 0 ? min(max_sweeps, 20) : sw;
      ++stages;
      cyc[1] += clock64() - t0;
      t0 = clock64();
      const bool ok = team_transform<NT>(tm, A, ell, c, false, tw, slot, sm);
      cyc[2] += clock64() - t0;
      t0 = clock64();
      if (!ok) return -1;
      bulk = false;
    }
    // Gram matrix of the vectors, by rows of A: S[p][q] = sum_i conj(a_p) a_q.  The first one only steers a step
    // whose own accuracy is 1e-8; later ones decide convergence.
    const OzPlanes g = oz_planes(tw.plP, tw.exP, c, ell, fine ? 8 : 5);
    auto vec = [&](int p, int k) { return A[size_t(p) * ell + k]; };
    if (fine)
      oz_split<NT, 8>(tm, g, ell, vec);
    else
      oz_split<NT, 5>(tm, g, ell, vec);
    tm.sync();
    oz_gemm<NT>(tm, g, g, true, fine ? 8 : 5, kOzHermT, tw.S, c, nullptr, sm);
    tm.sync();
    float fro = 0.f;
    {
      float part = 0.f;
      for (int j = threadIdx.x; j < c; j += NT) part += tw.S[size_t(j) * c + j].x.hi;
      fro = float(block_sum<NT>(double(part), sm.red));
    }
    const float tiny2 = fmaxf(fro * floor_t * floor_t, 1e-37f);
    float rmax = 0.f, kmax = 0.f;
    for (int e = gid; e < c * c; e += gthreads) {
      const int p = e / c, q = e - p * c;
      if (p > q) continue;
      cpx<float> vpq = czero<float>(), vqp = czero<float>();
      if (p != q) {
        const dd at_ = tw.S[size_t(p) * c + p].x, bt_ = tw.S[size_t(q) * c + q].x;
        const float a = at_.hi, b = bt_.hi;
        if (a > tiny2 && b > tiny2) {
          const cpx<dd> gv = tw.S[size_t(p) * c + q];
          const float sc = rsqrtf(a) * rsqrtf(b);
          const float hx = gv.x.hi * sc, hy = gv.y.hi * sc, r2 = fmaf(hx, hx, hy * hy), r = sqrtf(r2);
          rmax = fmaxf(rmax, r);
          if (r > tol) {
            const float rr = 1.f / r;
            const float z = 0.5f * ((bt_ - at_).hi * sc) * rr;
            const float z1 = fmaf(z, z, 1.f);
            const float t = fabsf(z) > 1e15f ? 0.5f / z : copysignf(1.f / (fabsf(z) + sqrtf(z1)), z);
            kmax = fmaxf(kmax, fabsf(t));
            const float ex = hx * rr, ey = -hy * rr;
            vqp = mkc<float>(-t * ex, -t * ey);
            vpq = mkc<float>(t * ex, -t * ey);
          }
        }
      }
      tw.V32[size_t(p) * c + q] = vqp;
      tw.V32[size_t(q) * c + p] = vpq;
    }
    rmax = team_max<NT>(tm, rmax, tw, slot, sm.red);
    kmax = team_max<NT>(tm, kmax, tw, slot, sm.red);
    tm.sync();
    cyc[0] += clock64() - t0;
    t0 = clock64();
    if (!(rmax < 2.f)) return -1;
    if (rmax <= tol && fine) return sweeps + 1;
    ++sweeps;
    const float far = fmaxf(rmax, kmax);  // as svd_local
    const bool last = fine && rmax * far * 8.f <= tol;
    // A += A K where the second order, which it leaves out, is below 2^-47
    // (beyond, or where K's entries are not all small: with its unitary factor)
    bool slight = far <= 1e-7f;
    if (slight)
      slight = team_row_sum<NT>(tm, c, [&](int r, int k) { return tw.V32[size_t(r) * c + k]; }, tw, slot, sm.red) <= kSlight;
    if (slight) {
      team_scales<NT>(tm, A, ell, c, tw);
      // K below 1e-7, so four digits of both leave 1e-16
      const OzPlanes k = oz_planes(tw.plQ, tw.exQ, c, c, 4), pa = oz_planes(tw.plP, tw.exP, ell, c, 4);
      oz_split<NT, 4>(tm, k, c, [&](int y, int p) {
        const cpx<float> v = tw.V32[size_t(y) * c + p];
        return mkc<dd>(dd(v.x * tw.cs[p]), dd(v.y * tw.cs[p]));
      });
      oz_split<NT, 4>(tm, pa, c, [&](int i, int p) { return dd_scale(A[size_t(p) * ell + i], 1.f / tw.cs[p]); });
      tm.sync();
      oz_gemm<NT>(tm, pa, k, false, 4, kOzTrans, A, ell, A, sm);
      tm.sync();
    } else if (rmax > 1e-3f && kmax > 0.3f && stages < kMaxStages) {
      bulk = true;
    } else if (!team_transform<NT>(tm, A, ell, c, true, tw, slot, sm)) {
      return -1;
    }
    cyc[2] += clock64() - t0;
    if (last) return sweeps + 1;
    fine = !bulk;
  }
  return -1;
}

}  // namespace tn
