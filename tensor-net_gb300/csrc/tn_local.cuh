// tn_local.cuh -- bond operations that fit the CTA's shared memory.
//
// Most bond operations of a trajectory are small (chain ends, early layers,
// strongly measured circuits), and their time is latency: barriers, scalar
// chains and round trips to global scratch, not arithmetic.  Here theta, the
// Jacobi vectors and every per-value array stay in shared memory, products
// have exactly as many terms as the bond has (no tile padding), and the SVD is
// split by precision:
//
//  1. float one-sided (Hestenes) Jacobi on a float copy of the vectors, the
//     rotations accumulated in V (hestenes): one barrier a round, no Gram matrix;
//  2. V made unitary to the working precision by a Newton-Schulz step
//     (unitarise), and A <- A Q in the working precision (apply_unitary): exact
//     to its rounding, so the float angles cost no accuracy;
//  3. refinement: the Gram matrix of A in the working precision gives every
//     remaining rotation at once, tan(theta) = t for each pair as in a Jacobi
//     rotation; I + K with K_qp = -t e, K_pq = t conj(e) is made unitary (by a
//     short series while K is small, unitary_step; else as in 2) and applied.
//     The off-diagonals fall quadratically; two steps usually reach the working
//     precision's threshold.
//
// The sweeps of 1 are the many, cheap ones; the working precision pays for two
// or three products instead of every rotation of every sweep.  Pairs that are
// degenerate to the float rounding cannot be separated by 3 (K would not be
// small); svd_local then reports so and the caller goes on with the block
// Jacobi on the (already unitarily transformed) vectors.
//
// Code size counts: an operation of a few vectors runs most of its code once.
// Sums unrolled four or eight times, with a copy per call, leave the warps
// waiting for instructions a third of the time that they are not at a barrier
// (46 % of the instruction cache's requests miss) and cost a quarter of such
// batches' time (304 trajectories at n = 64: 101 against 84 ms).  So one copy of
// every product, rolled loops where a loop is short, and unrolling only inside
// the float sweeps, where bonds of 16 and more vectors need it (5 %).
#pragma once

namespace tn {

// Float sweeps that are the last word end after one whose pairs leave nothing
// above the threshold (7e-7 to 1e-5): what a sweep leaves is of second order in
// what it found, r r' between vectors of different size (below 1e-9 with every r
// below kFloatDone) and r |t| between neighbours (r = |g| / (|a| |b|) before the
// rotation by the angle t; in a cluster of nearly equal values t is near 1 however
// small r is, and up to 2.6 times the threshold was left of a cluster of 128).
constexpr float kFloatDone = 3e-5f;
__device__ __forceinline__ bool pair_far(float a, float b, cpx<float> g, float tol, float tiny2) {
  if (!(a > tiny2 && b > tiny2)) return false;
  const float s = 1.f / (sqrtf(a) * sqrtf(b)), r = sqrtf(cabs2(g)) * s, d = fabsf(b - a) * s;
  if (!(r > tol)) return false;
  const float t = 2.f * r / (d + sqrtf(fmaf(d, d, 4.f * r * r)));
  return r > kFloatDone || 8.f * r * t > tol;
}
constexpr float kLastWord = 0.f;  // `done` of such sweeps

// ------------------------------------------------------------- arithmetic
// Arithmetic of the sums that need more than float but not float64's
// throughput cost (float64 issues at 1/64 of the float rate): double-float
// for float and dd, float64 only where the working precision is float64.
template <typename T>
struct RedType {
  using type = dd;
};
template <>
struct RedType<double> {
  using type = double;
};
// Arithmetic of bond_local: MIXED computes in double-float too, so that its
// rounding is that of the stored float Gammas.  (All in float it was a third
// faster, but the rotations' own rounding, sqrt(rotations) 2^-24, made its
// errors no smaller than before.)  Its vectors need orthogonality to 1e-8 only:
// what is left enters the recovered side as 1e-8 sigma_1 / sigma_j, of weight
// sigma_j.
template <typename TS>
struct LocalType {
  using type = dd;
};
template <>
struct LocalType<double> {
  using type = double;
};
__device__ __forceinline__ cpx<dd> widen(cpx<float> v) { return mkc<dd>(dd(v.x), dd(v.y)); }
__device__ __forceinline__ cpx<dd> widen(cpx<dd> v) { return v; }
__device__ __forceinline__ cpx<double> widen(cpx<double> v) { return v; }
template <typename TS, typename T>
__device__ __forceinline__ cpx<TS> narrow(cpx<T> v) {
  return mkc<TS>(TS(v.x), TS(v.y));
}
__device__ __forceinline__ float lead(float x) { return x; }
__device__ __forceinline__ float lead(double x) { return float(x); }
__device__ __forceinline__ float lead(dd x) { return x.hi; }
template <typename T>
__device__ __forceinline__ T from_dd(dd x) {
  return T(x);
}
template <>
__device__ __forceinline__ double from_dd<double>(dd x) {
  return double(x.hi) + double(x.lo);
}

// Sum of products of floats, every product exact, the sum in three floats
// (about 2^-60 of its largest term: V^H V - I cancels to 1e-6 and its own
// error is what V's unitarity is held to, in float64 too).
struct tacc {
  float hi, mid, lo;
};
__device__ __forceinline__ void tacc_add_prod(tacc &s, float a, float b) {
  float p, e, h, t, u;
  two_prod(a, b, p, e);
  two_sum(s.hi, p, h, t);
  s.hi = h;
  two_sum(s.mid, t, h, u);
  s.mid = h;
  s.lo = __fadd_rn(s.lo, __fadd_rn(u, e));
}
__device__ __forceinline__ dd tacc_fin(const tacc &s) {
  float h, e, m, f;
  two_sum(s.hi, s.mid, h, e);
  two_sum(e, s.lo, m, f);
  return dd_norm(h, m);
}
// acc + a w with w double-float
__device__ __forceinline__ void dacc_add_fdprod(dacc &s, float a, dd w) {
  float p, e, h, t;
  two_prod(a, w.hi, p, e);
  e = __fmaf_rn(a, w.lo, e);
  two_sum(s.hi, p, h, t);
  s.hi = h;
  s.lo = __fadd_rn(s.lo, __fadd_rn(t, e));
}

// Largest of the threads' non-negative values (uniform result).
template <int NT>
__device__ __forceinline__ float block_max(float v, double *red) {
  unsigned int *r = reinterpret_cast<unsigned int *>(red);
  // NaN compares above every number here (its bit pattern does), so a bad
  // value is seen by the caller's upper limits
  unsigned int m = __reduce_max_sync(0xffffffffu, __float_as_uint(v) & 0x7fffffffu);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = m;
  __syncthreads();
  m = r[threadIdx.x & (NT / 32 - 1)];
  m = __reduce_max_sync(0xffffffffu, m);
  return __uint_as_float(m);
}

// Sums of two values over the CTA in the arithmetic R (uniform result).
template <typename R, int NT>
__device__ __forceinline__ void block_sum2_in(R &a, R &b, double *red) {
  R *r = reinterpret_cast<R *>(red);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a = a + shfl_xor(a, o);
    b = b + shfl_xor(b, o);
  }
  __syncthreads();
  if (lane == 0) {
    r[warp] = a;
    r[NT / 32 + warp] = b;
  }
  __syncthreads();
  if (warp == 0) {
    a = lane < NT / 32 ? r[lane] : R(0);
    b = lane < NT / 32 ? r[NT / 32 + lane] : R(0);
#pragma unroll
    for (int o = NT / 64; o > 0; o >>= 1) {
      a = a + shfl_xor(a, o);
      b = b + shfl_xor(b, o);
    }
    if (lane == 0) {
      r[2 * (NT / 32)] = a;
      r[2 * (NT / 32) + 1] = b;
    }
  }
  __syncthreads();
  a = r[2 * (NT / 32)];
  b = r[2 * (NT / 32) + 1];
}

// Half of the smallest power of two that is at least n, within a warp: the
// first distance of a butterfly sum whose lanes from n on hold zeros.
__device__ __forceinline__ int warp_half(int n) { return n > 16 ? 16 : n > 1 ? 1 << (31 - __clz(n - 1)) : 0; }

// Upper-triangle entry e -> (p, q), p <= q < c, row by row.
__device__ __forceinline__ void tri_entry(int e, int c, int &p, int &q) {
  const float b = float(2 * c + 1);
  int r = int((b - sqrtf(fmaxf(b * b - 8.f * float(e), 0.f))) * 0.5f);
  r = max(0, min(r, c - 1));
  auto start = [&](int x) { return x * c - x * (x - 1) / 2; };
  while (r > 0 && start(r) > e) --r;
  while (r + 1 < c && start(r + 1) <= e) ++r;
  p = r;
  q = r + (e - start(r));
}

// C[x][y] = sum_k P(x, k) Q(y, k) over from(x, y) <= k < K (a triangular
// factor), one output a thread, exactly as many terms as there are.  Faster
// than the 64 x 64 tiles of gemm_nt while the outputs are at most a few per
// thread: a 16 x 16 x 16 double-float product is one pass of 16 terms here and
// a whole padded tile there.
template <typename T, int NT, class FK, class FP, class FQ, class FE>
__device__ void gemm_exact_from(int M, int N, FK from, int K, FP P, FQ Q, FE E) {
#pragma unroll 1
  for (int o = threadIdx.x; o < M * N; o += NT) {
    const int x = o / N, y = o - x * N;
    typename CAcc<T>::type acc = acc_zero<T>();
#pragma unroll 1
    for (int k = from(x, y); k < K; ++k) acc_fma<T>(acc, P(x, k), Q(y, k));
    E(x, y, acc_fin<T>(acc));
  }
  __syncthreads();
}

// ------------------------------------------------- 1. float Hestenes Jacobi
// One-sided Jacobi of the c float vectors As[j * pa + i] (length ell, in
// shared memory), rotations accumulated in the columns Vs[j * pv + i] (when
// Vs is set).  Round-robin ordering over the vectors sorted by decreasing norm
// (de Rijk); a pair belongs to LG lanes, which form the inner product and
// apply the rotation to their elements.  Norms are carried by a' = a - t |g|,
// b' = b + t |g| and recomputed each sweep.  Stops after a sweep without a
// pair above `done` (before its rotation), or by pair_far's rule (kLastWord).
// Returns the sweeps, -1 at the limit, -2 before a sweep whose sum of squared
// norms is below `least` or not below kNormMax (a NaN or an infinity among them;
// the vectors are as the sweep found them).
constexpr float kNormMax = 1e30f, kNormTiny = 1e-37f;
template <int NT>
__device__ __forceinline__ int hestenes(cpx<float> *As, int pa, int ell, cpx<float> *Vs, int pv, int c, float *nrm, int *ord,
                                        float floor_, float least, float tol, float done, int max_sweeps) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cp = c + (c & 1), np = cp >> 1, ring = cp - 1;
  int LG = 32;
  while (LG > 4 && (np * LG > NT || LG >= 2 * ell)) LG >>= 1;  // (short vectors need no more lanes)
  const int l = tid & (LG - 1), grp = tid / LG, ngrp = NT / LG;
  const int active = min(NT, ((np * LG + 31) >> 5) << 5);  // threads that own a pair (whole warps)
  const float tol2 = tol * tol, done2 = done * done;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
#pragma unroll 1
    for (int j = warp; j < c; j += NT / 32) {
      float s = 0.f;
#pragma unroll 1
      for (int i = lane; i < ell; i += 32) s += cabs2(As[j * pa + i]);
#pragma unroll 1
      for (int o = warp_half(ell); o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) nrm[j] = s;
    }
    __syncthreads();
    float fro = 0.f;
    {
      const float x = tid < c ? nrm[tid] : 0.f;  // (c <= NT)
      int rk = 0;  // as order_rank: below, every value is finite
#pragma unroll 4
      for (int i = 0; i < c; ++i) {
        const float y = nrm[i];
        fro += y;
        rk += (y > x || (y == x && i < tid)) ? 1 : 0;
      }
      if (!(fro >= least && fro < kNormMax)) return -2;  // uniform: every thread adds the same values in the same order
      if (tid < c) ord[rk] = tid;
    }
    const float tiny2 = fmaxf(fro * floor_ * floor_, kNormTiny);
    __syncthreads();
    int far = 0;
    if (tid < active) {
      for (int r = 0; r < ring; ++r) {
        for (int t0 = 0; t0 < np; t0 += ngrp) {
          const int t = t0 + grp;
          int a_ = t == 0 ? 0 : t + r, b_ = cp - 1 - t + r;  // circle positions t and cp - 1 - t
          if (a_ > ring) a_ -= ring;
          if (b_ > ring) b_ -= ring;
          const int lo = min(a_, b_), hi = max(a_, b_);
          const bool valid = t < np && hi < c;
          const int P = valid ? ord[lo] : 0, Q = valid ? ord[hi] : 0;
          cpx<float> *ap = As + P * pa, *aq = As + Q * pa;
          float gx = 0.f, gy = 0.f;
          for (int i = l; i < ell; i += LG) {
            const cpx<float> x = ap[i], y = aq[i];
            gx = fmaf(x.x, y.x, fmaf(x.y, y.y, gx));
            gy = fmaf(x.x, y.y, fmaf(-x.y, y.x, gy));
          }
          for (int o = LG >> 1; o > 0; o >>= 1) {
            gx += __shfl_xor_sync(0xffffffffu, gx, o);
            gy += __shfl_xor_sync(0xffffffffu, gy, o);
          }
          const float a = nrm[P], b = nrm[Q];
          __syncwarp();
          if (valid && a > tiny2 && b > tiny2) {
            // The rotation from the half difference d and h = sqrt(d^2 + |g|^2): cos^2 = (1 + |d| / h) / 2 and
            // s e = conj(g) / (2 h c); scaled by a + b, so that vectors of any size stay in range.  Two square
            // roots in a row instead of four special functions.
            const float sc = __fdividef(1.f, a + b);
            const float hx = gx * sc, hy = gy * sc, as = a * sc, bs = b * sc;
            const float g2 = fmaf(hx, hx, hy * hy), ab = as * bs;
            if (done > kLastWord) far |= int(g2 > done2 * ab);
            if (g2 > tol2 * ab) {
              const float d = 0.5f * (bs - as), h2 = fmaf(d, d, g2), rh = rsqrt_near(h2);
              const float c2 = fmaf(0.5f * fabsf(d), rh, 0.5f), rc = rsqrt_near(c2), cs = c2 * rc;
              if (done <= kLastWord) {  // pair_far, squared
                const float r2 = __fdividef(g2, ab), t2 = (1.f - c2) * rc * rc;
                far |= int(r2 > kFloatDone * kFloatDone || 64.f * r2 * t2 > tol2);
              }
              const float w = copysignf(0.5f * rh * rc, d);
              const cpx<float> se = mkc<float>(hx * w, -hy * w);
              for (int i = l; i < ell; i += LG) {
                const cpx<float> x = ap[i], y = aq[i];
                ap[i] = mkc<float>(cs * x.x - (se.x * y.x - se.y * y.y), cs * x.y - (se.x * y.y + se.y * y.x));
                aq[i] = mkc<float>(cs * y.x + (se.x * x.x + se.y * x.y), cs * y.y + (se.x * x.y - se.y * x.x));
              }
              if (Vs) {
                cpx<float> *vp = Vs + P * pv, *vq = Vs + Q * pv;
                for (int i = l; i < c; i += LG) {
                  const cpx<float> x = vp[i], y = vq[i];
                  vp[i] = mkc<float>(cs * x.x - (se.x * y.x - se.y * y.y), cs * x.y - (se.x * y.y + se.y * y.x));
                  vq[i] = mkc<float>(cs * y.x + (se.x * x.x + se.y * x.y), cs * y.y + (se.x * x.y - se.y * x.x));
                }
              }
              if (l == 0) {  // t |g| = |g|^2 / (|d| + h), signed as d
                const float u = copysignf(__fdividef(g2, fabsf(d) + h2 * rh), d) * (a + b);
                nrm[P] = a - u;
                nrm[Q] = b + u;
              }
            }
          }
        }
        if (active == 32)
          __syncwarp();
        else
          asm volatile("bar.sync 1, %0;" ::"r"(active) : "memory");
      }
    }
    if (!__syncthreads_or(far)) return sweep + 1;
  }
  return -1;
}

// ------------------------------------------------ 2. unitary to working precision
// V (I + W) is unitary for V^H V = I + S, S = D + O (D diagonal): V D_g with
// D_g = (I + D)^(-1/2) has V^H V - I = S1 = D_g O D_g, so
//   I + W = D_g (I - S1/2 + 3/8 S1^2 - 5/16 S1^3 + 35/128 S1^4 - ...).
// O is small, D may be larger: the approximate reciprocal square roots of the
// float rotations shrink every column a little (up to 1e-3 over long sweeps),
// and a rotation by t in I + K has D = t^2.  What a truncated series leaves is
// a power of S1's spectral norm, so its limits are on norms (Frobenius here,
// row sums in team_correction): entries alone say little, 64 x 64 of them at
// 2e-5 have norm 6e-4.  dg_minus1: (1 + x)^(-1/2) - 1 in double-float.
__device__ __forceinline__ dd dg_minus1(dd x) {
  // without cancellation: 1 / s - 1 = -x / (s (1 + s)), s = sqrt(1 + x)
  const dd s = sqrt(dd(1.f) + x);
  return -(x / (s * (dd(1.f) + s)));
}
// W[k][y] from S[k][y] (diagonal: x = S[k][k]), the factors dk, dy = D_g - 1 of
// k and y, and hi = (3/8 S1^2 - ...)[k][y].
__device__ __forceinline__ cpx<dd> unit_entry(bool diag, cpx<dd> s, dd dk, dd dy, cpx<float> hi) {
  const float gk = 1.f + dk.hi;
  if (diag) return mkc<dd>(dk + dd(gk * hi.x), dd(0.f, 0.f));
  // D_g,k S1 = (1 + dk)^2 O (1 + dy)
  const dd f = (dd(1.f) + dk) * (dd(1.f) + dk) * (dd(1.f) + dy);
  const dd ax = f * s.x, ay = f * s.y;
  return mkc<dd>(dd(-0.5f * ax.hi, -0.5f * ax.lo) + dd(gk * hi.x), dd(-0.5f * ay.hi, -0.5f * ay.lo) + dd(gk * hi.y));
}
// Frobenius norms of O and D: the third-order term is left out below kOffSquare
// (it is 2e-17 there), the fourth below kOffMax (4e-16 at the most; S1^2 in float
// errs by no more).
constexpr float kOffSquare = 3e-6f, kOffMax = 2e-4f, kDiagMax = 0.3f;

// Q (c x c, row-major with pitch pq) <- the unitary factor of V (float,
// columns Vs[k * pv + r]), V unitary to a few float roundings or I + K.
// S = V^H V - I is formed from exact float products; float Newton-Schulz
// steps bring its off-diagonals below kOffMax first where they are larger (I + K
// with a t near 1); then Q = V (I + W) by unit_entry.  dg: c double-float values
// of scratch.
// The correction V W is accumulated in double-float in every mode (W < 2e-4,
// so its error is below 1e-16).  Returns false (Q not written) when V is too
// far from unitary.
template <typename T, int NT>
__device__ __noinline__ bool unitarise(cpx<float> *Vs, int pv, int c, cpx<dd> *S, int ps, cpx<T> *Q, int pq, dd *dg,
                                       double *red) {
  Vs = as_shared(Vs);
  S = as_shared(S);
  Q = as_shared(Q);
  dg = as_shared(dg);
  cpx<float> *const tmp = reinterpret_cast<cpx<float> *>(Q);  // twice c x c floats, until Q is written
  float off = 0.f;
  const int tid = threadIdx.x;
  const int ntri = c * (c + 1) / 2;
  for (int it = 0;; ++it) {
    float o2 = 0.f, d2 = 0.f;
#pragma unroll 1
    for (int e = tid; e < ntri; e += NT) {
      int p, q;
      tri_entry(e, c, p, q);
      const cpx<float> *vp = Vs + p * pv, *vq = Vs + q * pv;
      tacc ax, ay;
      ax.mid = ax.lo = ay.hi = ay.mid = ay.lo = 0.f;
      ax.hi = p == q ? -1.f : 0.f;
#pragma unroll 1
      for (int k = 0; k < c; ++k) {
        const cpx<float> x = vp[k], y = vq[k];
        tacc_add_prod(ax, x.x, y.x);
        tacc_add_prod(ax, x.y, y.y);
        tacc_add_prod(ay, x.x, y.y);
        tacc_add_prod(ay, -x.y, y.x);
      }
      const dd sx = tacc_fin(ax), sy = tacc_fin(ay);
      S[p * ps + q] = mkc<dd>(sx, sy);
      if (p != q) S[q * ps + p] = mkc<dd>(sx, -sy);
      if (p == q)
        d2 = fmaf(sx.hi, sx.hi, d2);
      else
        o2 = fmaf(2.f * sx.hi, sx.hi, fmaf(2.f * sy.hi, sy.hi, o2));
    }
    block_sum2_in<float, NT>(o2, d2, red);  // (ends with S visible: its barriers follow the stores)
    off = sqrtf(o2);
    if (off <= kOffMax && d2 <= kDiagMax * kDiagMax) break;
    if (!(o2 <= 1.f && d2 <= 1.f) || it >= 6) return false;
#pragma unroll 1
    for (int o = tid; o < c * c; o += NT) {
      const int y = o / c, r = o - y * c;
      cpx<float> a = czero<float>();
#pragma unroll 1
      for (int k = 0; k < c; ++k) {
        const cpx<dd> s = S[k * ps + y];
        a = cfma(Vs[k * pv + r], mkc<float>(s.x.hi, s.y.hi), a);
      }
      const cpx<float> v = Vs[y * pv + r];
      tmp[o] = mkc<float>(fmaf(-0.5f, a.x, v.x), fmaf(-0.5f, a.y, v.y));
    }
    __syncthreads();
#pragma unroll 1
    for (int o = tid; o < c * c; o += NT) Vs[(o / c) * pv + o % c] = tmp[o];
    __syncthreads();
  }
  // W in place of S (the square and the cube in float)
  for (int k = tid; k < c; k += NT) dg[k] = dg_minus1(S[k * ps + k].x);
  __syncthreads();
#pragma unroll 1
  for (int o = tid; o < c * c; o += NT) {
    const int y = o / c, x = o - y * c;
    cpx<float> a = czero<float>();
#pragma unroll 1
    for (int k = 0; k < c; ++k) {
      if (k == x || k == y) continue;
      const cpx<dd> s = S[x * ps + k], t = S[k * ps + y];
      const float g = 1.f + dg[k].hi;
      a = cfma(mkc<float>(s.x.hi * (g * g), s.y.hi * (g * g)), mkc<float>(t.x.hi, t.y.hi), a);
    }
    const float g = (1.f + dg[x].hi) * (1.f + dg[y].hi);
    tmp[o] = mkc<float>(a.x * g, a.y * g);
  }
  __syncthreads();
  cpx<float> *const hi = off > kOffSquare ? tmp + c * c : tmp;
  const float w2 = off > kOffSquare ? 1.f : 0.375f;
  if (off > kOffSquare) {
#pragma unroll 1
    for (int o = tid; o < c * c; o += NT) {
      const int y = o / c, x = o - y * c;
      cpx<float> a = czero<float>();
#pragma unroll 1
      for (int k = 0; k < c; ++k) {
        if (k == x) continue;
        const cpx<dd> s = S[x * ps + k];
        const float g = 1.f + dg[k].hi;
        a = cfma(mkc<float>(s.x.hi * g, s.y.hi * g), tmp[y * c + k], a);
      }
      const float g = 0.3125f * (1.f + dg[x].hi);
      const cpx<float> q = tmp[o];
      hi[o] = mkc<float>(fmaf(0.375f, q.x, -g * a.x), fmaf(0.375f, q.y, -g * a.y));
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int o = tid; o < c * c; o += NT) {
    const int y = o / c, x = o - y * c;
    const cpx<float> h = hi[o];
    S[x * ps + y] = unit_entry(x == y, S[x * ps + y], dg[x], dg[y], mkc<float>(w2 * h.x, w2 * h.y));
  }
  __syncthreads();
#pragma unroll 1
  for (int o = tid; o < c * c; o += NT) {
    const int y = o / c, r = o - y * c;
    dacc ax, ay;
    ax.hi = ax.lo = ay.hi = ay.lo = 0.f;
#pragma unroll 1
    for (int k = 0; k < c; ++k) {
      const cpx<float> v = Vs[k * pv + r];
      const cpx<dd> w = S[k * ps + y];
      dacc_add_fdprod(ax, v.x, w.x);
      dacc_add_fdprod(ax, -v.y, w.y);
      dacc_add_fdprod(ay, v.x, w.y);
      dacc_add_fdprod(ay, v.y, w.x);
    }
    const cpx<float> v = Vs[y * pv + r];
    Q[r * pq + y] = mkc<T>(T(v.x) + from_dd<T>(dd_norm(ax.hi, ax.lo)), T(v.y) + from_dd<T>(dd_norm(ay.hi, ay.lo)));
  }
  __syncthreads();
  return true;
}

// Q <- the unitary factor of I + K for a refinement step: K anti-Hermitian,
// float, K[x][y] = Vs[y * pv + x] off the diagonal, of Frobenius norm at most
// kStepMax.  (I + K)(I - K^2)^(-1/2) = I + K + K^2 / 2 + K^3 / 2 + 3/8 K^4 +
// 3/8 K^5 ...: K is exact, K^2 is summed in double-float, what follows is below
// 5e-10, so floats do, and what is left out is below 4e-16.  Two passes instead
// of unitarise's five and its sums: a third of its time.  Y: c x c of scratch
// for K^2.
constexpr float kStepMax = 1e-3f;
template <typename T, int NT>
__device__ __noinline__ void unitary_step(const cpx<float> *Vs, int pv, int c, cpx<dd> *Y, int py, cpx<T> *Q, int pq) {
  Vs = as_shared(Vs);
  Y = as_shared(Y);
  Q = as_shared(Q);
#pragma unroll 1
  for (int o = threadIdx.x; o < c * c; o += NT) {
    const int y = o / c, x = o - y * c;
    dacc ax, ay;
    ax.hi = ax.lo = ay.hi = ay.lo = 0.f;
#pragma unroll 1
    for (int k = 0; k < c; ++k) {
      if (k == x || k == y) continue;
      const cpx<float> a = Vs[k * pv + x], b = Vs[y * pv + k];
      dacc_add_fdprod(ax, a.x, dd(b.x));
      dacc_add_fdprod(ax, -a.y, dd(b.y));
      dacc_add_fdprod(ay, a.x, dd(b.y));
      dacc_add_fdprod(ay, a.y, dd(b.x));
    }
    Y[x * py + y] = mkc<dd>(dd_norm(ax.hi, ax.lo), dd_norm(ay.hi, ay.lo));
  }
  __syncthreads();
#pragma unroll 1
  for (int o = threadIdx.x; o < c * c; o += NT) {
    const int y = o / c, x = o - y * c;
    cpx<float> z = czero<float>();
#pragma unroll 1
    for (int k = 0; k < c; ++k) {
      const cpx<dd> a = Y[x * py + k], b = Y[k * py + y];
      const cpx<float> v = k == y ? czero<float>() : Vs[y * pv + k];
      z = cfma(mkc<float>(a.x.hi, a.y.hi), mkc<float>(fmaf(0.5f, v.x, 0.375f * b.x.hi), fmaf(0.5f, v.y, 0.375f * b.y.hi)), z);
    }
    const cpx<dd> h = Y[x * py + y];
    const cpx<float> v = Vs[y * pv + x];  // (1 on the diagonal)
    const dd wx = dd(0.5f * h.x.hi, 0.5f * h.x.lo) + dd(z.x), wy = dd(0.5f * h.y.hi, 0.5f * h.y.lo) + dd(z.y);
    Q[x * pq + y] = mkc<T>(T(v.x) + from_dd<T>(wx), T(v.y) + from_dd<T>(wy));
  }
  __syncthreads();
}

// 32 rows [i0, i0 + 32) of the vectors A[j * ld + i] as stage[r * pt + j].
template <typename T, int NT>
__device__ __forceinline__ void stage_rows(const cpx<T> *A, int ld, int ell, int c, int i0, cpx<T> *stage, int pt) {
#pragma unroll 1
  for (int idx = threadIdx.x; idx < 32 * c; idx += NT) {
    const int r = idx & 31, p = idx >> 5;
    stage[r * pt + p] = i0 + r < ell ? A[size_t(p) * ld + i0 + r] : czero<T>();
  }
}

// A <- A Q, 32 rows at a time.
template <typename T, int NT>
__device__ void apply_unitary(cpx<T> *A, int ld, int ell, int c, const cpx<T> *Q, int pq, cpx<T> *stage, int pt) {
  for (int i0 = 0; i0 < ell; i0 += 32) {
    stage_rows<T, NT>(A, ld, ell, c, i0, stage, pt);
    __syncthreads();
    const int rows = min(32, ell - i0);
#pragma unroll 1
    for (int o = threadIdx.x; o < 32 * c; o += NT) {
      const int r = o & 31, y = o >> 5;
      if (r < rows) {
        typename CAcc<T>::type acc = acc_zero<T>();
#pragma unroll 2
        for (int p = 0; p < c; ++p) {
          if ((p & 1) == 0) acc_renorm(acc);
          acc_fma<T>(acc, stage[r * pt + p], Q[p * pq + y]);
        }
        A[size_t(y) * ld + i0 + r] = acc_fin<T>(acc);
      }
    }
    __syncthreads();
  }
}

// A <- A + A K for K (float, off-diagonal, K[p][y] = Ks[y * pk + p]) so small
// that the float correction of the leading parts is exact to the working
// precision (limit at the call).
template <typename T, int NT>
__device__ void apply_small(cpx<T> *A, int ld, int ell, int c, const cpx<float> *Ks, int pk, cpx<float> *stage,
                            int pt) {
  for (int i0 = 0; i0 < ell; i0 += 32) {
#pragma unroll 1
    for (int idx = threadIdx.x; idx < 32 * c; idx += NT) {
      const int r = idx & 31, p = idx >> 5;
      cpx<float> v = czero<float>();
      if (i0 + r < ell) {
        const cpx<T> x = A[size_t(p) * ld + i0 + r];
        v = mkc<float>(lead(x.x), lead(x.y));
      }
      stage[r * pt + p] = v;
    }
    __syncthreads();
    const int rows = min(32, ell - i0);
#pragma unroll 1
    for (int o = threadIdx.x; o < 32 * c; o += NT) {
      const int r = o & 31, y = o >> 5;
      if (r < rows) {
        cpx<float> a = czero<float>();
#pragma unroll 2
        for (int p = 0; p < c; ++p)
          if (p != y) a = cfma(stage[r * pt + p], Ks[y * pk + p], a);
        cpx<T> &x = A[size_t(y) * ld + i0 + r];
        const cpx<T> v = x;
        x = mkc<T>(v.x + T(a.x), v.y + T(a.y));
      }
    }
    __syncthreads();
  }
}

// G = A^H A (upper triangle G[p * pg + q], p <= q) in the working precision.
template <typename T, int NT>
__device__ void gram_local(const cpx<T> *A, int ld, int ell, int c, cpx<T> *G, int pg, cpx<T> *stage, int pt) {
  // (one entry a thread up to c = 31 at 512 threads; beyond, the rows are staged
  // again for every further group of entries: cheaper than the code of several
  // sums a thread, which all sizes would fetch)
  const int ntri = c * (c + 1) / 2;
#pragma unroll 1
  for (int e0 = 0; e0 < ntri; e0 += NT) {
    const int e = e0 + threadIdx.x;
    int p = 0, q = 0;
    if (e < ntri) tri_entry(e, c, p, q);
    typename CAcc<T>::type acc = acc_zero<T>();
#pragma unroll 1
    for (int i0 = 0; i0 < ell; i0 += 32) {
      if (e0 == 0 || ell > 32) {
        stage_rows<T, NT>(A, ld, ell, c, i0, stage, pt);
        __syncthreads();
      }
      const int rows = min(32, ell - i0);
      if (e < ntri) {
#pragma unroll 2
        for (int r = 0; r < rows; ++r) {
          if ((r & 1) == 0) acc_renorm(acc);
          acc_jfma<T>(acc, stage[r * pt + p], stage[r * pt + q]);
        }
      }
      if (ell > 32) __syncthreads();
    }
    if (e < ntri) G[p * pg + q] = acc_fin<T>(acc);
  }
  __syncthreads();
}

// ------------------------------------------------------------- the SVD
// Scratch of svd_local in bytes: the float vectors (or, later, a stage of 32
// rows and Q), the Gram matrix / S, V, norms and order.
template <typename T>
struct LocalSvd {
  static constexpr int MAXC = sizeof(T) == 4 ? 128 : 64;
  __host__ __device__ static constexpr size_t al(size_t x) { return (x + 15) & ~size_t(15); }
  __host__ __device__ static constexpr int odd(int x) { return x | 1; }
  __host__ __device__ static size_t as_bytes(int ell, int c) { return al(size_t(c) * odd(ell) * sizeof(cpx<float>)); }
  __host__ __device__ static size_t first_bytes(int ell, int c) {
    const size_t a = as_bytes(ell, c);
    const size_t b = sizeof(T) == 4 ? 0 : al(size_t(32) * odd(c) * sizeof(cpx<T>)) + al(size_t(c) * odd(c) * 16);
    return a > b ? a : b;
  }
  __host__ __device__ static size_t bytes(int ell, int c) {
    const size_t tail = al(size_t(c) * 8);
    if (sizeof(T) == 4) return first_bytes(ell, c) + tail;
    // (the factors dg share the norms' and the order's place)
    return first_bytes(ell, c) + al(size_t(c) * odd(c) * 16) + al(size_t(c) * odd(c) * 8) + tail;
  }
  // largest c of the refinement's fixed outputs per thread
  __host__ __device__ static int max_c(int nt) { return sizeof(T) == 4 ? MAXC : (nt >= 512 ? 64 : 32); }
};

// (svd_tolerance: the block Jacobi's threshold, 4 above the rounding of a Gram
// entry.)
template <typename T>
__device__ __forceinline__ float svd_tolerance(int ell) {
  return 4.f * sqrtf(float(ell)) * float(Eps<T>::v);
}

// Orthogonalises the c vectors A[j * ld + i] (length ell; any address space)
// by unitary column operations until |a_p^H a_q| <= tol |a_p| |a_q|.  scratch: LocalSvd<T>::bytes of shared memory,
// 16-byte aligned.  tail: so many further entries of each vector follow the
// operations without counting as its length (an appended identity becomes the
// accumulated unitary).  Returns the number of sweeps and refinement steps, or -1:
// A is then a unitary transform of the input that has not converged (a
// degenerate spectrum, or the sweep limit) or the input itself (norms that the
// float stage cannot hold, NaN), for the caller's block Jacobi.  svd_local_steps
// returns -2 for such norms.
template <typename T, int NT>
__device__ __forceinline__ int svd_local_steps(cpx<T> *A, int ld, int ell, int c, int max_sweeps, unsigned char *scratch,
                                               double *red, float tol, int tail) {
  using L = LocalSvd<T>;
  const int tid = threadIdx.x;
  const int pa = L::odd(ell), pc = L::odd(c);
  unsigned char *at = scratch;
  cpx<float> *As = reinterpret_cast<cpx<float> *>(at);
  at += L::first_bytes(ell, c);
  const float tolf = 4.f * sqrtf(float(ell)) * Eps<float>::v;
  auto load = [&]() {
#pragma unroll 1
    for (int idx = tid; idx < c * ell; idx += NT) {
      const int j = idx / ell, i = idx - j * ell;
      const cpx<T> x = A[size_t(j) * ld + i];
      As[j * pa + i] = mkc<float>(lead(x.x), lead(x.y));
    }
  };
  if constexpr (sizeof(T) == 4) {
    float *nrm = reinterpret_cast<float *>(at);
    int *ord = reinterpret_cast<int *>(nrm + c);
    load();
    __syncthreads();
    const int sw = hestenes<NT>(As, pa, ell, nullptr, 0, c, nrm, ord, float(sweep_floor<float>(ell)), 0.f, tolf,
                                kLastWord, max_sweeps);
    if (sw == -2) return -2;
    for (int idx = tid; idx < c * ell; idx += NT) {
      const int j = idx / ell, i = idx - j * ell;
      A[size_t(j) * ld + i] = As[j * pa + i];
    }
    __syncthreads();
    return sw;
  } else {
    cpx<T> *stage = reinterpret_cast<cpx<T> *>(scratch);
    cpx<T> *Q = reinterpret_cast<cpx<T> *>(scratch + L::al(size_t(32) * pc * sizeof(cpx<T>)));
    cpx<dd> *S = reinterpret_cast<cpx<dd> *>(at);
    cpx<T> *G = reinterpret_cast<cpx<T> *>(at);
    at += L::al(size_t(c) * pc * 16);
    cpx<float> *Vs = reinterpret_cast<cpx<float> *>(at);
    at += L::al(size_t(c) * pc * 8);
    float *nrm = reinterpret_cast<float *>(at);
    int *ord = reinterpret_cast<int *>(nrm + c);
    dd *dg = reinterpret_cast<dd *>(nrm);  // (not needed while the sweeps run)
    const float floor_t = float(sweep_floor<T>(ell));
    // float64: the float stage takes no vectors whose noise level is out of its
    // range.  The Gram matrix is scaled before its entries are compared in float:
    // tol times the smallest kept value squared is 4e-44 at norm 1.
    const float least2 = std::is_same<T, double>::value ? kNormTiny / (floor_t * floor_t) : 0.f;
    auto gram = [](T x) {
      if constexpr (std::is_same<T, double>::value)
        return lead(x * 0x1p66);
      else
        return lead(x);
    };
    // a correction formed in float is exact to the working precision below this angle
    // and its square, which that leaves out, is below the working precision
    constexpr float kFloatApply = std::is_same<T, double>::value ? 1e-9f : 3e-8f;
    constexpr int kMaxStages = 3, kMaxSteps = 10;
    int sweeps = 0, stages = 0;
    // what is due: a float stage, a product with the unitary factor of V (or
    // of I + K), a small correction; one copy of each in the loop
    bool bulk = true, small_step = false, near = false, last = false;
#pragma unroll 1
    for (int step = 0;; ++step) {
      if (bulk) {
        load();
#pragma unroll 1
        for (int idx = tid; idx < c * c; idx += NT) {
          const int y = idx / c, r = idx - y * c;
          Vs[y * pc + r] = mkc<float>(y == r ? 1.f : 0.f, 0.f);
        }
        __syncthreads();
        // the first stage leaves vectors at the float noise level alone; once A
        // holds them to its own precision the next one resolves them too
        const int sw = hestenes<NT>(As, pa, ell, Vs, pc, c, nrm, ord, stages == 0 ? Eps<float>::v : floor_t, least2,
                                    tolf, 1e-4f, min(max_sweeps, 20));
        if (sw == -2) return stages == 0 ? -2 : -1;
        sweeps += sw < 0 ? min(max_sweeps, 20) : sw;
        ++stages;
        bulk = false;
      }
      if (small_step) {
        apply_small<T, NT>(A, ld, ell + tail, c, Vs, pc, reinterpret_cast<cpx<float> *>(stage), pc);
      } else {
        if (near)
          unitary_step<T, NT>(Vs, pc, c, S, pc, Q, pc);
        else if (!unitarise<T, NT>(Vs, pc, c, S, pc, Q, pc, dg, red))
          return -1;
        apply_unitary<T, NT>(A, ld, ell + tail, c, Q, pc, stage, pc);
      }
      if (last) return sweeps + 1;
      if (step == kMaxSteps) return -1;
      gram_local<T, NT>(A, ld, ell, c, G, pc, stage, pc);
      float fro = 0.f;
      for (int j = 0; j < c; ++j) fro += gram(G[j * pc + j].x);
      if (!(fro < kNormMax)) return -1;
      const float tiny2 = fmaxf(fro * floor_t * floor_t, kNormTiny);
      // K of every pair above the threshold, r = |g| / (|a_p| |a_q|) and |t|.
      // Pairs below it, down to rounding, go along where their t is small (so
      // that all of them together stay below kFloatApply): what they leave would
      // enter the recovered side as r sigma_p / sigma_q, and with them a
      // trajectory's error against float64 is 2-10 times smaller.  k2: the
      // squared Frobenius norm of K.
      float rmax = 0.f, kmax = 0.f, k2 = 0.f, none = 0.f;
      const float least = tol < 1e-10f ? 0.03125f * tol : tol, along = kFloatApply / float(c);
#pragma unroll 1
      for (int e = tid; e < c * (c + 1) / 2; e += NT) {
        int p, q;
        tri_entry(e, c, p, q);
        if (p == q) {
          Vs[p * pc + p] = mkc<float>(1.f, 0.f);
          continue;
        }
        cpx<float> vpq = czero<float>(), vqp = czero<float>();
        const T at_ = G[p * pc + p].x, bt_ = G[q * pc + q].x;
        const float a = gram(at_), b = gram(bt_);
        if (a > tiny2 && b > tiny2) {
          const cpx<T> g = G[p * pc + q];
          const float sc = rsqrtf(a) * rsqrtf(b);
          const float hx = gram(g.x) * sc, hy = gram(g.y) * sc, r2 = fmaf(hx, hx, hy * hy), r = sqrtf(r2);
          rmax = fmaxf(rmax, r);
          if (r > least) {
            const float rr = 1.f / r;
            const float z = 0.5f * (gram(bt_ - at_) * sc) * rr;
            const float z1 = fmaf(z, z, 1.f);
            const float t = fabsf(z) > 1e15f ? 0.5f / z : copysignf(1.f / (fabsf(z) + sqrtf(z1)), z);
            const bool over = r > tol, take = over || fabsf(t) <= along;
            if (over) kmax = fmaxf(kmax, fabsf(t));
            if (take) {
              k2 = fmaf(2.f * t, t, k2);
              const float ex = hx * rr, ey = -hy * rr;
              vqp = mkc<float>(-t * ex, -t * ey);
              vpq = mkc<float>(t * ex, -t * ey);
            }
          }
        }
        Vs[p * pc + q] = vqp;  // column p, row q
        Vs[q * pc + p] = vpq;  // column q, row p
      }
      rmax = block_max<NT>(rmax, red);
      kmax = block_max<NT>(kmax, red);
      block_sum2_in<float, NT>(k2, none, red);
      if (!(rmax < 2.f)) return -1;  // not a number
      if (rmax <= tol) {
        if (!(k2 > 0.f)) return sweeps + 1;
        small_step = last = true;
        continue;
      }
      ++sweeps;
      // What is left after this step is of the order of the square: r r' between
      // vectors of different size (whose angles t are smaller than r), r t
      // between neighbours.
      const float far = fmaxf(rmax, kmax);
      small_step = far <= kFloatApply && k2 <= kFloatApply * kFloatApply;
      near = k2 <= kStepMax * kStepMax;
      // far from converged: vectors that the float stage had left alone
      bulk = !small_step && rmax > 1e-3f && kmax > 0.3f && stages < kMaxStages;
      last = !bulk && rmax * far * 8.f <= tol;
      if (bulk) {
        near = false;
        __syncthreads();
      }
    }
  }
}

// A scaled by 2^e (its ell entries, not the tail).
template <int NT>
__device__ __noinline__ void scale_vectors(cpx<double> *A, int ld, int ell, int c, int e) {
  for (int idx = threadIdx.x; idx < c * ell; idx += NT) {
    cpx<double> &x = A[size_t(idx / ell) * ld + idx % ell];
    x = mkc<double>(scalbn(x.x, e), scalbn(x.y, e));
  }
  __syncthreads();
}

// In float64, vectors out of the float stage's range (a gate or a state far from
// norm 1) are brought to norm 1 by a power of two for the time of the SVD.
template <typename T, int NT>
__device__ __forceinline__ int svd_local(cpx<T> *A, int ld, int ell, int c, int max_sweeps, unsigned char *scratch,
                                         double *red, float tol, int tail = 0) {
  if constexpr (!std::is_same<T, double>::value) {
    return max(-1, svd_local_steps<T, NT>(A, ld, ell, c, max_sweeps, scratch, red, tol, tail));
  } else {
    int e = 0, r;
#pragma unroll 1
    for (;;) {
      r = svd_local_steps<T, NT>(A, ld, ell, c, max_sweeps, scratch, red, tol, tail);
      if (r != -2 || e != 0) break;
      int top = 0;  // largest exponent field
      for (int idx = threadIdx.x; idx < c * ell; idx += NT) {
        const cpx<T> x = A[size_t(idx / ell) * ld + idx % ell];
        top = max(top, max(__double2hiint(fabs(x.x)), __double2hiint(fabs(x.y))) >> 20);
      }
      top = int(block_max<NT>(float(top), red));
      if (top == 0 || top == 2047 || top == 1023) break;  // zeros; not finite
      e = 1023 - top;
      scale_vectors<NT>(A, ld, ell, c, e);
    }
    if (e != 0) scale_vectors<NT>(A, ld, ell, c, -e);
    return max(-1, r);
  }
}

// The same for vectors in global memory (one copy for its several callers).
template <typename T, int NT>
__device__ __noinline__ int svd_local_global(cpx<T> *A, int ell, int c, int max_sweeps, unsigned char *scratch,
                                             double *red) {
  scratch = as_shared(scratch);
  red = as_shared(red);
  return svd_local<T, NT>(A, ell, ell, c, max_sweeps, scratch, red, svd_tolerance<T>(ell));
}

// In-place Cholesky S = L L^H of an n x n Hermitian matrix in shared memory
// (pitch ps; the lower triangle becomes L).  Same rule as cholesky_lower: false
// when a pivot falls below `rel` times its original diagonal.
template <typename T, int NT>
__device__ bool cholesky_local(cpx<T> *S, int ps, int n, float rel, T *diag0) {
#pragma unroll 1
  for (int i = threadIdx.x; i < n; i += NT) diag0[i] = S[i * ps + i].x;
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    const T d = S[k * ps + k].x;
    if (!(lead(d) > rel * lead(diag0[k])) || !(lead(d) > 0.f)) return false;  // uniform: every thread read the same
    __syncthreads();
    if (threadIdx.x < 32 || int(threadIdx.x & ~31u) < n - k - 1) {  // whole warps that hold a row below the pivot
      const T l = sqrt(d), il = T(1) / l;
#pragma unroll 1
      for (int i = k + 1 + threadIdx.x; i < n; i += NT) S[i * ps + k] = cscale(S[i * ps + k], il);
      if (threadIdx.x == 0) S[k * ps + k] = mkc<T>(l, T(0));
    }
    __syncthreads();
    const int rem = n - k - 1;
#pragma unroll 1
    for (int idx = threadIdx.x; idx < rem * rem; idx += NT) {
      const int i = k + 1 + idx / rem, j = k + 1 + idx % rem;
      if (j > i) continue;
      const cpx<T> li = S[i * ps + k], lj = S[j * ps + k];
      cpx<T> v = S[i * ps + j];
      v.x -= li.x * lj.x + li.y * lj.y;
      v.y -= li.y * lj.x - li.x * lj.y;
      S[i * ps + j] = v;
    }
    __syncthreads();
  }
  return true;
}

// ------------------------------------------------------------- bond operation
// Shared-memory plan of bond_local.  theta (T0) and the vectors (A) are
// vector-contiguous with an odd pitch, so that lanes that walk over vectors
// hit different banks.  Taken when theta is at most 64 x 64 (chi <= 32: beyond,
// the products want register tiles) and everything fits.
template <typename T>
struct LocalBond {
  static constexpr int MAXM = 64;
  unsigned theta, vec, svd, lam, vals, total;  // (below 2^20: at most 64 x 64)
  int c, ell;
  __host__ __device__ static unsigned al(unsigned x) { return (x + 15) & ~15u; }
  __host__ __device__ static unsigned most(unsigned a, unsigned b) { return a > b ? a : b; }
  __host__ __device__ bool plan(int cL, int cM, int cR, bool lq, size_t room, int nt) {
    const int m = 2 * cL, nc = 2 * cR, mn = m < nc ? m : nc;
    if (m > MAXM || nc > MAXM || cM > MAXM) return false;
    const unsigned e = sizeof(cpx<T>);
    // vectors and their length; theta with the same pitch.  (LQ: cM vectors of
    // length m, theta as columns; the general path takes what LQ declines.)
    c = lq ? cM : mn;
    ell = lq ? m : (m < nc ? nc : m);
    if (c > LocalSvd<T>::max_c(nt)) return false;
    theta = al((lq ? nc : mn) * (ell | 1) * e);
    vec = al(c * (ell | 1) * e);
    svd = unsigned(LocalSvd<T>::bytes(ell, c));
    svd = most(svd, al(cM * (cM | 1) * e) + al(cM * unsigned(sizeof(T))));  // S and its diagonal
    svd = most(svd, al(c * (lq ? nc : mn) * e));                            // the recovered side
    lam = al(2 * (cL + cM + cR) * unsigned(sizeof(T)));
    vals = al(mn * unsigned(3 * sizeof(double) + 3 * sizeof(T) + sizeof(int))) + 128;
    total = theta + vec + svd + lam + vals;
    return total <= room;
  }
};

// f[0], f[1] = 1 / sqrt of the block's sums of a and b (in order: the same bits
// for the same block).  terms: threads from this one on hold zeros; up to a
// warp's worth need no second stage.
template <typename R, typename T, int NT>
__device__ __forceinline__ void norms_in(R a, R b, int terms, double *red, T *f) {
  R *r = reinterpret_cast<R *>(red);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int o = warp_half(terms); o > 0; o >>= 1) {
    a = a + shfl_xor(a, o);
    b = b + shfl_xor(b, o);
  }
  if (terms > 32) {
    __syncthreads();
    if (lane == 0) {
      r[warp] = a;
      r[NT / 32 + warp] = b;
    }
    __syncthreads();
    if (warp == 0) {
      a = lane < NT / 32 ? r[lane] : R(0);
      b = lane < NT / 32 ? r[NT / 32 + lane] : R(0);
#pragma unroll 1
      for (int o = NT / 64; o > 0; o >>= 1) {
        a = a + shfl_xor(a, o);
        b = b + shfl_xor(b, o);
      }
    }
  }
  if (warp == 0) {
    const R x = R(1) / sqrt(lane & 1 ? b : a);
    if (lane < 2) f[lane] = T(x);
  }
  __syncthreads();
}

// What bond_local leaves behind.
struct LocalResult {
  bool done = false;  // the bond is finished; else theta and the vectors are in the global workspace
  bool declined = false;  // ... or nothing has happened (no LQ factor): the general path starts over
  bool svd_done = false;  // (general path) svd_local has orthogonalised the vectors
  bool lq = false, colmode = false;
  int ell = 0, c = 0, sweeps = 0;
};

}  // namespace tn
