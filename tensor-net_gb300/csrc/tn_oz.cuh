// tn_oz.cuh -- double-float matrix products on the tensor cores, and the team
// of CTAs that shares them.
//
// C[x][y] = sum_k P(x, k) Q(y, k) for double-float complex operands, exact to
// the double-float level (an Ozaki-style splitting, as update_ozaki): each row
// of P and of Q is written relative to a power of two above its largest entry
// as signed 7-bit digits, exact in bf16 (oz_split, once per operand, into
// planes in global memory); digit products of a pair (j, k) accumulate exactly
// in FP32 tensor memory, one accumulator per level j + k (kind::f16 MMAs of
// 128 x 64 x 16), and the levels are added from the largest in double-float.
// A level's sum over 256 real K values stays below 2^24 (first digit at most
// 2^7, the others 2^6, up to eight pairs a level: 40960 * 256 < 2^23.4), so
// accumulators are drained every 256.
//
// The complex product is one real product: P's row interleaves re and im along
// K; Q's row y becomes the two real rows (Qr, -Qi) and (Qi, Qr), made from the
// same planes when a tile is brought to shared memory (with conj: (Qr, Qi) and
// (-Qi, Qr)).
//
// Why: a double-float product costs 12 float operations a real term on the
// FP32 pipes (n = 512 on one SM: 26 ms); the digit products that matter (10 to
// 36 of 64, chosen by the caller from the accuracy it needs) run at the tensor
// rate, and an operand is split once instead of once per tile.
#pragma once

namespace tn {

// CTAs that work on one bond operation together: one, or a thread-block
// cluster.  Every thread of every member calls sync() the same number of
// times; what members read from each other goes through global memory.
struct Team {
  int rank = 0, size = 1;
  __device__ __forceinline__ void sync() const {
    if (size == 1) {
      __syncthreads();
    } else {
      __threadfence();
      asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  }
};

// Digit planes of an operand: nd planes of rows x ld bf16 values (ld = 2 K
// rounded up to 32, zero padded), and the rows' exponents.
struct OzPlanes {
  __nv_bfloat16 *p;
  int *expo;
  size_t stride;  // elements between planes
  int rows, ld, nd;
};
__host__ __device__ inline int oz_ld(int K) { return (2 * K + 31) & ~31; }
__device__ inline OzPlanes oz_planes(void *mem, int *expo, int rows, int K, int nd) {
  OzPlanes o;
  o.p = reinterpret_cast<__nv_bfloat16 *>(mem);
  o.expo = expo;
  o.rows = rows;
  o.ld = oz_ld(K);
  o.nd = nd;
  o.stride = size_t(rows) * o.ld;
  return o;
}

// Splits the rows get(row, k), k < K, into ND digits; a warp per row.  fixed
// >= -126: that exponent for every row instead of the row's own (a fixed-point
// rounding of the whole matrix).
template <int NT, int ND, class FG>
__device__ void oz_split(const Team &tm, const OzPlanes &o, int K, FG get, int fixed = -1000) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = NT / 32;
  for (int row = tm.rank * nw + warp; row < o.rows; row += tm.size * nw) {
    int E = fixed;
    if (fixed < -126) {
      float m = 0.f;
      for (int k = lane; k < K; k += 32) {
        const cpx<dd> v = get(row, k);
        m = fmaxf(m, fmaxf(fabsf(v.x.hi), fabsf(v.y.hi)));
      }
      m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
      // one above the largest entry: the low parts may carry past a power of two
      E = m > 0.f && isfinite(m) ? max(oz_exponent(m), -100) : 0;
    }
    if (lane == 0) o.expo[row] = E;
    __nv_bfloat162 *dst = reinterpret_cast<__nv_bfloat162 *>(o.p + size_t(row) * o.ld);
    const size_t st2 = o.stride / 2;
    for (int k = lane; k < o.ld / 2; k += 32) {
      float dx[ND], dy[ND];
      if (k < K) {
        const cpx<dd> v = get(row, k);
        oz_digits<ND>(v.x.hi, v.x.lo, E, dx);
        oz_digits<ND>(v.y.hi, v.y.lo, E, dy);
      } else {
#pragma unroll
        for (int j = 0; j < ND; ++j) dx[j] = dy[j] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < ND; ++j) dst[j * st2 + k] = __floats2bfloat162_rn(dx[j], dy[j]);
    }
  }
}

// Shared memory of oz_gemm: two stages of P planes (128 x 32) and of both real
// rows of Q (64 x 32), eight planes each.
constexpr int kOzM = 128, kOzN = 32, kOzKC = 32, kOzFlush = 256;
constexpr size_t kOzPBytes = size_t(8) * kOzM * kOzKC * 2, kOzQBytes = size_t(8) * 2 * kOzN * kOzKC * 2;
constexpr size_t kOzStage = kOzPBytes + kOzQBytes;
constexpr size_t kOzSmem = 2 * kOzStage;

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(n) : "memory");
}

// Waits for the MMAs committed to barrier s; bounded as wait_mma.
template <typename S>
__device__ void oz_wait(S &sm, int s) {
  const uint64_t t0 = tc::global_ns();
  while (!tc::mbar_try_wait(sm.gbar + s, (sm.gphase >> s) & 1u)) {
    if (tc::global_ns() - t0 > 10ull * 1000 * 1000 * 1000) {
      sm.tc_fail = true;
      break;
    }
  }
  sm.gphase ^= 1u << s;
}

// Where a product goes: C[x * ld + y], C[y * ld + x] (kOzTrans), or both
// triangles of a Hermitian result from its upper one (kOzHerm: C[x][y] = v;
// kOzHermT: its transpose).  add (same layout, not for the Hermitian ones): C =
// add + product; add may be C.
enum OzOut { kOzPlain, kOzTrans, kOzHerm, kOzHermT };

// The product, over the team's share of 128 x 32 tiles; levels j + k < nlev
// are kept (nlev <= digits of P + digits of Q - 1).  Two stages: a chunk of 32
// K values is brought in while the previous chunk's MMAs run.  Ends with a CTA
// barrier.
template <int NT, typename S>
__device__ __noinline__ void oz_gemm(const Team &tm, const OzPlanes &P, const OzPlanes &Q, bool conj, int nlev,
                                     OzOut out, cpx<dd> *C, int ldc, const cpx<dd> *add, S &sm_) {
  S sm = sm_.known();
  const bool tri = out == kOzHerm || out == kOzHermT;
  static_assert(NT == 512, "16 warps: 4 row quarters x 4 column quarters of a tile");
  constexpr uint32_t IDESC = tc::idesc_bf16(kOzM, 2 * kOzN);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nch = P.ld / kOzKC;
  const int tm_ = (P.rows + kOzM - 1) / kOzM, tn_ = (Q.rows + kOzN - 1) / kOzN;
  const int ndp = min(P.nd, nlev), ndq = min(Q.nd, nlev);
  unsigned char *base = as_shared(sm.r0);
  int mine = 0;
  for (int t = 0; t < tm_ * tn_; ++t) {
    const int i0 = (t % tm_) * kOzM, y0 = (t / tm_) * kOzN;
    if (tri && y0 + kOzN <= i0) continue;
    if (mine++ % tm.size != tm.rank) continue;
    const int row = 32 * (warp & 3) + lane, cq = warp >> 2;
    dacc acc[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) acc[c].hi = acc[c].lo = 0.f;
    bool pend0 = false, pend1 = false;
    bool fresh = true;  // the next MMA of each level overwrites its accumulator
    for (int ch = 0; ch < nch; ++ch) {
      const int s = ch & 1;
      if (s ? pend1 : pend0) oz_wait(sm, s);
      if (s)
        pend1 = false;
      else
        pend0 = false;
      __nv_bfloat16 *Ps = reinterpret_cast<__nv_bfloat16 *>(base + s * kOzStage);
      __nv_bfloat16 *Qs = Ps + kOzPBytes / 2;
      // pieces of 8 values (16 bytes): (plane, row, piece) -> 8-row core matrices
      for (int idx = tid; idx < ndp * kOzM * 4; idx += NT) {
        const int pc = idx & 3, r = (idx >> 2) & (kOzM - 1), d = idx >> 9;
        const bool ok = i0 + r < P.rows;
        const __nv_bfloat16 *src = P.p + d * P.stride + size_t(ok ? i0 + r : 0) * P.ld + ch * kOzKC + pc * 8;
        cp_async16(Ps + d * (kOzM * kOzKC) + oz_elem(r, pc * 8, kOzKC), src, ok);
      }
      for (int idx = tid; idx < ndq * kOzN * 4; idx += NT) {
        const int pc = idx & 3, y = (idx >> 2) & (kOzN - 1), d = idx >> 7;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (y0 + y < Q.rows)
          v = *reinterpret_cast<const uint4 *>(Q.p + d * Q.stride + size_t(y0 + y) * Q.ld + ch * kOzKC + pc * 8);
        // (re, im) words: re in the low half.  row 2y: (Qr, -Qi); row 2y + 1: (Qi, Qr); conj negates Qi
        const uint32_t neg0 = conj ? 0u : 0x80000000u, neg1 = conj ? 0x00008000u : 0u;
        uint4 a, b;
        a.x = v.x ^ neg0;
        a.y = v.y ^ neg0;
        a.z = v.z ^ neg0;
        a.w = v.w ^ neg0;
        b.x = __byte_perm(v.x, 0, 0x1032) ^ neg1;
        b.y = __byte_perm(v.y, 0, 0x1032) ^ neg1;
        b.z = __byte_perm(v.z, 0, 0x1032) ^ neg1;
        b.w = __byte_perm(v.w, 0, 0x1032) ^ neg1;
        __nv_bfloat16 *q = Qs + d * (2 * kOzN * kOzKC);
        *reinterpret_cast<uint4 *>(q + oz_elem(2 * y, pc * 8, kOzKC)) = a;
        *reinterpret_cast<uint4 *>(q + oz_elem(2 * y + 1, pc * 8, kOzKC)) = b;
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      tc::fence_smem_to_async();
      __syncthreads();
      if (tid == 0) {
        tc::fence_after_sync();
        for (int lv = 0; lv < nlev; ++lv) {
          bool first = fresh;
          for (int ja = max(0, lv - ndq + 1); ja <= min(lv, ndp - 1); ++ja) {
            const int jb = lv - ja;
#pragma unroll
            for (int ks = 0; ks < kOzKC / 16; ++ks) {
              const uint64_t ad =
                  tc::smem_desc(reinterpret_cast<char *>(Ps + ja * (kOzM * kOzKC)) + ks * 256, 128, kOzKC * 16);
              const uint64_t bd =
                  tc::smem_desc(reinterpret_cast<char *>(Qs + jb * (2 * kOzN * kOzKC)) + ks * 256, 128, kOzKC * 16);
              tc::mma_bf16(sm.tmem + uint32_t(64 * lv), ad, bd, IDESC, first ? 0u : 1u);
              first = false;
            }
          }
        }
        tc::mma_commit(sm.gbar + s);
      }
      fresh = false;
      if (s)
        pend1 = true;
      else
        pend0 = true;
      if (ch == nch - 1 || ((ch + 1) * kOzKC) % kOzFlush == 0) {  // drain the levels
        if (pend0 && s == 1) oz_wait(sm, 0);
        if (pend1 && s == 0) oz_wait(sm, 1);
        oz_wait(sm, s);
        pend0 = pend1 = false;
        tc::fence_after_sync();
#pragma unroll 1
        for (int lv = 0; lv < nlev; ++lv) {
          float t16[16];
          tc::tmem_ld16(sm.tmem + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(64 * lv + 16 * cq), t16);
          const float wgt = pow2f(-7 * lv);
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            float sum, e;
            two_sum(acc[c].hi, __fmul_rn(t16[c], wgt), sum, e);
            acc[c].hi = sum;
            acc[c].lo = __fadd_rn(acc[c].lo, e);
          }
        }
        tc::fence_before_sync();
        fresh = true;
        __syncthreads();
      }
    }
    const int x = i0 + row;
    if (x < P.rows) {
      const int ex = P.expo[x];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int y = y0 + 8 * cq + q;
        if (y < Q.rows) {
          const int sh = ex + Q.expo[y] - 14;
          const dd re = dd_norm(acc[2 * q].hi, acc[2 * q].lo), im = dd_norm(acc[2 * q + 1].hi, acc[2 * q + 1].lo);
          cpx<dd> v = mkc<dd>(dd(scale2f(re.hi, sh), scale2f(re.lo, sh)), dd(scale2f(im.hi, sh), scale2f(im.lo, sh)));
          if (tri) {
            if (y < x) continue;
            const cpx<dd> w = mkc<dd>(v.x, -v.y);
            C[size_t(x) * ldc + y] = out == kOzHerm ? v : w;
            if (x != y) C[size_t(y) * ldc + x] = out == kOzHerm ? w : v;
          } else {
            const size_t o = out == kOzTrans ? size_t(y) * ldc + x : size_t(x) * ldc + y;
            if (add) {
              const cpx<dd> a = add[o];
              v = mkc<dd>(a.x + v.x, a.y + v.y);
            }
            C[o] = v;
          }
        }
      }
    }
  }
  sm_.take(sm);
  __syncthreads();
}

}  // namespace tn
