// Batched thin SVD for the truncated tSVD (sm_103a).
//
// Replaces the per-sector LAPACK/Eigen SVD of full_svd_impl
// (src/Core/Tensor.cpp:494-521, src/Interfaces/PlainInterface_Eigen_impl.cpp:114-127).
//
// Algorithm: one-sided (Hestenes) Jacobi in FP32, then FP64 Newton-type refinement by matrix products.
// GB300 issues 64 times as many FP32 as FP64 multiply-adds (an FP64 warp instruction occupies its SM
// sub-partition for ~64 cycles), so the O(n^3) x sweeps work and the latency chains are FP32, and the
// FP64 work is a handful of n x n products spread over every SM (blocks up to kSmallN columns: inside
// one CTA).  Per block, op(A) = A when m >= n, else A^T (U and V swap roles):
//   1. A is scaled by a power of two (exact) so its largest entry is O(1); V32 = the right singular vectors of
//      op(A) in FP32, by a triangular factor and block-Jacobi sweeps until no pair's cosine exceeds kStop32
//      (jacobi32_cluster below).
//   2. V = V32 in FP64, W = op(A) V.
//   3. Up to kIters times: G = W^T W, E = V^T V - I; the first-order update Z of every pair,
//        z_pq + z_qp = -e_pq,  g_pp z_pq + g_qq z_qp = -g_pq,
//      restores V^T V = I and (W^T W)_pq = 0 up to second order; W <- W (I + Z), V <- V (I + Z).  (The
//      refinement of Ogita and Aishima, "Iterative refinement for singular value decomposition based on
//      matrix multiplication", J. Comput. Appl. Math. 369 (2020), in one-sided form.)  Pairs whose z is
//      not small (nearly equal singular values, or columns that FP32 could not resolve) only take the
//      orthogonality part -e/2.  Columns of a graded block that FP32 could not resolve (singular values
//      below ~1e-7 of the largest) are taken up by a second FP32 Jacobi pass, on W in place of op(A).
//   4. Pairs that still miss |w_p.w_q| <= tol |w_p||w_q| (singular values that agree to ~1e-7) are finished by
//      FP64 block-Jacobi sweeps, each rotation exactly orthogonal in FP64 (c = 1/sqrt(1+t^2) refined by
//      Newton steps, s = c t; its angle t comes from FP32 arithmetic on exactly rescaled inputs).
//   5. sigma_j = |w_j| sorted descending (ties by column), u_j = w_j / sigma_j, v_j = V[:, j]; every pair
//      sign-normalised (sign rule below).
// Blocks too large for a cluster's shared memory and at least kFactorN wide take FP64 Jacobi behind a column-pivoted QR
// instead (svd_factor_kernel).
// All control is on the device: every stage is launched once, reads the block's convergence state and
// returns when there is nothing to do, so the host neither waits nor decides.
//
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <new>
#include <stdexcept>
#include <cmath>
#include <string>
#include <mutex>
#include <vector>

#include "kernels.hpp"

namespace cg = cooperative_groups;

namespace xgb {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kCluster = 8;        // CTAs per block in the finishing kernel
constexpr int kMaxSweeps32 = 30;
constexpr int kMaxSweeps64 = 20;
constexpr int kIters = 6;          // refinement iterations at most (two usually do the work, the third checks)
// A sweep whose largest cosine stays below kStop32 is the last one: convergence is quadratic by then, and
// what is left (~1e-6) is the refinement's to remove.
constexpr float kStop32 = 1.0e-3f;
constexpr double kTol64 = 1.0e-13;
// Squared column norms at or below this fraction of the largest one are left out of the FP64
// convergence test and rotations: columns below 1e-15 of the largest are rounding noise of a
// rank-deficient block; rotating them never converges and changes no singular value or kept vector (the
// CTM truncation cuts at 1e-10).  Larger floors (1e-15) skipped directions the CTM keeps and changed its
// environments.
constexpr double kFloor64 = 1.0e-30;
constexpr int kSmemLimit = 220 * 1024;
// blocks up to kSmallN columns run start to finish in one CTA (svd_small_kernel)
constexpr int kSmallN = 24;
// blocks wider than this take the cooperative form (one launch per block) of the FP32 sweeps of pass 1 and of the
// FP64 sweeps
constexpr int kGridN = 512;
// blocks at least this wide whose columns no cluster holds take svd_factor_kernel
constexpr int kFactorN = 512;
constexpr int kFactorCols = 4;  // columns of its Jacobi blocks
constexpr int kFactorSweeps = 80;

template <class T>
__device__ __forceinline__ T wsum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void rr_pair(int round, int k, int N, int& p, int& q) {
  // circle method over N (even) slots: slot 0 fixed, 1..N-1 rotate
  auto pos = [&](int i) { return (round + i < N - 1 ? round + i : round + i - (N - 1)) + 1; };  // round < N - 1
  if (k == 0) { p = 0; q = pos(0); }
  else { p = pos(k); q = pos(N - 1 - k); }
}

__device__ __forceinline__ float ldg(const float* p) { return __ldcg(p); }
__device__ __forceinline__ double ldg(const double* p) { return __ldcg(p); }
__device__ __forceinline__ void stg(float* p, float v) { __stcg(p, v); }
__device__ __forceinline__ void stg(double* p, double v) { __stcg(p, v); }

// shared-memory or global (L1-bypassing) element access
template <class T, bool G>
__device__ __forceinline__ T ld(const T* p) { if constexpr (G) return ldg(p); else return *p; }
template <class T, bool G>
__device__ __forceinline__ void st(T* p, T v) { if constexpr (G) stg(p, v); else *p = v; }

// exact power of two 2^e as a double (|e| < 1000)
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
__device__ __forceinline__ int exponent_of(double x) { return int((__double_as_longlong(x) >> 52) & 0x7ff) - 1023; }

struct Ctx {
  int tid, lane, warp, rank, gw, gnw, gtid, gnt;
};

// FP32 rotation angle t = tan(theta) that zeroes w_p.w_q (Rutishauser's formula), from the difference be - al
// of the squared norms and the dot product ga, both scaled to at most O(1).  The difference is formed in the
// columns' own precision: rounded to FP32 first, squared norms that agree to 1e-7 gave any angle, and such
// pairs did not converge in 20 sweeps.
__device__ __forceinline__ float angle32(float diff, float ga) {
  const float zeta = diff / (2.0f * ga);
  return copysignf(1.0f, zeta) / (fabsf(zeta) + hypotf(1.0f, zeta));
}

// One plane rotation between columns p and q (warp-cooperative).  Returns
// true if a rotation was applied.
// Pairs with a column whose squared norm is at most `floor` are left alone:
// such a column changes no singular value by more than its norm.
template <class T, bool G>
__device__ bool rotate(T* wp, T* wq, T* vp, T* vq, T* np, T* nq, int64_t mm, int nn, T tol, T floor, int lane) {
  const T al = ld<T, G>(np), be = ld<T, G>(nq);
  if (!(al > floor) || !(be > floor)) return false;
  T ga = 0;
  for (int64_t i = lane; i < mm; i += 32) ga = fma(ld<T, G>(wp + i), ld<T, G>(wq + i), ga);
  ga = wsum(ga);
  if (ga * ga <= tol * tol * al * be) return false;
  T cs, sn, t;
  if constexpr (sizeof(T) == 4) {
    t = angle32(be - al, ga);
    cs = rsqrtf(1.0f + t * t);
    sn = cs * t;
  } else {
    // exact rescaling by a power of two brings be - al and ga into FP32 range
    const double sc = pow2(-exponent_of(fmax(al, be)));
    t = double(angle32(float((be - al) * sc), float(ga * sc)));
    const double x = 1.0 + t * t;
    double r = double(rsqrtf(float(x)));
    r = r * (1.5 - 0.5 * x * r * r);
    r = r * (1.5 - 0.5 * x * r * r);
    cs = r;
    sn = r * t;
  }
  for (int64_t i = lane; i < mm; i += 32) {
    const T x = ld<T, G>(wp + i), y = ld<T, G>(wq + i);
    st<T, G>(wp + i, cs * x - sn * y);
    st<T, G>(wq + i, sn * x + cs * y);
  }
  for (int i = lane; i < nn; i += 32) {
    const T x = ld<T, G>(vp + i), y = ld<T, G>(vq + i);
    st<T, G>(vp + i, cs * x - sn * y);
    st<T, G>(vq + i, sn * x + cs * y);
  }
  __syncwarp();
  if (lane == 0) {
    st<T, G>(np, al - t * ga);
    st<T, G>(nq, be + t * ga);
  }
  __syncwarp();
  return true;
}

// Rotations of one outer round for the CTA's block pair, columns staged in
// shared memory: column c (< 2b) at W + c*mm, V + c*nn, N + c; block A is
// [0, la), block B is [b, b+lb).
template <class T>
__device__ bool round_rotations(const Ctx& c, T* W, T* V, T* N, int b, int la, int lb, bool inner, int64_t mm, int nn,
                                T tol, T floor) {
  bool any = false;
  if (inner) {
    // pairs inside block A and inside block B: circle method over each block
    const int pa = la + (la & 1), pb = lb + (lb & 1);
    const int rounds = max(pa, pb) - 1;
    for (int r = 0; r < rounds; ++r) {
      const int na = r < pa - 1 ? pa / 2 : 0, nb = r < pb - 1 ? pb / 2 : 0;
      for (int k = c.warp; k < na + nb; k += kWarps) {
        int p, q, base;
        if (k < na) { rr_pair(r, k, pa, p, q); base = 0; if (p >= la || q >= la) continue; }
        else { rr_pair(r, k - na, pb, p, q); base = b; if (p >= lb || q >= lb) continue; }
        p += base;
        q += base;
        any |= rotate<T, false>(W + p * mm, W + q * mm, V + p * nn, V + q * nn, N + p, N + q, mm, nn, tol, floor, c.lane);
      }
      __syncthreads();
    }
  }
  // cross pairs (i, (i + r) mod b), i in A, j in B
  for (int r = 0; r < b; ++r) {
    for (int i = c.warp; i < b; i += kWarps) {
      const int j = (i + r) % b;
      if (i >= la || j >= lb) continue;
      const int p = i, q = b + j;
      any |= rotate<T, false>(W + p * mm, W + q * mm, V + p * nn, V + q * nn, N + p, N + q, mm, nn, tol, floor, c.lane);
    }
    __syncthreads();
  }
  return any;
}

template <class T, class Group>
__device__ int block_jacobi(Group& cl, const Ctx& c, T* W, T* V, T* norms, int* flag, int64_t mm, int nn,
                            T tol, T rel_floor, int max_sweeps, T* smem, bool staged, int nblocks, int* perm) {
  // nblocks = 2 x (CTAs of the group): one block pair per CTA and round.  perm (nn ints): at the start
  // of every sweep the columns are ordered by decreasing norm (de Rijk's pivoting, as in LAPACK's
  // dgesvj) and the blocks are cut from that order, which keeps graded columns converging.
  const int b = (nn + nblocks - 1) / nblocks;
  auto col_of = [&](int idx) { return __ldcg(perm + idx); };
  int sweeps = 0;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    for (int j = c.gw; j < nn; j += c.gnw) {
      const T* w = W + int64_t(j) * mm;
      T a = 0;
      for (int64_t i = c.lane; i < mm; i += 32) { const T x = ldg(w + i); a = fma(x, x, a); }
      a = wsum(a);
      if (c.lane == 0) stg(norms + j, fmin(a, T(sizeof(T) == 4 ? 3.0e38 : 1.0e308)));  // (a NaN column is ordered, not lost)
    }
    if (c.rank == 0 && c.tid == 0) atomicExch(flag, 0);
    cl.sync();
    // columns below rel_floor * (largest squared column norm) are numerically zero at this precision
    T gmax = 0;
    for (int j = c.lane; j < nn; j += 32) gmax = fmax(gmax, ldg(norms + j));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gmax = fmax(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
    const T floor = rel_floor * gmax;
    for (int j = c.gw; j < nn; j += c.gnw) {
      const T nj = ldg(norms + j);
      int r = 0;
      for (int i = c.lane; i < nn; i += 32) {
        const T ni = ldg(norms + i);
        r += (ni > nj) || (ni == nj && i < j);
      }
      r = wsum(r);
      if (c.lane == 0) __stcg(perm + r, j);
    }
    cl.sync();
    for (int round = 0; round < nblocks - 1; ++round) {
      int ba, bb;
      rr_pair(round, c.rank, nblocks, ba, bb);
      const int ca = ba * b, cb = bb * b;
      const int la = max(0, min(b, nn - ca)), lb = max(0, min(b, nn - cb));
      auto gcol = [&](int col) {
        return col < b ? (col < la ? col_of(ca + col) : -1) : (col - b < lb ? col_of(cb + col - b) : -1);
      };
      bool any = false;
      if (staged) {
        T* sW = smem;                        // 2b columns of mm
        T* sV = sW + int64_t(2 * b) * mm;    // 2b columns of nn
        T* sN = sV + int64_t(2 * b) * nn;    // 2b norms
        for (int col = c.warp; col < 2 * b; col += kWarps) {
          const int g = gcol(col);
          for (int64_t i = c.lane; i < mm; i += 32) sW[col * mm + i] = g >= 0 ? ldg(W + int64_t(g) * mm + i) : T(0);
          for (int i = c.lane; i < nn; i += 32) sV[col * nn + i] = g >= 0 ? ldg(V + int64_t(g) * nn + i) : T(0);
          if (c.lane == 0) sN[col] = g >= 0 ? ldg(norms + g) : T(0);
        }
        __syncthreads();
        any = round_rotations<T>(c, sW, sV, sN, b, la, lb, round == 0, mm, nn, tol, floor);
        for (int col = c.warp; col < 2 * b; col += kWarps) {
          const int g = gcol(col);
          if (g < 0) continue;
          for (int64_t i = c.lane; i < mm; i += 32) stg(W + int64_t(g) * mm + i, sW[col * mm + i]);
          for (int i = c.lane; i < nn; i += 32) stg(V + int64_t(g) * nn + i, sV[col * nn + i]);
          if (c.lane == 0) stg(norms + g, sN[col]);
        }
      } else {
        // staging does not fit: rotate the columns in place in L2 with
        // per-pair pointers (the two blocks are not adjacent in memory)
        if (round == 0) {
          const int pa = la + (la & 1), pb = lb + (lb & 1);
          const int rounds = max(pa, pb) - 1;
          for (int r = 0; r < rounds; ++r) {
            const int na = r < pa - 1 ? pa / 2 : 0, nb = r < pb - 1 ? pb / 2 : 0;
            for (int k = c.warp; k < na + nb; k += kWarps) {
              int p, q, base;
              if (k < na) { rr_pair(r, k, pa, p, q); base = ca; if (p >= la || q >= la) continue; }
              else { rr_pair(r, k - na, pb, p, q); base = cb; if (p >= lb || q >= lb) continue; }
              p = col_of(p + base);
              q = col_of(q + base);
              any |= rotate<T, true>(W + int64_t(p) * mm, W + int64_t(q) * mm, V + int64_t(p) * nn, V + int64_t(q) * nn,
                                     norms + p, norms + q, mm, nn, tol, floor, c.lane);
            }
            __syncthreads();
          }
        }
        for (int r = 0; r < b; ++r) {
          for (int i = c.warp; i < b; i += kWarps) {
            const int j = (i + r) % b;
            if (i >= la || j >= lb) continue;
            const int p = col_of(ca + i), q = col_of(cb + j);
            any |= rotate<T, true>(W + int64_t(p) * mm, W + int64_t(q) * mm, V + int64_t(p) * nn, V + int64_t(q) * nn,
                                   norms + p, norms + q, mm, nn, tol, floor, c.lane);
          }
          __syncthreads();
        }
      }
      if (any && c.lane == 0) atomicExch(flag, 1);
      cl.sync();
    }
    ++sweeps;
    const int any = atomicAdd(flag, 0);
    cl.sync();  // every CTA has read the flag before the next sweep resets it
    if (!any) break;
  }
  return sweeps;
}

// ---------------------------------------------------------------- FP32 block Jacobi, columns in registers
// One plane rotation of two columns with squared norms al and be: what does not need their dot product is
// computed before it (Pre), so that only one square root, one reciprocal and one more square root follow the
// warp's sum.  With d = (be - al) / (al + be) and g = 2 ga / (al + be), t = g / (d + sign(d) sqrt(d^2 + g^2))
// is the smaller root of the rotation's quadratic; nothing here squares a norm, so columns down to 1e-18 of
// the largest stay in range.  Approximate reciprocals and square roots (2 ulp): the rotations leave V32
// orthogonal to ~1e-6, which the FP64 refinement restores.
__device__ __forceinline__ float rsq(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// cosines below the rounding of a dot product of mm terms are left alone
__device__ __forceinline__ float tol32(int64_t mm) { return sqrtf(float(mm)) * 6.0e-8f; }
struct Pre32 {
  float root, inv, d;  // sqrt(al be), 2 / (al + be), (be - al) / (al + be)
};
__device__ __forceinline__ Pre32 pre32(float al, float be) {
  Pre32 p;
  p.root = al > 0.0f && be > 0.0f ? al * rsq(al) * (be * rsq(be)) : 3.0e38f;
  const float i = rcp(al + be);
  p.inv = i + i;
  p.d = (be - al) * i;
  return p;
}
// 0: orthogonal to `tol` (or a zero column), 1: rotated, 2: rotated and above kStop32
__device__ __forceinline__ int plan32(float ga, const Pre32& p, float tol, float& cs, float& sn, float& t) {
  const float ag = fabsf(ga);
  if (!(ag > tol * p.root)) return 0;
  const float g = ga * p.inv, h2 = fmaf(g, g, p.d * p.d);
  t = __fmul_rn(g, rcp(p.d + copysignf(h2 * rsq(h2), p.d)));
  cs = rsq(fmaf(t, t, 1.0f));
  sn = cs * t;
  return ag > kStop32 * p.root ? 2 : 1;
}

// Two FP32 values per 64-bit register: one packed instruction does both.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pack2(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float sum2(f2 a) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a));
  return lo + hi;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// A column of the sweeps in registers: NV (even) units of 2 LP rows, zero padded; LP lanes hold it, lane l
// rows 4 l .. 4 l + 3 of every two units, and a warp works on 32 / LP pairs of columns at once.  A pair costs ~50
// instructions beside its rows' (the sum over the lanes, the angle), so short columns take few lanes: with a
// whole warp on each pair a step of 32 pairs of 64 rows was bound by instruction issue (920 cycles).  NV is a
// template argument so that the loops have no predicates: with a runtime row count every row cost a
// comparison and a predicate beside its six instructions (2060 cycles a step at 347 rows).
template <int NV>
struct Column {
  f2 v[NV];
};
template <int LP, int NV>
__device__ __forceinline__ void load_column(Column<NV>& x, const float* from, int l) {
  const ulonglong2* p = reinterpret_cast<const ulonglong2*>(from) + l;
#pragma unroll
  for (int u = 0; u < NV; u += 2) {
    const ulonglong2 t = p[u / 2 * LP];
    x.v[u] = t.x;
    x.v[u + 1] = t.y;
  }
}
template <int LP, int NV>
__device__ __forceinline__ void store_column(const Column<NV>& x, float* to, int l) {
  ulonglong2* p = reinterpret_cast<ulonglong2*>(to) + l;
#pragma unroll
  for (int u = 0; u < NV; u += 2) p[u / 2 * LP] = make_ulonglong2(x.v[u], x.v[u + 1]);
}
// sum over the LP lanes of a column (all lanes of the warp take part)
template <int LP>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
  for (int o = LP / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// product of the first NW units
template <int NW, int NV>
__device__ __forceinline__ float dot_units(const Column<NV>& x, const Column<NV>& y) {
  f2 a = mul2(x.v[0], y.v[0]), b = 0;
#pragma unroll
  for (int u = 1; u < NW; ++u) {
    if (u & 1) b = fma2(x.v[u], y.v[u], b);
    else a = fma2(x.v[u], y.v[u], a);
  }
  return sum2(a) + sum2(b);
}
template <int NV>
__device__ __forceinline__ void rotate_columns(Column<NV>& x, Column<NV>& y, float cs, float sn) {
  const f2 c2 = pack2(cs, cs), s2 = pack2(sn, sn), n2 = pack2(-sn, -sn);
#pragma unroll
  for (int u = 0; u < NV; ++u) {
    const f2 xv = x.v[u];
    x.v[u] = fma2(c2, xv, mul2(n2, y.v[u]));
    y.v[u] = fma2(s2, xv, mul2(c2, y.v[u]));
  }
}
// the same with y streamed from shared memory: columns too long to keep two of in registers
template <int LP, int NW, int NV>
__device__ __forceinline__ float dot_units(const Column<NV>& x, const float* Y, int l) {
  const ulonglong2* y = reinterpret_cast<const ulonglong2*>(Y) + l;
  f2 a = 0, b = 0;
#pragma unroll
  for (int u = 0; u < NW; u += 2) {
    const ulonglong2 t = y[u / 2 * LP];
    a = fma2(x.v[u], t.x, a);
    if (u + 1 < NW) b = fma2(x.v[u + 1], t.y, b);
  }
  return sum2(a) + sum2(b);
}
template <int LP, int NV>
__device__ __forceinline__ void rotate_columns(Column<NV>& x, float* Y, float cs, float sn, int l) {
  ulonglong2* y = reinterpret_cast<ulonglong2*>(Y) + l;
  const f2 c2 = pack2(cs, cs), s2 = pack2(sn, sn), n2 = pack2(-sn, -sn);
#pragma unroll
  for (int u = 0; u < NV; u += 2) {
    const ulonglong2 t = y[u / 2 * LP];
    const f2 xa = x.v[u], xb = x.v[u + 1];
    x.v[u] = fma2(c2, xa, mul2(n2, t.x));
    x.v[u + 1] = fma2(c2, xb, mul2(n2, t.y));
    y[u / 2 * LP] = make_ulonglong2(fma2(s2, xa, mul2(c2, t.x)), fma2(s2, xb, mul2(c2, t.y)));
  }
}
constexpr int kKeepUnits = 20;  // both columns of a pair in registers up to this height

// Rotation of the pair whose first column is x (registers) and second one Y (shared memory), squared norms al
// and *ny, by the product of their first NW units; `on`: the lanes' pair exists (the others only take part in
// the sum).  Returns plan32's class.
template <int LP, int NW, int NV>
__device__ __forceinline__ int rotate_pair(Column<NV>& x, float& al, float* Y, float* ny, bool on, float tol, int l) {
  const float be = *ny;
  const Pre32 pre = pre32(al, be);
  float cs, sn, t, ga;
  int k;
  if constexpr (NV <= kKeepUnits) {
    Column<NV> y;
    load_column<LP>(y, Y, l);
    ga = lanes_sum<LP>(dot_units<NW>(x, y));
    k = on ? plan32(ga, pre, tol, cs, sn, t) : 0;
    if (k) {
      rotate_columns(x, y, cs, sn);
      store_column<LP>(y, Y, l);
    }
  } else {
    ga = lanes_sum<LP>(dot_units<LP, NW>(x, Y, l));
    k = on ? plan32(ga, pre, tol, cs, sn, t) : 0;
    if (k) rotate_columns<LP>(x, Y, cs, sn, l);
  }
  if (k) {
    al -= t * ga;
    if (l == 0) *ny = be + t * ga;
  }
  return k;
}

// The steps of one round: the LP lanes `col` hold column col (of la) of the first block in x and meet the lb
// columns of the second block in shared memory, one per step; one barrier of the warps that hold columns a step.
template <int LP, int NW, int NV>
__device__ __forceinline__ int cross_steps(Column<NV>& x, float& al, float* sB, float* nB, int stride, int b, int la,
                                           int lb, float tol, int col, int l) {
  const int warps = (b + 32 / LP - 1) / (32 / LP);
  int worst = 0, j = col < b ? col : 0;
  for (int r = 0; r < b; ++r) {
    const bool on = col < la && j < lb;
    worst = max(worst, rotate_pair<LP, NW>(x, al, sB + j * stride, nB + j, on, tol, l));
    if (++j == b) j = 0;
    asm volatile("bar.sync 1, %0;" ::"r"(32 * warps) : "memory");
  }
  return worst;
}

// The pairs inside two blocks of b columns in shared memory, circle method (`a` null: the block at bb alone);
// called by all threads.
template <int LP, int NW, int NV>
__device__ __forceinline__ int inner_steps(float* a, float* na, int la, float* bb, float* nb, int lb, int stride, int b,
                                           float tol, int col, int l) {
  const int pp = b + (b & 1), lanes = a ? pp : pp / 2;
  const bool first = a && col < pp / 2;
  const int lim = first ? la : lb, me = a && !first ? col - pp / 2 : col;
  float* base = first ? a : bb;
  float* nbase = first ? na : nb;
  int worst = 0;
  for (int r = 0; r < pp - 1; ++r) {
    if (col - col % (32 / LP) < lanes) {  // warp-uniform
      int p = 0, q = 0;
      if (col < lanes) rr_pair(r, me, pp, p, q);
      const bool on = col < lanes && p < lim && q < lim;
      if (!on) p = q = 0;
      Column<NV> x;
      load_column<LP>(x, base + p * stride, l);
      float al = nbase[p];
      const int k = rotate_pair<LP, NW>(x, al, base + q * stride, nbase + q, on, tol, l);
      if (k) {
        store_column<LP>(x, base + p * stride, l);
        if (l == 0) nbase[p] = al;
      }
      worst = max(worst, k);
    }
    __syncthreads();
  }
  return worst;
}

// How a block's columns are held: LP lanes, NU units, P CTAs of 2b columns each; `wide`: floats between the
// columns of the matrix (those of its triangular factor lie 2 LP NU apart).
struct Shape32 {
  int lp, nu, P, b, wide;
};
// compiled (LP, NU): 8 x 2, 4, .. 10 and 16 x 6, 8, .. 20 in pass 0, 16 x 2, 4, .. 12 in pass 1
// The fewest CTAs (a power of two: each exchange costs more than a longer stretch of steps) with at most 32
// pairs each (beyond that a step's loads and arithmetic add up: 1090 cycles at 55 pairs of 110 rows against 520
// at 32 of 64) whose shared memory holds the columns and their successors; P = 0: no such shape up to `most`.
__host__ __device__ __forceinline__ Shape32 shape32(int pass, int64_t mm, int64_t nn, int most, int64_t smem) {
  Shape32 s;
  s.P = 0;
  if (nn > (pass ? 384 : 640) || (pass && mm > 384)) return s;
  s.lp = nn <= 160 && !pass ? 8 : 16;
  const int unit = 4 * s.lp;  // rows of two units
  // the matrix's columns in as many registers as its factor's, when they are little longer
  const bool same = pass || (mm <= (s.lp == 8 ? 160 : 640) && 4 * mm <= 5 * nn);
  s.nu = 2 * int(((same ? mm : nn) + unit - 1) / unit);
  const int64_t narrow = 2 * s.lp * s.nu * (pass ? 2 : 1), rows = (mm + unit - 1) / unit * unit;
  const int64_t wide = rows > narrow ? rows : narrow;
  for (int P = 1; P <= most; P *= 2) {
    const int64_t b = (nn + 2 * P - 1) / (2 * P);
    if (b > 32 || 4 * (2 * b * (wide + narrow) + 4 * b + 2 * (2 * b * P) + 8 + 2 * wide) > smem) continue;
    s.P = P;
    s.b = int(b);
    s.wide = int(wide);
    return s;
  }
  return s;
}

// FP32 singular vectors of op(A) over a cluster of P CTAs whose shared memory holds its columns throughout.
//
// 1. op(A) = Q R by modified Gram-Schmidt, one column after the other: w_k goes to every CTA, the lanes of
//    column j > k take R_kj = q_k . w_j (q_k = w_k / |w_k|) and w_j -= R_kj q_k, and row k of R becomes column k
//    of X = R^T.  (R is as accurate as Householder's: A. Bjorck, BIT 7 (1967).)  Q is not needed.
// 2. One-sided block Jacobi on X: its columns are closer to orthogonal than op(A)'s (the preconditioning of
//    Drmac and Veselic, SIAM J. Matrix Anal. Appl. 29 (2008): 8 sweeps where graded op(A) took 13 to 23), they
//    are nn long and not mm + nn: X = U_X S V_X^T gives R = V_X S U_X^T, so the right singular vectors of op(A)
//    are U_X, the normalised rotated columns, and no rotation is accumulated.  A column of R below 1e-12 (the
//    matrix is scaled to O(1)) is replaced by 1e-12 times its unit vector, so that every column of U_X exists.
//
// The nn columns form 2P blocks of b columns in the order of decreasing norm (de Rijk's pivoting, as in
// LAPACK's dgesvj, renewed every sweep).  In each of a sweep's 2P - 1 rounds a CTA owns one pair of blocks
// (circle method) and visits its b^2 pairs in b steps (cross_steps); the pairs inside a block are visited in
// round 0.  A sweep is about nn steps whatever P is, and every round adds an exchange of the blocks (each CTA
// pulls its next two out of the cluster's shared memory into its other buffer; one cluster barrier).  What
// bounds it: the latency of a step (the lanes' sum, one square root, one reciprocal, one square root, one
// barrier), with long columns instruction issue.
// init(j, i) is op(A); the vectors leave as out(j, i, value), j < nn columns in some order.
//
// NV = 2 NU (pass 1, on columns that are already graded and nearly orthogonal): no triangular factor; the
// sweeps run on the columns themselves with the rotations accumulated in their second half, since only the
// product of the rotations keeps the small mixing of a large column into a small one to full relative
// accuracy, and it is what leaves.
// Measured on GB300, cycles a sweep: 23k + 16k + 5k (pairs inside the blocks, across them, the rest) for 64
// columns, 21k + 86k + 56k for 134 (4 CTAs), 42k + 333k + 200k for 347 (8 CTAs); both blocks in shared memory
// and the columns through L2 every round took 200k for 76 columns and 2.1M for 347, and twice the sweeps.  The
// triangular factor takes 72k, 340k and 1.4M.
template <int LP, int NU, int NV, class Init, class Out>
__device__ int jacobi32_cluster(cg::cluster_group& cl, const Ctx& c, const Shape32& sh, int mm, int nn, float tol,
                                int max_sweeps, float* sm, Init init, Out out) {
  constexpr bool kAcc = NV > NU;
  constexpr int kPer = 32 / LP, kHalf = 2 * LP * NU, kStride = 2 * LP * NV, kGroups = kWarps * kPer;
  const int P = sh.P, b = sh.b, nblocks = 2 * P, slots = 2 * b, wide = sh.wide;
  const int lane = c.lane, warp = c.warp, l = lane % LP, col = warp * kPer + lane / LP;
  float* buf0 = sm;  // 2b columns each: op(A)'s (stride wide) at first, and X's
  float* buf1 = sm + slots * wide;
  float* wk0 = buf1 + slots * kStride;  // copies of another CTA's w_k, alternating
  float* wk1 = wk0 + wide;
  float* norm0 = wk1 + wide;
  float* norm1 = norm0 + slots;
  float* table = norm1 + slots;                            // the cluster's norms (2b P), -1: no column
  int* order = reinterpret_cast<int*>(table + slots * P);  // position -> CTA and slot of the column
  int* any = order + slots * P;                            // this CTA saw a cosine above kStop32
  float* nk = reinterpret_cast<float*>(any + 4);           // |w_k|^2, alternating; [2, 3]: copies
  const int first = c.rank * slots;  // slot u of CTA k holds column 2b k + u
  const int own = max(0, min(slots, nn - first));
  for (int u = warp; u < slots; u += kWarps) {
    float* w = kAcc ? buf1 + u * kStride : buf0 + u * wide;
    for (int i = lane; i < (kAcc ? kHalf : wide); i += 32) w[i] = u < own && i < mm ? init(first + u, i) : 0.f;
    float* v = buf1 + u * kStride + (kAcc ? kHalf : 0);
    for (int i = lane; i < kHalf; i += 32) v[i] = kAcc && i == first + u ? 1.f : 0.f;
  }
  if (c.tid == 0) *any = 1;
  __syncthreads();

  if constexpr (!kAcc) {
    // ---- R by modified Gram-Schmidt
    const bool held = wide == kStride;  // columns of op(A) fit the registers of X's
    const int quads = wide / (4 * LP);
    // |w_u|^2 of this warp's columns u
    auto square = [&](int u) {
      f2 s0 = 0, s1 = 0;
      const ulonglong2* p = reinterpret_cast<const ulonglong2*>(buf0 + u * wide) + l;
      for (int e = 0; e < quads; ++e) {
        const ulonglong2 t = p[e * LP];
        s0 = fma2(t.x, t.x, s0);
        s1 = fma2(t.y, t.y, s1);
      }
      return lanes_sum<LP>(sum2(s0) + sum2(s1));
    };
    if (warp == 0) {
      const float a = square(0);
      if (lane == 0) nk[0] = a;
    }
    for (int k = 0; k < nn; ++k) {
      const int owner = k / slots, uk = k - owner * slots;
      const float* wk = buf0 + uk * wide;
      const float* ak = nk + (k & 1);
      if (P > 1) {
        cl.sync();
        if (owner != c.rank) {
          float* to = k & 1 ? wk1 : wk0;
          const ulonglong2* from = reinterpret_cast<const ulonglong2*>(cl.map_shared_rank(buf0, owner) + uk * wide);
          for (int e = c.tid; e < wide / 4; e += kThreads) reinterpret_cast<ulonglong2*>(to)[e] = from[e];
          if (c.tid == 0) nk[2 + (k & 1)] = cl.map_shared_rank(nk, owner)[k & 1];
          wk = to;
          ak = nk + 2 + (k & 1);
        }
      }
      __syncthreads();
      const float a = *ak;
      const bool live = a > 1.0e-24f;
      const float inv = live ? rsq(a) : 0.f;
      float* x = cl.map_shared_rank(buf1, owner) + uk * kStride;  // row k of R
      if (owner == c.rank && c.tid == kThreads - 1) x[k] = live ? a * inv : 1.0e-12f;
      Column<NU> q;
      if (held && first + own - 1 > k) load_column<LP>(q, wk, l);
      for (int u0 = warp * kPer; u0 < own; u0 += kGroups) {
        if (first + u0 + kPer - 1 <= k) continue;  // warp-uniform: columns already done
        const int u = u0 + lane / LP;
        const bool on = u < own && first + u > k;
        float* w = buf0 + min(u, own - 1) * wide;
        const bool next = first + u0 <= k + 1 && k + 1 < first + u0 + kPer;  // warp-uniform: column k + 1 is here
        float r, sq = 0.f;
        if (held) {
          Column<NU> y;
          load_column<LP>(y, w, l);
          r = lanes_sum<LP>(dot_units<NU>(q, y)) * inv;
          const float f = -r * inv;
          const f2 f22 = pack2(f, f);
  #pragma unroll
          for (int e = 0; e < NU; ++e) y.v[e] = fma2(f22, q.v[e], y.v[e]);
          if (on) store_column<LP>(y, w, l);
          if (next) sq = lanes_sum<LP>(dot_units<NU>(y, y));
        } else {
          const ulonglong2* qp = reinterpret_cast<const ulonglong2*>(wk) + l;
          ulonglong2* wp = reinterpret_cast<ulonglong2*>(w) + l;
          f2 s0 = 0, s1 = 0;
  #pragma unroll 2
          for (int e = 0; e < quads; ++e) {
            const ulonglong2 t = wp[e * LP], v = qp[e * LP];
            s0 = fma2(t.x, v.x, s0);
            s1 = fma2(t.y, v.y, s1);
          }
          r = lanes_sum<LP>(sum2(s0) + sum2(s1)) * inv;
          const float f = -r * inv;
          const f2 f22 = pack2(f, f);
          if (on)
  #pragma unroll 2
            for (int e = 0; e < quads; ++e) {
              const ulonglong2 t = wp[e * LP], v = qp[e * LP];
              wp[e * LP] = make_ulonglong2(fma2(f22, v.x, t.x), fma2(f22, v.y, t.y));
            }
          if (next) {
            __syncwarp();
            sq = square(min(u, own - 1));
          }
        }
        if (on && l == 0) {
          x[first + u] = r;
          if (first + u == k + 1) nk[(k + 1) & 1] = sq;
        }
      }
    }
    if (P > 1) cl.sync();
  }

  // ---- Jacobi sweeps on X
  int s = 1, sweeps = 0, pos_a = 0, pos_b = 0;  // current buffer; sorted positions of this CTA's two blocks
  int la = min(b, own), lb = max(0, own - b);
  for (;;) {
    float* buf = s ? buf1 : buf0;
    float* norm = s ? norm1 : norm0;
    __syncthreads();
    for (int u0 = warp * kPer; u0 < slots; u0 += kGroups) {
      const int u = u0 + lane / LP;
      Column<NV> x;
      load_column<LP>(x, buf + min(u, slots - 1) * kStride, l);
      const float a = lanes_sum<LP>(dot_units<NU>(x, x));
      const bool on = u < b ? u < la : u - b < lb;
      if (l == 0 && u < slots) norm[u] = on ? fminf(a, 3.0e38f) : -1.f;  // (a NaN column is ordered, not lost)
    }
    cl.sync();
    int again = 0;
    for (int k = c.tid; k < P; k += kThreads) again |= *cl.map_shared_rank(any, k);
    for (int u = c.tid; u < slots * P; u += kThreads) table[u] = cl.map_shared_rank(norm, u / slots)[u % slots];
    again = __syncthreads_or(again);
    if (!again || sweeps == max_sweeps) break;  // the same in every CTA
    for (int u = c.tid; u < slots * P; u += kThreads) {
      const float nu = table[u];
      int r = 0;
#pragma unroll 8
      for (int v = 0; v < slots * P; ++v) {
        const float nv = table[v];
        r += (nv > nu) || (nv == nu && v < u);
      }
      order[r] = (u / slots) << 16 | u % slots;
    }
    __syncthreads();
    int worst = 0;
    for (int round = 0; round < nblocks - 1; ++round) {
      int ba, bb;
      rr_pair(round, c.rank, nblocks, ba, bb);
      la = max(0, min(b, nn - ba * b));
      lb = max(0, min(b, nn - bb * b));
      // CTA and slot of column `col` of a block: by the order at first, then where the previous round left it
      auto source = [&](int blk) {
        if (round == 0) return order[blk * b + col];
        if (blk == 0) return col;
        int i = blk - round;
        if (i < 0) i += nblocks - 1;
        return i == 0 ? b + col : i < P ? i << 16 | col : (nblocks - 1 - i) << 16 | (b + col);
      };
      buf = s ? buf1 : buf0;
      norm = s ? norm1 : norm0;
      s ^= 1;
      float* sA = s ? buf1 : buf0;
      float* sB = sA + b * kStride;
      float* nA = s ? norm1 : norm0;
      float* nB = nA + b;
      Column<NV> x = {};
      float al = 0.f;
      if (col < la) {
        const int at = source(ba);
        load_column<LP>(x, cl.map_shared_rank(buf, at >> 16) + (at & 0xffff) * kStride, l);
        al = cl.map_shared_rank(norm, at >> 16)[at & 0xffff];
      }
      if (col < lb) {
        const int at = source(bb);
        Column<NV> y;
        load_column<LP>(y, cl.map_shared_rank(buf, at >> 16) + (at & 0xffff) * kStride, l);
        const float nb = cl.map_shared_rank(norm, at >> 16)[at & 0xffff];
        store_column<LP>(y, sB + col * kStride, l);
        if (l == 0) nB[col] = nb;
      }
      if (round == 0 && b > 1) {
        if (col < la) {
          store_column<LP>(x, sA + col * kStride, l);
          if (l == 0) nA[col] = al;
        }
        __syncthreads();
        worst = max(worst, inner_steps<LP, NU, NV>(sA, nA, la, sB, nB, lb, kStride, b, tol, col, l));
        if (col < la) {
          al = nA[col];
          load_column<LP>(x, sA + col * kStride, l);
        }
      }
      __syncthreads();
      if (warp * kPer < b) worst = max(worst, cross_steps<LP, NU>(x, al, sB, nB, kStride, b, la, lb, tol, col, l));
      if (col < la) {
        store_column<LP>(x, sA + col * kStride, l);
        if (l == 0) nA[col] = al;
      }
      pos_a = ba * b;
      pos_b = bb * b;
      if (round + 1 == nblocks - 1) {
        const int saw = __syncthreads_or(worst == 2);
        if (c.tid == 0) *any = saw;
      } else {
        cl.sync();
      }
    }
    ++sweeps;
  }
  const float* buf = s ? buf1 : buf0;
  for (int u = warp; u < slots; u += kWarps) {
    const int j = u < b ? (u < la ? pos_a + u : -1) : (u - b < lb ? pos_b + u - b : -1);
    if (j < 0) continue;
    const float inv = kAcc ? 1.f : rsq(fmaxf((s ? norm1 : norm0)[u], 1.0e-37f));
    for (int i = lane; i < nn; i += 32) out(j, i, buf[u * kStride + (kAcc ? kHalf : 0) + i] * inv);
  }
  cl.sync();  // no CTA leaves while another reads its norms
  return sweeps;
}

// The sweeps on op(A) itself with its rotations accumulated, the stacked columns [W; V] in global memory (L2)
// between rounds, for a cooperative grid of P CTAs or a cluster whose shared memory cannot hold them: W
// (mm x nn) and V (nn x nn) column-major, each padded to H units of 64 rows in registers, norms and perm nn
// each.  b <= 16 columns per block.
__host__ __device__ __forceinline__ int64_t global32_bytes(int64_t nn, int P, int H) {
  const int64_t b = (nn + 2 * P - 1) / (2 * P);
  return 4 * b * (128 * H + 1);
}

template <int H, class Group>
__device__ int jacobi32_global(Group& g, const Ctx& c, int P, float* W, float* V, float* norms, int* perm, int* flag,
                               int mm, int nn, float tol, int max_sweeps, float* sm, int smem_bytes) {
  constexpr int Lp = 128 * H;
  const int nblocks = 2 * P, b = (nn + nblocks - 1) / nblocks;
  const bool two = 2 * global32_bytes(nn, P, H) <= smem_bytes;  // both blocks fit for the pairs inside them
  float* sA = sm;
  float* sB = two ? sm + b * Lp : sm;
  float* nB = sm + (two ? 2 : 1) * b * Lp;
  float* nA = nB + b;  // (two only)
  const int lane = c.lane, warp = c.warp;
  auto pull = [&](Column<2 * H>& x, int gc) {
    const float* w = W + int64_t(gc) * mm;
    const float* v = V + int64_t(gc) * nn;
#pragma unroll
    for (int u = 0; u < 2 * H; ++u) {
      const int h = u < H ? u : u - H, i = h / 2 * 128 + 4 * lane + h % 2 * 2, lim = u < H ? mm : nn;
      const float* p = u < H ? w : v;
      x.v[u] = pack2(i < lim ? __ldcg(p + i) : 0.f, i + 1 < lim ? __ldcg(p + i + 1) : 0.f);
    }
  };
  auto push = [&](const Column<2 * H>& x, int gc) {
    float* w = W + int64_t(gc) * mm;
    float* v = V + int64_t(gc) * nn;
#pragma unroll
    for (int u = 0; u < 2 * H; ++u) {
      const int h = u < H ? u : u - H, i = h / 2 * 128 + 4 * lane + h % 2 * 2, lim = u < H ? mm : nn;
      float* p = u < H ? w : v;
      float lo, hi;
      asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x.v[u]));
      if (i < lim) __stcg(p + i, lo);
      if (i + 1 < lim) __stcg(p + i + 1, hi);
    }
  };
  int sweeps = 0;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    for (int j = c.gw; j < nn; j += c.gnw) {
      const float* w = W + int64_t(j) * mm;
      float a = 0;
      for (int i = lane; i < mm; i += 32) {
        const float x = __ldcg(w + i);
        a = fmaf(x, x, a);
      }
      a = wsum(a);
      if (lane == 0) __stcg(norms + j, fminf(a, 3.0e38f));  // (a NaN column is ordered, not lost)
    }
    if (c.rank == 0 && c.tid == 0) atomicExch(flag, 0);
    g.sync();
    for (int j = c.gw; j < nn; j += c.gnw) {
      const float nj = __ldcg(norms + j);
      int r = 0;
      for (int i = lane; i < nn; i += 32) {
        const float ni = __ldcg(norms + i);
        r += (ni > nj) || (ni == nj && i < j);
      }
      r = wsum(r);
      if (lane == 0) __stcg(perm + r, j);
    }
    g.sync();
    for (int round = 0; round < nblocks - 1; ++round) {
      int ba, bb;
      rr_pair(round, c.rank, nblocks, ba, bb);
      const int ca = ba * b, cb = bb * b;
      const int la = max(0, min(b, nn - ca)), lb = max(0, min(b, nn - cb));
      const int ga = warp < la ? __ldcg(perm + ca + warp) : -1, gb = warp < lb ? __ldcg(perm + cb + warp) : -1;
      int worst = 0;
      Column<2 * H> x;
      float al = 0.f;
      bool held = false;
      if (round == 0 && b > 1) {
        // pairs inside each block, circle method: both blocks at once when they fit, else one after the other
        for (int which = two ? 1 : 0; which < 2; ++which) {
          const int gc = two ? ga : which ? gb : ga;
          if (gc >= 0) {
            pull(x, gc);
            store_column<32>(x, (two ? sA : sB) + warp * Lp, lane);
            if (lane == 0) (two ? nA : nB)[warp] = __ldcg(norms + gc);
          }
          if (two && gb >= 0) {
            pull(x, gb);
            store_column<32>(x, sB + warp * Lp, lane);
            if (lane == 0) nB[warp] = __ldcg(norms + gb);
          }
          __syncthreads();
          worst = max(worst, inner_steps<32, H, 2 * H>(two ? sA : nullptr, nA, la, sB, nB, two || which ? lb : la, Lp, b, tol,
                                                warp, lane));
          if (!two && gc >= 0) {  // each warp reads its own column back below
            load_column<32>(x, sB + warp * Lp, lane);
            push(x, gc);
            if (lane == 0) __stcg(norms + gc, nB[warp]);
            __syncwarp();
          }
          if (!two) __syncthreads();
        }
        held = two;
      }
      if (gb >= 0 && !held) {
        pull(x, gb);
        store_column<32>(x, sB + warp * Lp, lane);
        if (lane == 0) nB[warp] = __ldcg(norms + gb);
      }
      if (ga >= 0) {
        if (held) {
          load_column<32>(x, sA + warp * Lp, lane);
          al = nA[warp];
        } else {
          pull(x, ga);
          al = __ldcg(norms + ga);
        }
      }
      __syncthreads();
      if (warp < b) worst = max(worst, cross_steps<32, H>(x, al, sB, nB, Lp, b, la, lb, tol, warp, lane));
      if (ga >= 0) {
        push(x, ga);
        if (lane == 0) __stcg(norms + ga, al);
      }
      __syncthreads();
      if (gb >= 0) {
        load_column<32>(x, sB + warp * Lp, lane);
        push(x, gb);
        if (lane == 0) __stcg(norms + gb, nB[warp]);
      }
      if (worst == 2 && lane == 0) atomicExch(flag, 1);
      g.sync();
    }
    ++sweeps;
    const int any = atomicAdd(flag, 0);
    g.sync();  // every CTA has read the flag before the next sweep resets it
    if (!any) break;
  }
  return sweeps;
}

// Sign rule shared with the CPU oracle: s = sign(r . u) with the fixed
// generic vector r_i = frac((i+1) * 0.7548776662466927) + 0.25; if r.u is
// negligible against sum_i r_i |u_i| (u nearly orthogonal to r), the sign
// of the first largest-magnitude entry is used instead.
template <bool G>
__device__ double sign_of(const double* u, int64_t len, double scale, int lane) {
  double dot = 0, mag = 0, best = -1, bval = 0;
  long long bidx = 0;
  for (int64_t i = lane; i < len; i += 32) {
    const double x = ld<double, G>(u + i) * scale;
    const double y = double(i + 1) * 0.7548776662466927;
    const double r = (y - floor(y)) + 0.25;
    dot = fma(r, x, dot);
    mag = fma(r, fabs(x), mag);
    if (fabs(x) > best) { best = fabs(x); bval = x; bidx = i; }
  }
  dot = wsum(dot);
  mag = wsum(mag);
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const double ov = __shfl_xor_sync(0xffffffffu, bval, o);
    const long long oi = __shfl_xor_sync(0xffffffffu, bidx, o);
    if (ob > best || (ob == best && oi < bidx)) { best = ob; bval = ov; bidx = oi; }
  }
  if (fabs(dot) > 1.0e-8 * mag) return dot < 0 ? -1.0 : 1.0;
  return bval < 0 ? -1.0 : 1.0;
}

// whether value a comes before b in descending order (NaN last, ties by position)
__device__ __forceinline__ int ranks_above(double a, double b, bool first) {
  const double x = a == a ? a : -1.0, y = b == b ? b : -1.0;
  return x > y || (x == y && first);
}

// Last phase of the wider blocks: sigma_j = |w_j| sorted descending (ties by column), u_j = w_j / sigma_j,
// v_j = V[:, j] (roles swapped when op(A) = A^T), every pair sign-normalised; `sval` is scratch (nn).
template <class Group>
__device__ void finish_svd(Group& cl, const Ctx& c, const xgb_svd_desc& d, bool tr, int64_t mm, int nn,
                           const double* W64, const double* V, double* sval, double* __restrict__ U,
                           double* __restrict__ S, double* __restrict__ Vt) {
  for (int j = c.gw; j < nn; j += c.gnw) {
    const double* w = W64 + int64_t(j) * mm;
    double a = 0;
    for (int64_t i = c.lane; i < mm; i += 32) { const double x = ldg(w + i); a = fma(x, x, a); }
    a = wsum(a);
    if (c.lane == 0) stg(sval + j, sqrt(a));
  }
  cl.sync();
  const int64_t k = nn;
  for (int j = c.gw; j < nn; j += c.gnw) {
    const double sj = ldg(sval + j);
    int r = 0;
    for (int i = c.lane; i < nn; i += 32) {
      r += ranks_above(ldg(sval + i), sj, i < j);
    }
    r = wsum(r);
    const double inv = sj > 0 ? 1.0 / sj : 0.0;
    const double* ucol = tr ? V + int64_t(j) * nn : W64 + int64_t(j) * mm;
    const double uscale = tr ? 1.0 : inv;
    const int64_t ulen = tr ? nn : mm;
    const double sg = sign_of<true>(ucol, ulen, uscale, c.lane);
    for (int64_t i = c.lane; i < ulen; i += 32) U[d.u_off + i + int64_t(r) * d.m] = sg * uscale * ldg(ucol + i);
    const double* vcol = tr ? W64 + int64_t(j) * mm : V + int64_t(j) * nn;
    const double vscale = tr ? inv : 1.0;
    const int64_t vlen = tr ? mm : nn;
    for (int64_t cc = c.lane; cc < vlen; cc += 32) Vt[d.vt_off + r + cc * k] = sg * vscale * ldg(vcol + cc);
    if (c.lane == 0) S[d.s_off + r] = sj;
  }
}

// ---------------------------------------------------------------- state of one block
// Workspace of a block wider than kSmallN (doubles): W0 mm*nn | V0 nn*nn | G nn*nn | E nn*nn | n64 nn | misc 10 | the
// FP32 columns W32 (mm*nn floats) of a pass 0 that no cluster holds, from a 32-byte sector on (columns across sectors:
// 3000 x 400 graded 761 ms instead of 511); their rotations V32 lie in E.  Later W32 is room for partial Gram sums.
// The second W / V pair of the refinement is the block's own U / V^T output, written only once A has been read for
// the last time (W = op(A) V): an output may overlap its block of A.
struct Block {
  int64_t mm, lda;
  int nn;
  bool tr;
  const double* A;
  double *W0, *V0, *G, *E, *n64, *W1, *V1;
  float* W32;
  int* misc;  // 0: Jacobi flag, 2-3: largest |entry| (bits), per iteration kUnconv and kZmax (float bits), kBig
};
constexpr int kPass2 = 1;  // the iteration after whose test unresolved blocks go through FP32 sweeps again
constexpr int kUnconv = 4, kZmax = kUnconv + kIters, kBig = kZmax + kIters;
constexpr int kState = 20;
static_assert(kBig < kState, "state words of a block");

__device__ __forceinline__ Block block_of(const xgb_svd_desc& d, int64_t off, const double* A, double* U, double* Vt,
                                          double* work) {
  Block k;
  k.tr = d.m < d.n;
  k.mm = k.tr ? d.n : d.m;
  k.nn = int(k.tr ? d.m : d.n);
  k.A = A + d.a_off;
  k.lda = d.m;
  const int64_t nn2 = int64_t(k.nn) * k.nn;
  k.W0 = work + off;
  k.V0 = k.W0 + k.mm * k.nn;
  k.G = k.V0 + nn2;
  k.E = k.G + nn2;
  k.n64 = k.E + nn2;
  k.misc = reinterpret_cast<int*>(k.n64 + k.nn);
  // (one column takes no sweeps, and its workspace has no room to spare)
  const uintptr_t unit = k.nn > 1 ? 32 : 8;
  k.W32 = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(k.misc + kState) + unit - 1) / unit * unit);
  k.W1 = k.tr ? Vt + d.vt_off : U + d.u_off;
  k.V1 = k.tr ? U + d.u_off : Vt + d.vt_off;
  return k;
}

// Whether refinement iteration `it` changes the block: the first one always, a later one if the one before
// it did and either pairs missed the tolerance or that update was too large for its square to vanish.
__device__ __forceinline__ bool iter_on(const int* misc, int it) {
  for (int i = 1; i <= it; ++i)
    if (!(__ldcg(misc + kUnconv + i) > 0 || __int_as_float(__ldcg(misc + kZmax + i - 1)) > 1.0e-8f)) return false;
  return true;
}
__device__ __forceinline__ int iters_done(const int* misc, int upto) {
  int n = 0;
  while (n < upto && iter_on(misc, n)) ++n;
  return n;
}

// Largest |z| taken as a small rotation, per iteration: the square of what is accepted has to vanish in the
// iterations that remain, since the last ones must leave V orthogonal to FP64 rounding.
__device__ __forceinline__ float z_limit(int it) {
  return it <= 2 ? 1.0e-2f : it == 3 ? 1.0e-3f : it == 4 ? 1.0e-5f : 3.0e-8f;
}
// V32 is off by ~1e-6, so W's columns carry that fraction of the largest one, and before the first update
// removes it the products of two small columns mean nothing: pairs whose squared norms differ by less than
// this fraction of the largest wait for the second iteration.
__device__ __forceinline__ double z_gap(int it, double gmax) { return it == 0 ? 1.0e-9 * gmax : 0.0; }

// The power of two by which the Gram entries enter z_pair: their products with one another stay in range for blocks
// down to 1e-140 and up to 1e150 (unscaled ones left it at 1e77).
__device__ __forceinline__ double z_scale(double gmax) { return pow2(-min(exponent_of(gmax), 1000)); }

// First-order update of the pair (p, q), and whether it misses the tolerance (1) or is unresolved (2: far
// from orthogonal and not a small rotation).
__device__ __forceinline__ int z_pair(double g, double gp, double gq, double e, double floor, float lim, double gap,
                                      double& zpq, double& zqp) {
  int state = 0;
  const bool live = gp > floor && gq > floor;
  const double gg = g * g, pq = gp * gq;
  if (live && !(gg <= kTol64 * kTol64 * pq)) state = 1;
  // nothing to rotate: the orthogonality part alone leaves (w_p.w_q) = -num + e (gp - gq) / 2 far below the
  // tolerance (equal singular values, whose z would be a quotient of rounding errors)
  const double num = gq * e - g, part = e * (gp - gq), few = 0.001 * kTol64 * kTol64 * pq;
  const bool still = num * num <= few && part * part <= few;
  const double z = num / (gp - gq);
  zpq = z;
  zqp = -e - z;
  const bool small = fabsf(float(z)) <= lim && fabs(gp - gq) >= gap;
  if (still || !small) {
    zpq = zqp = -0.5 * e;
    if (!still && state && gg > 1.0e-8 * pq) state = 2;
  }
  return state;
}

enum { kFormCluster, kFormGrid };
// clusters up to this size share a launch; blocks that need more CTAs have their own (a cluster of 16 waits
// for 16 free SMs of one GPC, also where its block takes two of them)
constexpr int kNarrow = 4, kMostCtas = 16;
template <int N>
struct Int {
  static constexpr int value = N;
};

// FP32 sweeps on op(A) (pass 0: V0 = V32) or on the current W (pass 1, blocks that iteration kPass2 found
// unresolved: E = V32, the factor that updates W and V).
template <int kForm, class Group>
__device__ void fp32_pass(Group& g, const Ctx& c, int P, const Block& k, int pass, float* sm, int smem_bytes, int* st6) {
  const long long t0 = clock64();
  unsigned long long* amax = reinterpret_cast<unsigned long long*>(k.misc + 2);
  const int64_t mm = k.mm;
  const int nn = k.nn;
  auto opA = [&](int64_t i, int64_t j) { return k.tr ? k.A[j + i * k.lda] : k.A[i + j * k.lda]; };
  // pass 1 comes after one update: W and V lie in W1 and V1, W0 and V0 are free
  static_assert(kPass2 == 1, "W and V after one update");
  const double* src = k.W1;
  float* W32 = pass ? reinterpret_cast<float*>(k.W0) : k.W32;
  float* V32 = reinterpret_cast<float*>(pass ? k.V0 : k.E);
  int* perm = reinterpret_cast<int*>(k.G);
  float* n32 = reinterpret_cast<float*>(k.G) + nn;
  if (pass == 0) {
    if (c.rank == 0 && c.tid < kState) k.misc[c.tid] = 0;
    g.sync();
    // power-of-two scale: the FP32 squares stay inside the FP32 range
    unsigned long long m = 0;
    for (int64_t e = c.gtid; e < mm * nn; e += c.gnt) {  // op(A) and A hold the same entries
      const unsigned long long b = (unsigned long long)__double_as_longlong(fabs(k.A[e]));
      m = b > m ? b : m;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long x = __shfl_xor_sync(0xffffffffu, m, o);
      m = x > m ? x : m;
    }
    if (c.lane == 0 && m) atomicMax(amax, m);
    g.sync();
  }
  const double amaxv = __longlong_as_double((long long)atomicAdd(amax, 0ull));
  const double scale = amaxv > 0.0 ? pow2(-exponent_of(amaxv)) : 1.0;
  double* out = pass ? k.E : k.V0;
  int sw = 0;
  bool held = false;
  const float tol = tol32(mm);
  if constexpr (kForm == kFormCluster) {
    const Shape32 sh = shape32(pass, mm, nn, P, smem_bytes);
    held = sh.P == P;
    if (held) {
      auto init = [&](int j, int i) { return float((pass ? ldg(src + int64_t(j) * mm + i) : opA(i, j)) * scale); };
      auto put = [&](int j, int i, float v) { stg(out + int64_t(j) * nn + i, double(v)); };
      auto go = [&](auto lp, auto nu, auto acc) {
        constexpr int LP = decltype(lp)::value, NU = decltype(nu)::value;
        return jacobi32_cluster<LP, NU, (decltype(acc)::value ? 2 : 1) * NU>(g, c, sh, int(mm), nn, tol, kMaxSweeps32, sm,
                                                                            init, put);
      };
      switch (pass * 10000 + sh.lp * 100 + sh.nu) {
        case 802: sw = go(Int<8>(), Int<2>(), Int<0>()); break;
        case 804: sw = go(Int<8>(), Int<4>(), Int<0>()); break;
        case 806: sw = go(Int<8>(), Int<6>(), Int<0>()); break;
        case 808: sw = go(Int<8>(), Int<8>(), Int<0>()); break;
        case 810: sw = go(Int<8>(), Int<10>(), Int<0>()); break;
        case 1606: sw = go(Int<16>(), Int<6>(), Int<0>()); break;
        case 1608: sw = go(Int<16>(), Int<8>(), Int<0>()); break;
        case 1610: sw = go(Int<16>(), Int<10>(), Int<0>()); break;
        case 1612: sw = go(Int<16>(), Int<12>(), Int<0>()); break;
        case 1614: sw = go(Int<16>(), Int<14>(), Int<0>()); break;
        case 1616: sw = go(Int<16>(), Int<16>(), Int<0>()); break;
        case 1618: sw = go(Int<16>(), Int<18>(), Int<0>()); break;
        case 1620: sw = go(Int<16>(), Int<20>(), Int<0>()); break;
        case 11602: sw = go(Int<16>(), Int<2>(), Int<1>()); break;
        case 11604: sw = go(Int<16>(), Int<4>(), Int<1>()); break;
        case 11606: sw = go(Int<16>(), Int<6>(), Int<1>()); break;
        case 11608: sw = go(Int<16>(), Int<8>(), Int<1>()); break;
        case 11610: sw = go(Int<16>(), Int<10>(), Int<1>()); break;
        default: sw = go(Int<16>(), Int<12>(), Int<1>()); break;
      }
    }
  }
  if (!held) {
    for (int j = c.gw; j < nn; j += c.gnw) {
      for (int64_t i = c.lane; i < mm; i += 32)
        __stcg(W32 + int64_t(j) * mm + i, float((pass ? ldg(src + int64_t(j) * mm + i) : opA(i, j)) * scale));
      for (int i = c.lane; i < nn; i += 32) __stcg(V32 + int64_t(j) * nn + i, i == j ? 1.f : 0.f);
    }
    g.sync();
    const int b = (nn + 2 * P - 1) / (2 * P);
    auto fits = [&](int h) { return mm <= 64 * h && b <= kWarps && global32_bytes(nn, P, h) <= smem_bytes; };
    if (nn == 1) sw = 0;
    else if (kForm == kFormGrid && fits(10))
      sw = jacobi32_global<10>(g, c, P, W32, V32, n32, perm, k.misc, int(mm), nn, tol, kMaxSweeps32, sm, smem_bytes);
    else if (kForm == kFormGrid && fits(20))
      sw = jacobi32_global<20>(g, c, P, W32, V32, n32, perm, k.misc, int(mm), nn, tol, kMaxSweeps32, sm, smem_bytes);
    else if (kForm == kFormCluster && fits(8))
      sw = jacobi32_global<8>(g, c, P, W32, V32, n32, perm, k.misc, int(mm), nn, tol, kMaxSweeps32, sm, smem_bytes);
    else  // longer columns: both blocks of a pair in shared memory, or rotated in place in L2
      sw = block_jacobi<float>(g, c, W32, V32, n32, k.misc, mm, nn, tol, 0.0f, kMaxSweeps32, sm,
                               int64_t(2 * b) * (mm + nn + 1) * 4 <= smem_bytes, 2 * P, perm);
    for (int j = c.gw; j < nn; j += c.gnw)
      for (int i = c.lane; i < nn; i += 32) stg(out + int64_t(j) * nn + i, double(__ldcg(V32 + int64_t(j) * nn + i)));
  }
  if (c.rank == 0 && c.tid == 0) {
    if (pass) k.misc[kZmax + kPass2] = __float_as_int(1.0f);  // another iteration follows
    if (st6) {
      st6[0] = pass ? st6[0] + sw : sw;
      if (!pass) st6[1] = st6[3] = st6[4] = st6[5] = 0;
      st6[2] = (pass ? st6[2] : 0) + int((clock64() - t0) >> 10);  // cycles / 1024 on CTA 0's SM
    }
  }
}

__device__ __forceinline__ Ctx make_ctx(int rank, int ctas) {
  Ctx c;
  c.tid = threadIdx.x;
  c.lane = c.tid & 31;
  c.warp = c.tid >> 5;
  c.rank = rank;
  c.gw = rank * kWarps + c.warp;
  c.gnw = ctas * kWarps;
  c.gtid = rank * kThreads + c.tid;
  c.gnt = ctas * kThreads;
  return c;
}

// whether a block is the small kernel's (host and device): its columns, twice, and four nn x nn matrices
// fit shared memory
__host__ __device__ __forceinline__ bool small_block(int64_t mm, int64_t nn) {
  return nn <= kSmallN && 8 * (2 * (mm | 1) * nn + 4 * (nn | 1) * nn) <= kSmemLimit;
}

// ---------------------------------------------------------------- small blocks: one CTA, shared memory
// The whole algorithm for a block of at most kSmallN columns (the bonds of a simple update, thin sectors):
// no cluster, no global round trip; every pair of a Jacobi round has its own warp, every entry of a
// refinement product its own thread.  Bound by latency: a Jacobi round takes ~400 cycles.  The same block
// on an 8-CTA cluster spent ~30k cycles per sweep on barriers and L2 staging: the 24 decompositions of a simple
// update at D = 6 (2 to 12 columns) took 10.5 ms there and take 0.95 ms here.
__device__ void svd_small(const xgb_svd_desc& d, const double* __restrict__ A, double* __restrict__ U,
                          double* __restrict__ S, double* __restrict__ Vt, int* st6, unsigned char* smem_raw) {
  __shared__ double red[kWarps];
  __shared__ float n32[kSmallN];
  __shared__ double n64[kSmallN];
  __shared__ int perm[kSmallN], flag, unconv, unresolved, zbits;
  const bool tr = d.m < d.n;
  const int mm = int(tr ? d.n : d.m), nn = int(tr ? d.m : d.n), ldw = mm | 1, ldv = nn | 1;
  const Ctx c = make_ctx(0, 1);
  const int tid = c.tid, lane = c.lane, warp = c.warp;
  double* Wa = reinterpret_cast<double*>(smem_raw);  // columns at stride ldw (odd: no bank conflicts along rows)
  double* Wb = Wa + ldw * nn;
  double* Va = Wb + ldw * nn;
  double* Vb = Va + ldv * nn;
  double* G = Vb + ldv * nn;
  double* E = G + ldv * nn;
  // op(A) into Wa, the power-of-two scale of the FP32 copy
  double amax = 0;
  for (int64_t e = tid; e < int64_t(mm) * nn; e += kThreads) {
    const double v = A[d.a_off + e];
    const int i = int(tr ? e / nn : e % mm), j = int(tr ? e % nn : e / mm);
    Wa[i + j * ldw] = v;
    amax = fmax(amax, fabs(v));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (lane == 0) red[warp] = amax;
  __syncthreads();
  for (int w = 0; w < kWarps; ++w) amax = fmax(amax, red[w]);
  const double scale = amax > 0.0 ? pow2(-exponent_of(amax)) : 1.0;
  const int np = nn + (nn & 1);

  // FP32 Jacobi of the columns of src (stride ldw); W32 and V32 are scratch, V32 holds the rotations afterwards
  auto sweeps = [&](const double* src, float* W32, float* V32) {
    for (int e = tid; e < mm * nn; e += kThreads) W32[e % mm + (e / mm) * ldw] = float(src[e % mm + (e / mm) * ldw] * scale);
    for (int e = tid; e < nn * nn; e += kThreads) V32[e % nn + (e / nn) * ldv] = e % nn == e / nn ? 1.f : 0.f;
    __syncthreads();
    const float tol = tol32(mm);
    int sw = 0;
    for (; sw < kMaxSweeps32 && nn > 1;) {
      for (int j = warp; j < nn; j += kWarps) {
        float a = 0;
        for (int i = lane; i < mm; i += 32) a = fmaf(W32[i + j * ldw], W32[i + j * ldw], a);
        a = wsum(a);
        if (lane == 0) n32[j] = fminf(a, 3.0e38f);  // (a NaN column is ordered, not lost)
      }
      if (tid == 0) flag = 0;
      __syncthreads();
      if (tid < nn) {
        int r = 0;
        for (int i = 0; i < nn; ++i) r += (n32[i] > n32[tid]) || (n32[i] == n32[tid] && i < tid);
        perm[r] = tid;
      }
      __syncthreads();
      int worst = 0;
      for (int r = 0; r < np - 1; ++r) {
        if (warp < np / 2) {
          int p, q;
          rr_pair(r, warp, np, p, q);
          if (p < nn && q < nn) {
            p = perm[p];
            q = perm[q];
            float *x = W32 + p * ldw, *y = W32 + q * ldw;
            const float al = n32[p], be = n32[q];
            const Pre32 pre = pre32(al, be);
            float ga = 0;
            for (int i = lane; i < mm; i += 32) ga = fmaf(x[i], y[i], ga);
            ga = wsum(ga);
            float cs, sn, t;
            const int k = plan32(ga, pre, tol, cs, sn, t);
            if (k) {
              worst = max(worst, k);
              for (int i = lane; i < mm; i += 32) {
                const float xv = x[i], yv = y[i];
                x[i] = cs * xv - sn * yv;
                y[i] = fmaf(sn, xv, cs * yv);
              }
              if (lane < nn) {
                float *vx = V32 + p * ldv, *vy = V32 + q * ldv;
                const float xv = vx[lane], yv = vy[lane];
                vx[lane] = cs * xv - sn * yv;
                vy[lane] = fmaf(sn, xv, cs * yv);
              }
              if (lane == 0) {
                n32[p] = al - t * ga;
                n32[q] = be + t * ga;
              }
            }
          }
        }
        __syncthreads();
      }
      ++sw;
      if (worst == 2) flag = 1;
      __syncthreads();
      const int any = flag;
      __syncthreads();
      if (!any) break;
    }
    return sw;
  };
  static_assert(kSmallN <= 32 && kSmallN / 2 <= kWarps, "one lane per row of V, one warp per pair");

  const long long t0 = clock64();
  int sw32 = sweeps(Wa, reinterpret_cast<float*>(Wb), reinterpret_cast<float*>(Vb));
  const long long t1 = clock64();
  for (int e = tid; e < nn * nn; e += kThreads)
    Va[e % nn + (e / nn) * ldv] = double(reinterpret_cast<float*>(Vb)[e % nn + (e / nn) * ldv]);
  __syncthreads();
  auto product = [&](const double* X, int ldx, int rows, const double* B, double* out) {  // out = X B (rows x nn)
    for (int e = tid; e < rows * nn; e += kThreads) {
      const int i = e % rows, j = e / rows;
      double a = 0;
      for (int l = 0; l < nn; ++l) a = fma(X[i + l * ldx], B[l + j * ldv], a);
      out[i + j * ldx] = a;
    }
  };
  product(Wa, ldw, mm, Va, Wb);  // the FP32 columns in Wb are no longer needed
  __syncthreads();
  double *W = Wb, *Wn = Wa, *V = Va, *Vn = Vb;
  float zprev = 1.0f;
  int it = 0;
  // Gram entries: a thread each, or, in tall blocks of few columns, a warp each.  FP64 warp instructions of an SM quarter:
  // mm for every 128 entries, or (mm / 32 + 10) for every 4 (5000 x 1: 516 us with one thread over all rows, 121 so).
  const int entries = nn * (nn + 1) / 2;
  const bool tall = mm >= 256 && 4 * ((entries + 127) / 128) * mm > entries * (mm / 32 + 10);
  auto pair_of = [](int e, int& p, int& q) {
    q = int((sqrtf(8.0f * float(e) + 1.0f) - 1.0f) * 0.5f);
    while ((q + 1) * (q + 2) / 2 <= e) ++q;
    while (q * (q + 1) / 2 > e) --q;
    p = e - q * (q + 1) / 2;
  };
  for (; it < kIters; ++it) {
    for (int e = tid; e < entries; e += kThreads) {
      int p, q;
      pair_of(e, p, q);
      double g = 0, v = 0;
      if (!tall)
        for (int i = 0; i < mm; ++i) g = fma(W[i + p * ldw], W[i + q * ldw], g);
      for (int i = 0; i < nn; ++i) v = fma(V[i + p * ldv], V[i + q * ldv], v);
      if (!tall) G[p + q * ldv] = g;
      E[p + q * ldv] = v;
    }
    for (int e = warp; tall && e < entries; e += kWarps) {
      int p, q;
      pair_of(e, p, q);
      double g = 0;
      for (int i = lane; i < mm; i += 32) g = fma(W[i + p * ldw], W[i + q * ldw], g);
      g = wsum(g);
      if (lane == 0) G[p + q * ldv] = g;
    }
    if (tid == 0) unconv = unresolved = zbits = 0;
    __syncthreads();
    double gmax = 0;
    for (int j = 0; j < nn; ++j) gmax = fmax(gmax, G[j * (ldv + 1)]);
    const double sc = z_scale(gmax), floor = kFloor64 * (sc * gmax);
    const float lim = z_limit(it);
    const double gap = z_gap(it, sc * gmax);
    float zmax = 0.f;
    for (int e = tid; e < nn * nn; e += kThreads) {
      const int p = e % nn, q = e / nn;
      if (p > q) continue;
      if (p == q) {
        const double z = -0.5 * (E[p * (ldv + 1)] - 1.0);
        E[p * (ldv + 1)] = 1.0 + z;
        zmax = fmaxf(zmax, fabsf(float(z)));
        continue;
      }
      double zpq, zqp;
      const int s = z_pair(sc * G[p + q * ldv], sc * G[p * (ldv + 1)], sc * G[q * (ldv + 1)], E[p + q * ldv], floor, lim,
                           gap, zpq, zqp);
      if (s) atomicAdd(&unconv, 1);
      if (s == 2) atomicAdd(&unresolved, 1);
      E[p + q * ldv] = zpq;
      E[q + p * ldv] = zqp;
      zmax = fmaxf(zmax, fmaxf(fabsf(float(zpq)), fabsf(float(zqp))));
    }
    if (zmax > 0.f) atomicMax(&zbits, __float_as_int(zmax));
    __syncthreads();
    const float z = __int_as_float(zbits);
    const bool on = it == 0 || unconv > 0 || zprev > 1.0e-8f;
    const bool again = it == kPass2 && unresolved > 0;
    __syncthreads();  // everyone has read the state
    if (!on) break;
    zprev = z;
    if (again) {
      // columns that FP32 could not resolve: FP32 sweeps on W, whose rotations become the update
      sw32 += sweeps(W, reinterpret_cast<float*>(Wn), reinterpret_cast<float*>(Vn));
      for (int e = tid; e < nn * nn; e += kThreads)
        E[e % nn + (e / nn) * ldv] = double(reinterpret_cast<float*>(Vn)[e % nn + (e / nn) * ldv]);
      zprev = 1.0f;
      __syncthreads();
    }
    product(W, ldw, mm, E, Wn);
    product(V, ldv, nn, E, Vn);
    __syncthreads();
    double* x = W; W = Wn; Wn = x;
    x = V; V = Vn; Vn = x;
  }
  int sw64 = 0;
  if (it == kIters) {  // pairs that the refinement left: FP64 Jacobi
    for (; sw64 < kMaxSweeps64 && nn > 1;) {
      for (int j = warp; j < nn; j += kWarps) {
        double a = 0;
        for (int i = lane; i < mm; i += 32) a = fma(W[i + j * ldw], W[i + j * ldw], a);
        a = wsum(a);
        if (lane == 0) n64[j] = fmin(a, 1.0e308);
      }
      if (tid == 0) flag = 0;
      __syncthreads();
      double gmax = 0;
      for (int j = 0; j < nn; ++j) gmax = fmax(gmax, n64[j]);
      if (tid < nn) {
        int r = 0;
        for (int i = 0; i < nn; ++i) r += (n64[i] > n64[tid]) || (n64[i] == n64[tid] && i < tid);
        perm[r] = tid;
      }
      __syncthreads();
      bool any = false;
      for (int r = 0; r < np - 1; ++r) {
        if (warp < np / 2) {
          int p, q;
          rr_pair(r, warp, np, p, q);
          if (p < nn && q < nn) {
            p = perm[p];
            q = perm[q];
            any |= rotate<double, false>(W + p * ldw, W + q * ldw, V + p * ldv, V + q * ldv, n64 + p, n64 + q, mm, nn,
                                         kTol64, kFloor64 * gmax, lane);
          }
        }
        __syncthreads();
      }
      ++sw64;
      if (any) flag = 1;
      __syncthreads();
      const int again = flag;
      __syncthreads();
      if (!again) break;
    }
  }
  const long long t3 = clock64();
  // sort, sign, write
  for (int j = warp; j < nn; j += kWarps) {
    double a = 0;
    for (int i = lane; i < mm; i += 32) a = fma(W[i + j * ldw], W[i + j * ldw], a);
    a = wsum(a);
    if (lane == 0) n64[j] = sqrt(a);
  }
  __syncthreads();
  for (int j = warp; j < nn; j += kWarps) {
    const double sj = n64[j];
    int r = 0;
    for (int i = lane; i < nn; i += 32) r += ranks_above(n64[i], sj, i < j);
    r = wsum(r);
    const double inv = sj > 0 ? 1.0 / sj : 0.0;
    const double* ucol = tr ? V + j * ldv : W + j * ldw;
    const double us = tr ? 1.0 : inv, vs = tr ? inv : 1.0;
    const int ulen = tr ? nn : mm, vlen = tr ? mm : nn;
    const double sg = sign_of<false>(ucol, ulen, us, lane);
    for (int i = lane; i < ulen; i += 32) U[d.u_off + i + int64_t(r) * d.m] = sg * us * ucol[i];
    const double* vcol = tr ? W + j * ldw : V + j * ldv;
    for (int i = lane; i < vlen; i += 32) Vt[d.vt_off + r + int64_t(i) * nn] = sg * vs * vcol[i];
    if (lane == 0) S[d.s_off + r] = sj;
  }
  if (st6 && tid == 0) {
    st6[0] = sw32;
    st6[1] = sw64;
    st6[2] = int((t1 - t0) >> 10);
    st6[3] = it;
    st6[4] = int((t3 - t1) >> 10);
    st6[5] = int((clock64() - t3) >> 10);
  }
}

// a batch's small blocks, one CTA each
__global__ void __launch_bounds__(kThreads)
    svd_small_kernel(const xgb_svd_desc* __restrict__ descs, const double* __restrict__ A, double* __restrict__ U,
                     double* __restrict__ S, double* __restrict__ Vt, int* __restrict__ sweep_stats) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const xgb_svd_desc d = descs[blockIdx.x];
  const int64_t mm = max(d.m, d.n), nn = min(d.m, d.n);
  if (nn == 0 || !small_block(mm, nn)) return;
  svd_small(d, A, U, S, Vt, sweep_stats ? sweep_stats + 6 * blockIdx.x : nullptr, smem_raw);
}

// CTAs of a block's FP32 sweeps on a cluster of at most `most`
__host__ __device__ __forceinline__ int sweep_ctas(int pass, int64_t mm, int64_t nn, int most) {
  const Shape32 sh = shape32(pass, mm, nn, most, kSmemLimit);
  if (sh.P) return sh.P;
  // too large for any: jacobi32_global or block_jacobi on all of them, but no more than give each of their 2P column
  // blocks a column (with 16 CTAs eight columns met in 31 rounds of one pair instead of seven of four: 1000000 x 8
  // 780 ms instead of 322), unless two single columns fit shared memory where two blocks do not (20000 x 30 graded 41
  // ms on 16 CTAs, 92 on 8)
  auto staged = [&](int P) { return 8 * ((nn + 2 * P - 1) / (2 * P)) * (mm + nn + 1) <= kSmemLimit; };
  int P = 1;
  while (2 * P <= most && 4 * P <= nn) P *= 2;
  if (staged(most))
    while (!staged(P)) P *= 2;
  return P;
}

// Whether a block takes svd_factor_kernel; `grid_most`: most CTAs per cluster, 0 where no cooperative grid is launched.
__host__ __device__ __forceinline__ bool factored(int64_t mm, int64_t nn, int grid_most) {
  return grid_most && nn >= kFactorN && shape32(0, mm, nn, grid_most, kSmemLimit).P == 0;
}

// FP32 sweeps of the blocks that take lo < CTAs <= hi, one cluster of `hi` CTAs per block; the CTAs that a
// block does not take leave at once (a cluster barrier waits for the threads that have not exited).  The launch
// with lo = 0 also decomposes the small blocks, start to finish, beside the others' sweeps.  `widest`: blocks of
// more columns take the cooperative grid (pass 1).
__global__ void __launch_bounds__(kThreads)
    svd_sweeps_kernel(const xgb_svd_desc* __restrict__ descs, const int64_t* __restrict__ work_off,
                      const double* __restrict__ A, double* __restrict__ U, double* __restrict__ S,
                      double* __restrict__ Vt, double* __restrict__ work, int* __restrict__ sweep_stats, int pass, int lo,
                      int most, int widest, int grid_most, int smem_bytes) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cg::cluster_group cl = cg::this_cluster();
  const int ctas = int(cl.num_blocks()), sector = int(blockIdx.x) / ctas;
  const Block k = block_of(descs[sector], work_off[sector], A, U, Vt, work);
  if (k.nn == 0 || k.nn > widest || factored(k.mm, k.nn, grid_most)) return;  // uniform across the cluster
  int* st6 = sweep_stats ? sweep_stats + 6 * sector : nullptr;
  if (small_block(k.mm, k.nn)) {
    if (pass == 0 && lo == 0 && cl.block_rank() == 0) svd_small(descs[sector], A, U, S, Vt, st6, smem_raw);
    return;
  }
  const int P = sweep_ctas(pass, k.mm, k.nn, most);
  if (P <= lo || P > ctas || int(cl.block_rank()) >= P) return;
  if (pass && __ldcg(k.misc + kBig) == 0) return;
  const Ctx c = make_ctx(int(cl.block_rank()), P);
  fp32_pass<kFormCluster>(cl, c, P, k, pass, reinterpret_cast<float*>(smem_raw), smem_bytes, st6);
}

// Pass 1 of one block wider than kGridN: a cooperative grid of nn / 32 CTAs with grid barriers.
__global__ void __launch_bounds__(kThreads)
    svd_sweeps_grid_kernel(const xgb_svd_desc* __restrict__ descs, const int64_t* __restrict__ work_off, int sector,
                           const double* __restrict__ A, double* __restrict__ U, double* __restrict__ Vt,
                           double* __restrict__ work, int* __restrict__ sweep_stats, int smem_bytes) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cg::grid_group gg = cg::this_grid();
  const Block k = block_of(descs[sector], work_off[sector], A, U, Vt, work);
  if (__ldcg(k.misc + kBig) == 0) return;  // uniform across the grid
  const Ctx c = make_ctx(int(blockIdx.x), int(gridDim.x));
  fp32_pass<kFormGrid>(gg, c, int(gridDim.x), k, 1, reinterpret_cast<float*>(smem_raw), smem_bytes,
                  sweep_stats ? sweep_stats + 6 * sector : nullptr);
}

// ---------------------------------------------------------------- FP64 products of the refinement
// One kTile x kTile tile of C (M x N) = op(A) (M x K) B (K x N), column-major, 256 threads with one output
// each; two shared-memory stages, the next k step's operands in flight in registers.  Bound by the FP64 pipe
// (128 cycles of it per k value, under which the shared-memory reads hide), so the smallest tile is the best
// one: it wastes least at a block's edges and spreads the work most evenly over the SMs (tiles of 32 took
// 0.71 ms for op(A) V of blocks up to 600 x 560, half the pipe's rate; tiles of 16 take 0.41 ms).
constexpr int kTile = 16;
__device__ __forceinline__ void tile_product(const double* __restrict__ A, int64_t lda, bool ta,
                                             const double* __restrict__ B, int64_t ldb, double* __restrict__ C,
                                             int64_t ldc, int64_t M, int64_t N, int64_t K, int64_t tm, int64_t tn,
                                             double* sm) {
  constexpr int BK = 16, LD = kTile + 1;
  double* As = sm;                // [2][BK][LD]
  double* Bs = sm + 2 * BK * LD;  // [2][BK][LD]
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int64_t row0 = tm * kTile, col0 = tn * kTile;
  const int i = ta ? ty : tx, kk = ta ? tx : ty;  // this thread's staged entry of op(A); of B: (k tx, column ty)
  const int64_t gi = row0 + i, gj = col0 + ty;
  double acc = 0.0, ra, rb;
  auto fetch = [&](int64_t k0) {
    ra = gi < M && k0 + kk < K ? (ta ? A[k0 + kk + gi * lda] : A[gi + (k0 + kk) * lda]) : 0.0;
    rb = gj < N && k0 + tx < K ? B[k0 + tx + gj * ldb] : 0.0;
  };
  auto stash = [&](int st) {
    As[(st * BK + kk) * LD + i] = ra;
    Bs[(st * BK + tx) * LD + ty] = rb;
  };
  fetch(0);
  stash(0);
  __syncthreads();
  int st = 0;
  for (int64_t k0 = 0; k0 < K; k0 += BK) {
    const bool more = k0 + BK < K;
    if (more) fetch(k0 + BK);
    const double* a = As + st * BK * LD + tx;
    const double* b = Bs + st * BK * LD + ty;
    if (K - k0 >= BK) {
#pragma unroll
      for (int e = 0; e < BK; ++e) acc = fma(a[e * LD], b[e * LD], acc);
    } else {
      for (int e = 0; e < int(K - k0); ++e) acc = fma(a[e * LD], b[e * LD], acc);
    }
    if (more) stash(st ^ 1);
    __syncthreads();
    st ^= 1;
  }
  if (row0 + tx < M && gj < N) C[row0 + tx + gj * ldc] = acc;
}

__host__ __device__ __forceinline__ int64_t svd_tiles(int64_t x) { return (x + kTile - 1) / kTile; }

// Row ranges that the tiles of W^T W are cut into: a thin block has few tiles, and one CTA over all rows of each kept the
// other SMs waiting (1000000 x 2: 255 ms, of which about 200 for three Gram products; 42 cut).  Four CTAs per SM, at least 512
// rows each, and partial sums (from W32 on, free by then) that fit mm nn / 2 doubles.  Below 4096 rows the rest of an
// iteration is as long.
__host__ __device__ __forceinline__ int64_t gram_splits(int64_t mm, int64_t nn) {
  if (mm < 4096) return 1;
  const int64_t nt = svd_tiles(nn);
  int64_t s = 608 / (nt * (nt + 1) / 2);
  if (s > mm / 512) s = mm / 512;
  if (s > mm / (2 * nn)) s = mm / (2 * nn);
  return s > 1 ? s : 1;
}

enum { kProdAV, kProdGram, kProdGramUncut, kProdCut, kProdApply };

// W = op(A) V (kProdAV), G = W^T W and E = V^T V on and above the diagonal (kProdGram), or W (I + Z) and V (I + Z)
// (kProdApply, I + Z in E): one launch over all blocks, blockIdx.y = block.  Batches with blocks whose Gram product is
// cut take kProdCut for those and kProdGramUncut for the rest of G and E: in one kernel they cost every batch 19
// registers, 1.2 % of a plain CTM step.
template <int kMode>
__global__ void __launch_bounds__(256)
    svd_product_kernel(const xgb_svd_desc* __restrict__ descs, const int64_t* __restrict__ work_off,
                       const double* __restrict__ A, double* __restrict__ U, double* __restrict__ Vt,
                       double* __restrict__ work, int it, int grid_most) {
  __shared__ double sm[4 * 16 * (kTile + 1)];
  const int sector = blockIdx.y;
  const Block k = block_of(descs[sector], work_off[sector], A, U, Vt, work);
  if (k.nn == 0 || small_block(k.mm, k.nn) || factored(k.mm, k.nn, grid_most)) return;
  const int64_t nt = svd_tiles(k.nn), mt = svd_tiles(k.mm);
  int64_t t = blockIdx.x;
  const int64_t splits = kMode == kProdCut ? gram_splits(k.mm, k.nn) : 1;
  if (kMode == kProdCut && splits == 1) return;
  constexpr bool kGram = kMode == kProdGram || kMode == kProdGramUncut;
  if (t >= (kMode == kProdAV ? mt * nt : kGram ? 2 * nt * nt : kMode == kProdCut ? splits * nt * nt : mt * nt + nt * nt))
    return;
  auto run = [&](const double* a, int64_t lda, bool ta, const double* b, int64_t ldb, double* c, int64_t ldc, int64_t M,
                 int64_t K, int64_t tm, int64_t tn) {
    tile_product(a, lda, ta, b, ldb, c, ldc, M, k.nn, K, tm, tn, sm);
  };
  if (kMode == kProdAV) {
    run(k.A, k.lda, k.tr, k.V0, k.nn, k.W0, k.mm, k.mm, k.nn, t % mt, t / mt);
    return;
  }
  if (kMode != kProdApply ? (it > 0 && !iter_on(k.misc, it - 1)) : !iter_on(k.misc, it)) return;
  const int cur = iters_done(k.misc, it) & 1;
  const double* W = cur ? k.W1 : k.W0;
  const double* V = cur ? k.V1 : k.V0;
  if (kGram) {
    const bool e = t >= nt * nt;
    if (e) t -= nt * nt;
    if (t % nt > t / nt) return;
    if (e) run(V, k.nn, true, V, k.nn, k.E, k.nn, k.nn, k.nn, t % nt, t / nt);
    else if (kMode == kProdGram || gram_splits(k.mm, k.nn) == 1)
      run(W, k.mm, true, W, k.mm, k.G, k.nn, k.nn, k.mm, t % nt, t / nt);
    return;
  }
  if (kMode == kProdCut) {
    const int64_t part = t / (nt * nt), rows = (k.mm + splits - 1) / splits, r0 = part * rows;
    t -= part * nt * nt;
    if (t % nt > t / nt) return;
    run(W + r0, k.mm, true, W + r0, k.mm, reinterpret_cast<double*>(k.W32) + part * k.nn * k.nn, k.nn, k.nn,
        k.mm - r0 < rows ? k.mm - r0 : rows, t % nt, t / nt);
    return;
  }
  if (t < mt * nt) {
    run(W, k.mm, false, k.E, k.nn, cur ? k.W0 : k.W1, k.mm, k.mm, k.nn, t % mt, t / mt);
  } else {
    t -= mt * nt;
    run(V, k.nn, false, k.E, k.nn, cur ? k.V0 : k.V1, k.nn, k.nn, k.nn, t % nt, t / nt);
  }
}

// G of the blocks whose Gram product was cut: its row ranges' sums, added in order.
__global__ void __launch_bounds__(256)
    svd_gram_sum_kernel(const xgb_svd_desc* __restrict__ descs, const int64_t* __restrict__ work_off,
                        const double* __restrict__ A, double* __restrict__ U, double* __restrict__ Vt,
                        double* __restrict__ work, int it, int grid_most) {
  const int sector = blockIdx.y;
  const Block k = block_of(descs[sector], work_off[sector], A, U, Vt, work);
  if (k.nn == 0 || small_block(k.mm, k.nn) || factored(k.mm, k.nn, grid_most)) return;
  const int64_t splits = gram_splits(k.mm, k.nn), nn2 = int64_t(k.nn) * k.nn, e = int64_t(blockIdx.x) * 256 + threadIdx.x;
  if (splits == 1 || e >= nn2 || e % k.nn > e / k.nn) return;
  if (it > 0 && !iter_on(k.misc, it - 1)) return;
  const double* part = reinterpret_cast<const double*>(k.W32) + e;
  double g = part[0];
#pragma unroll 8
  for (int64_t s = 1; s < splits; ++s) g += part[s * nn2];
  k.G[e] = g;
}

// E <- I + Z from G and E, and the block's convergence state of this iteration.
__global__ void __launch_bounds__(256)
    svd_update_kernel(const xgb_svd_desc* __restrict__ descs, const int64_t* __restrict__ work_off,
                      const double* __restrict__ A, double* __restrict__ U, double* __restrict__ Vt,
                      double* __restrict__ work, int it, int grid_most) {
  __shared__ double red[8];
  const int sector = blockIdx.y;
  const Block k = block_of(descs[sector], work_off[sector], A, U, Vt, work);
  const int64_t nn = k.nn;
  if (nn == 0 || small_block(k.mm, nn) || int64_t(blockIdx.x) * 256 >= nn * nn) return;
  if (factored(k.mm, nn, grid_most)) return;
  if (it > 0 && !iter_on(k.misc, it - 1)) return;
  double gmax = 0;
  for (int64_t j = threadIdx.x; j < nn; j += 256) gmax = fmax(gmax, k.G[j * (nn + 1)]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) gmax = fmax(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = gmax;
  __syncthreads();
  for (int w = 0; w < 8; ++w) gmax = fmax(gmax, red[w]);
  const double sc = z_scale(gmax), floor = kFloor64 * (sc * gmax);
  const float lim = z_limit(it);
  const double gap = z_gap(it, sc * gmax);
  int unconv = 0, unresolved = 0;
  float zmax = 0.f;
  for (int64_t e = int64_t(blockIdx.x) * 256 + threadIdx.x; e < nn * nn; e += int64_t(gridDim.x) * 256) {
    const int64_t p = e % nn, q = e / nn;
    if (p > q) continue;
    if (p == q) {
      const double z = -0.5 * (k.E[e] - 1.0);
      k.E[e] = 1.0 + z;
      zmax = fmaxf(zmax, fabsf(float(z)));
      continue;
    }
    double zpq, zqp;
    const int s = z_pair(sc * k.G[e], sc * k.G[p * (nn + 1)], sc * k.G[q * (nn + 1)], k.E[e], floor, lim, gap, zpq, zqp);
    unconv += s != 0;
    unresolved += s == 2;
    k.E[e] = zpq;
    k.E[q + p * nn] = zqp;
    zmax = fmaxf(zmax, fmaxf(fabsf(float(zpq)), fabsf(float(zqp))));
  }
  unconv = __reduce_add_sync(0xffffffffu, unconv);
  unresolved = __reduce_add_sync(0xffffffffu, unresolved);
  const int zb = __reduce_max_sync(0xffffffffu, __float_as_int(zmax));
  if ((threadIdx.x & 31) == 0) {
    if (unconv) atomicAdd(k.misc + kUnconv + it, unconv);
    if (it == kPass2 && unresolved) atomicAdd(k.misc + kBig, unresolved);
    atomicMax(k.misc + kZmax + it, zb);
  }
}

// FP64 sweeps for what the refinement left (nothing in the usual case), then sort, sign and write.
template <class Group>
__device__ void polish(Group& g, const Ctx& c, const Block& k, int ctas, double* sm, int smem_bytes, int* st6) {
  const int done = iters_done(k.misc, kIters);
  if (done < kIters) return;  // the last test passed
  const int cur = done & 1;
  const int b = (k.nn + 2 * ctas - 1) / (2 * ctas);
  const bool staged = int64_t(2 * b) * (k.mm + k.nn + 1) * 8 <= smem_bytes;
  const long long t0 = clock64();
  const int sw = block_jacobi<double>(g, c, cur ? k.W1 : k.W0, cur ? k.V1 : k.V0, k.n64, k.misc, k.mm, k.nn, kTol64,
                                      kFloor64, kMaxSweeps64, sm, staged, 2 * ctas, reinterpret_cast<int*>(k.G));
  if (st6 && c.rank == 0 && c.tid == 0) {
    st6[1] = sw;
    st6[4] = int((clock64() - t0) >> 10);
  }
}

// The sweeps of `polish` for one block wider than kGridN, over a cooperative grid.
__global__ void __launch_bounds__(kThreads)
    svd_polish_grid_kernel(const xgb_svd_desc* __restrict__ descs, const int64_t* __restrict__ work_off, int sector,
                           const double* __restrict__ A, double* __restrict__ U, double* __restrict__ Vt,
                           double* __restrict__ work, int* __restrict__ sweep_stats, int smem_bytes) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cg::grid_group gg = cg::this_grid();
  const Block k = block_of(descs[sector], work_off[sector], A, U, Vt, work);
  const Ctx c = make_ctx(int(blockIdx.x), int(gridDim.x));
  polish(gg, c, k, int(gridDim.x), reinterpret_cast<double*>(smem_raw), smem_bytes,
         sweep_stats ? sweep_stats + 6 * sector : nullptr);
}

// `grid_min`: blocks at least this wide had their polish on the cooperative grid.
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kThreads)
    svd_finish_kernel(const xgb_svd_desc* __restrict__ descs, const int64_t* __restrict__ work_off,
                      const double* __restrict__ A, double* __restrict__ U, double* __restrict__ S,
                      double* __restrict__ Vt, double* __restrict__ work, int* __restrict__ sweep_stats,
                      int smem_bytes, int grid_min, int grid_most) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cg::cluster_group cl = cg::this_cluster();
  const int sector = blockIdx.x / kCluster;
  const xgb_svd_desc d = descs[sector];
  const Block k = block_of(d, work_off[sector], A, U, Vt, work);
  if (k.nn == 0 || small_block(k.mm, k.nn) || factored(k.mm, k.nn, grid_most)) return;  // uniform across the cluster
  const Ctx c = make_ctx(int(cl.block_rank()), kCluster);
  const long long t0 = clock64();
  int* st6 = sweep_stats ? sweep_stats + 6 * sector : nullptr;
  if (k.nn < grid_min) polish(cl, c, k, kCluster, reinterpret_cast<double*>(smem_raw), smem_bytes, st6);
  const int done = iters_done(k.misc, kIters);
  if (done & 1) {  // the current W and V lie in the outputs that finish_svd writes
    for (int64_t e = c.gtid; e < k.mm * k.nn; e += c.gnt) stg(k.W0 + e, ldg(k.W1 + e));
    for (int64_t e = c.gtid; e < int64_t(k.nn) * k.nn; e += c.gnt) stg(k.V0 + e, ldg(k.V1 + e));
    cl.sync();
  }
  finish_svd(cl, c, d, k.tr, k.mm, k.nn, k.W0, k.V0, k.n64, U, S, Vt);
  if (st6 && c.rank == 0 && c.tid == 0) {
    st6[3] = done;
    st6[5] = int((clock64() - t0) >> 10);
  }
}

// ---------------------------------------------------------------- wide blocks: QR, then Jacobi on R^T
// Blocks from kFactorN columns on that no cluster's shared memory holds (beyond 640 columns, or tall): FP64 throughout
// on a cooperative grid of one CTA per 2 kFactorCols columns (every SM at most), one launch per block.
//   1. Householder QR with column pivoting, op(A) P = Q R (Businger-Golub: the largest remaining column
//      norm is pivoted in; the norms are downdated and recomputed under cancellation, the rule of
//      LAPACK's xLAQP2).  Per step CTA 0 picks the pivot, swaps it into place and forms the reflector,
//      and then every warp applies it to one trailing column.
//   2. Block Jacobi on X = R^T (nn x nn): the rows of a column-pivoted R are graded, so the columns of X are close
//      to orthogonal and converge in 11 to 14 sweeps (the preconditioning of Drmac and Veselic).
//   3. X V = W with W_j = sigma_j u_j gives R = V Sigma U_X^T, so op(A) = (Q V) Sigma (P U_X)^T: each
//      warp applies the reflectors to one column [V_j; 0] (no barriers), and P U_X is a row scatter.
// Bound by the latency of the factor's column steps (two grid barriers each: 50k of 340k kilocycles at 864 columns) and
// of the sweeps' grid barriers and FP64 dot products.  Measured against FP32 sweeps of op(A) itself with accumulated
// rotations through L2 and FP64 refinement, which graded spectra (1e-12) take 50 sweeps in (ms):
//   864 x 864   graded 163, 444   power law 180, 186   Gaussian 167, 124   degenerate pairs 155, 526
//   1176 x 1176 graded 294, 688   power law 326, 296;   1400 x 520 graded 78, 577;   3000 x 540 graded 104, 1111
// Projector spectra are graded, and the refinement's bits are no better, so one form for all of them.  Narrower blocks
// too tall for a cluster stay on the sweeps (3000 x 400 graded 511, without either 1459).
constexpr double kQrRecompute = 1.4901161193847656e-08;  // sqrt(eps): norm downdates below this are recomputed

// sum over the 512 threads of a CTA, the same bits in every thread; red: kWarps doubles of shared memory
__device__ double block_sum(double v, double* red, const Ctx& c) {
  v = wsum(v);
  __syncthreads();  // red is free (an earlier call's readers are done)
  if (c.lane == 0) red[c.warp] = v;
  __syncthreads();
  double t = 0;
  for (int w = 0; w < kWarps; ++w) t += red[w];
  return t;
}

// Householder QR with column pivoting of H (mm x nn column-major, mm >= nn) in place: R on and above
// the diagonal, the reflectors v_k = (1, H[k+1:, k]) below it, H_k = I - tau_k v_k v_k^T; piv[k] = the
// column of the input at position k.  vn1 / vn2: partial column norms and their last exact values.
template <class Group>
__device__ void qr_pivoted(Group& gg, const Ctx& c, double* H, int64_t mm, int nn, double* tau, int* piv,
                           double* vn1, double* vn2, double* red, int* redi) {
  const unsigned full = 0xffffffffu;
  for (int j = c.gw; j < nn; j += c.gnw) {
    const double* h = H + int64_t(j) * mm;
    double a = 0;
    for (int64_t i = c.lane; i < mm; i += 32) {
      const double x = ldg(h + i);
      a = fma(x, x, a);
    }
    a = sqrt(wsum(a));
    if (c.lane == 0) {
      stg(vn1 + j, a);
      stg(vn2 + j, a);
      __stcg(piv + j, j);
    }
  }
  gg.sync();
  for (int k = 0; k < nn; ++k) {
    if (c.rank == 0) {
      // pivot: the largest remaining norm (the first such column on ties)
      double best = -1.0;
      int bi = k;
      for (int j = k + c.tid; j < nn; j += kThreads) {
        const double v = ldg(vn1 + j);
        if (v > best) {
          best = v;
          bi = j;
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(full, best, o);
        const int oi = __shfl_xor_sync(full, bi, o);
        if (ob > best || (ob == best && oi < bi)) {
          best = ob;
          bi = oi;
        }
      }
      __syncthreads();
      if (c.lane == 0) {
        red[c.warp] = best;
        redi[c.warp] = bi;
      }
      __syncthreads();
      best = red[0];
      bi = redi[0];
      for (int w = 1; w < kWarps; ++w)
        if (red[w] > best || (red[w] == best && redi[w] < bi)) {
          best = red[w];
          bi = redi[w];
        }
      const int p = bi;
      double* hk = H + int64_t(k) * mm;
      double* hp = H + int64_t(p) * mm;
      // swap columns k and p (every row: rows above k hold R's earlier entries), with the sum of squares of
      // the new column k below row k
      double ss = 0;
      for (int64_t i = c.tid; i < mm; i += kThreads) {
        const double x = ldg(hp + i);
        if (p != k) {
          stg(hp + i, ldg(hk + i));
          stg(hk + i, x);
        }
        if (i > k) ss = fma(x, x, ss);
      }
      ss = block_sum(ss, red, c);  // its barriers also order the swap before the reads below
      if (c.tid == 0 && p != k) {
        const double a1 = ldg(vn1 + k), a2 = ldg(vn2 + k);
        stg(vn1 + k, ldg(vn1 + p));
        stg(vn2 + k, ldg(vn2 + p));
        stg(vn1 + p, a1);
        stg(vn2 + p, a2);
        const int q = __ldcg(piv + k);
        __stcg(piv + k, __ldcg(piv + p));
        __stcg(piv + p, q);
      }
      // reflector: beta = -sign(alpha) |(alpha, x)|, tau = (beta - alpha) / beta, v = x / (alpha - beta)
      const double alpha = ldg(hk + k);
      double beta = alpha, t = 0.0, scal = 0.0;
      if (ss > 0.0) {
        beta = -copysign(sqrt(fma(alpha, alpha, ss)), alpha);
        t = (beta - alpha) / beta;
        scal = 1.0 / (alpha - beta);
        for (int64_t i = k + 1 + c.tid; i < mm; i += kThreads) stg(hk + i, ldg(hk + i) * scal);
      }
      if (c.tid == 0) {
        stg(hk + k, beta);
        stg(tau + k, t);
      }
    }
    gg.sync();
    // apply H_k to the trailing columns (one warp each) and downdate their norms
    const double tk = ldg(tau + k);
    const double* v = H + int64_t(k) * mm;
    for (int j = k + 1 + c.gw; j < nn; j += c.gnw) {
      double* h = H + int64_t(j) * mm;
      const double hkj = ldg(h + k);
      double w = 0.0;
      if (tk != 0.0) {
        double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
        int64_t i = k + 1 + c.lane;
        for (; i + 96 < mm; i += 128) {
          a0 = fma(ldg(v + i), ldg(h + i), a0);
          a1 = fma(ldg(v + i + 32), ldg(h + i + 32), a1);
          a2 = fma(ldg(v + i + 64), ldg(h + i + 64), a2);
          a3 = fma(ldg(v + i + 96), ldg(h + i + 96), a3);
        }
        for (; i < mm; i += 32) a0 = fma(ldg(v + i), ldg(h + i), a0);
        w = tk * (hkj + wsum((a0 + a1) + (a2 + a3)));
        for (int64_t i2 = k + 1 + c.lane; i2 < mm; i2 += 32) stg(h + i2, fma(-w, ldg(v + i2), ldg(h + i2)));
      }
      const double rkj = hkj - w;  // R(k, j)
      if (c.lane == 0) stg(h + k, rkj);
      const double n1 = ldg(vn1 + j);
      if (n1 != 0.0) {  // warp-uniform
        double r = fabs(rkj) / n1;
        r = fmax(0.0, (1.0 + r) * (1.0 - r));
        const double q = n1 / ldg(vn2 + j);
        double n1new;
        if (r * q * q <= kQrRecompute) {
          // each lane re-reads the rows it wrote above
          double a = 0;
          for (int64_t i2 = k + 1 + c.lane; i2 < mm; i2 += 32) {
            const double x = ldg(h + i2);
            a = fma(x, x, a);
          }
          n1new = sqrt(wsum(a));
          if (c.lane == 0) stg(vn2 + j, n1new);
        } else {
          n1new = n1 * sqrt(r);
        }
        if (c.lane == 0) stg(vn1 + j, n1new);
      }
    }
    gg.sync();
  }
}

__global__ void __launch_bounds__(kThreads)
    svd_factor_kernel(const xgb_svd_desc* __restrict__ descs, const int64_t* __restrict__ work_off, int sector,
                    const double* __restrict__ A, double* __restrict__ U, double* __restrict__ S,
                    double* __restrict__ Vt, double* __restrict__ work, int* __restrict__ sweep_stats,
                    int smem_bytes) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[kWarps];
  __shared__ int redi[kWarps];
  cg::grid_group gg = cg::this_grid();
  const xgb_svd_desc d = descs[sector];
  const bool tr = d.m < d.n;
  const int64_t mm = tr ? d.n : d.m;
  const int nn = int(tr ? d.m : d.n);
  if (nn == 0) return;  // uniform across the grid

  const Ctx c = make_ctx(int(blockIdx.x), int(gridDim.x));
  // workspace (doubles): H mm*nn | V nn*nn | T1 nn*nn | X nn*nn | n64 nn | misc 8 | Y mm*nn (svd_work_elems
  // adds Y for blocks this wide); T1: the Jacobi column order (nn ints), then tau, vn1, vn2 (nn each), piv
  const int64_t nn2 = int64_t(nn) * nn;
  double* H = work + work_off[sector];
  double* V64 = H + mm * nn;
  double* T1 = V64 + nn2;
  double* X = T1 + nn2;
  double* n64 = X + nn2;
  int* flag = reinterpret_cast<int*>(n64 + nn);
  double* Y = n64 + nn + 8;
  int* jorder = reinterpret_cast<int*>(T1);
  double* tau = T1 + nn;
  double* vn1 = tau + nn;
  double* vn2 = vn1 + nn;
  int* piv = reinterpret_cast<int*>(vn2 + nn);
  auto opA = [&](int64_t i, int64_t j) { return tr ? A[d.a_off + j + i * d.m] : A[d.a_off + i + j * d.m]; };
  const long long t0 = clock64();
  for (int j = c.gw; j < nn; j += c.gnw)
    for (int64_t i = c.lane; i < mm; i += 32) stg(H + int64_t(j) * mm + i, opA(i, j));
  gg.sync();
  qr_pivoted(gg, c, H, mm, nn, tau, piv, vn1, vn2, red, redi);
  // X = R^T (lower triangle), V = I
  for (int j = c.gw; j < nn; j += c.gnw)
    for (int i = c.lane; i < nn; i += 32) {
      stg(X + int64_t(j) * nn + i, i >= j ? ldg(H + int64_t(i) * mm + j) : 0.0);
      stg(V64 + int64_t(j) * nn + i, i == j ? 1.0 : 0.0);
    }
  gg.sync();
  const long long t1 = clock64();
  const int nblocks = 2 * int(gridDim.x);
  const int b = (nn + nblocks - 1) / nblocks;
  const bool staged = int64_t(2 * b) * (nn + nn + 1) * 8 <= smem_bytes;
  const int sw = nn > 1 ? block_jacobi<double>(gg, c, X, V64, n64, flag, nn, nn, 1.0e-13, kFloor64, kFactorSweeps,
                                               reinterpret_cast<double*>(smem_raw), staged, nblocks, jorder)
                        : 0;
  const long long t2 = clock64();
  // sigma_j = |x_j|
  for (int j = c.gw; j < nn; j += c.gnw) {
    const double* x = X + int64_t(j) * nn;
    double a = 0;
    for (int i = c.lane; i < nn; i += 32) {
      const double e = ldg(x + i);
      a = fma(e, e, a);
    }
    a = wsum(a);
    if (c.lane == 0) stg(n64 + j, sqrt(a));
  }
  gg.sync();
  // per Jacobi column j (one warp, no barriers): rank r among the sigmas (descending, ties by column),
  // Y_j = Q [V_j; 0] (reflectors H_{nn-1} first; lane ln owns rows ln + 32 t throughout), then U, S, V^T of
  // the block with the sign rule
  const int64_t kk = nn;
  for (int j = c.gw; j < nn; j += c.gnw) {
    const double sj = ldg(n64 + j);
    int r = 0;
    for (int i = c.lane; i < nn; i += 32) {
      const double si = ldg(n64 + i);
      r += ranks_above(si, sj, i < j);
    }
    r = wsum(r);
    const double inv = sj > 0 ? 1.0 / sj : 0.0;
    double* y = Y + int64_t(j) * mm;
    for (int64_t i = c.lane; i < mm; i += 32) stg(y + i, i < nn ? ldg(V64 + int64_t(j) * nn + i) : 0.0);
    for (int k = nn - 1; k >= 0; --k) {
      const double tk = ldg(tau + k);
      if (tk == 0.0) continue;  // uniform
      const double* v = H + int64_t(k) * mm;
      double a0 = 0, a1 = 0, yk = 0;
      int64_t i = c.lane;
      for (; i + 32 < mm; i += 64) {
        const double y0 = ldg(y + i), y1 = ldg(y + i + 32);
        if (i > k) a0 = fma(ldg(v + i), y0, a0);
        else if (i == k) yk = y0;
        if (i + 32 > k) a1 = fma(ldg(v + i + 32), y1, a1);
        else if (i + 32 == k) yk = y1;
      }
      for (; i < mm; i += 32) {
        const double y0 = ldg(y + i);
        if (i > k) a0 = fma(ldg(v + i), y0, a0);
        else if (i == k) yk = y0;
      }
      yk = __shfl_sync(0xffffffffu, yk, k & 31);
      const double w = tk * (yk + wsum(a0 + a1));
      for (int64_t i2 = c.lane; i2 < mm; i2 += 32) {
        if (i2 == k) stg(y + i2, yk - w);
        else if (i2 > k) stg(y + i2, fma(-w, ldg(v + i2), ldg(y + i2)));
      }
    }
    // op(A) = Y Sigma (P U_X)^T with U_X = X / sigma: column j of P U_X has X[i, j] / sigma_j at row piv[i]
    double* ucol = U + d.u_off + int64_t(r) * d.m;
    double sg;
    if (!tr) {
      sg = sign_of<true>(y, mm, 1.0, c.lane);
      for (int64_t i = c.lane; i < mm; i += 32) ucol[i] = sg * ldg(y + i);
      for (int i = c.lane; i < nn; i += 32)
        Vt[d.vt_off + r + int64_t(__ldcg(piv + i)) * kk] = sg * inv * ldg(X + int64_t(j) * nn + i);
    } else {
      // U = P U_X (nn rows): scattered, then read back for the sign
      for (int i = c.lane; i < nn; i += 32) stg(ucol + __ldcg(piv + i), inv * ldg(X + int64_t(j) * nn + i));
      __syncwarp();
      sg = sign_of<true>(ucol, nn, 1.0, c.lane);
      if (sg < 0)
        for (int i = c.lane; i < nn; i += 32) stg(ucol + i, -ldg(ucol + i));
      for (int64_t cc = c.lane; cc < mm; cc += 32) Vt[d.vt_off + r + cc * kk] = sg * ldg(y + cc);
    }
    if (c.lane == 0) S[d.s_off + r] = sj;
  }
  if (sweep_stats && c.rank == 0 && c.tid == 0) {
    int* st6 = sweep_stats + 6 * sector;
    st6[0] = 0;
    st6[1] = sw;
    st6[2] = int((t1 - t0) >> 10);  // QR cycles / 1024 on CTA 0's SM
    st6[3] = 0;
    st6[4] = int((t2 - t1) >> 10);
    st6[5] = int((clock64() - t2) >> 10);
  }
}

int* g_stats_dev = nullptr;
int g_stats_cap = 0;
int g_stats_n = 0;

int g_most_ctas[PerDevice::kMost];  // most CTAs per cluster, by device (set with its kernels' attributes)

void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int grid, int ctas, cudaStream_t s) {
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemLimit;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(ctas);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
}

void launch_clusters(int pass, int lo, int ctas, int most, int widest, int grid_most, int n, const xgb_svd_desc* descs,
                     const int64_t* off, const double* A, double* U, double* S, double* Vt, double* work, int* stats,
                     cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cluster_config(cfg, attr, n * ctas, ctas, s);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, svd_sweeps_kernel, descs, off, A, U, S, Vt, work, stats, pass, lo,
                                           most, widest, grid_most, int(kSmemLimit));
  if (e != cudaSuccess) throw std::runtime_error(std::string("svd sweeps launch: ") + cudaGetErrorString(e));
  count_launch();
}

void launch_grid(const void* kernel, int ctas, void** args, cudaStream_t s) {
  const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(unsigned(ctas)), dim3(kThreads), args,
                                                    size_t(kSmemLimit), s);
  if (e != cudaSuccess) throw std::runtime_error(std::string("svd grid launch: ") + cudaGetErrorString(e));
  count_launch();
}

// All stages of a batch, in stream order; allocates nothing.  grid: wide blocks may use
// cooperative launches (a side lane shares the SMs with the other lane's kernels, and a cooperative grid's
// CTAs wait on one another, so there every block stays on clusters, which take any width).
void svd_pipeline(const xgb_svd_desc* d_descs, const xgb_svd_desc* h_descs, const int64_t* d_off, int n,
                  const double* A, double* U, double* S, double* Vt, double* work, int* stats, bool grid,
                  cudaStream_t s) {
  static PerDevice configured;
  configured.once([] {
    for (const void* f : {reinterpret_cast<const void*>(svd_sweeps_kernel),
                          reinterpret_cast<const void*>(svd_sweeps_grid_kernel),
                          reinterpret_cast<const void*>(svd_polish_grid_kernel),
                          reinterpret_cast<const void*>(svd_factor_kernel),
                          reinterpret_cast<const void*>(svd_finish_kernel),
                          reinterpret_cast<const void*>(svd_small_kernel)})
      cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    // clusters of 16 CTAs (above the portable 8), where the GPU can place one
    cudaFuncSetAttribute(svd_sweeps_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cluster_config(cfg, attr, kMostCtas, kMostCtas, nullptr);
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, svd_sweeps_kernel, &cfg) != cudaSuccess) (void)cudaGetLastError();
    g_most_ctas[PerDevice::current()] = fit > 0 ? kMostCtas : 8;
  });
  const int most = g_most_ctas[PerDevice::current()];
  int64_t small_bytes = 0;
  int narrow[2] = {0, 0}, broad[2] = {0, 0};  // CTAs of the two sweep launches of each pass
  int64_t av = 0, gram = 0, cut = 0, sum = 0, apply = 0, upd = 0;
  std::vector<int> factor, wide;  // blocks of svd_factor_kernel; those whose pass 1 and polish take the cooperative grid
  const int widest[2] = {INT32_MAX, grid ? kGridN : INT32_MAX};
  const int grid_most = grid ? most : 0;
  for (int i = 0; i < n; ++i) {
    const int64_t mm = std::max(h_descs[i].m, h_descs[i].n), nn = std::min(h_descs[i].m, h_descs[i].n);
    if (nn == 0) continue;
    if (small_block(mm, nn)) {
      small_bytes = std::max<int64_t>(small_bytes, 8 * (2 * (mm | 1) * nn + 4 * (nn | 1) * nn));
      continue;
    }
    if (factored(mm, nn, grid_most)) {
      factor.push_back(i);
      continue;
    }
    for (int pass = 0; pass < 2; ++pass) {
      const int ctas = sweep_ctas(pass, mm, nn, most);
      if (nn > widest[pass]) wide.push_back(i);
      else if (ctas <= kNarrow) narrow[pass] = std::max(narrow[pass], ctas);
      else broad[pass] = std::max(broad[pass], ctas);
    }
    const int64_t nt = svd_tiles(nn), mt = svd_tiles(mm);
    av = std::max(av, mt * nt);
    const int64_t splits = gram_splits(mm, nn);
    gram = std::max(gram, 2 * nt * nt);
    if (splits > 1) {
      cut = std::max(cut, splits * nt * nt);
      sum = std::max(sum, (nn * nn + 255) / 256);
    }
    apply = std::max(apply, mt * nt + nt * nt);
    upd = std::max(upd, std::min<int64_t>((nn * nn + 255) / 256, 1024));
  }
  if (small_bytes && !narrow[0]) {  // (else they run beside the sweeps of the wider ones)
    svd_small_kernel<<<n, kThreads, size_t(small_bytes), s>>>(d_descs, A, U, S, Vt, stats);
    count_launch();
  }
  int smem = kSmemLimit;
  for (int sector : factor) {
    const int64_t nn = std::min(h_descs[sector].m, h_descs[sector].n);
    const int ctas = int(std::min<int64_t>(num_sms(), (nn + 2 * kFactorCols - 1) / (2 * kFactorCols)));
    void* args[] = {&d_descs, &d_off, &sector, const_cast<double**>(&A), &U, &S, &Vt, &work, &stats, &smem};
    launch_grid(reinterpret_cast<const void*>(svd_factor_kernel), ctas, args, s);
  }
  if (!av) return;
  auto sweeps = [&](int pass) {
    if (pass)
      for (int sector : wide) {
        const int64_t nn = std::min(h_descs[sector].m, h_descs[sector].n);
        const int ctas = int(std::min<int64_t>(num_sms(), (nn + 2 * kWarps - 1) / (2 * kWarps)));
        void* args[] = {&d_descs, &d_off, &sector, const_cast<double**>(&A), &U, &Vt, &work, &stats, &smem};
        launch_grid(reinterpret_cast<const void*>(svd_sweeps_grid_kernel), ctas, args, s);
      }
    if (broad[pass])
      launch_clusters(pass, kNarrow, broad[pass], most, widest[pass], grid_most, n, d_descs, d_off, A, U, S, Vt, work,
                      stats, s);
    if (narrow[pass])
      launch_clusters(pass, 0, narrow[pass], most, widest[pass], grid_most, n, d_descs, d_off, A, U, S, Vt, work,
                      stats, s);
  };
  sweeps(0);
  auto rows = [&](auto* kernel, int64_t x, int it) {
    in_grid_rows(n, [&](int first, unsigned count) {
      kernel<<<dim3(unsigned(x), count), 256, 0, s>>>(d_descs + first, d_off + first, A, U, Vt, work, it, grid_most);
      count_launch();
    });
  };
  rows(svd_product_kernel<kProdAV>, av, 0);
  for (int it = 0; it < kIters; ++it) {
    if (cut) {
      rows(svd_product_kernel<kProdGramUncut>, gram, it);
      rows(svd_product_kernel<kProdCut>, cut, it);
      rows(svd_gram_sum_kernel, sum, it);
    } else {
      rows(svd_product_kernel<kProdGram>, gram, it);
    }
    rows(svd_update_kernel, upd, it);
    if (it == kPass2) sweeps(1);
    rows(svd_product_kernel<kProdApply>, apply, it);
  }
  for (int sector : wide) {
    const int64_t nn = std::min(h_descs[sector].m, h_descs[sector].n);
    const int ctas = int(std::min<int64_t>(num_sms(), (nn + 7) / 8));
    void* args[] = {&d_descs, &d_off, &sector, const_cast<double**>(&A), &U, &Vt, &work, &stats, &smem};
    launch_grid(reinterpret_cast<const void*>(svd_polish_grid_kernel), ctas, args, s);
  }
  svd_finish_kernel<<<n * kCluster, kThreads, kSmemLimit, s>>>(d_descs, d_off, A, U, S, Vt, work, stats, smem,
                                                               wide.empty() ? INT32_MAX : kGridN + 1,
                                                               grid_most);
  count_launch();
}

}  // namespace

size_t svd_work_elems(int64_t m, int64_t n) {
  // Block above: W, V, G, E, norms and the state words take mm nn + 3 nn^2 + nn + 10, the FP32 columns up to
  // mm nn / 2 + 3 (alignment) behind them
  const int64_t mm = std::max(m, n), nn = std::min(m, n);
  const int64_t doubles = mm * nn + 3 * nn * nn + nn + 8;
  const int64_t floats = mm * nn + nn * nn + nn;
  // svd_factor_kernel keeps Q's columns (mm x nn) behind them
  return size_t(doubles + std::max((floats + 1) / 2 + 2, nn >= kFactorN ? mm * nn : 0));
}

void launch_svd(const xgb_svd_desc* d_descs, const xgb_svd_desc* h_descs, const int64_t* d_work_off, int n,
                const double* A, double* U, double* S, double* Vt, double* work, cudaStream_t s) {
  if (n <= 0) return;
  // sweep statistics of lane 0's calls only (a side lane records none: the buffer is not shared)
  int* stats = nullptr;
  if (lane() == 0) {
    if (g_stats_cap < n) {
      if (g_stats_dev) cudaFree(g_stats_dev);
      cudaMalloc(&g_stats_dev, sizeof(int) * 6 * n);
      g_stats_cap = n;
    }
    g_stats_n = n;
    stats = g_stats_dev;
  }
  svd_pipeline(d_descs, h_descs, d_work_off, n, A, U, S, Vt, work, stats, lane() == 0, s);
}

}  // namespace xgb

// ---------------------------------------------------------------------------
// Batched SVD for callers that cannot allocate device memory.
//
// Some embedders of this library may not call cudaMalloc at all: a plugin
// whose host framework owns every device allocation through its own memory
// pool, or a service that fixes its device-memory budget up front and
// forbids allocations on the request path.  For them the SVD workspace (and the small
// descriptor tables) live in one file-scope device array of kNoAllocDoubles
// doubles (16 MiB) that every GPU loading the library keeps until exit.  The
// array's device address is looked up once per device with
// cudaGetSymbolAddress on that device's first call (make that first call
// before any stream capture begins).  All calls share the array and it keeps
// the previous call's contents; the kernel overwrites every workspace entry
// it reads, so nothing needs clearing between calls.  Two calls whose work
// overlaps on the GPU (different streams, or concurrent host threads) race on
// the array and must be serialised by the caller.
namespace xgb {
namespace {
constexpr size_t kNoAllocDoubles = size_t(2) << 20;  // 16 MiB
__device__ __align__(256) double g_noalloc_scratch[kNoAllocDoubles];
double* g_noalloc_ptr[64] = {nullptr};
}  // namespace
}  // namespace xgb

extern "C" size_t xgb_batched_svd_noalloc_capacity_bytes(void) { return xgb::kNoAllocDoubles * sizeof(double); }

namespace xgb {
namespace {
int batched_svd_noalloc(int n, const xgb_svd_desc* descs, const double* A, double* U, double* S, double* Vt,
                        void* stream_) {
  if (!runtime_ready()) return set_error(XGB_E_NOINIT, "xgb_init was not called");
  if (n <= 0) return XGB_OK;
  if (!descs) return set_error(XGB_E_BADPLAN, "xgb_batched_svd_noalloc: descriptor array is NULL");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return set_error(XGB_E_CUDA, "xgb_batched_svd_noalloc: no current CUDA device");
  // bytes needed: descriptors, work offsets, then the per-block workspaces
  const size_t desc_doubles = (sizeof(xgb_svd_desc) * size_t(n) + 255) / 256 * 32;
  const size_t off_doubles = (sizeof(int64_t) * size_t(n) + 255) / 256 * 32;
  std::vector<int64_t> off(static_cast<size_t>(n));
  size_t work = 0;
  for (int i = 0; i < n; ++i) {
    if (descs[i].m < 0 || descs[i].n < 0) return set_error(XGB_E_BADPLAN, "xgb_batched_svd_noalloc: negative extent");
    if (std::min(descs[i].m, descs[i].n) > 8192)
      return set_error(XGB_E_UNSUPPORTED, "xgb_batched_svd_noalloc: SVD block larger than 8192 columns");
    off[i] = int64_t(work);
    work += svd_work_elems(descs[i].m, descs[i].n);
  }
  const size_t need = desc_doubles + off_doubles + work;
  if (need > kNoAllocDoubles)
    return set_error(XGB_E_UNSUPPORTED,
                     "xgb_batched_svd_noalloc: the batch needs " + std::to_string(need * 8) +
                         " bytes of workspace, above the fixed capacity of " + std::to_string(kNoAllocDoubles * 8) +
                         " bytes; use xgb_batched_svd with caller-provided workspace");
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return set_error(XGB_E_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    g_noalloc_ptr[dev] = static_cast<double*>(p);
  }
  double* base = g_noalloc_ptr[dev];
  auto* d_descs = reinterpret_cast<xgb_svd_desc*>(base);
  auto* d_off = reinterpret_cast<int64_t*>(base + desc_doubles);
  double* d_work = base + desc_doubles + off_doubles;
  cudaStream_t s = stream_ ? static_cast<cudaStream_t>(stream_) : stream();
  cudaError_t e = cudaMemcpyAsync(d_descs, descs, sizeof(xgb_svd_desc) * size_t(n), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_off, off.data(), sizeof(int64_t) * size_t(n), cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return set_error(XGB_E_CUDA, std::string("descriptor copy: ") + cudaGetErrorString(e));
  // the same stages as xgb_batched_svd, cooperative launches included: none of them allocates
  svd_pipeline(d_descs, descs, d_off, n, A, U, S, Vt, d_work, nullptr, lane() == 0, s);
  e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(XGB_E_CUDA, std::string("svd launch: ") + cudaGetErrorString(e));
  // no sweep statistics are recorded here: xgb_svd_last_sweeps reports none after this call
  g_stats_n = 0;
  // the descriptor copies read pageable host memory that the caller may free
  // on return, so wait for them (and the kernels) before returning
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return set_error(XGB_E_CUDA, std::string("svd: ") + cudaGetErrorString(e));
  return XGB_OK;
}
}  // namespace
}  // namespace xgb

extern "C" int xgb_batched_svd_noalloc(int n, const xgb_svd_desc* descs, const double* A, double* U, double* S,
                                       double* Vt, void* stream_) {
  try {
    return xgb::batched_svd_noalloc(n, descs, A, U, S, Vt, stream_);
  } catch (const std::bad_alloc&) {
    return xgb::set_error(XGB_E_OOM, "xgb_batched_svd_noalloc: host allocation failed");
  } catch (const std::exception& ex) {
    return xgb::set_error(XGB_E_BADPLAN, ex.what());
  }
}

extern "C" int xgb_svd_last_sweeps(int32_t* out, int cap) {
  using namespace xgb;
  if (!g_stats_dev || g_stats_n == 0) return 0;
  const int n = std::min(cap / 6, g_stats_n);
  cudaStreamSynchronize(stream());
  cudaMemcpy(out, g_stats_dev, sizeof(int) * 6 * n, cudaMemcpyDeviceToHost);
  return n;
}
