// Kernels of the randomized blockwise tSVD: the seeded Gaussian test
// matrices and the singular-vector sign convention applied after the
// sketch-space singular vectors are lifted back (U = Q U_B).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <string>

#include "kernels.hpp"

namespace cg = cooperative_groups;

namespace xgb {
namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  // splitmix64 finaliser (Steele, Lea, Flood 2014)
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

// Standard normal number `e` of stream `stream` under `seed`: Box-Muller on
// two counter-hashed uniforms u1 in (0, 1], u2 in [0, 1).
__device__ double gauss_at(uint64_t seed, uint64_t stream, uint64_t e) {
  const uint64_t base = mix64(seed ^ mix64(stream));
  const uint64_t h1 = mix64(base ^ (2 * e)), h2 = mix64(base ^ (2 * e + 1));
  const double u1 = double((h1 >> 11) + 1) * 0x1.0p-53;
  const double u2 = double(h2 >> 11) * 0x1.0p-53;
  return sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
}

__global__ void gauss_fill_kernel(const GaussBlock* __restrict__ blocks, int n_blocks, uint64_t seed,
                                  double* __restrict__ out) {
  const GaussBlock b = blocks[blockIdx.y];
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < b.count; e += int64_t(gridDim.x) * blockDim.x)
    out[b.offset + e] = gauss_at(seed, uint64_t(b.stream), uint64_t(e));
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Same rule as the batched SVD kernel: s = sign(r . u) with
// r_i = frac((i+1) * 0.7548776662466927) + 0.25, or the sign of the first
// largest-magnitude entry when |r . u| <= 1e-8 sum_i r_i |u_i|.
__global__ void sign_fix_kernel(const SignFixDesc* __restrict__ descs, double* __restrict__ U, double* __restrict__ Vt) {
  const SignFixDesc d = descs[blockIdx.y];
  const int lane = threadIdx.x & 31;
  const int64_t j = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (j >= d.k) return;
  double* u = U + d.u_off + j * d.m;
  double dot = 0, mag = 0, best = -1, bval = 0;
  long long bidx = 0;
  for (int64_t i = lane; i < d.m; i += 32) {
    const double x = u[i];
    const double y = double(i + 1) * 0.7548776662466927;
    const double r = (y - floor(y)) + 0.25;
    dot = fma(r, x, dot);
    mag = fma(r, fabs(x), mag);
    if (fabs(x) > best) { best = fabs(x); bval = x; bidx = i; }
  }
  dot = warp_sum_d(dot);
  mag = warp_sum_d(mag);
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const double ov = __shfl_xor_sync(0xffffffffu, bval, o);
    const long long oi = __shfl_xor_sync(0xffffffffu, bidx, o);
    if (ob > best || (ob == best && oi < bidx)) { best = ob; bval = ov; bidx = oi; }
  }
  const bool neg = fabs(dot) > 1.0e-8 * mag ? dot < 0 : bval < 0;
  if (!neg) return;
  for (int64_t i = lane; i < d.m; i += 32) u[i] = -u[i];
  double* v = Vt + d.v_off + j;
  for (int64_t c = lane; c < d.n; c += 32) v[c * d.k] = -v[c * d.k];
}

// dst[d.dst_off + c + j * d.dst_ld] = src[d.src_off + j + c * d.src_ld] for j < rows, c < cols
// (descriptor: rows = k rows of the source block, cols = n its columns)
__global__ void transpose_copy_kernel(const xgb_copy2d_desc* __restrict__ descs, const double* __restrict__ src,
                                      double* __restrict__ dst) {
  const xgb_copy2d_desc d = descs[blockIdx.y];
  const int64_t ne = d.rows * d.cols;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < ne; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t c = e % d.cols, j = e / d.cols;  // consecutive threads write consecutive dst rows
    dst[d.dst_off + c + j * d.dst_ld] = src[d.src_off + j + c * d.src_ld];
  }
}

// res[out_off + j] = || R[:, j] - s_j U[:, j] ||_2 for the k columns of one
// sector (R = A V, one warp per column); descriptor fields reused from
// SignFixDesc: m rows, k columns, u_off (U and R share offsets), v_off = s_off,
// n = out_off.
__global__ void residual_norms_kernel(const SignFixDesc* __restrict__ descs, const double* __restrict__ R,
                                      const double* __restrict__ U, const double* __restrict__ S,
                                      double* __restrict__ res) {
  const SignFixDesc d = descs[blockIdx.y];
  const int lane = threadIdx.x & 31;
  const int64_t j = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (j >= d.k) return;
  const double sj = S[d.v_off + j];
  const double* r = R + d.u_off + j * d.m;
  const double* u = U + d.u_off + j * d.m;
  double acc = 0;
  for (int64_t i = lane; i < d.m; i += 32) {
    const double x = r[i] - sj * u[i];
    acc = fma(x, x, acc);
  }
  acc = warp_sum_d(acc);
  if (lane == 0) res[d.n + j] = sqrt(acc);
}

// Middle factor of the SVD reverse rule for one k x k sector (column-major;
// S is the k x k diagonal block, s_i = S[i + i k]):
//   N  = dS + (F.X + (F.X)^T) S + S (F.Y + (F.Y)^T) - S^-1 Y^T
//   XS = X S^-1
// with F_ij = 1 / (s_j^2 - s_i^2) (d -> d / (d^2 + 1e-12) for |d| < 1e-12).
__global__ void svd_bwd_mid_kernel(const SvdBwdDesc* __restrict__ descs, const double* __restrict__ S,
                                   const double* __restrict__ X, const double* __restrict__ Y,
                                   const double* __restrict__ dS, double* __restrict__ N, double* __restrict__ XS) {
  const SvdBwdDesc d = descs[blockIdx.y];
  const int64_t k = d.k, kk = k * k;
  auto F = [&](int64_t i, int64_t j) {
    const double si = S[d.s_off + i * (k + 1)], sj = S[d.s_off + j * (k + 1)];
    const double dd = sj * sj - si * si;
    return fabs(dd) < 1e-12 ? dd / (dd * dd + 1e-12) : 1.0 / dd;
  };
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < kk; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = e % k, j = e / k;
    const double si = S[d.s_off + i * (k + 1)], sj = S[d.s_off + j * (k + 1)];
    const double xij = X[d.kk_off + i + j * k], xji = X[d.kk_off + j + i * k];
    const double yij = Y[d.kk_off + i + j * k], yji = Y[d.kk_off + j + i * k];
    const double fij = F(i, j), fji = F(j, i);
    const double jsym = fij * xij + fji * xji;  // (F.X + (F.X)^T)_ij
    const double ksym = fij * yij + fji * yji;
    N[d.kk_off + e] = dS[d.ds_off + i + j * d.ds_ld] + jsym * sj + si * ksym - yji / si;
    XS[d.kk_off + e] = xij / sj;
  }
}

// W (k x n) += S^-1 dVd  (rows scaled) and P (m x k) = dU S^-1 (columns scaled), one sector per grid row
__global__ void svd_bwd_scale_kernel(const SvdBwdDesc* __restrict__ descs, const double* __restrict__ S,
                                     const double* __restrict__ dVd, const double* __restrict__ dU,
                                     double* __restrict__ W, double* __restrict__ P) {
  const SvdBwdDesc d = descs[blockIdx.y];
  const int64_t kn = d.k * d.n, mk = d.m * d.k;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < kn + mk; e += int64_t(gridDim.x) * blockDim.x) {
    if (e < kn) {
      const int64_t i = e % d.k;
      W[d.w_off + e] += dVd[d.v_off + e] / S[d.s_off + i * (d.k + 1)];
    } else {
      const int64_t f = e - kn, j = f / d.m;
      P[d.p_off + f] = dU[d.u_off + f] / S[d.s_off + j * (d.k + 1)];
    }
  }
}

// Upper-triangular inverse factor of the Gram matrix of one sketch block, for
// CholeskyQR: G (l x l, column-major at d.g_off) = L L^T with L lower
// triangular after adding `shift` = rel_shift * (m l + l (l + 1)) * trace(G)
// to the diagonal (shifted CholeskyQR, Fukaya et al. 2020; rel_shift = 0 for
// the unshifted passes); Rinv (at the same offset) = L^-T, upper triangular,
// zeros below the diagonal.  A pivot at or below eps * trace / l (a direction
// the block does not span) becomes sqrt(eps * trace / l) with a zero column
// below it, so the factor stays finite and well scaled; such pivots are
// counted in *bad.
//
// Three forms: chol_narrow_kernel, chol_cluster_kernel, and beyond their widths chol_inv_body on global memory (right-
// looking: Cholesky by columns; the inverse in trinv_kernel by many CTAs, or, kInverse = true for lists wider than its
// registers allow, by forward elimination of the identity; blocks of such a list that fit shared memory use it,
// row-major with an odd leading dimension).
constexpr int kCholNarrow = 48;    // widest list for one CTA per block
constexpr int kCholCluster = 320;  // widest list for a cluster of eight per block (217 KB of shared memory each)
constexpr unsigned kFullWarp = 0xffffffffu;

// trace of G by one warp, groups of 32 in order
template <typename Diag>
__device__ __forceinline__ double chol_trace(int l, Diag diag) {
  const int lane = threadIdx.x & 31;
  double t = 0;
  for (int g0 = 0; g0 < l; g0 += 32) t += warp_sum_d(g0 + lane < l ? diag(g0 + lane) : 0.0);
  return t;
}
struct CholShift {
  double shift, floor_v;
  __device__ __forceinline__ CholShift(const CholDesc& d, double trace, double rel_shift) {
    const double l = double(d.l);
    shift = rel_shift * (double(d.m) * l + l * (l + 1)) * trace;
    floor_v = fmax(2.220446049250313e-16 * (trace > 0.0 ? trace / l : 0.0), 1e-300);
  }
};
struct CholPivot {
  double r, diag;  // 1 / L_jj, L_jj
  bool dead;       // at or below the floor, or NaN; tested on the bits
  __device__ __forceinline__ CholPivot(double x, const CholShift& sh) {
    const long long bits = __double_as_longlong(x);
    dead = !(bits > __double_as_longlong(sh.floor_v) && bits <= 0x7ff0000000000000ll);
    const double v = dead ? sh.floor_v : x;
    r = rsqrt(v);
    diag = v * r;
  }
};

template <bool kShared, bool kInverse>
__device__ void chol_inv_body(const CholDesc& d, double* __restrict__ Gg, double* __restrict__ Xg, double rel_shift,
                              int* __restrict__ bad, double* sm) {
  const int l = int(d.l), tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int ld = kShared ? (l | 1) : l;
  double* Ls = kShared ? sm : Gg;
  double* Xs = kShared ? sm + int64_t(ld) * l : Xg;
  // element accessors: shared row-major (ld odd) or global column-major (ld = l); symmetric G
  auto LA = [&](int i, int k) -> double& { return kShared ? Ls[i * ld + k] : Ls[i + int64_t(k) * l]; };
  auto XA = [&](int i, int k) -> double& { return kShared ? Xs[i * ld + k] : Xs[i + int64_t(k) * l]; };
  __shared__ double red[32];
  __shared__ double bcast;
  // G is read from its upper triangle (the Gram products compute only that one): LA(i, k) = G(min, max)
  if (kShared) {
    for (int e = tid; e < l * l; e += nt) {
      const int i = e % l, k = e / l;
      LA(i, k) = Gg[i <= k ? e : k + int64_t(i) * l];
    }
  } else {
    for (int e = tid; e < l * l; e += nt) {
      const int i = e % l, k = e / l;
      if (i > k) Gg[e] = Gg[k + int64_t(i) * l];
    }
  }
  if (kInverse)
    for (int e = tid; e < l * l; e += nt) XA(e % l, e / l) = (e % l == e / l) ? 1.0 : 0.0;
  __syncthreads();
  // the trace in the order of a 1024-thread block whatever blockDim is (one element per thread, butterfly
  // sums per 32 elements, added in order), so that blocks of any size give the same shift and the same bits
  __shared__ double trace_s;
  if (l <= 1024) {
    if (warp == 0) {
      double t = 0;
      for (int g0 = 0; g0 < l; g0 += 32) t += warp_sum_d(g0 + lane < l ? LA(g0 + lane, g0 + lane) : 0.0);
      if (lane == 0) trace_s = t;
    }
  } else {
    double tr = 0;
    for (int i = tid; i < l; i += nt) tr += LA(i, i);
    tr = warp_sum_d(tr);
    if (lane == 0) red[warp] = tr;
  }
  __syncthreads();
  __shared__ double floor_s;
  if (tid == 0) {
    double t = 0;
    if (l <= 1024) t = trace_s;
    else
      for (int w = 0; w < (nt >> 5); ++w) t += red[w];
    bcast = rel_shift * (double(d.m) * l + double(l) * (l + 1)) * t;
    const double avg = t > 0.0 ? t / l : 0.0;
    floor_s = fmax(2.220446049250313e-16 * avg, 1e-300);
  }
  __syncthreads();
  const double shift = bcast, dfloor = floor_s;
  for (int i = tid; i < l; i += nt) LA(i, i) += shift;
  __syncthreads();
  // Cholesky (right-looking, one column of look-ahead), lower triangle in place.  Iteration j, with
  // column j final (updated by every earlier column and scaled by its pivot's reciprocal):
  //   warp 0 finishes the diagonal element j + 1 and forms its pivot, warp 1 applies column j to the
  //   rest of column j + 1 and scales it with the pivot's reciprocal (two-warp barrier in between),
  //   warps 2.. apply column j to the trailing columns j + 2 .. l - 1,
  // and one barrier ends the iteration.  The pivot chain - on GB300 a dependent FP64 operation takes
  // 65 cycles, sqrt 595 and a division 560, so the pivot is r = rsqrt(d) (380) with L_jj = d r and
  // 1 / L_jj = r - runs beside the trailing update instead of between two barriers.  Every element sees
  // the same FMAs in the same order as in the unblocked column algorithm.
  const unsigned full_warp = 0xffffffffu;
  auto panel = [&](int c) {  // warp 0: pivot of column c and its scaling (first column); lane ln owns rows c + ln + 32 r
    double r = 0.0;
    int dd = 0;
    if (lane == 0) {
      const double dj = LA(c, c);
      dd = !(dj > dfloor);  // also true for NaN
      if (dd) atomicAdd(bad, 1);
      const double v = dd ? dfloor : dj;
      r = rsqrt(v);
      LA(c, c) = v * r;
    }
    r = __shfl_sync(full_warp, r, 0);
    dd = __shfl_sync(full_warp, dd, 0);
    for (int i = c + lane; i < l; i += 32)
      if (i > c) LA(i, c) = dd ? 0.0 : LA(i, c) * r;
    __syncwarp();
  };
  if (warp == 0 && l > 0) panel(0);
  __syncthreads();
  // warp 0 forms the next pivot (one lane: the diagonal's last FMA, then rsqrt) while warp 1 applies
  // column j to the rest of column j + 1; a two-warp barrier hands the reciprocal over for the scaling
  __shared__ double piv_r;
  __shared__ int piv_dead;
  for (int j = 0; j + 1 < l; ++j) {
    const int nc = j + 1;  // the next column
    if (warp == 0) {
      if (lane == 0) {
        const double ljj = LA(nc, j);
        const double dj = fma(-ljj, ljj, LA(nc, nc));  // row nc of the column update, as in the unblocked order
        const int dd = !(dj > dfloor);               // also true for NaN
        if (dd) atomicAdd(bad, 1);
        const double v = dd ? dfloor : dj;
        const double r = rsqrt(v);
        LA(nc, nc) = v * r;
        piv_r = r;
        piv_dead = dd;
      }
      asm volatile("bar.sync 1, 64;" ::: "memory");
    } else if (warp == 1) {
      const double ljj = LA(nc, j);
      for (int i = nc + 1 + lane; i < l; i += 32) LA(i, nc) = fma(-LA(i, j), ljj, LA(i, nc));
      asm volatile("bar.sync 1, 64;" ::: "memory");
      const double r = piv_r;
      const bool dd = piv_dead != 0;
      for (int i = nc + 1 + lane; i < l; i += 32) LA(i, nc) = dd ? 0.0 : LA(i, nc) * r;
    } else {
      // trailing lower triangle (rows i >= k >= j + 2) folded into whole columns: column c and column
      // t-1-c together hold t+1 elements; an odd t leaves the middle column alone
      const int t = l - j - 2, half = t >> 1;
      const int total = (t + 1) * half + ((t & 1) ? (t + 1) >> 1 : 0);
      for (int e = tid - 64; e < total; e += nt - 64) {
        int i, k;
        if (e < (t + 1) * half) {
          const int r = e % (t + 1), c = e / (t + 1);
          if (r < t - c) { i = c + r; k = c; } else { i = (t - 1 - c) + (r - (t - c)); k = t - 1 - c; }
        } else {
          k = (t - 1) >> 1;
          i = k + (e - (t + 1) * half);
        }
        i += j + 2;
        k += j + 2;
        LA(i, k) = fma(-LA(i, j), LA(k, j), LA(i, k));
      }
    }
    __syncthreads();
  }
  if constexpr (!kInverse) {
    if (kShared)  // L back to G, column-major, lower triangle and diagonal
      for (int e = tid; e < l * l; e += nt) {
        const int i = e % l, k = e / l;
        if (i >= k) Gg[e] = LA(i, k);
      }
    return;
  } else {
    // X = L^-1 by forward elimination of the identity: row j of X is final after
    // dividing by L[j][j]; then rows i > j subtract L[i][j] * row j (columns c <= j)
    __shared__ double inv_s[1];
    for (int j = 0; j < l; ++j) {
      if (tid == 0) inv_s[0] = 1.0 / LA(j, j);
      __syncthreads();
      const double inv = inv_s[0];
      for (int c = tid; c <= j; c += nt) XA(j, c) *= inv;
      __syncthreads();
      const int t = l - j - 1;
      for (int e = tid; e < t * (j + 1); e += nt) {
        const int i = j + 1 + e % t, c = e / t;
        XA(i, c) = fma(-LA(i, j), XA(j, c), XA(i, c));
      }
      __syncthreads();
    }
    // Rinv = X^T, column-major l x l: Rinv[c + i l] = X[i][c]
    if (kShared) {
      for (int e = tid; e < l * l; e += nt) {
        const int c = e % l, i = e / l;
        Xg[e] = XA(i, c);
      }
    } else {
      for (int e = tid; e < l * l; e += nt) {
        const int i = e % l, c = e / l;
        if (i > c) {
          const double a = Xg[i + int64_t(c) * l], b = Xg[c + int64_t(i) * l];
          Xg[i + int64_t(c) * l] = b;
          Xg[c + int64_t(i) * l] = a;
        }
      }
    }
  }
}

template <bool kInverse>
__global__ void __launch_bounds__(1024) chol_inv_kernel(const CholDesc* __restrict__ descs, double* __restrict__ G,
                                                      double* __restrict__ Rinv, double rel_shift,
                                                      int* __restrict__ bad, int smem_cap_l) {
  extern __shared__ double sm[];
  const CholDesc d = descs[blockIdx.x];
  if (d.l <= smem_cap_l)
    chol_inv_body<true, kInverse>(d, G + d.g_off, Rinv + d.g_off, rel_shift, bad, sm);
  else
    chol_inv_body<false, kInverse>(d, G + d.g_off, Rinv + d.g_off, rel_shift, bad, sm);
}

// Narrow blocks: factor and inverse together, in one CTA's shared memory.
//
// Iteration j starts with columns <= j of L final and finishes column j + 1 (all of it in warp 0, which forms the
// pivot between its multiply-add and the scaling), applies column j to the columns behind and row j - 1 of X to the
// rows behind while warp 1 finishes row j of X; one barrier ends it.  The other warps take a row each, lanes along its
// columns of X and L: no index is divided.  What bounds it is the chain of warp 0 (on GB300 a dependent FP64 operation
// takes 65 cycles and rsqrt 380, so about 700 cycles a column).  So the warps that share warp 0's quarter of the SM
// stay out of the updates, and the pivot test is on the bits (a comparison is an FP64 instruction).
// Measured (two blocks, widths about 16 / 32 / 48, factor and inverse): 63 / 85 / 158 us with one warp per block and a
// second kernel for the inverse, 25 / 29 / 44 now.
__global__ void __launch_bounds__(512) chol_narrow_kernel(const CholDesc* __restrict__ descs,
                                                          const double* __restrict__ G, double* __restrict__ Rinv,
                                                          double rel_shift, int* __restrict__ bad) {
  extern __shared__ double sm[];
  __shared__ double trace_s, pivots[kCholNarrow];  // pivots: 1 / L_jj
  constexpr int kSlots = (kCholNarrow + 31) / 32;
  const CholDesc d = descs[blockIdx.x];
  const int l = int(d.l), ld = l | 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (l == 0) return;
  const double* Gg = G + d.g_off;
  double* Ls = sm;
  double* Xs = sm + l * ld;
  for (int k = warp; k < l; k += warps)  // row k of the lower triangle from column k of G's upper one
    for (int i = lane; i <= k; i += 32) {
      Ls[k * ld + i] = Gg[i + k * l];
      Xs[k * ld + i] = i == k ? 1.0 : 0.0;
    }
  __syncthreads();
  if (warp == 0) {
    const double t = chol_trace(l, [&](int i) { return Ls[i * (ld + 1)]; });
    if (lane == 0) trace_s = t;
  }
  __syncthreads();
  const CholShift sh(d, trace_s, rel_shift);
  for (int i = threadIdx.x; i < l; i += blockDim.x) Ls[i * (ld + 1)] += sh.shift;
  __syncthreads();
  // warp 0: the pivot of column c and its scaling, lane's rows c + lane + 32 s in x
  auto finish = [&](int c, const double* x) {
    const CholPivot p(__shfl_sync(kFullWarp, x[0], 0), sh);
    if (lane == 0) {
      Ls[c * (ld + 1)] = p.diag;
      pivots[c] = p.r;
      if (p.dead) atomicAdd(bad, 1);
    }
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
      const int i = c + lane + 32 * s;
      if (i > c && i < l) Ls[i * ld + c] = p.dead ? 0.0 : x[s] * p.r;
    }
  };
  if (warp == 0) {
    double x[kSlots];
#pragma unroll
    for (int s = 0; s < kSlots; ++s) x[s] = lane + 32 * s < l ? Ls[(lane + 32 * s) * ld] : 0.0;
    finish(0, x);
  }
  __syncthreads();
  const int rows = warps - (warps >> 2) - 1, rank = warp - 2 - (warp >> 2);
  for (int j = 0; j < l; ++j) {
    if (warp == 0) {
      const int c = j + 1;
      if (c < l) {
        double x[kSlots];
        const double ljj = Ls[c * ld + j];
#pragma unroll
        for (int s = 0; s < kSlots; ++s) {
          x[s] = 0.0;
          if (c + 32 * s >= l) break;
          const int i = min(c + lane + 32 * s, l - 1);
          x[s] = fma(-Ls[i * ld + j], ljj, Ls[i * ld + c]);
        }
        finish(c, x);
      }
    } else if (warp == 1) {  // row j of X: the last update and the scaling
      const double r = pivots[j], a = j > 0 ? Ls[j * ld + j - 1] : 0.0;
      for (int c = lane; c <= j; c += 32) {
        double x = Xs[j * ld + c];
        if (c < j) x = fma(-a, Xs[(j - 1) * ld + c], x);
        Xs[j * ld + c] = x * r;
      }
    } else if (warp & 3) {  // rows behind: X by row j - 1, L (columns j + 2 .. the diagonal) by column j
      for (int i = j + 1 + rank; i < l; i += rows) {
        double* Li = Ls + i * ld;
        const double b = Li[j], a = j > 0 ? Li[j - 1] : 0.0;
        for (int q = lane; q < i - 1; q += 32) {
          const int k = q + 2;  // = j + 2 + q - j
          double* p = q < j ? Xs + i * ld + q : Li + k;
          const double m = q < j ? Xs[(j - 1) * ld + q] : Ls[k * ld + j];
          *p = fma(q < j ? -a : -b, m, *p);
        }
      }
    }
    __syncthreads();
  }
  double* Xg = Rinv + d.g_off;  // Rinv = X^T, column-major: Rinv[c + i l] = X[i][c]
  for (int i = warp; i < l; i += warps)
    for (int c = lane; c < l; c += 32) Xg[c + i * l] = c <= i ? Xs[i * ld + c] : 0.0;
}

// Wide blocks: factor and inverse over a cluster, rows of 16 dealt out to its CTAs in turn, everything in their shared
// memory and in place (a row's columns of L give way to those of Y, with X_i = L_ii^-1 Y_i at the end).  Panel K:
//   the owner of row block K has factored the diagonal block and sent T = L_KK^-1 and Y_K to every CTA;
//   each CTA forms P_i = A_iK T^T (= L_iK) and M_i = P_i T of its rows, and sends P to every CTA;
//   A_iJ -= P_i P_J^T for K < J <= i, Y_iJ -= M_i Y_KJ for J < K, Y_iK = -M_i;
// where the owner of block K + 1 lets four warps (one per quarter of the SM) update and factor that diagonal block
// first, beside the update of its other rows; the owner of K stores X_K = T Y_K meanwhile.  Two cluster barriers a panel.
// The pivots are still a chain, 16 times 880 cycles a panel (1300 beside the updates), but the l^3 / 3 multiply-adds run
// on the pipes of all CTAs.  The sums' order does not depend on the cluster's size.  (Two rows of every block per CTA
// balance the updates, but need a third barrier and send more: as fast at 150 columns, 5 % slower at 125.)
// Measured, against a factorisation on one SM with the inverse in a second kernel: one block about 150 wide 357 ->
// 171 us, two about 125 wide 214 -> 119, two about 190 wide 894 -> 256; CTMRG D = 6, chi = 128 134 -> 89 us a call.
// One CTA is the faster up to 48 columns (its chain has no cluster barriers).
constexpr int kPan = 16;
__host__ __device__ constexpr int chol_cluster_elems(int l, int cluster) {
  const int nb = (l + kPan - 1) / kPan, lp = nb * kPan, own = (nb + cluster - 1) / cluster;
  return own * kPan * (lp + 2) + 2 * kPan * lp + 2 * kPan * kPan + 2 * own * kPan * kPan;
}

// threads 0..127: D (16 x 16, leading dimension ld, its first bs rows and columns used) -> T = L^-1 (row-major, zeros
// above the diagonal, the identity in rows behind bs), as in chol_narrow_kernel
__device__ __forceinline__ void chol_diag(double* D, int ld, int bs, double* T, double* pivots, const CholShift& sh,
                                          int* bad) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto team = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
  for (int e = tid; e < kPan * kPan; e += 128) T[e] = e / kPan == e % kPan ? 1.0 : 0.0;
  auto finish = [&](int c, double x) {
    const CholPivot p(__shfl_sync(kFullWarp, x, 0), sh);
    if (lane == 0) {
      D[c * (ld + 1)] = p.diag;
      pivots[c] = p.r;
      if (p.dead) atomicAdd(bad, 1);
    }
    const int i = c + lane;
    if (i > c && i < bs) D[i * ld + c] = p.dead ? 0.0 : x * p.r;
  };
  if (warp == 0) finish(0, lane < bs ? D[lane * ld] : 0.0);
  team();
  for (int j = 0; j < bs; ++j) {
    if (warp == 0) {
      const int c = j + 1;
      if (c < bs) {
        const int i = min(c + lane, bs - 1);
        finish(c, fma(-D[i * ld + j], D[c * ld + j], D[i * ld + c]));
      }
    } else if (warp == 1) {
      if (lane <= j) {
        double x = T[j * kPan + lane];
        if (lane < j) x = fma(-D[j * ld + j - 1], T[(j - 1) * kPan + lane], x);
        T[j * kPan + lane] = x * pivots[j];
      }
    } else {
      const int q = lane & 15;
      for (int i = j + 1 + (warp - 2) * 2 + (lane >> 4); i < bs; i += 4)
        if (q < i - 1) {
          double* p = q < j ? T + i * kPan + q : D + i * ld + q + 2;
          const double m = q < j ? T[(j - 1) * kPan + q] : D[(q + 2) * ld + j];
          *p = fma(-(q < j ? D[i * ld + j - 1] : D[i * ld + j]), m, *p);
        }
    }
    team();
  }
}

__global__ void __launch_bounds__(512) chol_cluster_kernel(const CholDesc* __restrict__ descs,
                                                           const double* __restrict__ G, double* __restrict__ Rinv,
                                                           double rel_shift, int* __restrict__ bad) {
  extern __shared__ __align__(16) double chol_sm[];
  __shared__ double pivots[kPan], partial[(kCholCluster + 31) / 32];
  cg::cluster_group cluster = cg::this_cluster();
  const int P = int(cluster.num_blocks()), me = int(cluster.block_rank());
  const CholDesc d = descs[blockIdx.x / P];
  const int l = int(d.l), nb = (l + kPan - 1) / kPan, lp = nb * kPan, ld = lp + 2, most = (nb + P - 1) / P;
  if (l == 0) return;  // the whole cluster
  cluster.barrier_arrive();  // completed before the first store to another CTA, which has to be running by then
  const int own = me < nb ? (nb - me + P - 1) / P : 0;  // row blocks me, me + P, ...
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  double* A = chol_sm;
  double* Bs = A + most * kPan * ld;            // two of 16 x lp: Y_K left of block K, P^T right of it
  double* Ts = Bs + 2 * kPan * lp;              // two of 16 x 16
  double* Pc = Ts + 2 * kPan * kPan;            // P and M of this CTA's rows
  double* Mc = Pc + most * kPan * kPan;
  const double* Gg = G + d.g_off;
  for (int k = warp; k < own * kPan; k += warps) {  // row i of the lower triangle from column i of G's upper one
    const int gb = me + (k / kPan) * P, i = gb * kPan + k % kPan;
#pragma unroll 5
    for (int c = lane; c < (gb + 1) * kPan; c += 32) A[k * ld + c] = i < l && c <= i ? __ldg(Gg + c + i * l) : 0.0;
  }
  const int groups = (l + 31) / 32;
  for (int g = warp; g < groups; g += warps) {
    const int i = g * 32 + lane;
    const double t = warp_sum_d(i < l ? Gg[i + i * l] : 0.0);
    if (lane == 0) partial[g] = t;
  }
  __syncthreads();
  double trace = 0.0;
  for (int g = 0; g < groups; ++g) trace += partial[g];
  const CholShift sh(d, trace, rel_shift);
  for (int k = tid; k < own * kPan; k += blockDim.x) {
    const int i = (me + (k / kPan) * P) * kPan + k % kPan;
    if (i < l) A[k * ld + i] += sh.shift;
  }
  __syncthreads();
  // factor diagonal block K (this CTA's): T goes to its slot
  auto diagonal = [&](int K) {
    double* D = A + (K / P) * kPan * ld + K * kPan;
    double* T = Ts + (K & 1) * kPan * kPan;
    chol_diag(D, ld, min(kPan, l - K * kPan), T, pivots, sh, bad);
  };
  // T of block K, and its Y (by `count` warps), to the other CTAs
  auto send_t = [&](int K) {
    double* T = Ts + (K & 1) * kPan * kPan;
    for (int p = 0; p < P; ++p)
      if (p != me && tid < kPan * kPan) cluster.map_shared_rank(T, p)[tid] = T[tid];
  };
  auto send_y = [&](int K, int rank, int count) {
    double* B = Bs + (K & 1) * kPan * lp;
    const double* Y = A + (K / P) * kPan * ld;
    const int half = K * kPan / 2;  // pairs of a row
    for (int p = 0; p < P; ++p) {
      double* Bp = cluster.map_shared_rank(B, p);
      for (int r = rank; r < kPan; r += count)
        for (int c = lane; c < half; c += 32)
          reinterpret_cast<double2*>(Bp + r * lp)[c] = reinterpret_cast<const double2*>(Y + r * ld)[c];
    }
  };
  // X_K = T [Y_K, I] by `count` warps of its CTA; Rinv = X^T, column-major: Rinv[c + i l] = X[i][c]
  double* Xg = Rinv + d.g_off;
  auto store_x = [&](int K, int rank, int count) {
    const double* T = Ts + (K & 1) * kPan * kPan;
    const double* Y = A + (K / P) * kPan * ld;
    const int chunks = (l + 31) / 32;
    for (int w = rank; w < kPan * chunks; w += count) {
      const int r = w / chunks, c = (w % chunks) * 32 + lane, i = K * kPan + r;
      if (i >= l || c >= l) continue;
      const double* t = T + r * kPan;
      double even = 0.0, odd = 0.0;  // T is zero behind r
      if (c < K * kPan) {
        for (int q = 0; q <= r; q += 2) {
          even = fma(t[q], Y[q * ld + c], even);
          odd = fma(t[q + 1], Y[(q + 1) * ld + c], odd);
        }
        even += odd;
      } else if (c <= i) {
        even = t[c - K * kPan];
      }
      Xg[c + i * l] = even;
    }
  };
  if (me == 0 && warp < 4) diagonal(0);
  cluster.barrier_wait();
  __syncthreads();
  if (me == 0) send_t(0);
  cluster.sync();
  for (int K = 0; K + 1 < nb; ++K) {
    const double* T = Ts + (K & 1) * kPan * kPan;
    double* B = Bs + (K & 1) * kPan * lp;
    for (int e = tid; e < own * kPan * kPan; e += blockDim.x) {
      const int b = e >> 8, c = (e >> 4) & 15, r = e & 15, gb = me + b * P;
      if (gb <= K) continue;
      const double* a = A + (b * kPan + r) * ld + K * kPan;
      double even = 0.0, odd = 0.0;  // two chains: T is zero behind c
      for (int k = 0; k <= c; k += 2) {
        even = fma(a[k], T[c * kPan + k], even);
        odd = fma(a[k + 1], T[c * kPan + k + 1], odd);
      }
      const double acc = even + odd;
      Pc[(b * kPan + r) * kPan + c] = acc;
      for (int p = 0; p < P; ++p) cluster.map_shared_rank(B, p)[c * lp + gb * kPan + r] = acc;
    }
    __syncthreads();
    cluster.barrier_arrive();
    for (int e = tid; e < own * kPan * kPan; e += blockDim.x) {
      const int b = e >> 8, c = e & 15;
      if (me + b * P <= K) continue;
      const double* p = Pc + (e & ~15);
      double acc = 0.0;
      for (int k = c; k < kPan; ++k) acc = fma(p[k], T[k * kPan + c], acc);
      Mc[e] = acc;
    }
    cluster.barrier_wait();
    __syncthreads();
    const int next = K + 1;
    const bool mine = next % P == me;
    if (mine) {  // the next diagonal block first, all warps
      const int b = next / P;
      for (int e = tid; e < kPan * kPan; e += blockDim.x) {
        const int r = e / kPan, c = e % kPan;
        if (c > r) continue;
        double* p = A + (b * kPan + r) * ld + next * kPan + c;
        const double* x = Pc + (b * kPan + r) * kPan;
        const double* y = Pc + (b * kPan + c) * kPan;
        double even = *p, odd = 0.0;
#pragma unroll
        for (int k = 0; k < kPan; k += 2) {
          even = fma(-x[k], y[k], even);
          odd = fma(-x[k + 1], y[k + 1], odd);
        }
        *p = even + odd;
      }
      __syncthreads();
    }
    if (mine && warp < 4) {
      diagonal(next);
    } else if (!mine || (warp & 3)) {
      const int team = mine ? warps - 4 - (warps - 4) / 4 : warps;
      const int rank = mine ? warp - 5 - (warp - 4) / 4 : warp;
      int at = 0;  // items (row pair, 32 columns) dealt out in turn over all row blocks
      for (int b = 0; b < own; ++b) {
        const int gb = me + b * P;
        if (gb <= K) continue;
        const int chunks = ((gb + 1) * kPan + 31) / 32, items = chunks * (kPan / 2);
        for (int w = (rank - at % team + team) % team; w < items; w += team) {
          const int r = (w / chunks) * 2, c = (w % chunks) * 32 + lane, cb = c / kPan;
          if (c >= (gb + 1) * kPan || (gb == next && cb == next)) continue;
          double* a0 = A + (b * kPan + r) * ld + c;
          const int o = (b * kPan + r) * kPan;
          if (cb == K) {
            a0[0] = -Mc[o + c % kPan];
            a0[ld] = -Mc[o + kPan + c % kPan];
            continue;
          }
          const double* co = (cb < K ? Mc : Pc) + o;
          double x = a0[0], y = a0[ld];
#pragma unroll
          for (int k = 0; k < kPan; ++k) {
            const double m = B[k * lp + c];
            x = fma(-co[k], m, x);
            y = fma(-co[kPan + k], m, y);
          }
          a0[0] = x;
          a0[ld] = y;
        }
        at += items;
        if (mine && gb == next) {  // its Y is final: to the other CTAs, beside the factorisation
          asm volatile("bar.sync 2, %0;" ::"r"(team * 32) : "memory");
          send_y(next, rank, team);
        }
      }
      if (K % P == me) store_x(K, rank, team);
    }
    __syncthreads();
    if (mine) send_t(next);
    cluster.sync();
  }
  if ((nb - 1) % P == me) store_x(nb - 1, warp, warps);
}

// Rinv = L^-T from the Cholesky factor L (column-major, lower triangle, in G): one warp per
// column c of X = L^-1, kTrinvCols columns per CTA, so the l^3/6 FMAs of a block spread over
// ceil(l / kTrinvCols) SMs.  Column c by forward substitution in the same operation order as
// the single-CTA elimination (x_k = r_k * (1 / L_kk), then r_i -= L_ik x_k for i > k), so
// both give the same bits; lane t keeps r_i for i = t + 32 j in registers (j < T).
constexpr int kTrinvCols = 8;
template <int T>
__global__ void __launch_bounds__(32 * kTrinvCols) trinv_kernel(const CholDesc* __restrict__ descs, int chunks,
                                                                 const double* __restrict__ G,
                                                                 double* __restrict__ Rinv) {
  extern __shared__ double tsm[];
  const int sector = blockIdx.x / chunks, c0 = (blockIdx.x % chunks) * kTrinvCols;
  const CholDesc d = descs[sector];
  const int l = int(d.l);
  if (c0 >= l) return;  // uniform over the CTA
  const int lt = l - c0;  // trailing order: rows / columns c0 .. l-1 are all this CTA reads
  double* inv_diag = tsm;
  const double* L = G + d.g_off;
  double* R = Rinv + d.g_off;
  for (int k = c0 + int(threadIdx.x); k < l; k += blockDim.x) inv_diag[k - c0] = 1.0 / L[k + int64_t(k) * l];
  __syncthreads();
  const int lane = threadIdx.x & 31, c = c0 + int(threadIdx.x >> 5);
  if (c >= l) return;
  double r[T];
#pragma unroll
  for (int j = 0; j < T; ++j) r[j] = (lane + 32 * j == c) ? 1.0 : 0.0;
  for (int k = c; k < l; ++k) {
    const int slot = k >> 5;
    double v = 0.0;
#pragma unroll
    for (int j = 0; j < T; ++j)
      if (j == slot) v = r[j];
    const double xk = __shfl_sync(0xffffffffu, v, k & 31) * inv_diag[k - c0];
    const double* Lk = L + int64_t(k) * l;
#pragma unroll
    for (int j = 0; j < T; ++j) {
      if (32 * j + 31 < k) continue;  // warp-uniform: rows of this slot are all finished
      const int i = lane + 32 * j;
      if (i == k) r[j] = xk;
      else if (i > k && i < l) r[j] = fma(-__ldg(Lk + i), xk, r[j]);
    }
  }
  // row c of Rinv (= column c of X): Rinv[c + i l] = X[i][c], zero for i < c
#pragma unroll
  for (int j = 0; j < T; ++j) {
    const int i = lane + 32 * j;
    if (i < l) R[c + int64_t(i) * l] = i >= c ? r[j] : 0.0;
  }
}

}  // namespace

void launch_chol_inv(const CholDesc* d_descs, int n, int64_t max_l, double* G, double* Rinv, double rel_shift,
                     int* bad, cudaStream_t s) {
  if (n <= 0 || max_l <= 0) return;
  static PerDevice attr;
  // Cholesky alone: one l x (l | 1) matrix in shared memory up to l = 167 (< 227 KB)
  constexpr int kCapChol = 167;
  // Cholesky and inverse in one CTA (blocks wider than the register-resident inverse allows):
  // two matrices up to l = 119
  constexpr int kCapBoth = 119;
  constexpr int kBytesChol = kCapChol * (kCapChol | 1) * int(sizeof(double));
  constexpr int kBytesBoth = 2 * kCapBoth * (kCapBoth | 1) * int(sizeof(double));
  attr.once([] {
    cudaFuncSetAttribute(chol_inv_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytesChol);
    cudaFuncSetAttribute(chol_inv_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytesBoth);
  });
  if (max_l > 64 * 32) {
    chol_inv_kernel<true><<<n, 1024, kBytesBoth, s>>>(d_descs, G, Rinv, rel_shift, bad, kCapBoth);
    count_launch();
    return;
  }
  if (max_l <= kCholNarrow) {
    constexpr int kBytes = 2 * kCholNarrow * (kCholNarrow | 1) * int(sizeof(double));
    static_assert(kBytes <= 48 * 1024);
    const int lw = int(max_l);
    chol_narrow_kernel<<<n, lw <= 32 ? 256 : 512, 2 * lw * (lw | 1) * int(sizeof(double)), s>>>(d_descs, G, Rinv,
                                                                                              rel_shift, bad);
    count_launch();
    return;
  }
  if (max_l <= kCholCluster) {
    const int cluster = max_l <= 4 * kPan ? 4 : 8;
    const int bytes = chol_cluster_elems(int(max_l), cluster) * int(sizeof(double));
    static PerDevice cattr;
    cattr.once([] {
      cudaFuncSetAttribute(chol_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           chol_cluster_elems(kCholCluster, 8) * int(sizeof(double)));
    });
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(n) * unsigned(cluster));
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = size_t(bytes);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim = {unsigned(cluster), 1, 1};
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, chol_cluster_kernel, d_descs, static_cast<const double*>(G), Rinv,
                                             rel_shift, bad);
    if (e != cudaSuccess) throw std::runtime_error(std::string("Cholesky launch: ") + cudaGetErrorString(e));
    count_launch();
    return;
  }
  chol_inv_kernel<false><<<n, 1024, kBytesChol, s>>>(d_descs, G, Rinv, rel_shift, bad, kCapChol);
  count_launch();
  const int chunks = int((max_l + kTrinvCols - 1) / kTrinvCols);
  const size_t sm = sizeof(double) * size_t(max_l);
  if (max_l <= 512)
    trinv_kernel<16><<<n * chunks, 32 * kTrinvCols, sm, s>>>(d_descs, chunks, G, Rinv);
  else if (max_l <= 1024)
    trinv_kernel<32><<<n * chunks, 32 * kTrinvCols, sm, s>>>(d_descs, chunks, G, Rinv);
  else
    trinv_kernel<64><<<n * chunks, 32 * kTrinvCols, sm, s>>>(d_descs, chunks, G, Rinv);
  count_launch();
}

void launch_svd_bwd_mid(const SvdBwdDesc* d_descs, int n, int64_t max_kk, const double* S, const double* X,
                        const double* Y, const double* dS, double* N, double* XS, cudaStream_t s) {
  if (n <= 0 || max_kk <= 0) return;
  const int64_t want = (max_kk + 255) / 256;
  dim3 grid(unsigned(want < 1024 ? want : 1024), unsigned(n));
  svd_bwd_mid_kernel<<<grid, 256, 0, s>>>(d_descs, S, X, Y, dS, N, XS);
  count_launch();
}

void launch_svd_bwd_scale(const SvdBwdDesc* d_descs, int n, int64_t max_elems, const double* S, const double* dVd,
                          const double* dU, double* W, double* P, cudaStream_t s) {
  if (n <= 0 || max_elems <= 0) return;
  const int64_t want = (max_elems + 255) / 256;
  dim3 grid(unsigned(want < 1024 ? want : 1024), unsigned(n));
  svd_bwd_scale_kernel<<<grid, 256, 0, s>>>(d_descs, S, dVd, dU, W, P);
  count_launch();
}

void launch_residual_norms(const SignFixDesc* d_descs, int n, int64_t max_k, const double* R, const double* U,
                           const double* S, double* res, cudaStream_t s) {
  if (n <= 0 || max_k <= 0) return;
  dim3 grid(unsigned((max_k + 7) / 8), unsigned(n));
  residual_norms_kernel<<<grid, 256, 0, s>>>(d_descs, R, U, S, res);
  count_launch();
}

void launch_transpose_copy(const xgb_copy2d_desc* d_descs, int n, int64_t max_elems, const double* src, double* dst,
                           cudaStream_t s) {
  if (n <= 0 || max_elems <= 0) return;
  const int64_t want = (max_elems + 255) / 256;
  dim3 grid(unsigned(want < 1024 ? want : 1024), unsigned(n));
  transpose_copy_kernel<<<grid, 256, 0, s>>>(d_descs, src, dst);
  count_launch();
}

void launch_gauss_fill(const GaussBlock* d_blocks, int n_blocks, int64_t max_count, uint64_t seed, double* out,
                       cudaStream_t s) {
  if (n_blocks <= 0 || max_count <= 0) return;
  const int64_t want = (max_count + 255) / 256;
  dim3 grid(unsigned(want < 1024 ? want : 1024), unsigned(n_blocks));
  gauss_fill_kernel<<<grid, 256, 0, s>>>(d_blocks, n_blocks, seed, out);
  count_launch();
}

void launch_sign_fix(const SignFixDesc* d_descs, int n, int64_t max_k, double* U, double* Vt, cudaStream_t s) {
  if (n <= 0 || max_k <= 0) return;
  dim3 grid(unsigned((max_k + 7) / 8), unsigned(n));
  sign_fix_kernel<<<grid, 256, 0, s>>>(d_descs, U, Vt);
  count_launch();
}

}  // namespace xgb
