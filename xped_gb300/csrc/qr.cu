// Batched Householder QR in FP64 with LAPACK's dlarfg sign convention (beta = -sign(alpha) ||x||), so Q
// and R agree with dgeqrf / dorgqr (Tensor::tQR, src/Core/Tensor.cpp:757-780).
//
// Two launches per batch (one where no block has more than four columns).  qr_factor_kernel: one cluster per block with the
// block's columns in its CTAs' shared memory (column j on CTA j mod P, fewer CTAs in crowded batches), a warp one to four
// trailing columns at a time.  The warp that holds column j + 1
// applies reflector j to it first and forms reflector j + 1 at once, beside the other columns' update, so a
// step is that warp's chain (a dot product, an update, a norm, a square root and a division: GB300's dependent
// FP64 operations take 65 cycles, a division 560, a square root 595), one cluster barrier and the copy of
// the reflector to the other CTAs, ~10k cycles together with 300 rows.  Reflectors stay unscaled (v = x with
// v_j = 1 / scal), which takes a pass over the column off that chain, unless x is far from one: then a power of two
// brings it there, so that its products with columns of any other scale stay in range.  qr_form_q_kernel: column c of Q is
// H_0 .. H_c e_c, independent of the others: one warp a column, four (one per SM sub-partition) a CTA, over
// all SMs.  One CTA per block (the kernel below, kept for blocks that no cluster's shared memory holds) was
// bound by a single SM's FP64 pipe: five blocks of 120 x 40 to 308 x 128 took 7.4 ms there and take
// 0.68 + 0.25 ms here.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <string>

#include "kernels.hpp"

namespace cg = cooperative_groups;

namespace xgb {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kMostCtas = 8;  // portable cluster size (16 gained 1 %: the chain bounds a step, not the update)
constexpr int64_t kSmemLimit = 220 * 1024;
constexpr int kQCols = 4;  // columns of Q per CTA
constexpr int kUnscaled = 32;  // largest |exponent| of a reflector that stays as it is

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Columns per CTA that a batch's blocks aim at (spread_of): blocks whose chain is at least `from` long, and the others.
struct Spread {
  int64_t from;
  int wide, rest;
};
// a block's chain of reflectors, in rows
__host__ __device__ __forceinline__ int64_t qr_chain(int64_t m, int64_t n) { return (m < n ? m : n) * (m + 256); }

// CTAs of a block's cluster: one per 16 columns (a warp each) or fewer in crowded batches, more when the columns need more
// shared memory; 0: no cluster holds them (a CTA's columns and its copy of the current reflector; kQCols columns of Q).
__host__ __device__ __forceinline__ int qr_ctas(int64_t m, int64_t n, const Spread& sp) {
  if (8 * m * kQCols > kSmemLimit) return 0;
  const int per = qr_chain(m, n) >= sp.from ? sp.wide : sp.rest;
  for (int p = 1; p <= kMostCtas; p *= 2) {
    const int64_t cols = (n + p - 1) / p;
    if ((cols <= per || p == kMostCtas) && 8 * m * (cols + 1) <= kSmemLimit) return p;
  }
  return 0;
}

// A workspace block (qr_work_elems): reflectors m x min(m, n) | tau | scal
__device__ __forceinline__ double* tau_of(double* w, int64_t m, int64_t n) { return w + m * n; }
__device__ __forceinline__ double* scal_of(double* w, int64_t m, int64_t n) { return w + m * n + (m < n ? m : n); }

// dot product of rows lo .. m-1, four partial sums a lane
__device__ __forceinline__ double column_dot(const double* x, const double* y, int lo, int m, int lane) {
  double a0 = 0, a1 = 0;
  int i = lo + lane;
  for (; i + 32 < m; i += 64) {
    a0 = fma(x[i], y[i], a0);
    a1 = fma(x[i + 32], y[i + 32], a1);
  }
  if (i < m) a0 = fma(x[i], y[i], a0);
  return warp_sum(a0 + a1);
}

// Reflector j (v below row j, tau t, scale sc) applied to N columns of a warp, `next` apart, with the bits of one column at a
// time.  What a crowded SM waits for is FP64 instructions: N sums share the steps of a butterfly (six additions for four
// columns instead of twenty), and the lanes of each column's part compute its factors at once.  300 blocks of 30 x 500
// 4.03 ms one column at a time, 2.62 so; one of 20 x 4000 1.21 and 0.59.
template <int N>
__device__ __forceinline__ void apply_reflector(const double* v, double* c, int64_t next, int j, int m, double t, double sc,
                                                int lane) {
  double a0[N] = {}, a1[N] = {};
  int i = j + 1 + lane;
  for (; i + 32 < m; i += 64) {
    const double x = v[i], y = v[i + 32];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      a0[k] = fma(x, c[i + k * next], a0[k]);
      a1[k] = fma(y, c[i + 32 + k * next], a1[k]);
    }
  }
  if (i < m) {
    const double x = v[i];
#pragma unroll
    for (int k = 0; k < N; ++k) a0[k] = fma(x, c[i + k * next], a0[k]);
  }
#pragma unroll
  for (int k = 0; k < N; ++k) a0[k] += a1[k];
  int o = 16;
#pragma unroll
  for (int half = N / 2; half > 0; half /= 2, o /= 2) {  // lanes with bit o keep the upper half of the columns
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < half; ++k) {
      const double keep = up ? a0[k + half] : a0[k], send = up ? a0[k] : a0[k + half];
      a0[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (; o > 0; o /= 2) a0[0] += __shfl_xor_sync(0xffffffffu, a0[0], o);
  constexpr int kPart = 32 / N;  // lanes of a column
  double* cj = c + j + (lane / kPart) * next;
  const double w = t * (*cj + sc * a0[0]), ws = -w * sc;
  __syncwarp();
  if (lane % kPart == 0) *cj -= w;
  double f[N];
#pragma unroll
  for (int k = 0; k < N; ++k) f[k] = __shfl_sync(0xffffffffu, ws, k * kPart);
#pragma unroll 4
  for (i = j + 1 + lane; i < m; i += 32) {
    const double x = v[i];
#pragma unroll
    for (int k = 0; k < N; ++k) c[i + k * next] = fma(f[k], x, c[i + k * next]);
  }
  __syncwarp();
}

// Column c of Q = H_0 .. H_c e_c by one warp, in shared memory (y), from the reflectors W (m rows each).
__device__ __forceinline__ void form_q(double* q, int64_t c, int m, int kk, const double* W, const double* tau,
                                       const double* scal, double* y, int lane) {
  if (c >= kk) {
    for (int i = lane; i < m; i += 32) q[i] = 0.0;
    return;
  }
  for (int i = lane; i < m; i += 32) y[i] = i == c ? 1.0 : 0.0;
  __syncwarp();
  for (int k = int(c); k >= 0; --k) {
    const double t = tau[k], sc = scal[k];
    if (t == 0.0) continue;
    const double* v = W + int64_t(k) * m;
    const double w = t * (y[k] + sc * column_dot(v, y, k + 1, m, lane)), ws = -w * sc;
    __syncwarp();
    if (lane == 0) y[k] -= w;
#pragma unroll 4
    for (int i = k + 1 + lane; i < m; i += 32) y[i] = fma(ws, v[i], y[i]);
    __syncwarp();
  }
  for (int i = lane; i < m; i += 32) q[i] = y[i];
}

// kGroups: some CTA holds more columns than warps (the branch alone costs a step of the others 2 %).  whole: Q as well.
template <bool kGroups>
__global__ void __launch_bounds__(kThreads)
    qr_factor_kernel(const xgb_qr_desc* __restrict__ descs, const int64_t* __restrict__ work_off,
                     const double* __restrict__ A, double* __restrict__ Q, double* __restrict__ R,
                     double* __restrict__ work, Spread sp, bool whole) {
  extern __shared__ __align__(16) double qr_sm[];
  __shared__ double tau_s[2], scal_s[2];  // of the reflector that this CTA formed last, by parity of its column
  cg::cluster_group cl = cg::this_cluster();
  const int ctas = int(cl.num_blocks()), block = int(blockIdx.x) / ctas, rank = int(cl.block_rank());
  const xgb_qr_desc d = descs[block];
  const int P = qr_ctas(d.m, d.n, sp);
  if (P == 0 || rank >= P) return;  // (a cluster barrier waits for the threads that have not exited)
  const int m = int(d.m), n = int(d.n), kk = m < n ? m : n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int own = n > rank ? (n - rank + P - 1) / P : 0;  // columns rank, rank + P, ...
  double* cols = qr_sm + m;                               // after the copy of the current reflector
  double* W = work + work_off[block];
  double* tau = tau_of(W, m, n);
  double* scal = scal_of(W, m, n);
  for (int u = warp; u < own; u += kWarps)
    for (int i = lane; i < m; i += 32) cols[u * m + i] = A[d.a_off + i + int64_t(rank + u * P) * m];
  __syncthreads();
  // reflector of column j, by the warp that holds it (rows below j: x, left as they are)
  auto reflect = [&](int j) {
    double* x = cols + (j / P) * m;
    const double ss = column_dot(x, x, j + 1, m, lane), alpha = x[j];
    double t = 0.0, sc = 0.0, beta = alpha;
    if (ss > 0.0) {
      beta = -copysign(sqrt(fma(alpha, alpha, ss)), alpha);
      t = (beta - alpha) / beta;
      sc = 1.0 / (alpha - beta);
      const int e = ((__double2hiint(beta) >> 20) & 0x7ff) - 1023;
      if (abs(e) > kUnscaled && e <= 1023) {  // (1024: infinite or NaN; else |e| stays below 540)
        const double p = __hiloint2double((1023 - e) << 20, 0);  // 2^-e
        sc *= __hiloint2double((1023 + e) << 20, 0);
        for (int i = j + 1 + lane; i < m; i += 32) x[i] *= p;
      }
    }
    __syncwarp();
    if (lane == 0) {
      x[j] = beta;
      tau_s[j & 1] = t;
      scal_s[j & 1] = sc;
      tau[j] = t;
      scal[j] = sc;
    }
  };
  if (rank == 0 && warp == 0 && kk > 0) reflect(0);
  for (int j = 0; j < kk; ++j) {
    const int owner = j % P;
    const double* v = cols + (j / P) * m;
    double t, sc;
    if (P > 1) {
      cl.sync();
      const double* from = cl.map_shared_rank(cols, owner) + (j / P) * m;
      t = cl.map_shared_rank(tau_s, owner)[j & 1];
      sc = cl.map_shared_rank(scal_s, owner)[j & 1];
      if (owner != rank) {
        for (int i = j + 1 + tid; i < m; i += kThreads) qr_sm[i] = from[i];
        v = qr_sm;
      }
    }
    __syncthreads();
    if (P == 1) {
      t = tau_s[j & 1];
      sc = scal_s[j & 1];
    }
    // the warp of column j + 1 is its own CTA's first: column j + 1 is the lowest one left there
    const int lowest = j + 1 <= rank ? 0 : (j + 1 - rank + P - 1) / P;
    for (int u = lowest + warp; u < own; u += kWarps) {
      double* c = cols + u * m;
      if (kGroups && t != 0.0 && u + kWarps < own && rank + u * P != j + 1) {  // four or two columns of this warp
        if (u + 3 * kWarps < own) {
          apply_reflector<4>(v, c, int64_t(kWarps) * m, j, m, t, sc, lane);
          u += 3 * kWarps;
        } else {
          apply_reflector<2>(v, c, int64_t(kWarps) * m, j, m, t, sc, lane);
          u += kWarps;
        }
        continue;
      }
      if (t != 0.0) {
        const double w = t * (c[j] + sc * column_dot(v, c, j + 1, m, lane)), ws = -w * sc;
        __syncwarp();
        if (lane == 0) c[j] -= w;
#pragma unroll 4
        for (int i = j + 1 + lane; i < m; i += 32) c[i] = fma(ws, v[i], c[i]);
        __syncwarp();
      }
      if (rank + u * P == j + 1 && j + 1 < kk) reflect(j + 1);
    }
  }
  if (P > 1) cl.sync();  // no CTA leaves while another reads its last reflector
  __syncthreads();
  // R: the first min(m, n) rows on and above the diagonal; the reflectors for qr_form_q_kernel
  for (int u = warp; u < own; u += kWarps) {
    const int c = rank + u * P;
    for (int64_t i = lane; i < d.r_rows; i += 32)
      R[d.r_off + i + int64_t(c) * d.r_rows] = i < kk && i <= c ? cols[u * m + i] : 0.0;
    if (c < kk && !whole)
      for (int i = c + 1 + lane; i < m; i += 32) W[i + int64_t(c) * m] = cols[u * m + i];
  }
  if (whole && warp < d.q_cols)  // (P = 1)
    form_q(Q + d.q_off + int64_t(warp) * m, warp, m, kk, cols, tau, scal, cols + (n + warp) * m, lane);
}

__global__ void __launch_bounds__(32 * kQCols)
    qr_form_q_kernel(const xgb_qr_desc* __restrict__ descs, const int64_t* __restrict__ work_off,
                     double* __restrict__ Q, const double* __restrict__ work, Spread sp) {
  extern __shared__ __align__(16) double qr_sm[];
  const xgb_qr_desc d = descs[blockIdx.y];
  if (qr_ctas(d.m, d.n, sp) == 0) return;
  const int m = int(d.m), kk = int(d.m < d.n ? d.m : d.n);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t c = d.q_cols - 1 - (int64_t(blockIdx.x) * kQCols + warp);  // the longest products first
  if (c < 0) return;
  const double* W = work + work_off[blockIdx.y];
  const double* tau = W + d.m * d.n;
  form_q(Q + d.q_off + c * m, c, m, kk, W, tau, tau + kk, qr_sm + warp * m, lane);
}

// One CTA per block, the columns in global memory: blocks that no cluster's shared memory holds.
__global__ void __launch_bounds__(256) qr_kernel(const xgb_qr_desc* __restrict__ descs, const int64_t* __restrict__ work_off,
                                                 const double* __restrict__ A, double* __restrict__ Q,
                                                 double* __restrict__ R, double* __restrict__ work,
                                                 Spread sp) {
  const xgb_qr_desc d = descs[blockIdx.x];
  if (qr_ctas(d.m, d.n, sp) != 0) return;
  const int64_t m = d.m, n = d.n, kk = m < n ? m : n;
  double* W = work + work_off[blockIdx.x];  // m x n working copy (Householder vectors below diagonal)
  double* tau = W + m * n;                  // kk
  double* Qw = tau + kk;                    // m x m accumulation
  __shared__ double red[8];
  __shared__ double bcast[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int64_t e = tid; e < m * n; e += 256) W[e] = A[d.a_off + e];
  __syncthreads();
  auto block_sum = [&](double v) {
    v = warp_sum(v);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double r = 0;
    if (tid == 0) { for (int w = 0; w < 8; ++w) r += red[w]; bcast[0] = r; }
    __syncthreads();
    r = bcast[0];
    __syncthreads();
    return r;
  };
  for (int64_t j = 0; j < kk; ++j) {
    double* col = W + j * m;
    double part = 0;
    for (int64_t i = j + 1 + tid; i < m; i += 256) part = fma(col[i], col[i], part);
    double xnorm2 = block_sum(part);
    double alpha = col[j];
    double t = 0.0, beta = alpha;
    if (xnorm2 > 0.0) {
      beta = -copysign(sqrt(alpha * alpha + xnorm2), alpha);
      t = (beta - alpha) / beta;
      double scal = 1.0 / (alpha - beta);
      for (int64_t i = j + 1 + tid; i < m; i += 256) col[i] *= scal;
    }
    __syncthreads();
    if (tid == 0) { tau[j] = t; col[j] = beta; }
    __syncthreads();
    if (t != 0.0) {
      for (int64_t c = j + 1 + warp; c < n; c += 8) {
        double* cc = W + c * m;
        double w = (lane == 0) ? cc[j] : 0.0;
        for (int64_t i = j + 1 + lane; i < m; i += 32) w = fma(col[i], cc[i], w);
        w = warp_sum(w) * t;
        if (lane == 0) cc[j] -= w;
        for (int64_t i = j + 1 + lane; i < m; i += 32) cc[i] -= w * col[i];
      }
    }
    __syncthreads();
  }
  // R (r_rows x n): upper triangle of W in the first kk rows
  for (int64_t e = tid; e < d.r_rows * n; e += 256) {
    int64_t i = e % d.r_rows, c = e / d.r_rows;
    R[d.r_off + e] = (i < kk && i <= c) ? W[i + c * m] : 0.0;
  }
  // Q = H_0 H_1 ... H_{kk-1} applied to the first q_cols columns of I (backward accumulation)
  const int64_t qc = d.q_cols < m ? d.q_cols : m;
  for (int64_t e = tid; e < m * qc; e += 256) Qw[e] = ((e % m) == (e / m)) ? 1.0 : 0.0;
  __syncthreads();
  for (int64_t j = kk - 1; j >= 0; --j) {
    const double t = tau[j];
    if (t == 0.0) continue;
    const double* v = W + j * m;
    for (int64_t c = warp; c < qc; c += 8) {
      double* cc = Qw + c * m;
      double w = (lane == 0) ? cc[j] : 0.0;
      for (int64_t i = j + 1 + lane; i < m; i += 32) w = fma(v[i], cc[i], w);
      w = warp_sum(w) * t;
      if (lane == 0) cc[j] -= w;
      for (int64_t i = j + 1 + lane; i < m; i += 32) cc[i] -= w * v[i];
    }
    __syncthreads();
  }
  for (int64_t e = tid; e < m * d.q_cols; e += 256) {
    int64_t c = e / m;
    Q[d.q_off + e] = (c < qc && c < kk) ? Qw[e] : 0.0;
  }
}

// Blocks of so few columns that their CTA forms Q as fast as qr_form_q_kernel does (one warp per SM sub-partition): a batch of
// them is one launch (one block of 1 x 1: 22.8 -> 19.1 us).
bool whole_block(const xgb_qr_desc& d) {
  return d.n <= kQCols && d.q_cols <= kQCols && 8 * d.m * (d.n + 1 + kQCols) <= kSmemLimit;
}

// 16 columns a CTA keep a block's chain shortest; where the clusters of a batch are more CTAs than the SMs take at once they
// only share the FP64 pipes, and pay for their barriers.  So from 5/4 CTAs per SM on, blocks take fewer: first those with
// less than half of the longest chain, then all.  Measured (us, 16 / 32 / 64 columns): 38 of 60 x 60 409 / 429 / 465, 75 of
// them 698 / 509 / 544, 300 1951 / 1455 / 1169 (one CTA per block in global memory 1346); 20 of 120 x 120 (160 CTAs) 908
// / 955 / 1154, 75 2560 / 2375 / 1767; 300 of 300 x 60 3024 / 2360 / 2290.
Spread spread_of(const xgb_qr_desc* d, int n) {
  int64_t longest = 0, cols = kWarps;
  for (int i = 0; i < n; ++i) {
    longest = std::max(longest, qr_chain(d[i].m, d[i].n));
    cols = std::max(cols, std::min<int64_t>(d[i].n, INT32_MAX / 2));
  }
  Spread sp{(longest + 1) / 2, kWarps, kWarps};
  auto crowded = [&](bool all) {
    int64_t room = 5 * int64_t(num_sms() > 0 ? num_sms() : 152) / 4;
    for (int i = 0; i < n && room >= 0; ++i)
      if (all || qr_chain(d[i].m, d[i].n) >= sp.from) room -= qr_ctas(d[i].m, d[i].n, sp);
    return room < 0;
  };
  while (sp.rest < cols && crowded(true)) sp.rest *= 2;
  while (sp.wide < cols && crowded(false)) sp.wide *= 2;
  return sp;
}

}  // namespace

size_t qr_work_elems(int64_t m, int64_t n) { return size_t(m * n + std::min(m, n) + m * m); }

void launch_qr(const xgb_qr_desc* d_descs, const xgb_qr_desc* h_descs, const int64_t* d_work_off, int n,
               const double* A, double* Q, double* R, double* work, cudaStream_t s) {
  if (n <= 0) return;
  static PerDevice attr;
  attr.once([] {
    cudaFuncSetAttribute(qr_factor_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemLimit));
    cudaFuncSetAttribute(qr_factor_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemLimit));
    cudaFuncSetAttribute(qr_form_q_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemLimit));
  });
  const Spread sp = spread_of(h_descs, n);
  int ctas = 0;
  int64_t bytes = 0, whole_bytes = 0, q_bytes = 0, q_cols = 0;
  bool large = false, groups = false, whole = true;
  for (int i = 0; i < n; ++i) {
    const xgb_qr_desc& d = h_descs[i];
    const int p = qr_ctas(d.m, d.n, sp);
    if (p == 0) {
      large = true;
      continue;
    }
    ctas = std::max(ctas, p);
    whole = whole && whole_block(d);
    whole_bytes = std::max(whole_bytes, 8 * d.m * (d.n + 1 + kQCols));
    groups = groups || d.n > int64_t(p) * kWarps;
    bytes = std::max(bytes, 8 * d.m * ((d.n + p - 1) / p + 1));
    q_bytes = std::max(q_bytes, 8 * d.m * kQCols);
    q_cols = std::max(q_cols, d.q_cols);
  }
  if (ctas) {
    if (whole) bytes = whole_bytes;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(n * ctas));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = size_t(bytes);
    cfg.stream = s;
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeClusterDimension;
    a[0].val.clusterDim.x = unsigned(ctas);
    a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
    cfg.attrs = a;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, groups ? qr_factor_kernel<true> : qr_factor_kernel<false>, d_descs,
                                             d_work_off, A, Q, R, work, sp, whole);
    if (e != cudaSuccess) throw std::runtime_error(std::string("qr launch: ") + cudaGetErrorString(e));
    count_launch();
    if (q_cols > 0 && !whole) {
      in_grid_rows(n, [&](int first, unsigned count) {
        qr_form_q_kernel<<<dim3(unsigned((q_cols + kQCols - 1) / kQCols), count), 32 * kQCols, size_t(q_bytes), s>>>(
            d_descs + first, d_work_off + first, Q, work, sp);
        count_launch();
      });
    }
  }
  if (large) {
    qr_kernel<<<n, 256, 0, s>>>(d_descs, d_work_off, A, Q, R, work, sp);
    count_launch();
  }
}

}  // namespace xgb
