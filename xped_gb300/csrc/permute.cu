// Gather-permute with recoupling coefficients (Tensor::permute_impl, src/Core/Tensor.cpp:83-214): every output
// fusion-tree pair's sub-block is a strided copy (abelian symmetries) or a sum of strided copies (SU(2)).
//
// The host rewrites each task as a set of PLANES: legs of extent 1 are dropped, legs whose strides chain in the
// output and in every source are merged, and two of the remaining legs, A (the output's fast leg) and B, span a
// plane, cut into chunks; the other legs enumerate the planes.  A block decodes a batch of chunks, one per thread,
// into shared memory; then groups of G lanes move a chunk each, with affine addresses in both legs, so that an
// element costs an add, a load and a store.  (Rows of leg 0, decoded one by one, took 108 warp instructions per 32
// elements; this takes 18 on planes of 400.)
//  * direct form: B is the next leg in the output; the lanes run along A, several rows side by side where A is short,
//    eight elements a lane in flight.  Reads are runs of leg A, or strided when A is not the source's fast leg.
//  * transposed form, when another leg is the source's unit-stride one and both are at least 4 long (64 elements
//    together): that leg is B; a warp copies a tile of the plane along B into its shared memory (cp.async: what is in
//    flight takes no registers) and stores it along A, so that both sides move whole runs.  The direct form reads
//    every 32-byte sector of such a plane four times.
// Coefficients +-1 (every abelian permute) are sign flips in a loop of their own: a warp's FP64 instruction takes its
// pipe 64 cycles, predicated off or not, and multiplying made the 1.4 GB permutes 1.2 ms instead of 0.54.
// Bound by HBM where the tensor is large, by the number of warp instructions for sums over short legs, and for the
// smallest by the dependent loads of one batch (6.5 us under the profiler).  Measured, before -> now (U(1), 5 sectors,
// legs up to 60, 2.8 GB moved): (0,2,1,3) 803 -> 540 us, (2,3,0,1) 3440 -> 438, (2,0,3,1) 1475 -> 499; SU(2) 2.6 M
// elements: (2,0,3,1) with 270 sources of 158 sub-blocks 48 -> 41 us on inputs out of cache (35 repeated).
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <stdexcept>
#include <type_traits>
#include <vector>

#include "kernels.hpp"

namespace xgb {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTileElems = 528;     // transposed form: doubles of shared memory per warp
constexpr int kUnroll = 4;            // elements of a lane in flight, several sources
constexpr int kFlight = 8;            // one source

constexpr int resident(bool transpose, bool single) { return transpose ? (single ? 5 : 3) : 4; }  // CTAs per SM

// a block's batch of chunks: decoded one per thread, then moved by G lanes each.  The transposed form's tiles leave
// less room (three CTAs per SM).
template <bool kTranspose, bool kSingle>
struct Batch {
  static constexpr int kMost = kTranspose ? 64 : kThreads;    // chunks
  static constexpr int kSlots = kMost * (kSingle ? 1 : 4);    // their source offsets
  static constexpr int kStart = kTranspose ? 256 : 1024;      // prefix sums of the tasks' chunks, if they fit
  int64_t start[kStart], dst[kMost], src[kSlots];
  int32_t task[kMost], extent[kMost];  // extent: ni | nj << 16
  int next;
};

// the index arithmetic is shared with the host walk below
#define XGB_HD __host__ __device__ __forceinline__

// one plane's chunk and its outer leg indices
struct Plane {
  int i0, j0, ni, nj;
  int o[kPlaneOuter];
  int64_t dst;
};

// SI: 32-bit where a task's offsets and its number of chunks fit
template <typename SI>
XGB_HD Plane locate(const PlaneTask& t, int64_t q) {
  using Index = std::conditional_t<sizeof(SI) == 4, uint32_t, uint64_t>;
  Plane p;
  Index r = Index(q);
  int ic = 0, jc = 0;
  if (t.nci > 1) {
    ic = int(r % Index(t.nci));
    r /= Index(t.nci);
  }
  if (t.ncj > 1) {
    jc = int(r % Index(t.ncj));
    r /= Index(t.ncj);
  }
  p.i0 = ic * t.ci;
  p.j0 = jc * t.cj;
  p.ni = t.na - p.i0 < t.ci ? t.na - p.i0 : t.ci;
  p.nj = t.nb - p.j0 < t.cj ? t.nb - p.j0 : t.cj;
  SI at = SI(p.i0) * SI(t.dst_a) + SI(p.j0) * SI(t.dst_b);
#pragma unroll
  for (int k = 0; k < kPlaneOuter; ++k) {
    p.o[k] = 0;
    if (k < t.n_outer) {
      const Index d = Index(t.odim[k]), x = r / d;
      p.o[k] = int(r - x * d);
      r = x;
      at += SI(p.o[k]) * SI(t.odst[k]);
    }
  }
  p.dst = t.dst_base + at;
  return p;
}

template <typename SI>
XGB_HD int64_t source(const PlaneTask& t, const PlaneSource& s, const Plane& p) {
  SI at = SI(p.i0) * SI(s.a) + SI(p.j0) * SI(s.b);
#pragma unroll
  for (int k = 0; k < kPlaneOuter; ++k)
    if (k < t.n_outer) at += SI(p.o[k]) * SI(s.outer[k]);
  return s.base + at;
}

// +-1: the sign bit to flip; anything else: 2
__device__ __forceinline__ int unit_sign(double c) {  // by its bits: a comparison would be an FP64 instruction
  const unsigned long long b = (unsigned long long)__double_as_longlong(c);
  return b << 1 == 0x3ff0000000000000ull << 1 ? int(b >> 63) : 2;
}
__device__ __forceinline__ double flip(double v, int sign) {
  return __longlong_as_double(__double_as_longlong(v) ^ ((long long)sign << 63));
}

// which task holds plane p (start ascending, start[n] the number of planes)
XGB_HD int task_of(const int64_t* start, int n, int64_t p) {
  int a = 0, b = n - 1;
  while (a < b) {
    const int mid = (a + b + 1) >> 1;
    if (start[mid] <= p) a = mid;
    else b = mid - 1;
  }
  return a;
}

__device__ __forceinline__ void cp_async8(double* smem, const double* gmem) {
  const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(at), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <int G, bool kTranspose, bool kSingle, typename SI>
__global__ void __launch_bounds__(kThreads, resident(kTranspose, kSingle))
    permute_planes_kernel(const PlaneTask* __restrict__ tasks, const int64_t* __restrict__ start, int n_tasks,
                          int64_t n_planes, int batch, const PlaneSource* __restrict__ sources,
                          const double* __restrict__ src, double* __restrict__ dst) {
  static_assert(!kTranspose || G == 32, "a warp per tile");
  extern __shared__ double tile_sm[];
  using B = Batch<kTranspose, kSingle>;
  __shared__ B bt;
  const bool held = n_tasks <= B::kStart;
  if (held)
    for (int k = threadIdx.x; k < n_tasks; k += kThreads) bt.start[k] = start[k];
  __syncthreads();
  const int64_t* first = held ? bt.start : start;
  const int tid = int(threadIdx.x), l = tid % G;
  double* tile = kTranspose ? tile_sm + (tid / 32) * kTileElems : nullptr;
  for (int64_t p0 = int64_t(blockIdx.x) * batch; p0 < n_planes; p0 += int64_t(gridDim.x) * batch) {
    const int here = int(n_planes - p0 < batch ? n_planes - p0 : batch);
    if (tid == 0) bt.next = kWarps;
    if (tid < here) {
      const int at = task_of(first, n_tasks, p0 + tid);
      const PlaneTask& t = tasks[at];
      const Plane pl = locate<SI>(t, p0 + tid - first[at]);
      bt.dst[tid] = pl.dst;
      bt.task[tid] = at;
      bt.extent[tid] = pl.ni | pl.nj << 16;
      const int keep = kSingle ? 1 : min(t.n_source, B::kSlots / batch);
      for (int k = 0; k < keep; ++k) bt.src[k * batch + tid] = source<SI>(t, sources[t.source0 + k], pl);
    }
    __syncthreads();
    // a warp takes the next chunk when it has done one: their sizes differ
    auto next = [&](int c) {
      if (G < 32) return c + kThreads / G;
      int got = 0;
      if (l == 0) got = atomicAdd(&bt.next, 1);
      return __shfl_sync(0xffffffffu, got, 0);
    };
    for (int c = tid / G; c < here; c = next(c)) {
      const PlaneTask& t = tasks[bt.task[c]];
      double* to = dst + bt.dst[c];
      const int ni = bt.extent[c] & 0xffff, nj = bt.extent[c] >> 16;
      // la lanes along A and ia along B; transposed: lb lanes along B and ib along A on the reading side.  The direction
      // with more steps is the unrolled one (y), the other (x) is outside.
      const int fast = kTranspose ? t.lb : t.la, rows = kTranspose ? t.ib : t.ia;
      const int slow = (l * (kTranspose ? t.rb : t.ra)) >> 16, f = l - slow * fast;
      const SI da = SI(t.dst_a), db = SI(t.dst_b);
      const int ld = nj | 1;
      const bool y_is_a = t.y_is_a;
      const bool y_fast = y_is_a != kTranspose;  // y is the direction that the lanes run along
      const int y_end = y_is_a ? ni : nj, x_end = y_is_a ? nj : ni;
      const int y_step = y_fast ? fast : rows, x_step = y_fast ? rows : fast;
      const int y0 = y_fast ? f : slow, x0 = slow >= rows ? x_end : y_fast ? slow : f;  // lanes left over: none
      const SI yd = kTranspose ? SI(y_is_a ? ld : 1) : y_is_a ? da : db;
      const SI xd = kTranspose ? SI(y_is_a ? 1 : ld) : y_is_a ? db : da;
      if (kSingle) {
        const PlaneSource& o = sources[t.source0];
        const SI ys = y_is_a ? SI(o.a) : SI(o.b), xs = y_is_a ? SI(o.b) : SI(o.a);
        const double* from = src + bt.src[c];
        const double coeff = o.coeff;
        const int sign = unit_sign(coeff);
        const SI ss = SI(y_step) * ys, sd = SI(y_step) * yd;
        if (kTranspose) {
          for (int x = x0; x < x_end; x += x_step) {
            const double* sp = from + (SI(x) * xs + SI(y0) * ys);
            double* dp = tile + (SI(x) * xd + SI(y0) * yd);
            for (int y = y0; y < y_end; y += y_step) {
              cp_async8(dp, sp);
              sp += ss;
              dp += sd;
            }
          }
          cp_async_wait_all();
          __syncwarp();
          const int sj = (l * t.ra) >> 16, fi = l - sj * t.la;
          auto put = [&](auto scale) {
            for (int i = fi; i < ni; i += t.la) {
              const double* tp = tile + i * ld + sj;
              double* dp = to + (SI(i) * da + SI(sj) * db);
              const SI step = SI(t.ia) * db;
              for (int j = sj; j < nj; j += t.ia) {
                *dp = decltype(scale)::value ? *tp * coeff : flip(*tp, sign);
                tp += t.ia;
                dp += step;
              }
            }
          };
          if (sj < t.ia) {
            if (sign == 2) put(std::true_type{});
            else put(std::false_type{});
          }
          __syncwarp();
          continue;
        }
        auto move = [&](auto scale) {
          for (int x = x0; x < x_end; x += x_step) {
            const double* sp = from + (SI(x) * xs + SI(y0) * ys);
            double* dp = to + (SI(x) * xd + SI(y0) * yd);
            for (int y = y0; y < y_end; y += kFlight * y_step) {
              double v[kFlight];
#pragma unroll
              for (int u = 0; u < kFlight; ++u)
                if (y + u * y_step < y_end) v[u] = __ldg(sp + SI(u) * ss);
#pragma unroll
              for (int u = 0; u < kFlight; ++u)
                if (y + u * y_step < y_end) dp[SI(u) * sd] = decltype(scale)::value ? v[u] * coeff : flip(v[u], sign);
              sp += SI(kFlight) * ss;
              dp += SI(kFlight) * sd;
            }
          }
        };
        if (sign == 2) move(std::true_type{});
        else move(std::false_type{});
        continue;
      }
      // several sources, added in their fixed order (the sum's rounding is the plan's)
      double* into = kTranspose ? tile : to;
      const SI sd = SI(y_step) * yd;
      auto sum = [&](int x, int y, auto unroll) {
        constexpr int U = decltype(unroll)::value;
        double v[U] = {};
        for (int k = 0; k < t.n_source; ++k) {
          const PlaneSource& o = sources[t.source0 + k];
          const SI ys = y_is_a ? SI(o.a) : SI(o.b), xs = y_is_a ? SI(o.b) : SI(o.a);
          int64_t base;
          if (k < B::kSlots / batch) base = bt.src[k * batch + c];
          else base = source<SI>(t, o, locate<SI>(t, p0 + c - first[bt.task[c]]));
          const double* sp = src + base + (SI(x) * xs + SI(y) * ys);
          const SI ss = SI(y_step) * ys;
          const double coeff = o.coeff;
          double w[U];
#pragma unroll
          for (int u = 0; u < U; ++u) w[u] = __ldg(sp + SI(u) * ss);
#pragma unroll
          for (int u = 0; u < U; ++u) v[u] = fma(coeff, w[u], v[u]);
        }
        double* dp = into + (SI(x) * xd + SI(y) * yd);
#pragma unroll
        for (int u = 0; u < U; ++u) dp[SI(u) * sd] = v[u];
      };
      // whole fours, then one by one: a warp's FP64 instruction takes the pipe 64 cycles, also for lanes that are off
      for (int x = x0; x < x_end; x += x_step) {
        int y = y0;
        for (; y + (kUnroll - 1) * y_step < y_end; y += kUnroll * y_step) sum(x, y, std::integral_constant<int, kUnroll>{});
        for (; y < y_end; y += y_step) sum(x, y, std::integral_constant<int, 1>{});
      }
      if (kTranspose) {
        __syncwarp();
        const int sj = (l * t.ra) >> 16, fi = l - sj * t.la;
        if (sj < t.ia)
          for (int i = fi; i < ni; i += t.la)
            for (int j = sj; j < nj; j += t.ia) to[SI(i) * da + SI(j) * db] = tile[i * ld + j];
        __syncwarp();
      }
    }
    __syncthreads();
  }
}

template <int G, bool kTranspose, bool kSingle, typename SI>
void launch_form(const PlaneTask* d_tasks, const int64_t* d_start, int n_tasks, int64_t n_planes, int max_source,
                 const PlaneSource* d_sources, const double* src, double* dst, cudaStream_t s) {
  using B = Batch<kTranspose, kSingle>;
  const int sms = num_sms() > 0 ? num_sms() : 152;
  // batches: five or more for each resident block where there are chunks enough (a batch's decoding is a chain of
  // dependent loads), one chunk or more per group of lanes, and no larger than its slots
  const int64_t wanted = n_planes / (5 * int64_t(sms) * resident(kTranspose, kSingle));
  const int64_t most = std::max(1, std::min(B::kMost, B::kSlots / std::max(1, max_source)));
  const int batch = int(std::min(most, std::max<int64_t>(kThreads / G, wanted)));
  const unsigned blocks = unsigned(std::min<int64_t>((n_planes + batch - 1) / batch, int64_t(1) << 20));
  constexpr int bytes = kTranspose ? kWarps * kTileElems * int(sizeof(double)) : 0;
  if constexpr (kTranspose) {
    static PerDevice attr;
    attr.once([] {
      if (cudaFuncSetAttribute(permute_planes_kernel<G, kTranspose, kSingle, SI>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
        throw std::runtime_error("permute: shared memory not granted");
    });
  }
  permute_planes_kernel<G, kTranspose, kSingle, SI>
      <<<blocks, kThreads, bytes, s>>>(d_tasks, d_start, n_tasks, n_planes, batch, d_sources, src, dst);
  count_launch();
}

}  // namespace

void launch_permute(const PlaneTask* d_tasks, const int64_t* d_start, int n_tasks, int64_t n_planes, PlaneForm form,
                    const PlaneSource* d_sources, const double* src, double* dst, cudaStream_t s) {
  if (n_planes <= 0 || n_tasks <= 0) return;
  auto pick = [&](auto single) {
    constexpr bool kSingle = decltype(single)::value;
    // Tiles copied from a single source: 64-bit offsets make the copy loop plain pointer additions, and are the faster
    // from 4 M elements on (us, 32- / 64-bit offsets: 2.7 M elements 17.1 / 18.3, 7.3 M 40.4 / 35.9, 23 M 94 / 80,
    // 177 M 638 / 499); below, and for sums (34.5 / 37.8 at 2.6 M), decoding in 32 bits is.
    constexpr int64_t kWideFrom = 4 << 20;
    if (form.transpose) {
      if (form.narrow && (!kSingle || form.elems < kWideFrom)) return launch_form<32, true, kSingle, int32_t>;
      return launch_form<32, true, kSingle, int64_t>;
    }
    if (!form.narrow) return launch_form<32, false, kSingle, int64_t>;
    switch (form.group) {
      case 32: return launch_form<32, false, kSingle, int32_t>;
      case 16: return launch_form<16, false, kSingle, int32_t>;
      case 8: return launch_form<8, false, kSingle, int32_t>;
      default: return launch_form<4, false, kSingle, int32_t>;
    }
  };
  auto* launch = form.single ? pick(std::true_type{}) : pick(std::false_type{});
  launch(d_tasks, d_start, n_tasks, n_planes, form.max_source, d_sources, src, dst, s);
}

namespace {

// Planes of the output's two fast legs smaller than this take the longest of the other legs in place of the second: a
// plane costs its decoding, some 100 instructions, whatever it holds.  Measured (us, second leg / longest leg): [2, 5 M, 3]
// -> (0,2,1) 1680 / 203, twenty of [3, 200, 2, 200] -> (0,2,1,3) 56 / 38, a hundred of [2^5, 1000] -> (0,2,1,4,3,5) 62 /
// 51; planes of 36 ([6, 6, 200, 200] -> (0,1,3,2)) 42 either way.
constexpr int64_t kSmallPlane = 32;

// lanes x (of g) along a leg of extent n, r = g / x along one of extent m: few left over, runs not too short, that is
// the largest share of busy lanes, n m / (g ceil(n / x) ceil(m / r)), times x / (x + 8).  For each r only the largest x
// can be the best: ten candidates of 32.
int lanes_along(int g, int n, int m) {
  int best = 1;
  int64_t num = 0, den = 1;
  for (int x = std::min(g, n); x > 0;) {
    const int r = g / x;
    const int64_t d = int64_t(x + 8) * ((n + x - 1) / x) * ((m + r - 1) / r);
    if (x * den > num * d) {
      num = x;
      den = d;
      best = x;
    }
    x = g / (r + 1);
  }
  return best;
}

}  // namespace

PlanePlan plan_planes(const xgb_perm_task* tasks, int n_tasks, const xgb_perm_contrib* contribs) {
  PlanePlan plan;
  const int sms = num_sms() > 0 ? num_sms() : 152;
  double total = 0;
  size_t n_sources = 0;
  for (int t = 0; t < n_tasks; ++t) {
    total += double(tasks[t].nelem);
    n_sources += size_t(std::max(tasks[t].n_contrib, 0));
  }
  plan.tasks.reserve(size_t(n_tasks));
  plan.start.reserve(size_t(n_tasks) + 1);
  plan.sources.reserve(n_sources);
  // legs of each task: extent 1 dropped, ascending output stride, chained ones merged (`from`: the first leg of
  // the input that a merged leg begins with, whose strides are the merged leg's)
  struct Shape {
    int n = 0, leg[XGB_MAX_LEGS];
    int64_t dim[XGB_MAX_LEGS];
    int fast = -1;  // position of the source's unit-stride leg, -1: none (or not the same in all sources)
  };
  std::vector<Shape> shapes(static_cast<size_t>(n_tasks));
  double gain = 0;  // elements in tasks that the transposed form suits
  for (int t = 0; t < n_tasks; ++t) {
    const xgb_perm_task& k = tasks[t];
    Shape& sh = shapes[t];
    int order[XGB_MAX_LEGS], n = 0;
    for (int i = 0; i < k.rank; ++i)
      if (k.dims[i] != 1) order[n++] = i;
    for (int i = 1; i < n; ++i)  // by ascending output stride
      for (int j = i; j > 0 && k.dst_stride[order[j]] < k.dst_stride[order[j - 1]]; --j) std::swap(order[j], order[j - 1]);
    for (int i = 0; i < n; ++i) {
      const int leg = order[i];
      bool chain = sh.n > 0;
      if (chain) {
        const int prev = sh.leg[sh.n - 1];
        const int64_t len = sh.dim[sh.n - 1];
        chain = len * k.dims[leg] <= INT32_MAX && k.dst_stride[leg] == k.dst_stride[prev] * len;
        for (int c = 0; c < k.n_contrib && chain; ++c) {
          const xgb_perm_contrib& cc = contribs[k.contrib0 + c];
          chain = cc.src_stride[leg] == cc.src_stride[prev] * len;
        }
      }
      if (chain) {
        sh.dim[sh.n - 1] *= k.dims[leg];
      } else {
        sh.leg[sh.n] = leg;
        sh.dim[sh.n++] = k.dims[leg];
      }
    }
    for (int i = 0; i < sh.n; ++i) {
      bool unit = k.n_contrib > 0;
      for (int c = 0; c < k.n_contrib; ++c) unit = unit && contribs[k.contrib0 + c].src_stride[sh.leg[i]] == 1;
      if (unit) sh.fast = i;
    }
    if (sh.fast > 0 && sh.dim[0] >= 4 && sh.dim[sh.fast] >= 4 && sh.dim[0] * sh.dim[sh.fast] >= 64)
      gain += double(k.nelem);
  }
  // one form per plan: the legs move alike in all tasks, only short ones differ
  plan.form.transpose = gain > 0.5 * total;
  // chunks: enough of them for every SM's warps, at least four elements a lane and at most 2048 elements
  const int64_t chunk = std::min<int64_t>(2048, std::max<int64_t>(128, int64_t(total / (8.0 * sms))));
  const int64_t side = chunk >= 1024 ? 32 : 16;
  double elems = 0, weighted = 0;
  plan.start.assign(1, 0);
  for (int t = 0; t < n_tasks; ++t) {
    const xgb_perm_task& k = tasks[t];
    const Shape& sh = shapes[t];
    if (k.nelem <= 0) continue;
    // offsets inside the sub-block in 32 bits, with room for the lanes past a chunk's end
    auto narrow = [&](const int64_t* stride) {
      int64_t span = 0;
      for (int i = 0; i < k.rank; ++i) {
        if (k.dims[i] == 1) continue;  // such a leg is not walked
        if (std::abs(stride[i]) > INT32_MAX) return false;
        span += std::abs(stride[i]) * (int64_t(k.dims[i]) + 32 * kFlight);
      }
      return span <= INT32_MAX;
    };
    int b = sh.n < 2 ? -1 : plan.form.transpose && sh.fast > 0 ? sh.fast : 1;
    if (b == 1 && sh.dim[0] * sh.dim[1] < kSmallPlane)
      for (int i = 2; i < sh.n; ++i)
        if (sh.dim[i] > sh.dim[b]) b = i;
    PlaneTask& p = plan.tasks.emplace_back();
    p.dst_base = k.dst_base;
    p.na = sh.n > 0 ? int32_t(sh.dim[0]) : 1;
    p.nb = b > 0 ? int32_t(sh.dim[b]) : 1;
    p.dst_a = sh.n > 0 ? k.dst_stride[sh.leg[0]] : 0;
    p.dst_b = b > 0 ? k.dst_stride[sh.leg[b]] : 0;
    if (plan.form.transpose) {  // tiles about side/2 x side, a short side made up for by the other
      p.cj = int32_t(std::min<int64_t>(p.nb, std::max<int64_t>(side, side * side / 2 / std::min<int64_t>(p.na, side / 2))));
      p.ci = int32_t(std::min<int64_t>(p.na, std::max<int64_t>(side / 2, side / 2 * (side + 1) / (p.cj | 1))));
    } else {
      p.ci = int32_t(std::min<int64_t>(p.na, chunk));
      p.cj = int32_t(std::min<int64_t>(p.nb, std::max<int64_t>(1, chunk / p.ci)));
    }
    p.nci = (p.na + p.ci - 1) / p.ci;
    p.ncj = (p.nb + p.cj - 1) / p.cj;
    p.source0 = int32_t(plan.sources.size());
    p.n_source = k.n_contrib;
    int64_t planes = int64_t(p.nci) * p.ncj;
    for (int i = 1; i < sh.n; ++i) {
      if (i == b) continue;
      p.odim[p.n_outer] = int32_t(sh.dim[i]);
      p.odst[p.n_outer++] = k.dst_stride[sh.leg[i]];
      planes *= sh.dim[i];
    }
    if (planes > INT32_MAX) plan.form.narrow = false;
    for (int c = 0; c < k.n_contrib; ++c) {
      const xgb_perm_contrib& cc = contribs[k.contrib0 + c];
      PlaneSource& s = plan.sources.emplace_back();
      s.base = cc.src_base;
      s.coeff = cc.coeff;
      s.a = sh.n > 0 ? cc.src_stride[sh.leg[0]] : 0;
      s.b = b > 0 ? cc.src_stride[sh.leg[b]] : 0;
      int o = 0;
      for (int i = 1; i < sh.n; ++i)
        if (i != b) s.outer[o++] = cc.src_stride[sh.leg[i]];
      if (!narrow(cc.src_stride)) plan.form.narrow = false;
    }
    if (!narrow(k.dst_stride)) plan.form.narrow = false;
    plan.form.max_source = std::max(plan.form.max_source, k.n_contrib);
    if (k.n_contrib != 1) plan.form.single = false;
    const double size = double(p.ci) * double(p.cj);
    elems += double(k.nelem);
    weighted += double(k.nelem) * size;
    plan.start.push_back(plan.start.back() + planes);
  }
  plan.form.elems = int64_t(elems);
  // lanes per chunk: about four elements each or more
  const double avg = elems > 0 ? weighted / elems : 1.0;
  plan.form.group = plan.form.transpose || !plan.form.narrow || avg >= 96 ? 32 : avg >= 48 ? 16 : avg >= 24 ? 8 : 4;
  // A call waits for its plan: tasks whose chunks have extents seen before (a leg has few degeneracies) take the lanes
  // found then.  With this, ten candidates and no copies of the entries a task takes 90 ns instead of 570 (x86).
  struct Lanes { int32_t ci = 0, cj = 0, la = 0, lb = 0; };
  std::array<Lanes, 256> seen;
  for (PlaneTask& p : plan.tasks) {
    Lanes& f = seen[size_t(p.ci * 37 + p.cj) % seen.size()];
    if (f.ci != p.ci || f.cj != p.cj)
      f = {p.ci, p.cj, lanes_along(plan.form.group, p.ci, p.cj), lanes_along(plan.form.group, p.cj, p.ci)};
    p.la = int16_t(f.la);
    p.lb = int16_t(f.lb);
    p.ia = int16_t(plan.form.group / p.la);
    p.ib = int16_t(plan.form.group / p.lb);
    p.ra = 65536 / p.la + 1;  // l / la = l ra >> 16 for l < 32
    p.rb = 65536 / p.lb + 1;
    const int step_a = plan.form.transpose ? p.ib : p.la, step_b = plan.form.transpose ? p.lb : p.ia;
    p.y_is_a = p.ci * step_b > p.cj * step_a;
  }
  return plan;
}

void permute_planes_host(const PlanePlan& plan, const double* src, double* dst) {
  const int n = int(plan.tasks.size());
  for (int64_t p = 0; p < plan.start.back(); ++p) {
    const int at = task_of(plan.start.data(), n, p);
    const PlaneTask& t = plan.tasks[size_t(at)];
    const int64_t q = p - plan.start[size_t(at)];
    const Plane pl = plan.form.narrow ? locate<int32_t>(t, q) : locate<int64_t>(t, q);
    for (int j = 0; j < pl.nj; ++j)
      for (int i = 0; i < pl.ni; ++i) {
        double v = 0.0;
        for (int k = 0; k < t.n_source; ++k) {
          const PlaneSource& s = plan.sources[size_t(t.source0 + k)];
          v = std::fma(s.coeff, src[(plan.form.narrow ? source<int32_t>(t, s, pl) : source<int64_t>(t, s, pl)) + i * s.a + j * s.b], v);
        }
        dst[pl.dst + i * t.dst_a + j * t.dst_b] = v;
      }
  }
}

}  // namespace xgb
