// CUDA kernels of the GB300 block-sparse tensor backend (sm_103a) and the
// kernel-level C-ABI declared in include/xgb.h.
//
// Data layout: one flat column-major FP64 buffer per tensor, one block per
// coupled sector at a known element offset (the reference's contiguous
// storage, include/Xped/Core/storage/StorageType_contiguous.hpp:79-122).
// Every kernel processes all sectors of one tensor operation in a single
// launch driven by a descriptor table.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <map>
#include <mutex>
#include <stdexcept>
#include <thread>
#include <new>
#include <string>
#include <vector>

#include "kernels.hpp"

namespace xgb {

// ======================================================================= runtime
namespace {
struct Runtime {
  bool ready = false;
  int device = 0;
  int sms = 152;
  cudaStream_t stream = nullptr;  // lane 0
  double* scratch = nullptr;      // 64 doubles of device scratch per lane
  cudaStream_t side[kLanes - 1] = {nullptr, nullptr};
  double* side_scratch[kLanes - 1] = {nullptr, nullptr};
  cudaEvent_t fork_ev = nullptr, join_ev[kLanes - 1] = {nullptr, nullptr};
};
Runtime g_rt;
std::atomic<int64_t> g_launches{0};
std::atomic<bool> g_lanes_used{false};
thread_local std::string g_err;
thread_local int t_lane = 0;
thread_local cudaStream_t t_alloc = nullptr;  // stream of an AllocScope

// The worker host thread of lane 1: runs one task at a time, handed over under a mutex.
class LaneWorker {
 public:
  ~LaneWorker() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    if (th_.joinable()) th_.join();
  }
  void start(std::function<void()> f) {
    std::lock_guard<std::mutex> lk(mu_);
    if (!th_.joinable()) th_ = std::thread([this] { loop(); });
    task_ = std::move(f);
    err_ = nullptr;
    has_ = true;
    done_ = false;
    cv_.notify_all();
  }
  void wait() {
    std::unique_lock<std::mutex> lk(mu_);
    cv_.wait(lk, [this] { return done_; });
    if (err_) {
      std::exception_ptr e = err_;
      err_ = nullptr;
      std::rethrow_exception(e);
    }
  }

 private:
  void loop() {
    std::unique_lock<std::mutex> lk(mu_);
    for (;;) {
      cv_.wait(lk, [this] { return stop_ || has_; });
      if (stop_) return;
      std::function<void()> f = std::move(task_);
      has_ = false;
      lk.unlock();
      std::exception_ptr e;
      try {
        cudaSetDevice(g_rt.device);  // the current device is per host thread
        f();
      } catch (...) {
        e = std::current_exception();
      }
      lk.lock();
      err_ = e;
      done_ = true;
      cv_.notify_all();
    }
  }
  std::mutex mu_;
  std::condition_variable cv_;
  std::thread th_;
  std::function<void()> task_;
  std::exception_ptr err_;
  bool has_ = false, done_ = true, stop_ = false;
};

LaneWorker& lane_worker() {
  static LaneWorker w;
  return w;
}
std::mutex g_pair_mu;  // one fork-join section at a time
}  // namespace

cudaStream_t stream() { return t_lane == 0 ? g_rt.stream : g_rt.side[t_lane - 1]; }
int lane() { return t_lane; }
LaneScope::LaneScope(int l) : saved(t_lane) { t_lane = l; }
LaneScope::~LaneScope() { t_lane = saved; }
bool lanes_used() { return g_lanes_used.load(); }
bool runtime_ready() { return g_rt.ready; }
int num_sms() { return g_rt.sms; }
double* scalar_scratch() { return t_lane == 0 ? g_rt.scratch : g_rt.side_scratch[t_lane - 1]; }
void count_launch(int n) { g_launches += n; }

void run_pair(const std::function<void()>& a, const std::function<void()>& b) {
  if (t_lane != 0) throw std::runtime_error("run_pair: called from a side lane");
  std::lock_guard<std::mutex> lk(g_pair_mu);
  g_lanes_used = true;
  if (cudaEventRecord(g_rt.fork_ev, g_rt.stream) != cudaSuccess ||
      cudaStreamWaitEvent(g_rt.side[0], g_rt.fork_ev, 0) != cudaSuccess ||
      cudaStreamWaitEvent(g_rt.side[1], g_rt.fork_ev, 0) != cudaSuccess)
    throw std::runtime_error("run_pair: fork failed");
  LaneWorker& w = lane_worker();
  w.start([&a] {
    LaneScope ls(1);
    a();
  });
  std::exception_ptr eb, ea;
  try {
    LaneScope ls(2);
    b();
  } catch (...) {
    eb = std::current_exception();
  }
  try {
    w.wait();
  } catch (...) {
    ea = std::current_exception();
  }
  for (int i = 0; i < kLanes - 1; ++i) {
    cudaEventRecord(g_rt.join_ev[i], g_rt.side[i]);
    cudaStreamWaitEvent(g_rt.stream, g_rt.join_ev[i], 0);
  }
  if (ea) std::rethrow_exception(ea);
  if (eb) std::rethrow_exception(eb);
}

void order_after_lanes(cudaStream_t s) {
  for (int l = 0; l < kLanes; ++l) {
    cudaStream_t o = l == 0 ? g_rt.stream : g_rt.side[l - 1];
    if (o == s || !o) continue;
    cudaEvent_t e;
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) continue;
    cudaEventRecord(e, o);
    cudaStreamWaitEvent(s, e, 0);
    cudaEventDestroy(e);  // released once the wait has been satisfied
  }
}

int set_error(int code, const std::string& msg) {
  g_err = msg;
  return code;
}

int check_cuda(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return XGB_OK;
  return set_error(e == cudaErrorMemoryAllocation ? XGB_E_OOM : XGB_E_CUDA,
                   std::string(what) + ": " + cudaGetErrorString(e));
}

AllocScope::AllocScope(cudaStream_t s) : saved(t_alloc) { t_alloc = s; }
AllocScope::~AllocScope() { t_alloc = saved; }

void* dev_alloc(size_t bytes) {
  if (bytes == 0) bytes = 8;
  void* p = nullptr;
  cudaError_t e = cudaMallocAsync(&p, bytes, t_alloc ? t_alloc : stream());
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    set_error(XGB_E_OOM, std::string("cudaMallocAsync: ") + cudaGetErrorString(e));
    throw std::bad_alloc();
  }
  return p;
}

void dev_free(void* p) {
  if (p && g_rt.ready) cudaFreeAsync(p, t_alloc ? t_alloc : stream());
}

// ======================================================================= instrumentation
namespace {
struct ProfEvent {
  int kind;
  cudaEvent_t a, b;
  double work;
};
bool g_prof_on = false;
std::mutex g_prof_mu;
std::vector<ProfEvent> g_prof_events;
std::vector<cudaEvent_t> g_event_pool;
int64_t g_prof_launches[K_COUNT] = {0};
double g_prof_work[K_COUNT] = {0};
double g_prof_ms[K_COUNT] = {0};
cudaEvent_t g_pending_a[K_COUNT] = {nullptr};
cudaEvent_t g_user_events[16] = {nullptr};

cudaEvent_t pool_event() {
  if (!g_event_pool.empty()) {
    cudaEvent_t e = g_event_pool.back();
    g_event_pool.pop_back();
    return e;
  }
  cudaEvent_t e;
  cudaEventCreate(&e);
  return e;
}

void prof_drain() {
  for (auto& ev : g_prof_events) {
    float ms = 0.f;
    cudaEventSynchronize(ev.b);
    cudaEventElapsedTime(&ms, ev.a, ev.b);
    g_prof_ms[ev.kind] += ms;
    g_event_pool.push_back(ev.a);
    g_event_pool.push_back(ev.b);
  }
  g_prof_events.clear();
}
}  // namespace

bool profiling() { return g_prof_on; }

void prof_begin(int kind, cudaStream_t s) {
  if (!g_prof_on) return;
  g_pending_a[kind] = pool_event();
  cudaEventRecord(g_pending_a[kind], s);
}

void prof_end(int kind, cudaStream_t s, double work) {
  {
    std::lock_guard<std::mutex> lk(g_prof_mu);  // lanes count concurrently (profiling itself runs on lane 0)
    g_prof_launches[kind] += 1;
    g_prof_work[kind] += work;
  }
  if (!g_prof_on || !g_pending_a[kind]) return;
  cudaEvent_t b = pool_event();
  cudaEventRecord(b, s);
  g_prof_events.push_back({kind, g_pending_a[kind], b, work});
  g_pending_a[kind] = nullptr;
  if (g_prof_events.size() > 4096) prof_drain();
}

// ======================================================================= GEMM
// Grouped GEMM on the CUDA cores: C_g = alpha*op(A_g)op(B_g) + beta*C_g.  One
// CTA per TILE x TILE output tile of one group; 256 threads, each owning a
// (TILE/16)^2 micro-tile.  T = double is the FP64 form, bound by GB300's narrow
// FP64 pipe (two multiply-adds per clock and SM): it reaches 0.96 of that rate on
// nine blocks 36 to 616 wide (1013 us; 1399 us when edge tiles were multiplied
// whole and the tiles were 64 wide).  T = float is the FP32 form (operands
// rounded to FP32 as they are staged, FP32 accumulation, alpha/beta and the
// store in FP64).
// A warp owns 8 x 4 outputs of every 16 x 16 sub-block of the tile, and multiplies only the sub-blocks where some of
// its outputs lie inside the block: a warp's FP64 instruction takes the pipe 64 cycles whatever its active lanes, and
// predicated off as well, so the count of sub-blocks is a template argument of the inner loop.  An edge tile costs its
// extents rounded up to 8 x 4 instead of the whole tile (64-wide tiles on blocks 36 to 616 wide: 17 % of the time).
// Unrolled eight times so that the next operands are read ahead of the pipe: 1089 us without, 1010 with.
template <int R, int RM, int CM, int LD, typename T>
__device__ __forceinline__ void multiply(const T (*As)[LD], const T (*Bs)[LD], int kmax, int row, int col, T (*acc)[R]) {
#pragma unroll 8
  for (int kk = 0; kk < kmax; ++kk) {
    T a[RM], b[CM];
#pragma unroll
    for (int r = 0; r < RM; ++r) a[r] = As[kk][row + 16 * r];
#pragma unroll
    for (int c = 0; c < CM; ++c) b[c] = Bs[kk][col + 16 * c];
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
      for (int c = 0; c < CM; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
  }
}
template <int R, int RM, int LD, typename T>
__device__ __forceinline__ void multiply_cols(int cm, const T (*As)[LD], const T (*Bs)[LD], int kmax, int row, int col,
                                              T (*acc)[R]) {
  if (cm == 1) multiply<R, RM, 1, LD>(As, Bs, kmax, row, col, acc);
  if constexpr (R >= 2)
    if (cm == 2) multiply<R, RM, 2, LD>(As, Bs, kmax, row, col, acc);
  if constexpr (R >= 4) {
    if (cm == 3) multiply<R, RM, 3, LD>(As, Bs, kmax, row, col, acc);
    if (cm == 4) multiply<R, RM, 4, LD>(As, Bs, kmax, row, col, acc);
  }
}
template <int R, int LD, typename T>
__device__ __forceinline__ void multiply_live(int rm, int cm, const T (*As)[LD], const T (*Bs)[LD], int kmax, int row,
                                              int col, T (*acc)[R]) {
  if (rm == 1) multiply_cols<R, 1, LD>(cm, As, Bs, kmax, row, col, acc);
  if constexpr (R >= 2)
    if (rm == 2) multiply_cols<R, 2, LD>(cm, As, Bs, kmax, row, col, acc);
  if constexpr (R >= 4) {
    if (rm == 3) multiply_cols<R, 3, LD>(cm, As, Bs, kmax, row, col, acc);
    if (rm == 4) multiply_cols<R, 4, LD>(cm, As, Bs, kmax, row, col, acc);
  }
}

template <int TILE, typename T>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const xgb_gemm_desc* __restrict__ descs,
                                                        const GemmTile* __restrict__ tiles, const double* __restrict__ A,
                                                        const double* __restrict__ B, double* __restrict__ C,
                                                        double alpha, double beta, double* __restrict__ ws) {
  constexpr int BK = 16;
  constexpr int R = TILE / 16;
  constexpr int PER = TILE * BK / 256;  // staged elements of A (and of B) per thread and k step
  // two stages: the global loads of k step s + 1 are in flight (in registers) while step s is
  // multiplied out of shared memory, and one barrier per step separates the stages
  __shared__ T As[2][BK][TILE + 1];
  __shared__ T Bs[2][BK][TILE + 1];
  const GemmTile t = tiles[blockIdx.x];
  const xgb_gemm_desc d = descs[t.g];
  const int64_t kbeg = t.k0, kend = t.k1 < 0 ? d.k : t.k1;
  const int tid = threadIdx.x;
  const int64_t row0 = int64_t(t.tm) * TILE, col0 = int64_t(t.tn) * TILE;
  // FP64: warps w and w + 4 (one quarter of the SM) hold the two row halves of a column group; the groups rotate with
  // the tile so that the CTAs of an SM do not all have their fuller warps on the same quarter.  FP32 (not bound by its
  // pipe): 16 x 2 outputs of every sub-block, and all sub-blocks of a warp with any live output.
  constexpr bool kNarrowPipe = sizeof(T) == 8;
  const int warp = tid >> 5, lane = tid & 31;
  const int wrow = kNarrowPipe ? (warp >> 2) * 8 : 0;
  const int wcol = kNarrowPipe ? ((warp + int(blockIdx.x)) & 3) * 4 : warp * 2;
  const int tx = kNarrowPipe ? wrow + (lane & 7) : tid & 15;
  const int ty = kNarrowPipe ? wcol + (lane >> 3) : tid >> 4;
  const int64_t rows = d.m - row0 - wrow, cols = d.n - col0 - wcol;
  const int rm = rows <= 0 ? 0 : int(rows + 15 < TILE ? (rows + 15) / 16 : R);
  const int cm = cols <= 0 ? 0 : int(cols + 15 < TILE ? (cols + 15) / 16 : R);
  bool live = kNarrowPipe;
  if constexpr (!kNarrowPipe) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < R; ++c) live |= row0 + tx + 16 * r < d.m && col0 + ty + 16 * c < d.n;
  }
  const bool warp_live = __any_sync(0xffffffffu, live);
  T acc[R][R];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < R; ++j) acc[i][j] = T(0);

  T ra[PER], rb[PER];
  auto fetch = [&](int64_t k0) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = tid + 256 * u;
      int i, kk;
      if (d.trans_a) { kk = e % BK; i = e / BK; } else { i = e % TILE; kk = e / TILE; }
      const int64_t gi = row0 + i, gk = k0 + kk;
      double v = 0.0;
      if (gi < d.m && gk < kend) v = d.trans_a ? A[d.a_off + gk + gi * d.lda] : A[d.a_off + gi + gk * d.lda];
      ra[u] = T(v);
      int j, kb;
      if (d.trans_b) { j = e % TILE; kb = e / TILE; } else { kb = e % BK; j = e / BK; }
      const int64_t gj = col0 + j, gkb = k0 + kb;
      double w = 0.0;
      if (gj < d.n && gkb < kend) w = d.trans_b ? B[d.b_off + gj + gkb * d.ldb] : B[d.b_off + gkb + gj * d.ldb];
      rb[u] = T(w);
    }
  };
  auto stash = [&](int st) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = tid + 256 * u;
      int i, kk;
      if (d.trans_a) { kk = e % BK; i = e / BK; } else { i = e % TILE; kk = e / TILE; }
      As[st][kk][i] = ra[u];
      int j, kb;
      if (d.trans_b) { j = e % TILE; kb = e / TILE; } else { kb = e % BK; j = e / BK; }
      Bs[st][kb][j] = rb[u];
    }
  };
  if (kbeg < kend) {
    fetch(kbeg);
    stash(0);
  }
  __syncthreads();
  int st = 0;
  for (int64_t k0 = kbeg; k0 < kend; k0 += BK) {
    const bool more = k0 + BK < kend;
    if (more) fetch(k0 + BK);
    const int kmax = !kNarrowPipe && !warp_live ? 0 : (kend - k0) < BK ? int(kend - k0) : BK;
    if constexpr (kNarrowPipe) multiply_live<R, TILE + 1>(rm, cm, As[st], Bs[st], kmax, tx, ty, acc);
    else
      for (int kk = 0; kk < kmax; ++kk) {
        T a[R], b[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = As[st][kk][tx + 16 * r];
#pragma unroll
        for (int c = 0; c < R; ++c) b[c] = Bs[st][kk][ty + 16 * c];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < R; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
      }
    if (more) stash(st ^ 1);
    __syncthreads();
    st ^= 1;
  }
  if (t.slot >= 0) {  // split-K partial: the whole tile, raw sums, column-major TILE x TILE
    double* w = ws + int64_t(t.slot) * TILE * TILE;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < R; ++c) w[(tx + 16 * r) + (ty + 16 * c) * TILE] = double(acc[r][c]);
    return;
  }
  // FP64 operations go through GB300's narrow FP64 pipe: alpha = 1, beta = 0 stores the sums as they are
  const bool scaled = alpha != 1.0, accumulate = beta != 0.0;
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < R; ++c) {
      int64_t i = row0 + tx + 16 * r, j = col0 + ty + 16 * c;
      if (i < d.m && j < d.n) {
        double* p = C + d.c_off + i + j * d.ldc;
        double v = scaled ? alpha * double(acc[r][c]) : double(acc[r][c]);
        if (accumulate) v += beta * (*p);
        *p = v;
      }
    }
}

void launch_gemm_f64(const xgb_gemm_desc* d_descs, const GemmTile* d_tiles, int n_tiles, int tile, const double* A,
                     const double* B, double* C, double alpha, double beta, cudaStream_t s) {
  if (n_tiles <= 0) return;
  if (tile == 64) gemm_simt_kernel<64, double><<<n_tiles, 256, 0, s>>>(d_descs, d_tiles, A, B, C, alpha, beta, nullptr);
  else if (tile == 32) gemm_simt_kernel<32, double><<<n_tiles, 256, 0, s>>>(d_descs, d_tiles, A, B, C, alpha, beta, nullptr);
  else gemm_simt_kernel<16, double><<<n_tiles, 256, 0, s>>>(d_descs, d_tiles, A, B, C, alpha, beta, nullptr);
  count_launch();
}

// C tile = alpha * (sum of its partial slots in slot order) + beta * C: the result does not
// depend on which CTA finished first
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const xgb_gemm_desc* __restrict__ descs,
                                                            const SplitReduce* __restrict__ red, int tile,
                                                            const double* __restrict__ ws, double* __restrict__ C,
                                                            double alpha, double beta) {
  const SplitReduce r = red[blockIdx.x];
  const xgb_gemm_desc d = descs[r.g];
  const int64_t tt = int64_t(tile) * tile;
  for (int64_t e = threadIdx.x; e < tt; e += blockDim.x) {
    const int64_t i = int64_t(r.tm) * tile + e % tile, j = int64_t(r.tn) * tile + e / tile;
    if (i >= d.m || j >= d.n) continue;
    const double* part = ws + int64_t(r.first) * tt + e;
    double acc = part[0];
    for (int p = 1; p < r.count; p += 8) {  // eight loads in flight
      double x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (p + u < r.count) x[u] = __ldg(part + int64_t(p + u) * tt);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (p + u < r.count) acc += x[u];
    }
    double* c = C + d.c_off + i + j * d.ldc;
    double v = alpha == 1.0 ? acc : alpha * acc;
    if (beta != 0.0) v += beta * (*c);
    *c = v;
  }
}

void launch_gemm_f64_splitk(const xgb_gemm_desc* d_descs, const GemmTile* d_tiles, int n_tiles, int tile,
                            const SplitReduce* d_reduce, int n_reduce, const double* A, const double* B, double* C,
                            double* ws, double alpha, double beta, cudaStream_t s) {
  if (n_tiles <= 0) return;
  if (tile == 64) gemm_simt_kernel<64, double><<<n_tiles, 256, 0, s>>>(d_descs, d_tiles, A, B, C, alpha, beta, ws);
  else if (tile == 32) gemm_simt_kernel<32, double><<<n_tiles, 256, 0, s>>>(d_descs, d_tiles, A, B, C, alpha, beta, ws);
  else gemm_simt_kernel<16, double><<<n_tiles, 256, 0, s>>>(d_descs, d_tiles, A, B, C, alpha, beta, ws);
  count_launch();
  if (n_reduce <= 0) return;
  splitk_reduce_kernel<<<n_reduce, 256, 0, s>>>(d_descs, d_reduce, tile, ws, C, alpha, beta);
  count_launch();
}

void launch_gemm_f32(const xgb_gemm_desc* d_descs, const GemmTile* d_tiles, int n_tiles, int tile, const double* A,
                     const double* B, double* C, double alpha, double beta, cudaStream_t s) {
  if (n_tiles <= 0) return;
  if (tile == 64) gemm_simt_kernel<64, float><<<n_tiles, 256, 0, s>>>(d_descs, d_tiles, A, B, C, alpha, beta, nullptr);
  else if (tile == 32) gemm_simt_kernel<32, float><<<n_tiles, 256, 0, s>>>(d_descs, d_tiles, A, B, C, alpha, beta, nullptr);
  else gemm_simt_kernel<16, float><<<n_tiles, 256, 0, s>>>(d_descs, d_tiles, A, B, C, alpha, beta, nullptr);
  count_launch();
}

void order_tiles_by_work(std::vector<GemmTile>& tiles, const xgb_gemm_desc* descs) {
  // stable counting sort on the k extent, longest first: a list holds few distinct extents but up to
  // ~10^5 tiles, and the plans of a step whose shapes changed are built while the GPU waits
  auto extent = [&](const GemmTile& t) { return int64_t(t.k1 < 0 ? descs[t.g].k : t.k1) - t.k0; };
  std::map<int64_t, size_t, std::greater<int64_t>> slot;  // extent -> first position, descending
  for (const auto& t : tiles) ++slot[extent(t)];
  if (slot.size() <= 1) return;
  size_t off = 0;
  for (auto& [e, c] : slot) {
    const size_t n = c;
    c = off;
    off += n;
  }
  std::vector<GemmTile> out(tiles.size());
  int64_t last_e = -1;
  size_t* last_slot = nullptr;
  for (const auto& t : tiles) {
    const int64_t e = extent(t);
    if (e != last_e) {  // runs of equal extents are common: one map lookup per run
      last_slot = &slot.find(e)->second;
      last_e = e;
    }
    out[(*last_slot)++] = t;
  }
  tiles.swap(out);
}

int choose_gemm_tile(const xgb_gemm_desc* descs, int n) {
  // FP32 form: the largest tile edge that still yields >= 2 CTAs per SM (operand reuse, then SMs in use)
  const int target = 2 * (g_rt.sms > 0 ? g_rt.sms : 152);
  for (int tile : {64, 32}) {
    int64_t cnt = 0;
    for (int g = 0; g < n; ++g) cnt += ((descs[g].m + tile - 1) / tile) * ((descs[g].n + tile - 1) / tile);
    if (cnt >= target) return tile;
  }
  return 16;
}

int choose_f64_tile(const xgb_gemm_desc* descs, int n) {
  // The FP64 pipe is the bound, so what counts is that the SMs end together and that edges are not rounded up far:
  // 16-wide tiles are the fastest or within 1 % of it on every list measured from 20 to 1000 wide, with and without
  // split-K (us, 16 / 32 / 64 wide: nine blocks of 36 to 616 1010 / 1037 / 1159, nine of 9 to 154 31 / 49 / 166, one
  // of 1000 1657 / 1829 / 2024).  Lists of very many tiles take 32 (nine blocks of 72 to 1232, 18900 tiles: 7907 /
  // 7864 / 8379), which also keeps their tables short: they are built while the GPU waits.
  constexpr int64_t kMost = 16384;
  int64_t cnt = 0;
  for (int g = 0; g < n; ++g) cnt += ((descs[g].m + 15) / 16) * ((descs[g].n + 15) / 16);
  return cnt > kMost ? 32 : 16;
}

// ======================================================================= shared helpers
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ======================================================================= truncation
// cutoff_matrices on the device (src/Core/Tensor.cpp:523-633).  The global
// descending order of all singular values is made deterministic and robust
// to last-bit differences: values are ranked exactly (ties by position),
// consecutive values within kTieRtol (relative) form a tie group, and inside
// a group entries keep their (sector, index) position order.  Then: keep the
// first max_keep, drop values < eps, optionally cut the last multiplet, fall
// back to the first value of the first sector when nothing survives, and
// count kept values per sector.  One CTA; n is the number of singular values
// of one tensor (thousands at most).
//
// Bound by latency (one CTA, a few block barriers).  Everything lives in shared memory up to
// kTruncSmem values (a global workspace beyond), the ranks count 64-bit integer keys that order like
// the doubles (a double comparison occupies the narrow FP64 pipe), and the tie groups and the kept list
// come from block-wide prefix scans.  Measured on GB300 for one tSVD: 178 us with 324 values and 2.0 ms
// with 1414 when one thread walked the sorted list through global memory; 22 us and 123 us now.
constexpr double kTieRtol = 1.0e-12;
constexpr int kTruncThreads = 1024;
constexpr int64_t kTruncSmem = 8192;  // values held in shared memory: 24 bytes each (196,608 of 227 KB)

// A double as an unsigned integer of the same order; NaN lies below every number, -0.0 equals 0.0.
__device__ __forceinline__ unsigned long long order_key(double v) {
  if (v != v) return 0ull;
  const long long b = __double_as_longlong(v);
  if (b == (long long)0x8000000000000000ull) return 0x8000000000000000ull;
  return b < 0 ? ~(unsigned long long)b : (unsigned long long)b | 0x8000000000000000ull;
}

// Inclusive scans over the CTA's threads (sum / max); `part` holds one int per warp.
template <bool kMax>
__device__ __forceinline__ int block_scan(int v, int* part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v = kMax ? max(v, u) : v + u;
  }
  __syncthreads();  // part is free again (an earlier scan's readers are done)
  if (lane == 31) part[warp] = v;
  __syncthreads();
  if (warp == 0) {
    int w = part[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w = kMax ? max(w, u) : w + u;
    }
    part[lane] = w;
  }
  __syncthreads();
  if (warp > 0) v = kMax ? max(v, part[warp - 1]) : v + part[warp - 1];
  return v;
}

// `ws`: 3 * total 8-byte words, used when `in_smem` is 0.
__global__ void __launch_bounds__(kTruncThreads) truncate_kernel(int n_sectors, const int64_t* __restrict__ s_begin,
                                                                 const int32_t* __restrict__ deg,
                                                                 const double* __restrict__ s, int total,
                                                                 int64_t max_keep, double eps, int preserve,
                                                                 int32_t* __restrict__ keep, double* __restrict__ out2,
                                                                 unsigned long long* __restrict__ ws, int in_smem) {
  extern __shared__ unsigned long long trunc_sm[];
  __shared__ double red_w[32], red_e[32];
  __shared__ int part[32];
  __shared__ int kept_n;
  unsigned long long* base = in_smem ? trunc_sm : ws;
  unsigned long long* key = base;                     // key[i]: order of value i
  int* exact = reinterpret_cast<int*>(base + total);  // exact[r] = index with exact rank r; later the kept list
  int* gstart = exact + total;                        // first position of the tie group of each exact position
  int* order = gstart + total;                        // order[f] = index at final position f
  int* flag = order + total;                          // flag[i]: bit 0 kept, bit 1 counts as truncated weight
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = kTruncThreads;
  for (int g = tid; g < n_sectors; g += nt) keep[g] = 0;
  for (int i = tid; i < total; i += nt) {
    key[i] = order_key(s[i]);
    flag[i] = 0;
  }
  __syncthreads();
  // exact ranks under a total order (ties by index), so that `exact` is a permutation whatever the values are
  for (int i = tid; i < total; i += nt) {
    const unsigned long long ki = key[i];
    int r = 0;
#pragma unroll 8
    for (int j = 0; j < total; ++j) {
      const unsigned long long kj = key[j];
      r += (kj > ki) || (kj == ki && j < i);
    }
    exact[r] = i;
  }
  __syncthreads();
  // tie groups: a value more than kTieRtol below its predecessor opens one (running maximum of the openings)
  for (int p0 = 0, carry = 0; p0 < total; p0 += nt) {
    const int p = p0 + tid;
    int open = 0;
    if (p < total && p > 0) {
      const double prev = s[exact[p - 1]], cur = s[exact[p]];
      if (prev - cur > kTieRtol * prev) open = p;
    }
    const int g = max(carry, block_scan<true>(open, part));
    if (p < total) gstart[p] = g;
    carry = max(carry, part[31]);
  }
  __syncthreads();
  for (int p = tid; p < total; p += nt) {
    const int i = exact[p], g0 = gstart[p];
    int f = g0;
    for (int q = g0; q < total && gstart[q] == g0; ++q) f += (exact[q] < i);
    order[f] = i;
  }
  __syncthreads();
  const int lim = total < max_keep ? total : int(max_keep);
  // kept list in final order, stored compactly at the front of `exact`
  int nk = 0;
  for (int f0 = 0; f0 < lim; f0 += nt) {
    const int f = f0 + tid;
    const int i = f < lim ? order[f] : 0;
    const int on = f < lim && !(eps > 0.0 && s[i] < eps);
    const int at = nk + block_scan<false>(on, part);
    if (on) exact[at - 1] = i;
    nk += part[31];
  }
  __syncthreads();
  if (tid == 0) {
    if (preserve) {
      int end = -1;
      for (int k = nk - 1; k > 0; --k) {
        const double a = s[exact[k - 1]], b = s[exact[k]];
        if (2.0 * (a - b) / (a + b) > 0.1) { end = k; break; }
      }
      if (end != -1) nk = end;
    }
    if (nk == 0) { exact[0] = 0; nk = 1; }  // first entry: first value of the first sector
    kept_n = nk;
  }
  __syncthreads();
  nk = kept_n;
  for (int k = tid; k < nk; k += nt) flag[exact[k]] = 1;
  __syncthreads();
  // positions >= max_keep contribute to the truncated weight
  for (int f = max(lim, 0) + tid; f < total; f += nt) flag[order[f]] |= 2;
  __syncthreads();
  double wsum = 0.0, esum = 0.0;
  for (int i = tid; i < total; i += nt) {
    const int fl = flag[i];
    if (fl == 0) continue;
    int lo = 0, hi = n_sectors - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s_begin[mid] <= i) lo = mid; else hi = mid - 1;
    }
    const double v = s[i];
    if (fl & 2) wsum += deg[lo] * v * v;
    if (fl & 1) {
      atomicAdd(&keep[lo], 1);
      esum += -deg[lo] * v * v * log(v * v);
    }
  }
  wsum = warp_sum(wsum);
  esum = warp_sum(esum);
  if (lane == 0) { red_w[warp] = wsum; red_e[warp] = esum; }
  __syncthreads();
  if (tid == 0) {
    double a = 0, b = 0;
    for (int w = 0; w < nt / 32; ++w) { a += red_w[w]; b += red_e[w]; }
    out2[0] = a;
    out2[1] = b;
  }
}

void launch_truncate(int n_sectors, const int64_t* d_s_begin, const int32_t* d_deg, const double* s, int64_t total,
                     int64_t max_keep, double eps, int preserve, int32_t* keep, double* out2, cudaStream_t st) {
  if (total > INT32_MAX / 4) throw std::runtime_error("truncate: too many singular values");
  static PerDevice attr;
  attr.once([] {
    cudaFuncSetAttribute(truncate_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTruncSmem) * 24);
  });
  const bool in_smem = total <= kTruncSmem;
  const size_t bytes = size_t(std::max<int64_t>(total, 1)) * 24;
  auto* ws = in_smem ? nullptr : static_cast<unsigned long long*>(dev_alloc(bytes));
  truncate_kernel<<<1, kTruncThreads, in_smem ? bytes : 0, st>>>(n_sectors, d_s_begin, d_deg, s, int(total), max_keep,
                                                                 eps, preserve, keep, out2, ws, in_smem ? 1 : 0);
  count_launch();
  if (ws) dev_free(ws);
}

// ======================================================================= elementwise
__global__ void absmax_kernel(const double* __restrict__ x, int64_t n, unsigned long long* __restrict__ out) {
  double m = 0.0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    m = fmax(m, fabs(x[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  // non-negative doubles order like their bit patterns
  if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(out, __double_as_longlong(m));
}

void launch_absmax(const double* x, int64_t n, double* out, cudaStream_t s) {
  cudaMemsetAsync(out, 0, sizeof(double), s);
  if (n <= 0) return;
  int blocks = int(std::min<int64_t>((n + 255) / 256, int64_t(num_sms()) * 8));
  absmax_kernel<<<blocks, 256, 0, s>>>(x, n, reinterpret_cast<unsigned long long*>(out));
  count_launch();
}

__global__ void scale_by_inv_kernel(double* __restrict__ x, int64_t n, const double* __restrict__ m) {
  const double mv = *m;
  if (mv == 0.0) return;
  const double inv = 1.0 / mv;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) x[i] *= inv;
}

void launch_scale_by_inv(double* x, int64_t n, const double* m, cudaStream_t s) {
  if (n <= 0) return;
  int blocks = int(std::min<int64_t>((n + 255) / 256, int64_t(num_sms()) * 8));
  scale_by_inv_kernel<<<blocks, 256, 0, s>>>(x, n, m);
  count_launch();
}

__global__ void scale_kernel(double* __restrict__ x, int64_t n, double a) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) x[i] *= a;
}

void launch_scale(double* x, int64_t n, double alpha, cudaStream_t s) {
  if (n <= 0) return;
  int blocks = int(std::min<int64_t>((n + 255) / 256, int64_t(num_sms()) * 8));
  scale_kernel<<<blocks, 256, 0, s>>>(x, n, alpha);
  count_launch();
}

__global__ void copy2d_kernel(const xgb_copy2d_desc* __restrict__ descs, const double* __restrict__ src,
                              double* __restrict__ dst) {
  const xgb_copy2d_desc d = descs[blockIdx.y];
  const int64_t ne = d.rows * d.cols;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < ne; e += int64_t(gridDim.x) * blockDim.x) {
    int64_t i = e % d.rows, j = e / d.rows;
    dst[d.dst_off + i + j * d.dst_ld] = src[d.src_off + i + j * d.src_ld];
  }
}

void launch_copy2d(const xgb_copy2d_desc* d_descs, int n, int64_t max_elems, const double* src, double* dst, cudaStream_t s) {
  if (n <= 0 || max_elems <= 0) return;
  dim3 grid(unsigned(std::min<int64_t>((max_elems + 255) / 256, 1024)), unsigned(n));
  copy2d_kernel<<<grid, 256, 0, s>>>(d_descs, src, dst);
  count_launch();
}

__device__ __forceinline__ double diag_fn(int fn, double x) {
  switch (fn) {
    case XGB_DIAG_SQRT: return sqrt(x);
    case XGB_DIAG_INV: return 1.0 / x;
    default: return 1.0 / sqrt(x);
  }
}

__global__ void diag_from_vec_kernel(const xgb_copy2d_desc* __restrict__ descs, int fn, const double* __restrict__ src,
                                     double* __restrict__ dst) {
  const xgb_copy2d_desc d = descs[blockIdx.y];
  const int64_t k = d.rows;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < k * k; e += int64_t(gridDim.x) * blockDim.x) {
    int64_t i = e % k, j = e / k;
    dst[d.dst_off + e] = (i == j) ? (fn < 0 ? src[d.src_off + i] : diag_fn(fn, src[d.src_off + i])) : 0.0;
  }
}

void launch_diag_from_vec(const xgb_copy2d_desc* d_descs, int n, int64_t max_k, int fn, const double* src, double* dst,
                          cudaStream_t s) {
  if (n <= 0 || max_k <= 0) return;
  dim3 grid(unsigned(std::min<int64_t>((max_k * max_k + 255) / 256, 1024)), unsigned(n));
  diag_from_vec_kernel<<<grid, 256, 0, s>>>(d_descs, fn, src, dst);
  count_launch();
}

__global__ void diag_apply_kernel(const xgb_copy2d_desc* __restrict__ descs, int fn, double* __restrict__ x) {
  const xgb_copy2d_desc d = descs[blockIdx.y];
  const int64_t r = d.rows, c = d.cols;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < r * c; e += int64_t(gridDim.x) * blockDim.x) {
    int64_t i = e % r, j = e / r;
    double* p = x + d.dst_off + i + j * d.dst_ld;
    *p = (i == j) ? diag_fn(fn, *p) : 0.0;
  }
}

void launch_diag_apply(const xgb_copy2d_desc* d_descs, int n, int64_t max_k, int fn, double* x, cudaStream_t s) {
  if (n <= 0 || max_k <= 0) return;
  dim3 grid(unsigned(std::min<int64_t>((max_k * max_k + 255) / 256, 1024)), unsigned(n));
  diag_apply_kernel<<<grid, 256, 0, s>>>(d_descs, fn, x);
  count_launch();
}

// A Tensor<2,3> with a diagonal Tensor<1,1> on each of its first four legs: y = (((x wL) wT) wR) wB entry by entry, one
// warp per 256 entries of a fusion-tree pair's sub-block (found in the prefix sums of the pairs' chunks, so that the
// tables do not grow with the degeneracies).  Each weight costs one multiplication where contracting it
// takes a permute of the tensor to the leg, a product with the weight's blocks and a permute back (13 launches of small
// kernels instead of one; a D = 6 simple-update step 6.2 ms instead of 4.0).  Bound by launch and load latency for such
// tensors, by HBM for large ones.
__global__ void __launch_bounds__(256) leg_weights_kernel(const LegWeightTask* __restrict__ tasks, int n,
                                                          int64_t chunks, const int64_t* __restrict__ start,
                                                          LegWeights w, const double* __restrict__ x,
                                                          double* __restrict__ y) {
  constexpr int kHeld = 512;
  __shared__ int64_t start_s[kHeld];
  const bool held = n <= kHeld;
  if (held)
    for (int i = threadIdx.x; i < n; i += blockDim.x) start_s[i] = start[i];
  __syncthreads();
  const int64_t c = int64_t(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (c >= chunks) return;
  const int64_t* at = held ? start_s : start;
  int a = 0, b = n - 1;
  while (a < b) {
    const int mid = (a + b + 1) >> 1;
    if (at[mid] <= c) a = mid;
    else b = mid - 1;
  }
  const LegWeightTask& k = tasks[a];
  const int64_t first = (c - at[a]) * kLegWeightChunk;
  const int64_t last = first + kLegWeightChunk < k.entries ? first + kLegWeightChunk : k.entries;
  const int lane = threadIdx.x & 31;
  auto entries = [&](auto index) {  // 32-bit divisions where the sub-block's entries fit
    using Index = decltype(index);
    for (int64_t e = first + lane; e < last; e += 32) {
      Index r = Index(e);
      int64_t src = k.src, dst = k.dst;
      int i[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        const Index d = Index(k.dims[m]), next = r / d;
        i[m] = int(r - next * d);
        r = next;
        src += i[m] * k.src_stride[m];
        dst += i[m] * k.dst_stride[m];
      }
      double v = x[src];
#pragma unroll
      for (int m = 0; m < 4; ++m) v *= w.data[m][k.weight[m] + i[m] * k.weight_step[m]];
      y[dst] = v;
    }
  };
  if (k.entries <= INT32_MAX) entries(uint32_t(0));
  else entries(uint64_t(0));
}

void launch_leg_weights(const LegWeightTask* d_tasks, const int64_t* d_start, int n, int64_t chunks, const LegWeights& w,
                        const double* x, double* y, cudaStream_t s) {
  if (n <= 0 || chunks <= 0) return;
  leg_weights_kernel<<<unsigned((chunks + 7) / 8), 256, 0, s>>>(d_tasks, n, chunks, d_start, w, x, y);
  count_launch();
}

// ======================================================================= C-ABI helpers
namespace {
template <class T>
T* upload(const T* host, size_t n, cudaStream_t s) {
  T* d = static_cast<T*>(dev_alloc(sizeof(T) * std::max<size_t>(n, 1)));
  if (n) cudaMemcpyAsync(d, host, sizeof(T) * n, cudaMemcpyHostToDevice, s);
  return d;
}
cudaStream_t pick(void* s) { return s ? static_cast<cudaStream_t>(s) : g_rt.stream; }
#define XGB_REQUIRE_INIT() \
  if (!g_rt.ready) return set_error(XGB_E_NOINIT, "xgb_init was not called")
#define XGB_GUARD_BEGIN try {
#define XGB_GUARD_END                                                         \
  }                                                                           \
  catch (const std::bad_alloc&) {                                             \
    return XGB_E_OOM;                                                         \
  }                                                                           \
  catch (const std::exception& ex) {                                          \
    return set_error(XGB_E_BADPLAN, ex.what());                               \
  }
}  // namespace

}  // namespace xgb

using namespace xgb;

extern "C" {

int xgb_init(int device) {
  if (g_rt.ready) return XGB_OK;
  int rc = check_cuda(cudaSetDevice(device), "cudaSetDevice");
  if (rc) return rc;
  cudaDeviceProp prop{};
  if ((rc = check_cuda(cudaGetDeviceProperties(&prop, device), "cudaGetDeviceProperties"))) return rc;
  g_rt.sms = prop.multiProcessorCount;
  g_rt.device = device;
  if ((rc = check_cuda(cudaStreamCreateWithFlags(&g_rt.stream, cudaStreamNonBlocking), "cudaStreamCreate"))) return rc;
  for (int i = 0; i < kLanes - 1; ++i) {
    if ((rc = check_cuda(cudaStreamCreateWithFlags(&g_rt.side[i], cudaStreamNonBlocking), "cudaStreamCreate"))) return rc;
    if ((rc = check_cuda(cudaMalloc(&g_rt.side_scratch[i], 64 * sizeof(double)), "cudaMalloc scratch"))) return rc;
    if ((rc = check_cuda(cudaEventCreateWithFlags(&g_rt.join_ev[i], cudaEventDisableTiming), "cudaEventCreate")))
      return rc;
  }
  if ((rc = check_cuda(cudaEventCreateWithFlags(&g_rt.fork_ev, cudaEventDisableTiming), "cudaEventCreate"))) return rc;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
    uint64_t thr = ~0ull;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    // memory freed on one lane is not handed to another lane's allocation behind an inserted wait
    // (that would serialise the lanes); it is reused there once its free has completed
    int no = 0;
    cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &no);
  }
  if ((rc = check_cuda(cudaMalloc(&g_rt.scratch, 64 * sizeof(double)), "cudaMalloc scratch"))) return rc;
  g_rt.ready = true;
  return XGB_OK;
}

int xgb_shutdown(void) {
  if (!g_rt.ready) return XGB_OK;
  cudaStreamSynchronize(g_rt.stream);
  for (int i = 0; i < kLanes - 1; ++i) {
    cudaStreamSynchronize(g_rt.side[i]);
    cudaFree(g_rt.side_scratch[i]);
    cudaStreamDestroy(g_rt.side[i]);
    cudaEventDestroy(g_rt.join_ev[i]);
  }
  cudaEventDestroy(g_rt.fork_ev);
  cudaFree(g_rt.scratch);
  cudaStreamDestroy(g_rt.stream);
  g_rt = Runtime{};
  g_lanes_used = false;
  return XGB_OK;
}

const char* xgb_last_error(void) { return g_err.c_str(); }

int xgb_synchronize(void) {
  XGB_REQUIRE_INIT();
  return check_cuda(cudaStreamSynchronize(g_rt.stream), "cudaStreamSynchronize");
}

int64_t xgb_launch_count(void) { return g_launches.load(); }

int xgb_profile_enable(int on) {
  XGB_REQUIRE_INIT();
  if (!on) prof_drain();
  g_prof_on = on != 0;
  return XGB_OK;
}

int xgb_profile_reset(void) {
  XGB_REQUIRE_INIT();
  cudaStreamSynchronize(g_rt.stream);
  prof_drain();
  for (int k = 0; k < K_COUNT; ++k) { g_prof_launches[k] = 0; g_prof_work[k] = 0; g_prof_ms[k] = 0; }
  return XGB_OK;
}

int xgb_profile_read(int kind, int64_t* launches, double* ms, double* work) {
  XGB_REQUIRE_INIT();
  if (kind < 0 || kind >= K_COUNT) return set_error(XGB_E_BADPLAN, "kernel kind out of range");
  cudaStreamSynchronize(g_rt.stream);
  prof_drain();
  *launches = g_prof_launches[kind];
  *ms = g_prof_ms[kind];
  *work = g_prof_work[kind];
  return XGB_OK;
}

int xgb_event_record(int slot) {
  XGB_REQUIRE_INIT();
  if (slot < 0 || slot >= 16) return set_error(XGB_E_BADPLAN, "event slot out of range");
  if (!g_user_events[slot]) cudaEventCreate(&g_user_events[slot]);
  return check_cuda(cudaEventRecord(g_user_events[slot], g_rt.stream), "cudaEventRecord");
}

double xgb_event_elapsed_ms(int a, int b) {
  if (a < 0 || a >= 16 || b < 0 || b >= 16 || !g_user_events[a] || !g_user_events[b]) return -1.0;
  cudaEventSynchronize(g_user_events[b]);
  float ms = -1.f;
  if (cudaEventElapsedTime(&ms, g_user_events[a], g_user_events[b]) != cudaSuccess) return -1.0;
  return ms;
}

void* xgb_stream_handle(void) { return g_rt.stream; }

int xgb_malloc(void** ptr, size_t bytes) {
  XGB_REQUIRE_INIT();
  return check_cuda(cudaMalloc(ptr, bytes ? bytes : 8), "cudaMalloc");
}
int xgb_free(void* ptr) {
  XGB_REQUIRE_INIT();
  cudaStreamSynchronize(g_rt.stream);
  return check_cuda(cudaFree(ptr), "cudaFree");
}
int xgb_memcpy_h2d(void* dst, const void* src, size_t bytes) {
  XGB_REQUIRE_INIT();
  int rc = check_cuda(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, g_rt.stream), "h2d");
  if (rc) return rc;
  return check_cuda(cudaStreamSynchronize(g_rt.stream), "h2d sync");
}
int xgb_memcpy_d2h(void* dst, const void* src, size_t bytes) {
  XGB_REQUIRE_INIT();
  int rc = check_cuda(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, g_rt.stream), "d2h");
  if (rc) return rc;
  return check_cuda(cudaStreamSynchronize(g_rt.stream), "d2h sync");
}
int xgb_memset_zero(void* dst, size_t bytes) {
  XGB_REQUIRE_INIT();
  return check_cuda(cudaMemsetAsync(dst, 0, bytes, g_rt.stream), "memset");
}

int xgb_grouped_gemm(int precision, int n_groups, const xgb_gemm_desc* descs, const double* A, const double* B,
                     double* C, double alpha, double beta, void* stream_) {
  XGB_REQUIRE_INIT();
  if (!gemm_precision_available(precision))
    return set_error(XGB_E_UNSUPPORTED, "precision form not available through this entry");
  if (n_groups < 0) return set_error(XGB_E_BADPLAN, "n_groups < 0");
  XGB_GUARD_BEGIN
  cudaStream_t s = pick(stream_);
  AllocScope alloc(s);
  for (int g = 0; g < n_groups; ++g)
    if (descs[g].m < 0 || descs[g].n < 0 || descs[g].k < 0) return set_error(XGB_E_BADPLAN, "negative GEMM extent");
  if (precision == XGB_PREC_F64TC) {
    OzPlanHost op = build_oz_plan(descs, n_groups);
    if (op.tiles.empty()) return XGB_OK;
    double flops = 0;
    for (int g = 0; g < n_groups; ++g) flops += 2.0 * double(descs[g].m) * double(descs[g].n) * double(descs[g].k);
    auto* dd = upload(descs, size_t(n_groups), s);
    auto* dg = upload(op.groups.data(), op.groups.size(), s);
    auto* dk = upload(op.tasks.data(), op.tasks.size(), s);
    auto* dt = upload(op.tiles.data(), op.tiles.size(), s);
    auto* dr = upload(op.red.data(), op.red.size(), s);
    auto* rm = static_cast<unsigned long long*>(dev_alloc(sizeof(unsigned long long) * size_t(std::max<int64_t>(op.rowmax, 1))));
    auto* ap = static_cast<unsigned char*>(dev_alloc(size_t(std::max<int64_t>(op.a_bytes, 16))));
    auto* bp = static_cast<unsigned char*>(dev_alloc(size_t(std::max<int64_t>(op.b_bytes, 16))));
    prof_begin(K_GEMM_OZ, s);
    launch_gemm_oz(dd, dg, dk, int(op.tasks.size()), op.pack_cluster, dt, int(op.tiles.size()), dr, int(op.red.size()), op.slots, A, B,
                   rm, ap, bp, C, alpha, beta, s);
    prof_end(K_GEMM_OZ, s, flops);
    for (void* p : {static_cast<void*>(dd), static_cast<void*>(dg), static_cast<void*>(dk), static_cast<void*>(dt),
                    static_cast<void*>(dr), static_cast<void*>(rm), static_cast<void*>(ap), static_cast<void*>(bp)})
      dev_free(p);
    return check_cuda(cudaGetLastError(), "f64tc gemm launch");
  }
  if (precision == XGB_PREC_3XTF32 || precision == XGB_PREC_BF16X9) {
    const int form = precision == XGB_PREC_BF16X9 ? 1 : 0;
    TcPlanHost tp = build_tc_plan(descs, n_groups, form);
    if (tp.tiles.empty()) return XGB_OK;
    double flops = 0;
    for (int g = 0; g < n_groups; ++g) flops += 2.0 * double(descs[g].m) * double(descs[g].n) * double(descs[g].k);
    auto* dd = upload(descs, size_t(n_groups), s);
    auto* dg = upload(tp.groups.data(), tp.groups.size(), s);
    auto* dk = upload(tp.tasks.data(), tp.tasks.size(), s);
    auto* dt = upload(tp.tiles.data(), tp.tiles.size(), s);
    auto* ap = static_cast<float*>(dev_alloc(sizeof(float) * size_t(std::max<int64_t>(tp.a_floats, 4))));
    auto* bp = static_cast<float*>(dev_alloc(sizeof(float) * size_t(std::max<int64_t>(tp.b_floats, 4))));
    prof_begin(K_GEMM_TC, s);
    launch_gemm_tc(dd, dg, dk, int(tp.tasks.size()), dt, int(tp.tiles.size()), A, B, ap, bp, C, alpha, beta, s, form);
    prof_end(K_GEMM_TC, s, flops);
    for (void* p : {static_cast<void*>(dd), static_cast<void*>(dg), static_cast<void*>(dk), static_cast<void*>(dt),
                    static_cast<void*>(ap), static_cast<void*>(bp)})
      dev_free(p);
    return check_cuda(cudaGetLastError(), "tensor-core gemm launch");
  }
  if (precision == XGB_PREC_FP64) {
    // FP64: the built-in shape (no split-K) or, with autotuning on, the tuned one of the list's bucket
    const F64Config cfg = gemm_f64_config(descs, n_groups, A, B, {choose_f64_tile(descs, n_groups), 0}, s);
    run_gemm_f64_config(descs, n_groups, cfg, A, B, C, alpha, beta, s);
    return check_cuda(cudaGetLastError(), "gemm launch");
  }
  const int tile = choose_gemm_tile(descs, n_groups);
  std::vector<GemmTile> tiles;
  for (int g = 0; g < n_groups; ++g) {
    int64_t tm = (descs[g].m + tile - 1) / tile, tn = (descs[g].n + tile - 1) / tile;
    for (int64_t j = 0; j < tn; ++j)
      for (int64_t i = 0; i < tm; ++i) tiles.push_back({g, int32_t(i), int32_t(j), tile});
  }
  if (tiles.empty()) return XGB_OK;
  order_tiles_by_work(tiles, descs);
  auto* dd = upload(descs, size_t(n_groups), s);
  auto* dt = upload(tiles.data(), tiles.size(), s);
  double flops = 0;  // XGB_PREC_FP32 (the other forms returned above)
  for (int g = 0; g < n_groups; ++g) flops += 2.0 * double(descs[g].m) * double(descs[g].n) * double(descs[g].k);
  prof_begin(K_GEMM_F32, s);
  launch_gemm_f32(dd, dt, int(tiles.size()), tile, A, B, C, alpha, beta, s);
  prof_end(K_GEMM_F32, s, flops);
  dev_free(dd);
  dev_free(dt);
  return check_cuda(cudaGetLastError(), "gemm launch");
  XGB_GUARD_END
}

int xgb_gemm_tc_status(void) {
  XGB_REQUIRE_INIT();
  XGB_GUARD_BEGIN
  cudaStreamSynchronize(stream());
  return gemm_tc_error(true) ? set_error(XGB_E_TIMEOUT, "tensor-core GEMM: a CTA gave up waiting for its MMAs") : XGB_OK;
  XGB_GUARD_END
}

static int check_permute(int n_tasks, const xgb_perm_task* tasks, int n_contrib) {
  for (int t = 0; t < n_tasks; ++t) {
    if (tasks[t].rank < 0 || tasks[t].rank > XGB_MAX_LEGS) return set_error(XGB_E_BADPLAN, "task rank out of range");
    if (tasks[t].contrib0 < 0 || tasks[t].contrib0 + tasks[t].n_contrib > n_contrib)
      return set_error(XGB_E_BADPLAN, "contribution index out of range");
    int64_t prod = 1;
    for (int k = 0; k < tasks[t].rank; ++k) {
      if (tasks[t].dims[k] <= 0) return set_error(XGB_E_BADPLAN, "task extent must be positive");
      prod *= tasks[t].dims[k];
    }
    if (prod != tasks[t].nelem) return set_error(XGB_E_BADPLAN, "task nelem differs from the product of its extents");
  }
  return XGB_OK;
}

int xgb_permute(int n_tasks, const xgb_perm_task* tasks, int n_contrib, const xgb_perm_contrib* contribs,
                const double* src, double* dst, void* stream_) {
  XGB_REQUIRE_INIT();
  XGB_GUARD_BEGIN
  cudaStream_t s = pick(stream_);
  AllocScope alloc(s);
  if (const int rc = check_permute(n_tasks, tasks, n_contrib)) return rc;
  const PlanePlan plan = plan_planes(tasks, n_tasks, contribs);
  if (plan.start.back() == 0) return XGB_OK;
  auto* dt = upload(plan.tasks.data(), plan.tasks.size(), s);
  auto* ds = upload(plan.start.data(), plan.start.size(), s);
  auto* dc = upload(plan.sources.data(), plan.sources.size(), s);
  launch_permute(dt, ds, int(plan.tasks.size()), plan.start.back(), plan.form, dc, src, dst, s);
  dev_free(dt);
  dev_free(ds);
  dev_free(dc);
  return check_cuda(cudaGetLastError(), "permute launch");
  XGB_GUARD_END
}

int xgb_permute_walk_host(int n_tasks, const xgb_perm_task* tasks, int n_contrib, const xgb_perm_contrib* contribs,
                          const double* src, double* dst, int* transposed) {
  XGB_GUARD_BEGIN
  if (const int rc = check_permute(n_tasks, tasks, n_contrib)) return rc;
  const PlanePlan plan = plan_planes(tasks, n_tasks, contribs);
  permute_planes_host(plan, src, dst);
  if (transposed) *transposed = plan.form.transpose;
  return XGB_OK;
  XGB_GUARD_END
}

size_t xgb_svd_workspace_bytes(int n, const xgb_svd_desc* descs) {
  size_t e = 0;
  for (int i = 0; i < n; ++i) e += svd_work_elems(descs[i].m, descs[i].n);
  return e * sizeof(double);
}

int xgb_batched_svd(int n, const xgb_svd_desc* descs, const double* A, double* U, double* S, double* Vt, void* work,
                    void* stream_) {
  XGB_REQUIRE_INIT();
  XGB_GUARD_BEGIN
  cudaStream_t s = pick(stream_);
  AllocScope alloc(s);
  std::vector<int64_t> off(size_t(std::max(n, 0)), 0);
  int64_t acc = 0, maxk = 0;
  for (int i = 0; i < n; ++i) {
    if (descs[i].m < 0 || descs[i].n < 0) return set_error(XGB_E_BADPLAN, "negative SVD extent");
    off[i] = acc;
    acc += int64_t(svd_work_elems(descs[i].m, descs[i].n));
    maxk = std::max(maxk, std::min(descs[i].m, descs[i].n));
  }
  if (maxk > 8192) return set_error(XGB_E_UNSUPPORTED, "SVD block larger than 8192 columns");
  if (n == 0) return XGB_OK;
  auto* dd = upload(descs, size_t(n), s);
  auto* dof = upload(off.data(), off.size(), s);
  launch_svd(dd, descs, dof, n, A, U, S, Vt, static_cast<double*>(work), s);
  dev_free(dd);
  dev_free(dof);
  return check_cuda(cudaGetLastError(), "svd launch");
  XGB_GUARD_END
}

int xgb_truncate(int n_sectors, const int64_t* s_begin_host, const int32_t* degeneracy_host, const double* s,
                 int64_t max_keep, double eps_svd, int preserve_multiplets, int32_t* keep_dev, double* out2_dev,
                 void* stream_) {
  XGB_REQUIRE_INIT();
  XGB_GUARD_BEGIN
  if (n_sectors <= 0) return set_error(XGB_E_BADPLAN, "truncation needs at least one sector");
  cudaStream_t st = pick(stream_);
  AllocScope alloc(st);
  const int64_t total = s_begin_host[n_sectors];
  if (total <= 0) return set_error(XGB_E_BADPLAN, "no singular values");
  auto* db = upload(s_begin_host, size_t(n_sectors) + 1, st);
  auto* dg = upload(degeneracy_host, size_t(n_sectors), st);
  launch_truncate(n_sectors, db, dg, s, total, max_keep, eps_svd, preserve_multiplets, keep_dev, out2_dev, st);
  dev_free(db);
  dev_free(dg);
  return check_cuda(cudaGetLastError(), "truncate launch");
  XGB_GUARD_END
}

size_t xgb_qr_workspace_bytes(int n, const xgb_qr_desc* descs) {
  size_t e = 0;
  for (int i = 0; i < n; ++i) e += qr_work_elems(descs[i].m, descs[i].n);
  return e * sizeof(double);
}

int xgb_batched_qr(int n, const xgb_qr_desc* descs, const double* A, double* Q, double* R, void* work, void* stream_) {
  XGB_REQUIRE_INIT();
  XGB_GUARD_BEGIN
  cudaStream_t s = pick(stream_);
  AllocScope alloc(s);
  std::vector<int64_t> off(size_t(std::max(n, 0)), 0);
  int64_t acc = 0;
  for (int i = 0; i < n; ++i) {
    off[i] = acc;
    acc += int64_t(qr_work_elems(descs[i].m, descs[i].n));
  }
  if (n == 0) return XGB_OK;
  auto* dd = upload(descs, size_t(n), s);
  auto* dof = upload(off.data(), off.size(), s);
  launch_qr(dd, descs, dof, n, A, Q, R, static_cast<double*>(work), s);
  dev_free(dd);
  dev_free(dof);
  return check_cuda(cudaGetLastError(), "qr launch");
  XGB_GUARD_END
}

int xgb_absmax(const double* x, int64_t n, double* out_dev, void* stream_) {
  XGB_REQUIRE_INIT();
  launch_absmax(x, n, out_dev, pick(stream_));
  return check_cuda(cudaGetLastError(), "absmax launch");
}

int xgb_scale_by_inv_absmax(double* x, int64_t n, double* scratch_dev, void* stream_) {
  XGB_REQUIRE_INIT();
  cudaStream_t s = pick(stream_);
  launch_absmax(x, n, scratch_dev, s);
  launch_scale_by_inv(x, n, scratch_dev, s);
  return check_cuda(cudaGetLastError(), "scale launch");
}

int xgb_scale(double* x, int64_t n, double alpha, void* stream_) {
  XGB_REQUIRE_INIT();
  launch_scale(x, n, alpha, pick(stream_));
  return check_cuda(cudaGetLastError(), "scale launch");
}

int xgb_copy2d_batched(int n, const xgb_copy2d_desc* descs, const double* src, double* dst, void* stream_) {
  XGB_REQUIRE_INIT();
  XGB_GUARD_BEGIN
  if (n <= 0) return XGB_OK;
  cudaStream_t s = pick(stream_);
  AllocScope alloc(s);
  int64_t mx = 0;
  for (int i = 0; i < n; ++i) mx = std::max(mx, descs[i].rows * descs[i].cols);
  auto* dd = upload(descs, size_t(n), s);
  launch_copy2d(dd, n, mx, src, dst, s);
  dev_free(dd);
  return check_cuda(cudaGetLastError(), "copy2d launch");
  XGB_GUARD_END
}

int xgb_diag_from_vec(int n, const xgb_copy2d_desc* descs, int fn, const double* src, double* dst, void* stream_) {
  XGB_REQUIRE_INIT();
  XGB_GUARD_BEGIN
  if (n <= 0) return XGB_OK;
  cudaStream_t s = pick(stream_);
  AllocScope alloc(s);
  int64_t mx = 0;
  for (int i = 0; i < n; ++i) mx = std::max(mx, descs[i].rows);
  auto* dd = upload(descs, size_t(n), s);
  launch_diag_from_vec(dd, n, mx, fn, src, dst, s);
  dev_free(dd);
  return check_cuda(cudaGetLastError(), "diag launch");
  XGB_GUARD_END
}

int xgb_diag_apply(int n, const xgb_copy2d_desc* descs, int fn, double* x, void* stream_) {
  XGB_REQUIRE_INIT();
  XGB_GUARD_BEGIN
  if (n <= 0) return XGB_OK;
  cudaStream_t s = pick(stream_);
  AllocScope alloc(s);
  int64_t mx = 0;
  for (int i = 0; i < n; ++i) mx = std::max(mx, std::max(descs[i].rows, descs[i].cols));
  auto* dd = upload(descs, size_t(n), s);
  launch_diag_apply(dd, n, mx, fn, x, s);
  dev_free(dd);
  return check_cuda(cudaGetLastError(), "diag launch");
  XGB_GUARD_END
}

}  // extern "C"
