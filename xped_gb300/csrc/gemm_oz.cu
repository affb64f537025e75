// FP64-accurate grouped GEMM on the 5th-generation tensor cores from exact BF16 slices.
//
// C_g = alpha op(A_g) op(B_g) + beta C_g for FP64 column-major blocks.  Every row i of op(A) is
// written relative to a power of two 2^e_i above its largest entry (taken over the whole k range)
// and cut into seven balanced base-128 digits, a_ik = 2^e_i (sum_s m_s 2^(-7 s) + O(2^-50)) with
// integers |m_1| <= 128 and |m_s| <= 64 for s >= 2; every column of op(B) likewise (2^f_j).  A slice
// m_s 2^(-7 s) is exact in BF16, the product of two slices is exact in FP32, and all products of a
// "level" L = s + t share the unit 2^(-7 L).  Per k value a level adds at most 2 x 128 x 64 + 5 x 64 x 64
// = 36864 units, so a sum over 448 k values (28 K slices) stays below 2^24 and is exact in the FP32
// tensor-memory accumulator whatever order the tensor core adds in.  The row and column scales
// 2^(e_i + f_j) go into the exponent field when the tile is stored.  This is the slicing scheme of
// Ozaki, Ogita, Oishi and Rump ("Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication and its applications", Numer. Algorithms 59 (2012)), with BF16
// tcgen05.mma as the fast routine.
//
// GB300 runs FP64 arithmetic at a small fraction of its FP32 and tensor rates, so nothing here
// computes in FP64 but the one addition that joins the two FP32 halves of a result: the row
// maxima, scales and slices are integer operations on the IEEE bits.
//
// Kernels (one launch each, all groups of the list):
//  * oz_pack_kernel: the row scales, and the seven slices of every entry as BF16 in the K-major,
//    unswizzled canonical layout the MMA reads (8-row x 16-byte core matrices), zero padded past the
//    block edges; the slices come from integer arithmetic on the FP64 significand (|x| rounded to 49
//    bits below the row's scale, balanced digits, every slice with the sign of its entry);
//  * oz_gemm_kernel: one CTA (18 warps) per 128 x 64 output tile and K range.  Warp 16 streams the
//    slices of each 16-wide K slice of the tile's rows and columns into a 5-stage shared-memory ring
//    (42 KB per stage, bulk copies counted on mbarriers); warp 17 issues, per K slice, the 28
//    BF16 MMAs of the slice pairs with s + t <= 8 into seven 64-column TMEM accumulators (one per
//    level, 448 of 512 columns); after every 28 K slices (the exactness bound) and at the end of the
//    range warps 0-15 read the seven levels and add them into double-FP32 (hi + lo) register sums, two
//    values per instruction, and the next chunk starts from zero on the levels that have been read.
//    The slice rounding (2^-50 of the row / column scale), the dropped pairs (s + t > 8) and the
//    double-FP32 sums bound the error of an element by a small multiple of
//    2^-49 k max_k |a_ik| max_k |b_kj|: about 5e-14 of ||C|| for Gaussian blocks, against ~1e-15 for
//    an FP64 dot product and ~3e-7 for 3xTF32.
// Bound by the MMA rate: nine blocks of 144 to 2464 take 2042 us with 8 draining warps, a 2-stage ring
// and MMAs in the order in which they open the levels, 1640 now (1.16 ms at the rate of a plain BF16
// product of 28 times the size; slicing 0.24, drains and epilogues about 0.15).
//
// Every mbarrier wait is bounded; on timeout the CTA records an error flag (shared with the 3xTF32
// kernel, xgb_gemm_tc_status), skips the epilogue and still frees its TMEM.
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

constexpr int OM = 128, ON = 64, OK = 16;          // output tile rows / columns, K per slice
constexpr int kPieces = 7, kBits = 7;               // seven 7-bit slices per entry
constexpr int kLevels = kPieces;                    // levels s + t = 2 .. 8 (1-based slices)
constexpr int kChunk = 28;                          // K slices per exact TMEM accumulation (448 x 36864 < 2^24)
constexpr int kMinSplit = 8;                        // smallest K range of a split-K CTA, in K slices
constexpr int kAPieceBytes = OM * OK * 2;           // 4 KB
constexpr int kBPieceBytes = ON * OK * 2;           // 2 KB
constexpr int kOzStageBytes = kPieces * (kAPieceBytes + kBPieceBytes);  // 42 KB
constexpr int kOzStages = 5;
constexpr int kOzSmem = kOzStages * kOzStageBytes + 1024;
constexpr uint32_t kOzTmemCols = 512;               // 7 levels x 64 columns used
constexpr int kOzDrainWarps = 16, kOzProducer = kOzDrainWarps, kOzMma = kOzDrainWarps + 1;
constexpr int kOzWarps = kOzDrainWarps + 2, kOzThreads = kOzWarps * 32;
constexpr int kDrainCols = ON / (kOzDrainWarps / 4);  // columns of a drain warp
constexpr long long kOzSpin = 1ll << 26;
constexpr int kReduceThreads = 256;
constexpr int kPackRows = 32;                       // rows of a slicing cluster
constexpr int kPackCluster = 8;                     // its CTAs at most
constexpr uint32_t kSboBytes = 128;                 // next 8-row group
// A: seven separate 128-row pieces.  B: the seven 64-row pieces stacked into one 448-row operand (row
// group g of piece s is row group 8 s + g), so that pieces t .. t + c - 1 form one N = 64 c operand
constexpr uint32_t kLboA = (OM / 8) * 128;          // next 16-byte K group, 128-row pieces
constexpr uint32_t kBPieceStride = (ON / 8) * 128;  // 1 KB: next B piece within a K group
constexpr uint32_t kLboB = kPieces * kBPieceStride; // 7 KB: next 16-byte K group of the stacked B
static_assert(kLevels * ON <= int(kOzTmemCols), "level accumulators fit TMEM");
static_assert(kOzSmem <= 227 * 1024, "stages fit shared memory");

__device__ __forceinline__ uint32_t s_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ uint64_t oz_desc(uint32_t saddr, uint32_t lbo) {
  uint64_t d = 0;
  d |= uint64_t((saddr >> 4) & 0x3FFF);
  d |= uint64_t((lbo >> 4) & 0x3FFF) << 16;
  d |= uint64_t((kSboBytes >> 4) & 0x3FFF) << 32;
  d |= uint64_t(1) << 46;  // tcgen05 descriptor version; base offset 0, no swizzle
  return d;
}

// FP32 accumulate, BF16 A and B (kind::f16), both K-major, M = 128, N = 64 NC (NC stacked B pieces)
template <int NC>
__host__ __device__ constexpr uint32_t oz_idesc() {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t((ON * NC) >> 3) << 17) | (uint32_t(OM >> 4) << 24);
}

__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s_u32(bar)), "r"(count));
}

__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t a = s_u32(bar);
  for (long long it = 0; it < kOzSpin; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void bar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(s_u32(dst_smem)),
      "l"(src_gmem), "r"(bytes), "r"(s_u32(bar))
      : "memory");
}

template <int NC>
__device__ __forceinline__ void mma_bf16_oz(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(oz_idesc<NC>()), "r"(acc));
}

// 16 columns of this warp's 32 lanes; the registers hold them after tcgen05.wait::ld
__device__ __forceinline__ void tmem_load16(uint32_t addr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(addr));
}

// waits for the loads; the values pass through so that no use moves ahead of it
__device__ __forceinline__ void tmem_wait16(uint32_t* v) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
               :
               : "memory");
}

// two FP32 additions at once, each rounded as __fadd_rn
__device__ __forceinline__ unsigned long long pair(uint32_t a, uint32_t b) {
  return uint64_t(a) | uint64_t(b) << 32;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

__device__ __forceinline__ void commit_to(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s_u32(bar))
               : "memory");
}

// ----------------------------------------------------------------------------- row scales and slices
// exponent e with |x| < 2^e for every entry of the row, from the bits of its largest |entry|
// m = f 2^e, f in [0.5, 1): the biased exponent less 1022.  A zero row, or one whose largest entry
// is subnormal (its slices are all zero), gets 0.
__device__ __forceinline__ int row_scale(unsigned long long bits) {
  const int be = int((bits >> 52) & 0x7FF);
  return be == 0 ? 0 : be - 1022;
}

// Seven balanced base-128 digits of x relative to 2^e (|x| < 2^e): x = 2^e sum_s m_s 2^(-7 s) + O(2^(e - 50)),
// |m_1| <= 128, |m_s| <= 64 for s >= 2.  Adding 64 at each of the six lower digits turns the balanced digits of |x| into
// the plain 7-bit fields of one integer: lo holds fields 7, 6, 5, 4 (four of 7 bits), hi fields 3, 2 and the leading one.
__device__ __forceinline__ void digits7(double x, int e, uint32_t& lo, uint32_t& hi) {
  const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(x));
  const int ex = int((bits >> 52) & 0x7FF);
  unsigned long long q = 64ull * (1 + (1ull << 7) + (1ull << 14) + (1ull << 21) + (1ull << 28) + (1ull << 35));
  if (ex != 0) {  // normal numbers (subnormals are below every slice of any realistic row)
    const unsigned long long mant = (bits & ((1ull << 52) - 1)) | (1ull << 52);
    // x = mant 2^(ex - 1075); |x| rounded to the nearest multiple of 2^(e - 49) (ties up): shift right
    // by sh = e - 49 - (ex - 1075) >= 4 (|x| < 2^e) with one guard bit; at most 2^49
    const int sh = e - 49 - (ex - 1075);
    if (sh < 64) q += ((mant >> (sh - 1)) + 1ull) >> 1;
  }
  lo = uint32_t(q);
  hi = uint32_t(q >> 28);
}

// digit s (1-based) times 2^(-7 s) as a float, from its 7-bit (leading: 8-bit) field: the field below 2^23 in a
// significand, and one exact multiply-add that takes the offset off and scales
template <int S>
__device__ __forceinline__ uint32_t digit_float(uint32_t lo, uint32_t hi) {
  constexpr float k = 1.0f / float(1ull << (7 * S));
  constexpr float c = -(8388608.0f + (S == 1 ? 0.0f : 64.0f)) * k;
  const uint32_t f = S == 1 ? hi >> 14 : S <= 3 ? (hi >> (7 * (3 - S))) & 127u : (lo >> (7 * (7 - S))) & 127u;
  return __float_as_uint(fmaf(__uint_as_float(0x4B000000u | f), k, c));
}

// slice S of eight consecutive entries as BF16 (exact: at most 8 significant bits, the upper half of the float), with
// the entries' signs
template <int S>
__device__ __forceinline__ void store_slice(unsigned char* at, int stride, const uint32_t* lo, const uint32_t* hi,
                                            const uint32_t* sign) {
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    w[j] = __byte_perm(digit_float<S>(lo[2 * j], hi[2 * j]), digit_float<S>(lo[2 * j + 1], hi[2 * j + 1]), 0x7632) ^ sign[j];
  *reinterpret_cast<uint4*>(at + (S - 1) * stride) = make_uint4(w[0], w[1], w[2], w[3]);
  if constexpr (S < kPieces) store_slice<S + 1>(at, stride, lo, hi, sign);
}

// One cluster per (group, 32 rows of op(A) or of op(B)^T): its CTAs share the K range in groups of eight, a thread a row
// and every eighth group.  The row maxima (on the IEEE bits: integer order is numeric
// order) meet in distributed shared memory; then the same entries are read again, from L2, and sliced.  Bound by the
// 14 bytes written per entry for large operands, by the reads' latency for small ones.
// Measured (nine blocks of 100 to 1729 squared, both operands): 233 us as a maximum kernel (with atomics) and a slicing
// kernel with 64-bit digit arithmetic, 114 now.
// A list of few rows and a long k (a full contraction) has no CTAs for all SMs in clusters of eight: kMax and kSlice do the
// two halves in launches of their own, over any number of CTAs per task, with the maxima in `rowmax` (cleared before).
enum PackForm { kWhole, kMax, kSlice };
template <PackForm kForm>
__global__ void __launch_bounds__(256) oz_pack_kernel(int ctas, const xgb_gemm_desc* __restrict__ descs,
                                                       const OzGroup* __restrict__ groups,
                                                       const TcPackTask* __restrict__ tasks,
                                                       const double* __restrict__ A, const double* __restrict__ B,
                                                       unsigned long long* __restrict__ rowmax,
                                                       unsigned char* __restrict__ apack,
                                                       unsigned char* __restrict__ bpack) {
  __shared__ unsigned long long part[256], own[kPackRows];
  cg::cluster_group cluster = cg::this_cluster();
  const int P = kForm == kWhole ? int(cluster.num_blocks()) : ctas;
  const int me = kForm == kWhole ? int(cluster.block_rank()) : int(blockIdx.x % unsigned(P));
  const TcPackTask t = tasks[blockIdx.x / unsigned(P)];
  const xgb_gemm_desc d = descs[t.g];
  const OzGroup gr = groups[t.g];
  const bool isB = t.which != 0;
  const bool sb = isB != (gr.swap != 0);  // the rows of this role are op(B)^T's (columns of op(B))
  const int64_t ld = sb ? d.ldb : d.lda, rows = sb ? d.n : d.m;
  const bool rowfast = sb ? d.trans_b != 0 : d.trans_a == 0;
  constexpr int tr = kPackRows, nq = 256 / kPackRows;
  const int r = int(threadIdx.x) % tr, q = int(threadIdx.x) / tr;
  const int64_t row = int64_t(t.tile) * tr + r;
  const bool live = row < rows;
  const double* src = (sb ? B + d.b_off : A + d.a_off) + (live ? (rowfast ? row : row * ld) : 0);
  const int64_t step = rowfast ? ld : 1;
  const int n8 = gr.slices * (OK / 8), per = (n8 + P - 1) / P, first = min(n8, me * per) + q, last = min(n8, (me + 1) * per);
  auto load8 = [&](int g, double* x) {
    const int64_t k = int64_t(g) * 8;
    const double* at = src + k * step;
    if (live && k + 8 <= d.k) {
      if (!rowfast && (reinterpret_cast<uintptr_t>(at) & 15) == 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double2 v = __ldg(reinterpret_cast<const double2*>(at) + j);
          x[2 * j] = v.x;
          x[2 * j + 1] = v.y;
        }
        return;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = __ldg(at + j * step);
      return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = live && k + j < d.k ? __ldg(at + j * step) : 0.0;
  };
  unsigned long long* rmax = rowmax + (isB ? gr.b_rowmax : gr.a_rowmax) + row;
  unsigned long long m = 0;
  for (int g = first; kForm != kSlice && g < last; g += nq) {
    double x[8];
    load8(g, x);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x[j])) & 0x7FFFFFFFFFFFFFFFull;
      m = m > b ? m : b;
    }
  }
  if constexpr (kForm == kSlice) {
    if (int(threadIdx.x) < tr) part[r] = live ? *rmax : 0ull;
    __syncthreads();
  } else {
    part[threadIdx.x] = m;
    __syncthreads();
    if (int(threadIdx.x) < tr) {
      for (int p = 1; p < nq; ++p) m = m > part[p * tr + r] ? m : part[p * tr + r];
      own[r] = m;
    }
    if constexpr (kForm == kMax) {
      if (int(threadIdx.x) < tr && live && m) atomicMax(rmax, m);
      return;
    }
    cluster.sync();
    if (int(threadIdx.x) < tr) {
      for (int p = 0; p < P; ++p) {
        const unsigned long long o = cluster.map_shared_rank(own, p)[r];
        m = m > o ? m : o;
      }
      part[r] = m;
      if (me == 0 && live) *rmax = m;
    }
    cluster.sync();  // `own` of every CTA has been read
  }
  const int e = row_scale(part[r]);
  // block of one (tile, K slice): kPieces pieces of tr x OK BF16, each in canonical layout
  const int piece_bytes = isB ? kBPieceBytes : kAPieceBytes;
  const int piece_stride = isB ? int(kBPieceStride) : kAPieceBytes;
  const uint32_t lbo = isB ? kLboB : kLboA;
  const int per_tile = (isB ? ON : OM) / tr, in_tile = (t.tile % per_tile) * tr + r;  // row of the output tile
  unsigned char* base = (isB ? bpack + gr.b_pack : apack + gr.a_pack) +
                        int64_t(t.tile / per_tile) * gr.slices * (kPieces * piece_bytes) + in_tile * 16;
  for (int g = first; g < last; g += nq) {
    double x[8];
    load8(g, x);
    uint32_t lo[8], hi[8], sign[4];
#pragma unroll
    for (int j = 0; j < 8; ++j) digits7(x[j], e, lo[j], hi[j]);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      sign[j] = (uint32_t(__double2hiint(x[2 * j])) & 0x80000000u) >> 16 | (uint32_t(__double2hiint(x[2 * j + 1])) & 0x80000000u);
    store_slice<1>(base + int64_t(g / (OK / 8)) * (kPieces * piece_bytes) + (g % (OK / 8)) * lbo, piece_stride, lo,
                   hi, sign);
  }
}

// the maxima of each task's rows to zero
__global__ void oz_clear_kernel(const xgb_gemm_desc* __restrict__ descs, const OzGroup* __restrict__ groups,
                                const TcPackTask* __restrict__ tasks, unsigned long long* __restrict__ rowmax) {
  const TcPackTask t = tasks[blockIdx.x];
  const OzGroup gr = groups[t.g];
  const bool sb = (t.which != 0) != (gr.swap != 0);
  const int64_t row = int64_t(t.tile) * kPackRows + threadIdx.x;
  if (row < (sb ? descs[t.g].n : descs[t.g].m)) rowmax[(t.which ? gr.b_rowmax : gr.a_rowmax) + row] = 0;
}

// ----------------------------------------------------------------------------- gemm
// the rare cases of scaled_double (subnormal, infinite or out-of-range results), out of line so that
// the common path is never if-converted into the FP64 conversion and ldexp
__device__ __noinline__ double scaled_double_slow(float v, int sc) { return ldexp(double(v), sc); }

// v 2^sc as a double, assembled from the FP32 bits (exact; no FP64 arithmetic) while the result is a
// normal double, else through ldexp
__device__ __forceinline__ double scaled_double(float v, int sc) {
  const uint32_t b = __float_as_uint(v);
  const int e8 = int((b >> 23) & 0xFF);
  if ((b & 0x7FFFFFFFu) == 0u) return __longlong_as_double(static_cast<long long>(uint64_t(b >> 31) << 63));
  const int e = e8 - 127 + 1023 + sc;
  if (e8 == 0 || e8 == 255 || e <= 0 || e >= 2047) return scaled_double_slow(v, sc);
  return __longlong_as_double(static_cast<long long>((uint64_t(b >> 31) << 63) | (uint64_t(e) << 52) |
                                                     (uint64_t(b & 0x7FFFFFu) << 29)));
}

__global__ void __launch_bounds__(kOzThreads, 1)
    oz_gemm_kernel(const xgb_gemm_desc* __restrict__ descs, const OzGroup* __restrict__ groups,
                   const GemmTile* __restrict__ tiles, const unsigned char* __restrict__ apack,
                   const unsigned char* __restrict__ bpack, const unsigned long long* __restrict__ rowmax,
                   double* __restrict__ C, double alpha, double beta, double* __restrict__ ws,
                   int* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t full[kOzStages], empty[kOzStages], accf, acce[2], done;
  __shared__ uint32_t tmem_slot;
  __shared__ int fail, issued, consumed;
  __shared__ int rsc[OM], csc[ON];  // row and column scale exponents of the tile
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  const GemmTile t = tiles[blockIdx.x];
  const xgb_gemm_desc d = descs[t.g];
  const OzGroup gr = groups[t.g];
  const int64_t m0 = int64_t(t.tm) * OM, n0 = int64_t(t.tn) * ON;
  // extents of the computed product: C, or C^T for a swapped group (element (r, c) of C^T is C[c + r ldc])
  const bool swp = gr.swap != 0;
  const int64_t pm = swp ? d.n : d.m, pn = swp ? d.m : d.n;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // split-K: this CTA takes K slices [ks, ks + nk) and, with a slot, stores its raw partial tile
  const int ks = t.k0, nk = (t.k1 < 0 ? gr.slices : t.k1) - t.k0;
  const int nchunks = (nk + kChunk - 1) / kChunk;

  for (int i = threadIdx.x; i < OM + ON; i += kOzThreads) {
    if (i < OM) rsc[i] = m0 + i < pm ? row_scale(rowmax[gr.a_rowmax + m0 + i]) : 0;
    else csc[i - OM] = n0 + (i - OM) < pn ? row_scale(rowmax[gr.b_rowmax + n0 + (i - OM)]) : 0;
  }
  if (warp == kOzMma) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(&tmem_slot)),
                 "r"(kOzTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kOzStages; ++s) {
      bar_init(&full[s], 1);
      bar_init(&empty[s], 1);
    }
    bar_init(&accf, 1);
    for (int h = 0; h < 2; ++h) bar_init(&acce[h], kOzDrainWarps);
    bar_init(&done, 1);
    fail = 0;
    issued = 0;
    consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  // drain-warp state: TMEM lane quarter (rows) and column group; double-FP32 sums of 16 columns
  const int quarter = warp & 3, colg = warp >> 2;
  unsigned long long hi2[kDrainCols / 2], lo2[kDrainCols / 2];  // two floats each
#pragma unroll
  for (int j = 0; j < kDrainCols / 2; ++j) { hi2[j] = 0; lo2[j] = 0; }

  if (nk > 0 && warp == kOzProducer) {
    if (lane == 0) {
      const unsigned char* a_base =
          apack + gr.a_pack + (int64_t(t.tm) * gr.slices + ks) * kPieces * kAPieceBytes;
      const unsigned char* b_base =
          bpack + gr.b_pack + (int64_t(t.tn) * gr.slices + ks) * kPieces * kBPieceBytes;
      for (int kc = 0; kc < nk; ++kc) {
        const int s = kc % kOzStages, round = kc / kOzStages;
        if (round > 0 && !bar_wait(&empty[s], uint32_t((round - 1) & 1))) { atomicExch(&fail, 1); break; }
        unsigned char* st = smem + s * kOzStageBytes;
        bar_expect_tx(&full[s], kOzStageBytes);
        bulk_g2s(st, a_base + int64_t(kc) * kPieces * kAPieceBytes, kPieces * kAPieceBytes, &full[s]);
        bulk_g2s(st + kPieces * kAPieceBytes, b_base + int64_t(kc) * kPieces * kBPieceBytes, kPieces * kBPieceBytes,
                 &full[s]);
        issued = kc + 1;
      }
    }
  } else if (nk > 0 && warp == kOzMma) {
    if (lane == 0) {
      for (int kc = 0; kc < nk; ++kc) {
        const int s = kc % kOzStages, cs = kc % kChunk, ch = kc / kChunk;
        if (!bar_wait(&full[s], uint32_t((kc / kOzStages) & 1))) { atomicExch(&fail, 1); break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t abase = s_u32(smem + s * kOzStageBytes);
        const uint32_t bbase = abase + kPieces * kAPieceBytes;
        // slice pairs (i, j), j <= 6 - i, in MMAs of up to four stacked B pieces: the product of A piece
        // i with B pieces j0 .. j0 + c - 1 lands in levels i + j0 .. i + j0 + c - 1, the adjacent
        // 64-column accumulators from column 64 (i + j0); ten MMAs cover the 28 pairs.  Narrow ones first:
        // an MMA of N = 64 or 128 waits for its operands, and the wide ones behind hide that (k = 144 to
        // 2464, without the drains: 1.66 ms as the levels are opened, 1.73 from wide to narrow, 1.49 so)
        const uint64_t ad[kPieces] = {
            oz_desc(abase + 0 * kAPieceBytes, kLboA), oz_desc(abase + 1 * kAPieceBytes, kLboA),
            oz_desc(abase + 2 * kAPieceBytes, kLboA), oz_desc(abase + 3 * kAPieceBytes, kLboA),
            oz_desc(abase + 4 * kAPieceBytes, kLboA), oz_desc(abase + 5 * kAPieceBytes, kLboA),
            oz_desc(abase + 6 * kAPieceBytes, kLboA)};
        auto bd = [&](int j0) { return oz_desc(bbase + j0 * kBPieceStride, kLboB); };
        auto col = [&](int lvl) { return tmem + uint32_t(lvl * ON); };
        // The first slice of a chunk opens the levels with its i = 0 MMAs, each once the previous chunk has
        // been drained from it: the levels 4-6 are drained first and multiplied while 0-3 are read.
        const uint32_t drained = uint32_t((ch - 1) & 1);
        if (cs == 0) {
          if (ch > 0 && !bar_wait(&acce[0], drained)) { atomicExch(&fail, 1); break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          mma_bf16_oz<3>(col(4), ad[0], bd(4), 0u);
        }
        mma_bf16_oz<1>(col(6), ad[6], bd(0), 1u);
        mma_bf16_oz<1>(col(6), ad[2], bd(4), 1u);
        mma_bf16_oz<2>(col(5), ad[5], bd(0), 1u);
        mma_bf16_oz<2>(col(5), ad[1], bd(4), 1u);
        mma_bf16_oz<3>(col(4), ad[4], bd(0), 1u);
        if (cs == 0) {
          if (ch > 0 && !bar_wait(&acce[1], drained)) { atomicExch(&fail, 1); break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          mma_bf16_oz<4>(col(0), ad[0], bd(0), 0u);
        } else {
          mma_bf16_oz<3>(col(4), ad[0], bd(4), 1u);
        }
        mma_bf16_oz<4>(col(3), ad[3], bd(0), 1u);
        mma_bf16_oz<4>(col(2), ad[2], bd(0), 1u);
        mma_bf16_oz<4>(col(1), ad[1], bd(0), 1u);
        if (cs != 0) mma_bf16_oz<4>(col(0), ad[0], bd(0), 1u);
        commit_to(&empty[s]);
        if (cs == kChunk - 1 || kc == nk - 1) commit_to(&accf);
        consumed = kc + 1;
      }
      commit_to(&done);
    }
  } else if (nk > 0 && warp < kOzDrainWarps) {
    for (int ch = 0; ch < nchunks; ++ch) {
      const bool got = __all_sync(0xffffffffu, bar_wait(&accf, uint32_t(ch & 1)));
      if (!got) {
        if (lane == 0) atomicExch(&fail, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // smallest contributions first; the next level's load is in flight while one is added
      static_assert(kDrainCols == 16, "the loads below");
      uint32_t next[kDrainCols];
      const uint32_t tcol = tmem + (uint32_t(quarter * 32) << 16) + uint32_t(colg * kDrainCols);
      tmem_load16(tcol + uint32_t((kLevels - 1) * ON), next);
#pragma unroll
      for (int level = kLevels - 1; level >= 0; --level) {
        uint32_t v[kDrainCols];
        tmem_wait16(next);
#pragma unroll
        for (int j = 0; j < kDrainCols; ++j) v[j] = next[j];
        if (level == 4 || level == 0) {  // levels 4-6, then 0-3 have been read
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s_u32(&acce[level == 0])) : "memory");
        }
        if (level > 0) tmem_load16(tcol + uint32_t((level - 1) * ON), next);
#pragma unroll
        for (int j = 0; j < kDrainCols / 2; ++j) {
          // two-sum of hi and the exact level partial; the rounding error goes to lo
          const unsigned long long x = pair(v[2 * j], v[2 * j + 1]);
          const unsigned long long t = add2(hi2[j], x), bb = sub2(t, hi2[j]);
          lo2[j] = add2(lo2[j], add2(sub2(hi2[j], sub2(t, bb)), sub2(x, bb)));
          hi2[j] = t;
        }
      }
#pragma unroll
      for (int j = 0; j < kDrainCols / 2; ++j) {  // renormalise: |lo| stays below one unit of hi
        const unsigned long long t = add2(hi2[j], lo2[j]);
        lo2[j] = sub2(lo2[j], sub2(t, hi2[j]));
        hi2[j] = t;
      }
    }
  }
  bool ok = true;
  if (nk > 0) ok = bar_wait(&done, 0);
  __syncthreads();
  ok = ok && (fail == 0);
  ok = __syncthreads_and(ok);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  float hi[kDrainCols], lo[kDrainCols];
#pragma unroll
  for (int j = 0; j < kDrainCols; ++j) {
    hi[j] = __uint_as_float(uint32_t(hi2[j / 2] >> (32 * (j % 2))));
    lo[j] = __uint_as_float(uint32_t(lo2[j / 2] >> (32 * (j % 2))));
  }
  // 0: partial tile to the workspace, 1: C = acc, 2: C = alpha acc, 3: C = alpha acc + beta C
  const int mode = t.slot >= 0 ? 0 : beta != 0.0 ? 3 : alpha != 1.0 ? 2 : 1;
  if (ok && nk > 0 && warp < kOzDrainWarps) {
    const int64_t row = m0 + quarter * 32 + lane;
    const int ei = rsc[quarter * 32 + lane];
    if (mode != 0 && swp) {
      // transposed store through shared memory (the stages are idle now): thread (r, its columns) puts
      // its values at T[c][r] (row pitch 129 doubles), then each warp writes 32 consecutive rows of C
      double* T = reinterpret_cast<double*>(smem);
#pragma unroll
      for (int j = 0; j < kDrainCols; ++j) {
        const int c = colg * kDrainCols + j;
        const int sc = ei + csc[c];
        T[c * (OM + 1) + quarter * 32 + lane] = scaled_double(hi[j], sc) + scaled_double(lo[j], sc);
      }
      asm volatile("bar.sync 1, %0;" ::"n"(kOzDrainWarps * 32) : "memory");
      for (int e = threadIdx.x; e < OM * ON; e += kOzDrainWarps * 32) {
        const int c = e % ON, r = e / ON;  // C row n0 + c, C column m0 + r
        if (m0 + r < pm && n0 + c < pn) {
          const double acc = T[c * (OM + 1) + r];
          double* cp = C + d.c_off + (n0 + c) + (m0 + r) * d.ldc;
          if (mode == 1) *cp = acc;
          else if (mode == 2) *cp = alpha * acc;
          else *cp = fma(alpha, acc, beta * *cp);
        }
      }
    } else if (row < pm) {
#pragma unroll
      for (int j = 0; j < kDrainCols; ++j) {
        const int64_t col = n0 + colg * kDrainCols + j;
        if (col < pn) {
          const int sc = ei + csc[colg * kDrainCols + j];
          const double acc = scaled_double(hi[j], sc) + scaled_double(lo[j], sc);
          if (mode == 0) {  // split-K partial: raw sum, tile-local column-major OM x ON
            ws[int64_t(t.slot) * OM * ON + (quarter * 32 + lane) + int64_t(colg * kDrainCols + j) * OM] = acc;
          } else {
            double* cp = C + d.c_off + row + col * d.ldc;
            if (mode == 1) *cp = acc;
            else if (mode == 2) *cp = alpha * acc;
            else *cp = fma(alpha, acc, beta * *cp);
          }
        }
      }
    }
  } else if (ok && nk == 0) {
    for (int e = threadIdx.x; e < OM * ON; e += kOzThreads) {
      const int64_t row = m0 + e % OM, col = n0 + e / OM;
      if (row < pm && col < pn) {
        double* cp = C + d.c_off + (swp ? col + row * d.ldc : row + col * d.ldc);
        *cp = beta == 0.0 ? 0.0 : beta * *cp;
      }
    }
  }
  if (!ok && threadIdx.x == 0) {
    atomicExch(err, 1);
    for (int kc = consumed; kc < issued; ++kc) bar_wait(&full[kc % kOzStages], uint32_t((kc / kOzStages) & 1));
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kOzMma)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kOzTmemCols));
}

// C tile = alpha * (the split-K partials of the tile, added in slot order) + beta * C
__global__ void __launch_bounds__(256) oz_splitk_reduce_kernel(const xgb_gemm_desc* __restrict__ descs,
                                                                const OzGroup* __restrict__ groups,
                                                                const SplitReduce* __restrict__ red,
                                                                const double* __restrict__ ws, double* __restrict__ C,
                                                                double alpha, double beta) {
  const SplitReduce r = red[blockIdx.x];
  const xgb_gemm_desc d = descs[r.g];
  const bool swp = groups[r.g].swap != 0;
  const int64_t pm = swp ? d.n : d.m, pn = swp ? d.m : d.n;
  // blockIdx.y: 256 elements of the tile, one per thread (the sums are chains of dependent loads: four per thread took
  // 12 us on tiles cut nineteen ways); consecutive threads take consecutive rows of C (tile rows, or tile columns of a
  // swapped group)
  static_assert(OM * ON % kReduceThreads == 0);
  const int e = int(blockIdx.y) * kReduceThreads + int(threadIdx.x);
  const int li = swp ? e / ON : e % OM, lj = swp ? e % ON : e / OM;  // tile-local row / column
  const int64_t i = int64_t(r.tm) * OM + li, j = int64_t(r.tn) * ON + lj;
  if (i >= pm || j >= pn) return;
  const int64_t w = li + int64_t(lj) * OM;
  const double* part = ws + int64_t(r.first) * OM * ON + w;
  double acc = part[0];
  // eight loads in flight
  for (int p = 1; p < r.count; p += 8) {
    double x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (p + u < r.count) x[u] = __ldg(part + int64_t(p + u) * OM * ON);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (p + u < r.count) acc += x[u];
  }
  double* c = C + d.c_off + (swp ? j + i * d.ldc : i + j * d.ldc);
  *c = beta != 0.0 ? fma(alpha, acc, beta * *c) : alpha == 1.0 ? acc : alpha * acc;
}

PerDevice g_oz_attr;

}  // namespace

OzPlanHost build_oz_plan(const xgb_gemm_desc* descs, int n, bool allow_swap) {
  // A group is computed transposed (C^T = op(B)^T op(A)^T) when that needs at most 3/4 of the 128 x 64
  // output tiles (few rows, many columns: the 128-row tile would be mostly padding).
  auto tiles_of = [](int64_t r, int64_t c) { return ((r + OM - 1) / OM) * ((c + ON - 1) / ON); };
  std::vector<char> swap(size_t(n), 0);
  if (allow_swap)
    for (int g = 0; g < n; ++g) swap[g] = 4 * tiles_of(descs[g].n, descs[g].m) <= 3 * tiles_of(descs[g].m, descs[g].n);
  // rowmax layout: every group's rows of the "A" role first, then every group's rows of the "B" role
  // (columns of the product)
  OzPlanHost p;
  int64_t ra = 0, rb = 0;
  for (int g = 0; g < n; ++g) rb += swap[g] ? descs[g].n : descs[g].m;
  for (int g = 0; g < n; ++g) {
    const xgb_gemm_desc& d = descs[g];
    const int64_t pm = swap[g] ? d.n : d.m, pn = swap[g] ? d.m : d.n;  // extents of the computed product
    OzGroup gr{};
    gr.swap = swap[g];
    gr.a_tiles = int32_t((pm + OM - 1) / OM);
    gr.b_tiles = int32_t((pn + ON - 1) / ON);
    gr.slices = int32_t((d.k + OK - 1) / OK);
    gr.a_pack = p.a_bytes;
    gr.b_pack = p.b_bytes;
    gr.a_rowmax = ra;
    gr.b_rowmax = rb;
    ra += pm;
    rb += pn;
    p.a_bytes += int64_t(gr.a_tiles) * gr.slices * kPieces * kAPieceBytes;
    p.b_bytes += int64_t(gr.b_tiles) * gr.slices * kPieces * kBPieceBytes;
    // clusters that slice the operands: at most 128 k values per CTA, eight CTAs
    while (p.pack_cluster < kPackCluster && gr.slices * OK > 128 * p.pack_cluster) p.pack_cluster *= 2;
    for (int32_t t = 0; t < gr.a_tiles * (OM / kPackRows); ++t) p.tasks_a.push_back({g, t, 0, 0});
    for (int32_t t = 0; t < gr.b_tiles * (ON / kPackRows); ++t) p.tasks_b.push_back({g, t, 0, 1});
    p.groups.push_back(gr);
  }
  // few tasks over a long k: the slicing in launches of its own over four CTAs per SM, at least 512 k values each (the
  // whole product, us: 4 x 4 x 100000 581 in clusters of eight, 213 so; 1 x 1 x 10000 90 and 76; at k = 2000 the launches
  // cost more than the CTAs gain)
  const int64_t sms = num_sms() > 0 ? num_sms() : 152, n_tasks = int64_t(p.tasks_a.size() + p.tasks_b.size());
  int64_t kmax = 0;
  for (const auto& gr : p.groups) kmax = std::max<int64_t>(kmax, int64_t(gr.slices) * OK);
  if (n_tasks * kPackCluster < sms && kmax >= 1024 * kPackCluster)
    p.pack_cluster = int(std::min(kmax / 512, (4 * sms + n_tasks - 1) / n_tasks));
  // output tiles and their K ranges.  One CTA runs per SM (its stages and TMEM fill one), so the K
  // slices of all tiles are cut into ranges of at most `cap` slices (at least kMinSplit), the largest
  // tiles split the most: cap starts at total / SMs and grows until the CTAs fit one wave (a second,
  // partial wave costs a whole CTA's fixed part - first load, drain, epilogue - on the SMs it uses).
  // The partial tiles of a split tile are added by a fixed-order reduce.
  int64_t work = 0, smax = 0;
  for (const auto& gr : p.groups) {
    work += int64_t(gr.a_tiles) * gr.b_tiles * gr.slices;
    smax = std::max<int64_t>(smax, gr.slices);
  }
  auto ctas = [&](int64_t cp) {
    int64_t c = 0;
    for (const auto& gr : p.groups) c += int64_t(gr.a_tiles) * gr.b_tiles * std::max<int64_t>(1, (gr.slices + cp - 1) / cp);
    return c;
  };
  int64_t cap = std::max<int64_t>(kMinSplit, (work + sms - 1) / sms);
  while (cap < smax && ctas(cap) > sms) ++cap;
  for (int g = 0; g < n; ++g) {
    const OzGroup& gr = p.groups[g];
    const int64_t splits = std::max<int64_t>(1, (gr.slices + cap - 1) / cap);
    const int64_t per = (gr.slices + splits - 1) / splits;
    for (int32_t y = 0; y < gr.b_tiles; ++y)
      for (int32_t x = 0; x < gr.a_tiles; ++x) {
        if (splits == 1) {
          p.tiles.push_back({g, x, y, OM});
          continue;
        }
        const int32_t first = p.slots;
        for (int64_t k0 = 0; k0 < gr.slices; k0 += per)
          p.tiles.push_back({g, x, y, OM, int32_t(k0), int32_t(std::min<int64_t>(k0 + per, gr.slices)), p.slots++});
        p.red.push_back({g, x, y, first, p.slots - first, 0});
      }
  }
  // longest K ranges first: CTAs start in index order, so the short ones fill the tail of the wave
  auto range = [&](const GemmTile& t) { return (t.k1 < 0 ? p.groups[t.g].slices : t.k1) - t.k0; };
  std::stable_sort(p.tiles.begin(), p.tiles.end(),
                   [&](const GemmTile& a, const GemmTile& b) { return range(a) > range(b); });
  p.rowmax = rb;
  p.tasks = p.tasks_a;
  p.tasks.insert(p.tasks.end(), p.tasks_b.begin(), p.tasks_b.end());
  return p;
}

void launch_oz_pack(const xgb_gemm_desc* d_descs, const OzGroup* d_groups, const TcPackTask* d_tasks, int n_tasks,
                    int cluster, const double* A, const double* B, unsigned long long* rowmax, unsigned char* apack,
                    unsigned char* bpack, cudaStream_t s) {
  if (n_tasks <= 0) return;
  if (cluster > kPackCluster) {
    const unsigned grid = unsigned(n_tasks) * unsigned(cluster);
    oz_clear_kernel<<<n_tasks, kPackRows, 0, s>>>(d_descs, d_groups, d_tasks, rowmax);
    oz_pack_kernel<kMax><<<grid, 256, 0, s>>>(cluster, d_descs, d_groups, d_tasks, A, B, rowmax, apack, bpack);
    oz_pack_kernel<kSlice><<<grid, 256, 0, s>>>(cluster, d_descs, d_groups, d_tasks, A, B, rowmax, apack, bpack);
    count_launch(3);
    return;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(n_tasks) * unsigned(cluster));
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim = {unsigned(cluster), 1, 1};
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const cudaError_t e =
      cudaLaunchKernelEx(&cfg, oz_pack_kernel<kWhole>, 0, d_descs, d_groups, d_tasks, A, B, rowmax, apack, bpack);
  if (e != cudaSuccess) throw std::runtime_error(std::string("slicing launch: ") + cudaGetErrorString(e));
  count_launch();
}

void launch_oz_gemm(const xgb_gemm_desc* d_descs, const OzGroup* d_groups, const GemmTile* d_tiles, int n_tiles,
                    const SplitReduce* d_red, int n_red, int slots, const unsigned char* apack,
                    const unsigned char* bpack, const unsigned long long* rowmax, double* C, double alpha, double beta,
                    cudaStream_t s) {
  if (n_tiles <= 0) return;
  g_oz_attr.once([] {
    cudaFuncSetAttribute(oz_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kOzSmem);
  });
  double* ws = slots > 0 ? static_cast<double*>(dev_alloc(sizeof(double) * size_t(slots) * OM * ON)) : nullptr;
  oz_gemm_kernel<<<n_tiles, kOzThreads, kOzSmem, s>>>(d_descs, d_groups, d_tiles, apack, bpack, rowmax, C, alpha,
                                                     beta, ws, gemm_tc_error_flag());
  count_launch();
  if (n_red > 0) {
    oz_splitk_reduce_kernel<<<dim3(unsigned(n_red), OM * ON / kReduceThreads), kReduceThreads, 0, s>>>(d_descs, d_groups, d_red,
                                                                                            ws, C, alpha, beta);
    count_launch();
  }
  if (ws) dev_free(ws);
}

bool f64tc_heuristic(const xgb_gemm_desc* d, int n) {
  double flops = 0, out = 0;
  for (int g = 0; g < n; ++g) {
    flops += 2.0 * double(d[g].m) * double(d[g].n) * double(d[g].k);
    out += double(d[g].m) * double(d[g].n);
  }
  return out > 0 && flops / out >= 128.0;  // average k >= 64
}

void run_gemm_oz_host(const xgb_gemm_desc* h_descs, int n, const double* A, const double* B, double* C, double alpha,
                      double beta, cudaStream_t s) {
  if (n <= 0) return;
  OzPlanHost op = build_oz_plan(h_descs, n);
  if (op.tiles.empty()) return;
  auto up = [&](const void* h, size_t bytes) {
    void* d = dev_alloc(std::max<size_t>(bytes, 16));
    if (bytes) cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s);
    return d;
  };
  auto* dd = static_cast<xgb_gemm_desc*>(up(h_descs, sizeof(xgb_gemm_desc) * size_t(n)));
  auto* dg = static_cast<OzGroup*>(up(op.groups.data(), sizeof(OzGroup) * op.groups.size()));
  auto* dk = static_cast<TcPackTask*>(up(op.tasks.data(), sizeof(TcPackTask) * op.tasks.size()));
  auto* dt = static_cast<GemmTile*>(up(op.tiles.data(), sizeof(GemmTile) * op.tiles.size()));
  auto* dr = static_cast<SplitReduce*>(up(op.red.data(), sizeof(SplitReduce) * op.red.size()));
  auto* rm = static_cast<unsigned long long*>(dev_alloc(sizeof(unsigned long long) * size_t(std::max<int64_t>(op.rowmax, 1))));
  auto* ap = static_cast<unsigned char*>(dev_alloc(size_t(std::max<int64_t>(op.a_bytes, 16))));
  auto* bp = static_cast<unsigned char*>(dev_alloc(size_t(std::max<int64_t>(op.b_bytes, 16))));
  launch_gemm_oz(dd, dg, dk, int(op.tasks.size()), op.pack_cluster, dt, int(op.tiles.size()), dr, int(op.red.size()), op.slots, A, B,
                 rm, ap, bp, C, alpha, beta, s);
  for (void* p : {static_cast<void*>(dd), static_cast<void*>(dg), static_cast<void*>(dk), static_cast<void*>(dt),
                  static_cast<void*>(dr), static_cast<void*>(rm), static_cast<void*>(ap), static_cast<void*>(bp)})
    dev_free(p);
}

void launch_gemm_oz(const xgb_gemm_desc* d_descs, const OzGroup* d_groups, const TcPackTask* d_tasks, int n_tasks,
                    int cluster, const GemmTile* d_tiles, int n_tiles, const SplitReduce* d_red, int n_red, int slots,
                    const double* A, const double* B, unsigned long long* rowmax, unsigned char* apack, unsigned char* bpack, double* C, double alpha, double beta, cudaStream_t s) {
  if (n_tiles <= 0) return;
  launch_oz_pack(d_descs, d_groups, d_tasks, n_tasks, cluster, A, B, rowmax, apack, bpack, s);
  launch_oz_gemm(d_descs, d_groups, d_tiles, n_tiles, d_red, n_red, slots, apack, bpack, rowmax, C, alpha, beta, s);
}

}  // namespace xgb
