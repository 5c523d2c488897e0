// FP64 complex rank-64 updates C -= A B on the integer tensor cores (tcgen05 kind::i8), by splitting the
// operands into 8-bit digits.
//
// The GPU multiplies FP64 at 64 FMAs a cycle and SM, 8-bit integers exactly at 8192.  So every row of
// A and every column of B is scaled by a power of two to 62-bit integers and written as eight signed
// 8-bit digits (digit 0 the highest; digit splitting of the operands for error-free products is
// Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 95 (2012)).  The product of digit i of A and digit
// j of B has weight 256^-(i + j); the 36 products with i + j < 8 are kept.  Products of equal weight are
// summed exactly in 32-bit accumulators (8 x 128 x 2^14 < 2^31), and the eight sums are combined in FP64.
// An element keeps 62 bits below its row's (column's) largest one, and the products left out are below
// 2^-58 of the largest times the largest: an FP64 accumulation of the same 128 products rounds at
// about 2^-53 of its running sum, so the split is the more exact of the two unless a row of A and a column
// of B span a wide range against each other, which the balance of the inner indices (balance_kernel) takes
// out.  On updates of KKR matrices (fcc, 43 sites) with energies on a contour from -0.3 to 0.7 Ry the
// norm of the error is 0.4 to 1.4e-17 of that of |A| |B|, where FP64 has 0.4 to 1.9e-16; at E = 0.02 +
// 0.02 i, where the digits without the balance lose to FP64 (0.9 to 3.5e-16), 0.3 to 2.2e-17 against 0.3
// to 0.7e-16.  Whole solves, gradients and inverses are as close to 64 bits as with FP64 products (tau00 of
// contours 6.3e-13 with either).
//
// A complex C (m x n) is the real matrix with rows 2r, 2r + 1 = (re, im): C = At Bh with Bh column c =
// (Br[0], Bi[0], Br[1], ...) and At the 2 x 2 expansion [[ar, -ai], [ai, ar]] (as in tc_update.cu), K =
// 128 digits = one 128-byte row.
//
// A CTA takes a panel of 64 complex rows: A's eight digit planes (128 KB) stay in shared memory while B's
// column tiles (32 columns x 8 digits, 32 KB) stream through a two-stage ring, so the operand traffic is
// B's alone.  With the digits of a B tile stacked along N, one MMA multiplies digit i of A by digits
// 0 .. 7 - i of B (N = 32 (8 - i)) into the accumulators of weights i .. 7, which lie side by side in
// tensor memory (8 x 32 columns, two sets): 32 MMAs a tile, 2300 cycles of the tensor core.  Sixteen
// epilogue warps, eight for either set, combine the sums (64-bit integers first, so that FP64 does five
// operations an element) and update C, whose elements they request before the wait for the products.
// 31 jobs of N = 2160: the elimination 30.0 -> 22.9 ms against the FP64 tensor cores' tiles (dmma.cuh).  A tile
// takes 3.0 us of an SM, 1.2 us of them the tensor core's: what bounds it is the epilogue's arithmetic (some
// 60 instructions an element; with eight warps and the digit sums combined in FP64 a tile took 3.75 us).
// Work items (row panel, 4 to 32 column tiles) come from a counter, so that CTAs which start late
// (their SM still held by a diagonal inverse) take fewer.  Every wait is bounded; on expiry the CTA
// records an error flag, drains what it issued, frees tensor memory and returns.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"

namespace b200 {
namespace s8 {

constexpr int kDigits = kSplitDigits;
constexpr int kPanel = 64;                      // complex rows of a work item
constexpr int kTM = 2 * kPanel;                 // real rows: the MMA's M
constexpr int kTN = 32;                         // columns of a tile
constexpr int kRowBytes = kSplitRowBytes;       // K: 64 complex, re and im
constexpr int kABytes = kTM * kRowBytes;        // one digit plane of a panel
constexpr int kBBytes = kTN * kRowBytes;        // one digit plane of a column tile
constexpr int kStages = 2;
constexpr int kMinTiles = 4, kMaxTiles = 32;    // column tiles per work item
constexpr int kEpiWarps = 16;                   // per accumulator set two column halves of four warps
constexpr int kEpiCols = kTN / 2;
constexpr int kThreads = 64 + 32 * kEpiWarps;   // producer, MMA issuer, epilogue
constexpr int kQ = 4;                           // work-item ring
constexpr int kMaxBalance = 100;                // largest exponent of an inner index's balance
constexpr int kAccCols = kDigits * kTN;         // tensor-memory columns per accumulator set (two of them)
constexpr long kWaitBound = 1L << 22;

// C -= A B of one job: A m x K, B K x n, C m x n, column-major, K <= 64.
struct View {
  const double2 *A, *B;
  double2 *C;
  int lda, ldb, ldc, m, n, K;
};

// Op's view where the integer tensor cores take it: at least ELEMS elements (split_pays).
template <class Op, long ELEMS>
struct Large {
  __device__ bool operator()(const JobDev &J, int k, View &g) const {
    return Op()(J, k, g) && split_pays(g.m, g.n, ELEMS);
  }
};

struct __align__(1024) Smem {
  signed char a[kDigits][kABytes];
  signed char b[kStages][kDigits * kBBytes];
  unsigned long long a_full, a_empty, b_full[kStages], b_empty[kStages], acc_full[2], acc_empty[2], drain;
  unsigned long long q_full[kQ], q_empty[kQ];
  int q[kQ];
  unsigned tmem_base;
  volatile int abort;
};
static_assert(sizeof(Smem) + 1024 <= 232448, "split update shared memory above the per-block limit");

__device__ __forceinline__ unsigned su32(const void *p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(unsigned long long *b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned parity, long bound = kWaitBound) {
  for (long i = 0; i < bound; ++i) {
    unsigned ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(su32(b)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load(void *dst, const CUtensorMap *map, int y, int z, unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
          "r"(su32(dst)),
      "l"(map), "r"(0), "r"(y), "r"(z), "r"(su32(bar))
      : "memory");
}
// K-major operand, 128-byte rows with 128-byte swizzle: 8-row groups 1024 bytes apart, version 1, layout 2.
__device__ __forceinline__ uint64_t smem_desc(const void *p) {
  const uint64_t addr = su32(p);
  return ((addr >> 4) & 0x3FFFull) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}
// kind::i8: D = S32, A = B = S8, both K-major, M = 128, N columns.
__device__ __forceinline__ constexpr uint32_t idesc(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTM >> 4) << 24);
}
__device__ __forceinline__ void umma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p; }" ::"r"(d),
      "l"(a), "l"(b), "r"(id), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned long long *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
               : "memory");
}

// --- the digit planes -------------------------------------------------------------------------------
// x 2^(61 - E) rounded to an integer, as eight signed base-256 digits, one per byte (digit 0, the
// highest, in the top byte): adding 128 to every digit makes all bytes non-negative without carries.
__device__ __forceinline__ unsigned long long digits_of(long long q) {
  constexpr unsigned long long kBias = 0x8080808080808080ull;
  return ((unsigned long long)q + kBias) ^ kBias;
}
// The scale of a row or column whose largest element has the high word `hi`: E, clamped so that both
// 2^(61 - E) and 2^(E - 5) are normal numbers, and 2^(E - 5), or NaN where an element is not finite
// (or past 2^900, whose products overflow).
__device__ __forceinline__ int scale_exponent(unsigned hi) { return max(-900, min(900, (int)(hi >> 20) - 1023)); }
__device__ __forceinline__ double exp2i(int e) { return __hiloint2double((e + 1023) << 20, 0); }
__device__ __forceinline__ double scale_of(unsigned hi) {
  const int e = (int)(hi >> 20) - 1023;
  return e > 900 ? __longlong_as_double(0x7ff8000000000000ll) : exp2i(scale_exponent(hi) - 5);
}
// Byte s of four 64-bit digit words, as one 32-bit word.
__device__ __forceinline__ unsigned gather(const unsigned long long (&w)[4], int s) {
  const int y = kDigits - 1 - s, sel = (y & 3) | ((y & 3) + 4) << 4;  // byte y & 3 of two half words
  unsigned h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = (unsigned)(y >= 4 ? w[i] >> 32 : w[i]);
  return __byte_perm(__byte_perm(h[0], h[1], sel), __byte_perm(h[2], h[3], sel), 0x5410);
}

// The balance of the inner indices: A's column p is taken times 2^s and B's row p times 2^-s, s half the
// difference of their largest exponents, so that no row of A and column of B spans a wide range against
// each other (the l-dependence of G and t at energies near zero).  Both sides' maxima are those of 64
// rows (columns) in eight groups over the range: the balance is a matter of accuracy only, so a sample does.
// Grid (njobs), 256 threads.
template <class Op>
__global__ void __launch_bounds__(256) balance_kernel(const JobDev *__restrict__ jobs, int k, Op op, SplitBufs sb) {
  __shared__ unsigned s_a[kNb], s_b[kNb];
  View g;
  if (!op(jobs[blockIdx.x], k, g)) return;
  const int tid = threadIdx.x;
  if (tid < kNb) s_a[tid] = s_b[tid] = 0u;
  __syncthreads();
  auto sample = [](int i, int n) { return min((i >> 3) * (max(n - 8, 0) / 7) + (i & 7), n - 1); };  // i < 64
  auto high = [](double2 v) {
    return max((unsigned)__double2hiint(v.x) & 0x7fffffffu, (unsigned)__double2hiint(v.y) & 0x7fffffffu);
  };
  const int q = tid >> 6, i = tid & 63, r = sample(i, g.m);
  double2 a[16], b[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int p = q + 4 * e;  // A: inner index; B: sampled column, inner index i
    a[e] = p < g.K ? g.A[r + (size_t)p * g.lda] : make_double2(0.0, 0.0);
    b[e] = i < g.K ? g.B[i + (size_t)sample(p, g.n) * g.ldb] : make_double2(0.0, 0.0);
  }
  unsigned hb = 0;
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const unsigned ha = __reduce_max_sync(0xffffffffu, high(a[e]));
    if ((tid & 31) == 0) atomicMax(&s_a[q + 4 * e], ha);
    hb = max(hb, high(b[e]));
  }
  atomicMax(&s_b[i], hb);
  __syncthreads();
  if (tid < kNb) {
    const int s = ((int)(s_b[tid] >> 20) - (int)(s_a[tid] >> 20)) / 2;
    sb.balance[blockIdx.x * kNb + tid] = s_a[tid] && s_b[tid] ? max(-kMaxBalance, min(kMaxBalance, s)) : 0;
  }
}

// Grid (rows / 32, njobs), 128 threads: lane = one complex row of A, warp w its columns 16 w .. + 15:
// their digits as real rows 2r (ar, -ai, ...) and 2r + 1 (ai, ar, ...), and the row's scale.
template <class Op>
__global__ void __launch_bounds__(128) pack_a_kernel(const JobDev *__restrict__ jobs, int k, Op op, SplitBufs sb) {
  __shared__ unsigned s_hi[4][32];
  const JobDev &J = jobs[blockIdx.y];
  View g;
  if (!op(J, k, g)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = blockIdx.x * 32 + lane, p0 = 16 * warp;
  if ((int)blockIdx.x * 32 >= g.m) return;
  const double2 *a = g.A + r;
  double2 v[16];
  unsigned hi = 0;
#pragma unroll
  for (int p = 0; p < 16; ++p)
    v[p] = r < g.m && p0 + p < g.K ? a[(size_t)(p0 + p) * g.lda] : make_double2(0.0, 0.0);
#pragma unroll
  for (int p = 0; p < 16; ++p) {
    const double f = exp2i(sb.balance[blockIdx.y * kNb + p0 + p]);
    v[p].x *= f;
    v[p].y *= f;
  }
#pragma unroll
  for (int p = 0; p < 16; ++p)
    hi = max(hi, max((unsigned)__double2hiint(v[p].x) & 0x7fffffffu, (unsigned)__double2hiint(v[p].y) & 0x7fffffffu));
  s_hi[warp][lane] = hi;
  __syncthreads();
  hi = max(max(s_hi[0][lane], s_hi[1][lane]), max(s_hi[2][lane], s_hi[3][lane]));
  if (r >= g.m) return;
  const double sc = exp2i(61 - scale_exponent(hi));
  if (warp == 0) sb.a_scale[(size_t)blockIdx.y * sb.ld + r] = scale_of(hi);
  signed char *dst = sb.a + (size_t)blockIdx.y * sb.a_slot + (size_t)(2 * r) * kRowBytes + 2 * p0;
  const size_t plane = (size_t)2 * sb.ld * kRowBytes;
#pragma unroll
  for (int b = 0; b < 2; ++b) {  // 16 bytes (8 columns) of every plane's two rows
    uint4 o[kDigits][2];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      unsigned long long top[4], bot[4];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double2 x = v[8 * b + 2 * h + e];
        const long long qr = __double2ll_rn(x.x * sc), qi = __double2ll_rn(x.y * sc);
        top[2 * e] = bot[2 * e + 1] = digits_of(qr);
        top[2 * e + 1] = digits_of(-qi);
        bot[2 * e] = digits_of(qi);
      }
#pragma unroll
      for (int s = 0; s < kDigits; ++s) {
        reinterpret_cast<unsigned *>(&o[s][0])[h] = gather(top, s);
        reinterpret_cast<unsigned *>(&o[s][1])[h] = gather(bot, s);
      }
    }
#pragma unroll
    for (int s = 0; s < kDigits; ++s) {
      *reinterpret_cast<uint4 *>(dst + s * plane + 16 * b) = o[s][0];
      *reinterpret_cast<uint4 *>(dst + s * plane + kRowBytes + 16 * b) = o[s][1];
    }
  }
}

// Grid (columns / 8, njobs), 256 threads: a warp per column of B, its digits and its scale.
template <class Op>
__global__ void __launch_bounds__(256) pack_b_kernel(const JobDev *__restrict__ jobs, int k, Op op, SplitBufs sb) {
  const JobDev &J = jobs[blockIdx.y];
  View g;
  if (!op(J, k, g)) return;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= g.n) return;
  const double2 *b = g.B + (size_t)c * g.ldb;
  double2 v[2];
  unsigned hi = 0;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int p = 2 * lane + e;
    v[e] = p < g.K ? b[p] : make_double2(0.0, 0.0);
    const double f = exp2i(-sb.balance[blockIdx.y * kNb + p]);
    v[e].x *= f;
    v[e].y *= f;
    hi = max(hi, max((unsigned)__double2hiint(v[e].x) & 0x7fffffffu, (unsigned)__double2hiint(v[e].y) & 0x7fffffffu));
  }
  hi = __reduce_max_sync(0xffffffffu, hi);
  const double sc = exp2i(61 - scale_exponent(hi));
  if (lane == 0) sb.b_scale[(size_t)blockIdx.y * sb.ld + c] = scale_of(hi);
  unsigned long long w[4];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    w[2 * e] = digits_of(__double2ll_rn(v[e].x * sc));
    w[2 * e + 1] = digits_of(__double2ll_rn(v[e].y * sc));
  }
  signed char *dst = sb.b + (size_t)blockIdx.y * sb.b_slot + (size_t)c * kRowBytes + 4 * lane;
  const size_t plane = (size_t)sb.ld * kRowBytes;
#pragma unroll
  for (int s = 0; s < kDigits; ++s) *reinterpret_cast<unsigned *>(dst + s * plane) = gather(w, s);
}

// a 2^24 + b 2^16 + c 2^8 + d of sums below 2^24, exactly: a 64-bit integer below 2^50 by four wide
// multiply-adds, made a double by adding it to the bits of 1.5 x 2^52.
__device__ __forceinline__ double digit_sum(unsigned a, unsigned b, unsigned c, unsigned d) {
  long long v;
  asm("{ .reg .s64 t;\n\t"
      "mad.wide.s32 t, %4, 1, %5;\n\t"
      "mad.wide.s32 t, %3, 256, t;\n\t"
      "mad.wide.s32 t, %2, 65536, t;\n\t"
      "mad.wide.s32 %0, %1, 16777216, t; }"
      : "=l"(v)
      : "r"(a), "r"(b), "r"(c), "r"(d), "l"(0x4338000000000000ll));
  return __longlong_as_double(v) - 6755399441055744.0;
}

// --- the update ----------------------------------------------------------------------------------
// Work items of a launch: item = (job, row panel, chunk of `len` column tiles), sized for the largest
// job.  skip_first: without the first 64 x 64 of C.
struct Items {
  int panels, chunks, len, total, skip_first;
};
struct Item {
  int z, row0, t0, t1;  // job, first complex row, column tiles [t0, t1)
};
template <class Op>
__device__ __forceinline__ bool item_of(const JobDev *jobs, const Items &is, int k, const Op &op, int i, View &g,
                                        Item &it) {
  const int per = is.panels * is.chunks;
  it.z = i / per;
  const int r = i - it.z * per, pm = r / is.chunks, ch = r - pm * is.chunks;
  if (!op(jobs[it.z], k, g)) return false;
  it.row0 = pm * kPanel;
  it.t0 = ch * is.len;
  it.t1 = min(it.t0 + is.len, (g.n + kTN - 1) / kTN);
  if (is.skip_first && pm == 0) it.t0 = max(it.t0, kNb / kTN);
  return it.row0 < g.m && it.t0 < it.t1;
}

template <class Op>
__global__ void __launch_bounds__(kThreads, 1)
    split_update_kernel(const __grid_constant__ CUtensorMap tA, const __grid_constant__ CUtensorMap tB,
                        const JobDev *__restrict__ jobs, int k, Op op, Items is, SplitBufs sb, int *counter, int *err) {
  extern __shared__ __align__(1024) unsigned char s8_raw[];
  Smem &sm = *reinterpret_cast<Smem *>((reinterpret_cast<uintptr_t>(s8_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&sm.a_full, 1);
    mbar_init(&sm.a_empty, 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&sm.b_full[s], 1);
      mbar_init(&sm.b_empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&sm.acc_full[a], 1);
      mbar_init(&sm.acc_empty[a], kEpiWarps / 2);
    }
    mbar_init(&sm.drain, 1);
    for (int q = 0; q < kQ; ++q) {
      mbar_init(&sm.q_full[q], 1);
      mbar_init(&sm.q_empty[q], 1 + kEpiWarps);  // the MMA warp and the epilogue warps
    }
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&sm.tmem_base)),
                 "r"(2 * kAccCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sm.tmem_base;
  auto expired = [&]() {
    atomicOr(err, kErrUpdateWait);
    sm.abort = 1;
  };

  if (warp == 0) {
    if (lane == 0) {
      int items = 0;  // published
      long g = 0;     // B tiles requested
      View v;
      Item it;
      for (;;) {
        int i = atomicAdd(counter, 1);
        while (i < is.total && !item_of(jobs, is, k, op, i, v, it)) i = atomicAdd(counter, 1);
        const bool more = i < is.total && !sm.abort;
        const int q = items % kQ;
        if (items >= kQ && !mbar_wait(&sm.q_empty[q], (unsigned)(((items / kQ) - 1) & 1))) {
          expired();
          break;
        }
        sm.q[q] = more ? i : -1;
        mbar_arrive(&sm.q_full[q]);
        if (!more) break;
        if (items > 0 && !mbar_wait(&sm.a_empty, (unsigned)((items - 1) & 1))) {
          expired();
          break;
        }
        ++items;
        mbar_expect_tx(&sm.a_full, kDigits * kABytes);
        for (int s = 0; s < kDigits; ++s) tma_load(sm.a[s], &tA, 2 * (s * sb.ld + it.row0), it.z, &sm.a_full);
        bool ok = true;
        for (int t = it.t0; t < it.t1; ++t, ++g) {
          const int st = (int)(g % kStages);
          if (g >= kStages && !mbar_wait(&sm.b_empty[st], (unsigned)(((g / kStages) - 1) & 1))) {
            ok = false;
            break;
          }
          mbar_expect_tx(&sm.b_full[st], kDigits * kBBytes);
          for (int s = 0; s < kDigits; ++s)
            tma_load(sm.b[st] + s * kBBytes, &tB, s * sb.ld + t * kTN, it.z, &sm.b_full[st]);
        }
        if (!ok) {
          expired();
          break;
        }
      }
      // every issued load has landed before the CTA can exit (normally already true)
      if (items > 0 && !mbar_wait(&sm.a_full, (unsigned)((items - 1) & 1), kDrainPolls)) expired();
      for (long q = g > kStages ? g - kStages : 0; q < g; ++q)
        if (!mbar_wait(&sm.b_full[q % kStages], (unsigned)((q / kStages) & 1), kDrainPolls)) expired();
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int items = 0, li = 0;  // items and tiles started
      long g = 0;
      bool ok = true;
      View v;
      Item it;
      while (ok) {
        const int q = items % kQ;
        if (!mbar_wait(&sm.q_full[q], (unsigned)((items / kQ) & 1))) {
          expired();
          break;
        }
        const int i = sm.q[q];
        mbar_arrive(&sm.q_empty[q]);
        if (i < 0) break;
        item_of(jobs, is, k, op, i, v, it);
        ok = mbar_wait(&sm.a_full, (unsigned)(items & 1));
        ++items;
        for (int t = it.t0; ok && t < it.t1; ++t, ++g, ++li) {
          const int st = (int)(g % kStages), a = li & 1;
          ok = (li < 2 || mbar_wait(&sm.acc_empty[a], (unsigned)(((li >> 1) - 1) & 1))) &&
               mbar_wait(&sm.b_full[st], (unsigned)((g / kStages) & 1));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t d = tmem + (uint32_t)(a * kAccCols);
          const uint64_t db = smem_desc(sm.b[st]);
#pragma unroll
          for (int s = 0; s < kDigits; ++s) {
            const uint64_t da = smem_desc(sm.a[s]);
#pragma unroll
            for (int ks = 0; ks < kRowBytes / 32; ++ks)  // digit s of A by digits 0 .. 7 - s of B
              umma_i8(d + (uint32_t)(s * kTN), da + 2 * ks, db + 2 * ks, idesc(kTN * (kDigits - s)),
                      (s > 0 || ks > 0) ? 1u : 0u);
          }
          umma_commit(&sm.b_empty[st]);
          umma_commit(&sm.acc_full[a]);
        }
        if (!ok) {
          expired();
          break;
        }
        umma_commit(&sm.a_empty);
      }
      umma_commit(&sm.drain);
      if (!mbar_wait(&sm.drain, 0, kDrainPolls)) expired();
    }
  } else {
    // Four epilogue warps take 16 columns of accumulator set `grp`: warp w reads tensor-memory lanes
    // 32 (w % 4) .. + 31, lane = real row, in pieces of four columns.
    const int grp = ((warp - 2) >> 2) & 1, half = (warp - 2) >> 3, quarter = warp & 3, rr = 32 * quarter + lane;
    int items = 0, li = 0;
    bool ok = true;
    View v;
    Item it;
    while (ok) {
      const int q = items % kQ;
      int i = -1;
      if (lane == 0) {
        if (mbar_wait(&sm.q_full[q], (unsigned)((items / kQ) & 1))) {
          i = sm.q[q];
          mbar_arrive(&sm.q_empty[q]);
        } else {
          expired();
        }
      }
      i = __shfl_sync(0xffffffffu, i, 0);
      if (i < 0) break;
      ++items;
      item_of(jobs, is, k, op, i, v, it);
      const int r = it.row0 + (rr >> 1);  // complex row
      const bool row_in = r < v.m;
      // the row's scale, with the 2^-24 of the digit sums below
      const double as = row_in ? sb.a_scale[(size_t)it.z * sb.ld + r] * 5.9604644775390625e-08 : 0.0;
      double *Cr = reinterpret_cast<double *>(v.C + r) + (rr & 1);
      const size_t ldc = (size_t)2 * v.ldc;
      for (int t = it.t0; t < it.t1; ++t, ++li) {
        if ((li & 1) != grp) continue;
        const int c0 = t * kTN + half * kEpiCols, nc = row_in ? min(kEpiCols, v.n - c0) : 0;
        double *C = Cr + (size_t)c0 * ldc;
        // lane l < 16: the scale of column c0 + l
        const double bs =
            lane < kEpiCols && c0 + lane < v.n ? sb.b_scale[(size_t)it.z * sb.ld + c0 + lane] : 0.0;
        double cv[kEpiCols];
#pragma unroll
        for (int c = 0; c < kEpiCols; ++c) cv[c] = c < nc ? C[c * ldc] : 0.0;
        // the set's next tile of C on its way to L2: lane = (column, 128-byte half of the warp's rows)
        {
          const int pc = c0 + 2 * kTN + (lane >> 1), pr = it.row0 + 16 * quarter + 8 * (lane & 1);
          if (t + 2 < it.t1 && pc < v.n && pr < v.m)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(v.C + pr + (size_t)pc * v.ldc));
        }
        int fine = 1;
        if (lane == 0 && !mbar_wait(&sm.acc_full[grp], (unsigned)((li >> 1) & 1))) {
          expired();
          fine = 0;
        }
        ok = __shfl_sync(0xffffffffu, fine, 0) != 0;
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c4 = 0; c4 < kEpiCols; c4 += 4) {
          uint32_t d[kDigits][4];
#pragma unroll
          for (int s = 0; s < kDigits; ++s)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(d[s][0]), "=r"(d[s][1]), "=r"(d[s][2]), "=r"(d[s][3])
                         : "r"(tmem + ((uint32_t)(32 * quarter) << 16) +
                               (uint32_t)(grp * kAccCols + s * kTN + half * kEpiCols + c4))
                         : "memory");
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            // sum of the digit sums times 256^-w, w = 0 .. 7, times 2^24: h + l 2^-32
            const double h = digit_sum(d[0][e], d[1][e], d[2][e], d[3][e]);
            const double l = digit_sum(d[4][e], d[5][e], d[6][e], d[7][e]);
            cv[c4 + e] -= fma(l, 2.3283064365386963e-10, h) * (as * __shfl_sync(0xffffffffu, bs, c4 + e));
          }
        }
        // this part of the accumulator set has been read out
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.acc_empty[grp]);
#pragma unroll
        for (int c = 0; c < kEpiCols; ++c)
          if (c < nc) C[c * ldc] = cv[c];
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kAccCols) : "memory");
  }
}

// Packs and update of step k for every job: max_m x max_n bounds the jobs' C.  `counter`: one of sb's
// work counters, zero.
template <class Op>
cudaError_t launch_split_update(const SplitBufs &sb, const JobDev *jobs, int njobs, int k, int max_m, int max_n,
                                bool skip_first, int *counter, int *err, cudaStream_t s, const Op &op) {
  const int smem = (int)sizeof(Smem) + 1024;
  const cudaError_t e = ensure_smem(split_update_kernel<Op>, smem);
  if (e != cudaSuccess) return e;
  Items is;
  is.panels = (max_m + kPanel - 1) / kPanel;
  // two items or more per SM where there are few tiles, long ones (a panel is loaded once per item)
  // where there are many
  const int tiles = (max_n + kTN - 1) / kTN;
  is.len = (int)std::max<long>(kMinTiles, std::min<long>(kMaxTiles, (long)is.panels * tiles * njobs / (2 * tc_num_sms())));
  is.chunks = (tiles + is.len - 1) / is.len;
  is.total = is.panels * is.chunks * njobs;
  is.skip_first = skip_first ? 1 : 0;
  split_update_kernel<Op><<<std::min(is.total, tc_num_sms()), kThreads, smem, s>>>(sb.tA, sb.tB, jobs, k, op, is, sb,
                                                                                   counter, err);
  return cudaGetLastError();
}
template <class Op>
cudaError_t launch_split_pack(const SplitBufs &sb, const JobDev *jobs, int njobs, int k, int max_m, int max_n,
                              cudaStream_t s, const Op &op) {
  balance_kernel<Op><<<njobs, 256, 0, s>>>(jobs, k, op, sb);
  pack_a_kernel<Op><<<dim3((max_m + 31) / 32, njobs), 128, 0, s>>>(jobs, k, op, sb);
  pack_b_kernel<Op><<<dim3((max_n + 7) / 8, njobs), 256, 0, s>>>(jobs, k, op, sb);
  return cudaGetLastError();
}

}  // namespace s8
}  // namespace b200
