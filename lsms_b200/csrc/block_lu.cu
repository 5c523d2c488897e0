// Block elimination and iterative refinement for tau00 (batched over jobs).
//
// Restates the reference's block LU contract (zblock_lu_cpp.cpp:19-86, zblock_lu_CPU.f:2-82,
// block_inverse.cpp:24-47, tau_inv_postproc.f:1-77 / linearSolvers_CPU.cpp:299-330):
//   Delta = M0r Mrr^-1 Mr0,  tau00 = (1 - Delta)^-1 t0,  tau00_l = rotate(tau00 - t0).
// The reference eliminates bottom-up with pivoting restricted to each diagonal block (zgetrf on
// the block, zgetrs on its block row, zgemm on the rest; its CUDA variant
// zblock_lu_cuda_c.cu:56-353 re-blocks to 55 columns and inverts each diagonal block).
// Here M is stored with the central site last and eliminated top-down in 64-column steps on the
// factor storage F (FP64 or FP32):
//   diag_inverse_kernel   D = A11^-1, Gauss-Jordan with partial pivoting inside the block (FP64)
//   W = D A12 in place over the block row
//   A22 -= A21 W over the trailing matrix (the O(N^3) part)
// FP64 factors take both as tiles on the FP64 tensor cores (dmma.cuh); FP32 factors as FP32 tiles
// (zgemm_tile_kernel), or the update on the TF32 tensor cores (tc_update.cu).
// After n = N - b columns the trailing b x b block holds S = 1 - Delta and F holds, in place, the
// block factors {D_k in the diagonal blocks, A21_k below them, W_k to their right}.
// Without refinement, finalize solves S tau00 = t0.  With refinement (the reference's zcgesv /
// cusolverDnIRSXgesv idea, linearSolvers_CPU.cpp:148-174, linearSolvers_CUDA.cu:424-469, applied
// to the N x b system M X = [0; t0]):
//   X = F^-1 B;  repeat: R = B - M X (FP64, M unmodified), Y = F^-1 R, X += Y;
// where F^-1 is a forward sweep (Y_k = D_k R_k, R_below -= A21_k Y_k), the S solve, and a backward
// sweep (Y_above -= W Y_k), each one launch with a thread-block cluster per job (sweep.cu).
// tau00 = X[n:N].

#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "cluster.cuh"
#include "cplx.cuh"
#include "dmma.cuh"
#include "gj.cuh"
#include "split8.cuh"

namespace b200 {
namespace {

using namespace cx;

// ---------------------------------------------------------------------------------------------
// In-place inverse of the kb x kb diagonal block at (k, k) of F, kb <= 64: FP64 Gauss-Jordan with
// partial pivoting inside the block on |re| + |im| (izamax's measure; ties go to the lowest row).
// Rows are never interchanged: step p pivots on the not-yet-used row pv with the largest
// |A[pv][p]|, and the permutation is applied when the block is written back (for the in-place
// result P, A^-1[i][pv_k] = P[pv_i][k]).
// One step subtracts g u^T from every column but p, u = row pv, g_r = A[r][p] / d (d = A[pv][p]) and
// g_pv = 1 - 1/d, which leaves row pv divided by d; column p becomes -g_r, and 1/d in row pv.
//
// What bounds the kernel is the chain from one pivot to the next, so the block is taken in panels of
// eight columns.  One warp does a panel's eight steps in registers (lane l rows l and l + 32, columns
// rotating through the places so that the next one to search is always the first), where a step needs
// no barrier and no shared memory: the pivot is a warp argmax on 64-bit keys, beside which every lane
// computes the reciprocal of its own candidate, and row pv is shuffled out of its lane.  The panel's
// result X holds the columns e_pv of the eight steps' product, so every other column then takes
// C += X U, U = the panel's pivot rows, with those rows of C cleared first: 8 x 8 x 8 products on the FP64
// tensor cores.  All eight warps update the next panel; the other columns are updated by six warps, one
// block of eight columns each, while the next panel's steps run (the warp that would share the
// scheduler of the panel's stays idle).
// A full block takes 47.5 k cycles, 742 a step, against 75.7 k with every step over all 64 columns, where the
// eight warps wait for row pv to pass through shared memory (300 cycles of a step) and for a barrier; panels
// of four columns take 54.0 k.  A launch takes 33 us (45 us).  One mixed solve
// of N = 2160: 5.25 -> 4.85 ms; one of N = 240: 0.43 -> 0.38 ms.
// ---------------------------------------------------------------------------------------------
constexpr int kDiagThreads = 256;
static_assert(kDiagThreads == 256 && kNb == 64, "diagonal inverse layout: 2 rows per lane, 8 panels, 8 row tiles");

// PER_SM = blocks per SM the register budget allows: 1 (for the elimination that keeps one SM per job
// free for the inverses) or 2 (for the elimination with panel pivoting, which leaves fewer SMs to them).
template <typename T, int PER_SM>
__global__ void __launch_bounds__(kDiagThreads, PER_SM) diag_inverse_kernel(const JobDev *__restrict__ jobs, int k,
                                                                            int *info) {
  constexpr int NB = kNb, kStride = NB + 1, kMb = NB / 8;
  const JobDev &J = jobs[blockIdx.x];
  if (k >= J.n || J.inactive) return;
  const int kb = min(NB, J.n - k);
  const int np = (kb + 7) / 8, kbp = 8 * np;  // panels; rows and columns kb .. kbp - 1 are the identity's
  extern __shared__ __align__(16) double2 dyn_smem[];
  double2(*As)[kStride] = reinterpret_cast<double2(*)[kStride]>(dyn_smem);  // As[column][row]
  // Us[column][step]: 8 steps of a column in 192 bytes, so that a fragment's eight lanes (two columns,
  // four steps) hit eight 16-byte banks
  __shared__ double2 Us[NB][12];
  __shared__ int s_sing;
  __shared__ int s_pv[NB], s_inv[NB], s_hi[kDiagThreads / 32];
  T *__restrict__ Fk = static_cast<T *>(J.F) + (size_t)k + (size_t)k * J.ld;
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  constexpr int kPer = NB * NB / kDiagThreads;  // entries per thread of a full block
  // the block is inverted times a power of two that brings its largest element to 1 .. 2: the squares of
  // its pivots stay in range, and 1 - 1/d does not lose the digits of a large d
  double scale;
  {
    // all of a thread's loads in flight at once (a loop over them waits out one DRAM round trip
    // per entry)
    double2 v[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int e = tid + i * kDiagThreads, r = e % NB, c = e / NB;
      v[i] = r < kb && c < kb ? ldc(Fk + r + (size_t)c * J.ld) : make_double2(0.0, 0.0);
    }
    int hi = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      hi = max(hi, max(__double2hiint(v[i].x) & 0x7fffffff, __double2hiint(v[i].y) & 0x7fffffff));
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (l == 0) s_hi[w] = hi;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kDiagThreads / 32; ++i) hi = max(hi, s_hi[i]);
    const int e2 = hi >> 20;  // (0x7ff: an element is not finite)
    scale = e2 == 0x7ff ? 1.0 : __hiloint2double(max(1, 2046 - e2) << 20, 0);
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int e = tid + i * kDiagThreads, r = e % NB, c = e / NB;
      As[c][r] = r < kb && c < kb ? make_double2(v[i].x * scale, v[i].y * scale)
                                  : make_double2(r == c ? 1.0 : 0.0, 0.0);
    }
  }
  if (tid < NB) s_pv[tid] = s_inv[tid] = tid;  // every entry in range whatever the pivots
  if (tid == 0) s_sing = 0;
  __syncthreads();
  bool used0 = l >= kbp, used1 = l + 32 >= kbp;  // rows already pivoted on (warp 0)
  // C += X U for the 8 x 8 block (mb, nb) of A, X = the finished panel q
  auto update = [&](int mb, int nb, int q) {
    const int r = 8 * mb + (l >> 2);
    double2 *c0 = &As[8 * nb + 2 * (l & 3)][r], *c1 = c0 + kStride;
    double re[2], im[2];
    re[0] = c0->x, im[0] = c0->y, re[1] = c1->x, im[1] = c1->y;
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      const double2 x = As[8 * q + 4 * ks + (l & 3)][r], u = Us[8 * nb + (l >> 2)][4 * ks + (l & 3)];
      dm::mma_884(re[0], re[1], x.x, u.x);
      dm::mma_884(im[0], im[1], x.x, u.y);
      dm::mma_884(re[0], re[1], -x.y, u.y);
      dm::mma_884(im[0], im[1], x.y, u.x);
    }
    *c0 = make_double2(re[0], im[0]);
    *c1 = make_double2(re[1], im[1]);
  };
  for (int q = 0; q < np; ++q) {
    if (w == 0) {
      // the panel's eight steps; place j of a[.][] holds column 8q + ((p + j) & 7)
      double2 a[2][8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        a[0][j] = As[8 * q + j][l];
        a[1][j] = As[8 * q + j][l + 32];
      }
      // the unused row of largest |re| + |im| of the next column, as the largest 64-bit key, and 1/d;
      // beside the argmax every lane takes the reciprocal of its own candidate
      int pv;
      double2 dinv;
      auto search = [&](double2 x0, double2 x1) {
        const unsigned long long k0 = used0 ? 0ull : pivot_key(cabs1(x0), l);
        const unsigned long long k1 = used1 ? 0ull : pivot_key(cabs1(x1), l + 32);
        const bool first = k0 > k1;
        const double2 rl = reciprocal(first ? x0 : x1);
        pv = min(pivot_row(first ? k0 : k1), kbp - 1);  // (a row < kbp: some are unused)
        dinv.x = __shfl_sync(0xffffffffu, rl.x, pv & 31);
        dinv.y = __shfl_sync(0xffffffffu, rl.y, pv & 31);
      };
      search(a[0][0], a[1][0]);
#pragma unroll 1
      for (int p = 0; p < 8; ++p) {
        const int pc = pv, pl = pv & 31;
        const bool hi = pv >= 32, is0 = l == pv, is1 = l + 32 == pv;
        const double2 di = dinv, h0 = cmul(a[0][0], di), h1 = cmul(a[1][0], di);
        const double2 one = make_double2(1.0 - di.x, -di.y);
        const double2 g0 = is0 ? one : h0, g1 = is1 ? one : h1;
        used0 |= is0;
        used1 |= is1;
        {
          const double2 v = hi ? a[1][1] : a[0][1];
          double2 u;
          u.x = __shfl_sync(0xffffffffu, v.x, pl);
          u.y = __shfl_sync(0xffffffffu, v.y, pl);
          a[0][0] = cfnma(a[0][1], g0, u);
          a[1][0] = cfnma(a[1][1], g1, u);
        }
        search(a[0][0], a[1][0]);  // (after the last step: a finished column, not used)
#pragma unroll
        for (int j = 2; j < 8; ++j) {
          const double2 v = hi ? a[1][j] : a[0][j];
          double2 u;
          u.x = __shfl_sync(0xffffffffu, v.x, pl);
          u.y = __shfl_sync(0xffffffffu, v.y, pl);
          a[0][j - 1] = cfnma(a[0][j], g0, u);
          a[1][j - 1] = cfnma(a[1][j], g1, u);
        }
        a[0][7] = is0 ? di : make_double2(-h0.x, -h0.y);
        a[1][7] = is1 ? di : make_double2(-h1.x, -h1.y);
        if (l == 0) {
          s_pv[8 * q + p] = pc;
          s_inv[pc] = 8 * q + p;
          if (di.x == 0.0 && di.y == 0.0) s_sing = 1;
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        As[8 * q + j][l] = a[0][j];
        As[8 * q + j][l + 32] = a[1][j];
      }
    } else if (q > 0 && (w & 3)) {
      // meanwhile the step before, on the columns past the next panel: one block column a warp
      int nb = (w & 3) - 1 + (w > 4 ? 3 : 0);  // 0 .. 5 over the blocks other than q - 1 and q
      if (nb >= q - 1) nb += 2;
      if (nb < np)
#pragma unroll 2
        for (int mb = 0; mb < kMb; ++mb) update(mb, nb, q - 1);
    }
    __syncthreads();
    // U = the pivot rows, which A's update then builds from zero
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int e = tid + i * kDiagThreads, c = e >> 3, pr = s_pv[8 * q + (e & 7)];
      if ((c >> 3) != q) {
        Us[c][e & 7] = As[c][pr];
        As[c][pr] = make_double2(0.0, 0.0);
      }
    }
    __syncthreads();
    if (q + 1 < np) update(w, q + 1, q);
    else
      for (int nb = 0; nb < np - 1; ++nb) update(w, nb, q);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = tid + i * kDiagThreads, r = e % NB, c = e / NB;
    if (r < kb && c < kb) {
      const double2 v = As[s_inv[c]][s_pv[r]];
      stc(Fk + r + (size_t)c * J.ld, make_double2(v.x * scale, v.y * scale));
    }
  }
  if (s_sing && tid == 0) atomicCAS(&info[blockIdx.x], 0, k + 1);
}

template <typename T>
void launch_diag_inverse(bool packed, const JobDev *jobs, int njobs, int k, int *info, int smem, cudaStream_t s) {
  if (packed) diag_inverse_kernel<T, 2><<<njobs, kDiagThreads, smem, s>>>(jobs, k, info);
  else diag_inverse_kernel<T, 1><<<njobs, kDiagThreads, smem, s>>>(jobs, k, info);
}

// ---------------------------------------------------------------------------------------------
// Complex GEMM tile on FP32 factors (SIMT), C (m x n) = A (m x K) B (K x n)  [kOverwrite, in place over B]
//                                           C (m x n) -= A (m x K) B (K x n) [kSubtract]
// 64 x 64 complex tile per CTA, 256 threads, 4 x 4 complex accumulators per thread, each one packed
// (re, im) pair: a complex multiply-add is two packed FMAs (fma.rn.f32x2, the same four products and
// roundings as scalar FMAs), which leaves half the issue slots to the operand loads.  The whole
// K <= 64 of both operands is requested by cp.async at once, in four K chunks of 16 that are
// multiplied as they land, so a CTA waits out one memory round trip.  (31 mixed jobs of
// N = 2160: the elimination took 8.97 ms with scalar FMAs and a two-stage ring, 8.29 with these.)
// Thread (tx, ty) owns rows 2 tx, 2 tx + 1, 32 + 2 tx, 33 + 2 tx (16-byte shared-memory loads and
// stores) and columns ty + 16 j.
// ---------------------------------------------------------------------------------------------
constexpr int kTile = 64;
constexpr int kKc = 16;
constexpr int kTileBs = kNb + 2;  // B's columns in shared memory, padded to 16 bytes modulo 128
constexpr int kTileSmem = (kNb * kTile + kTile * kTileBs) * (int)sizeof(float2);
using dm::kOverwrite;
using dm::kSubtract;

// Optional second output of the W = D A12 tiles (FP32, tensor-core path): W's hi/lo TF32 split in
// the K-major operand layout of the trailing update (column c of the trailing block at
// b + z * slot + c * kTcKMax + k_off floats, (re, im) of row p at 2 p), job z = the launch's job
// index.  With shift_k >= 0 the trailing block is that of the next step shift_k (its columns
// start kb(shift_k) further right; W's columns left of it are not packed), and this step's rows
// go to K offset k_off: the first half of a two-step update's operand.
struct PackB {
  float *hi = nullptr, *lo = nullptr;
  size_t slot = 0;
  int shift_k = -1;
  int k_off = 0;
};

__device__ __forceinline__ float tf32_round(float x) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// Packed (x, y) pairs of FP32 in a 64-bit register, and d += a b elementwise.
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(unsigned long long &d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
// 16 bytes to shared memory of which the first `bytes` (0, 8 or 16) are read and the rest are zeros.
__device__ __forceinline__ void cp_async16_part(void *smem, const void *gmem, int bytes) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}

template <int MODE>
__device__ __forceinline__ void zgemm_tile_body(const JobDev &J, int k, int bx, int by, int bx0, int by0,
                                                const PackB &pk = PackB(), int z = 0) {
  using T = float2;
  const int N = J.N, ld = J.ld;
  if (k >= J.n || J.inactive) return;
  const int kb = min(kNb, J.n - k);
  const int K = kb;
  T *__restrict__ F = static_cast<T *>(J.F);
  int row0, m;
  const T *Ab;
  const int col0 = k + kb + (bx + bx0) * kTile;
  int n = N - col0;
  if (n <= 0) return;
  if (MODE == kOverwrite) {
    if (by != 0) return;
    row0 = k;
    m = kb;
    Ab = F + (size_t)k + (size_t)k * ld;  // D (kb x kb)
  } else {
    row0 = k + kb + (by + by0) * kTile;
    m = N - row0;
    if (m <= 0) return;
    Ab = F + (size_t)row0 + (size_t)k * ld;  // A21
  }
  const T *Bb = F + (size_t)k + (size_t)col0 * ld;  // A12 / W
  T *Cb = F + (size_t)row0 + (size_t)col0 * ld;
  m = min(m, kTile);
  n = min(n, kTile);

  extern __shared__ __align__(16) unsigned char zsm[];
  T(*As)[kTile] = reinterpret_cast<T(*)[kTile]>(zsm);                                    // As[kk][row]
  T(*Bs)[kTileBs] = reinterpret_cast<T(*)[kTileBs]>(zsm + kNb * kTile * sizeof(T));  // Bs[col][kk]
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int nchunks = (K + kKc - 1) / kKc;
  // rows of A start on an odd one (8 bytes off a 16-byte boundary) only after an odd last step
  const bool aligned = (row0 & 1) == 0;
#pragma unroll
  for (int ch = 0; ch < kNb / kKc; ++ch) {
    if (ch < nchunks) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int e = tid + q * 256;
        const int r = (e & 31) * 2, kk = ch * kKc + (e >> 5);
        const int left = kk < K ? max(0, min(2, m - r)) : 0;
        const T *src = left > 0 ? Ab + r + (size_t)kk * ld : Ab;
        if (aligned) {
          cp_async16_part(&As[kk][r], src, 8 * left);
        } else {
          As[kk][r] = left > 0 ? src[0] : make_float2(0.f, 0.f);
          As[kk][r + 1] = left > 1 ? src[1] : make_float2(0.f, 0.f);
        }
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int e = tid + q * 256;
        const int kk = ch * kKc + (e & 7) * 2, c = e >> 3;
        const int left = c < n ? max(0, min(2, K - kk)) : 0;
        cp_async16_part(&Bs[c][kk], left > 0 ? Bb + kk + (size_t)c * ld : Bb, 8 * left);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  if (MODE == kSubtract) {  // C's lines on their way to L2 while the product runs
    const int r = (tid & 3) * 16, c = tid >> 2;
    if (r < m && c < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(Cb + r + (size_t)c * ld));
  }

  unsigned long long acc2[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc2[i][j] = 0ull;
#pragma unroll
  for (int ch = 0; ch < kNb / kKc; ++ch) {
    if (ch >= nchunks) break;
    if (ch == 0) asm volatile("cp.async.wait_group 3;" ::: "memory");
    else if (ch == 1) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else if (ch == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int k2 = 0; k2 < kKc; k2 += 2) {
      const int kk = ch * kKc + k2;
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4 *>(&Bs[ty + 16 * j][kk]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 a01 = *reinterpret_cast<const float4 *>(&As[kk + h][2 * tx]);
        const float4 a23 = *reinterpret_cast<const float4 *>(&As[kk + h][32 + 2 * tx]);
        const float ar[4] = {a01.x, a01.z, a23.x, a23.z}, ai[4] = {a01.y, a01.w, a23.y, a23.w};
        unsigned long long bp[4], bs[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float br = h ? b[j].z : b[j].x, bi = h ? b[j].w : b[j].y;
          bp[j] = pack2(br, bi);
          bs[j] = pack2(-bi, br);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned long long ax = pack2(ar[i], ar[i]), ay = pack2(ai[i], ai[i]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            fma2(acc2[i][j], ax, bp[j]);
            fma2(acc2[i][j], ay, bs[j]);
          }
        }
      }
    }
  }
  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = unpack2(acc2[i][j]);
  // for kOverwrite every read of B = C (into shared memory) happened before the last __syncthreads
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = ty + 16 * j;
    if (c >= n) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 2 * tx + (i & 1) + 32 * (i >> 1);
      if (MODE == kOverwrite && pk.hi != nullptr) {
        // rows past kb pack as zero
        const int shift = pk.shift_k >= 0 ? min(kNb, J.n - pk.shift_k) : 0;
        const int prow = (bx + bx0) * kTile + c - shift;
        if (prow >= 0) {
          const float wr = r < m ? acc[i][j].x : 0.f, wi = r < m ? acc[i][j].y : 0.f;
          const float hr = tf32_round(wr), hi = tf32_round(wi);
          const size_t o = (size_t)z * pk.slot + (size_t)prow * kTcKMax + pk.k_off;
          reinterpret_cast<float2 *>(pk.hi + o)[r] = make_float2(hr, hi);
          reinterpret_cast<float2 *>(pk.lo + o)[r] = make_float2(wr - hr, wi - hi);
        }
      }
      if (r >= m) continue;
      T *dst = Cb + (size_t)r + (size_t)c * ld;
      if (MODE == kOverwrite) {
        *dst = acc[i][j];
      } else {
        const T cv = *dst;
        *dst = T{cv.x - acc[i][j].x, cv.y - acc[i][j].y};
      }
    }
  }
}

// One output tile per (bx, by, job).  Two resident CTAs per SM: with K = 64 per step each CTA runs
// only four K-chunks, so its operand prologue and C read-modify-write latencies are hidden by the
// other CTA's FMAs.  Tiles start at column tile bx0 and row tile by0 of the step's trailing block.
template <int MODE>
__global__ void __launch_bounds__(256, 2) zgemm_tile_kernel(const JobDev *__restrict__ jobs, int k, PackB pk, int bx0,
                                                            int by0 = 0) {
  zgemm_tile_body<MODE>(jobs[blockIdx.z], k, blockIdx.x, blockIdx.y, bx0, by0, pk, blockIdx.z);
}

// Step k's update of the two strips a paired step k2 = k + 64 needs before its own W (block
// pivoting): block column k2 below its diagonal block (CTAs x < t1: row tiles 1 .. t1) and block
// row k2 right of it (x >= t1: column tiles 1 .. t1), one grid of 2 t1 x njobs CTAs, so that the
// last wave of one strip shares the GPU with the other.
__global__ void __launch_bounds__(256, 2) zgemm_strips_kernel(const JobDev *__restrict__ jobs, int k, int t1) {
  const int x = blockIdx.x;
  if (x < t1) zgemm_tile_body<kSubtract>(jobs[blockIdx.z], k, 0, x, 0, 1);
  else zgemm_tile_body<kSubtract>(jobs[blockIdx.z], k, x - t1, 0, 1, 0);
}

// ---------------------------------------------------------------------------------------------
// The same products on FP64 factors, tiles on the FP64 tensor cores (dmma.cuh):
// step k's W = D A12 (kOverwrite) and A22 -= A21 W (kSubtract).
// ---------------------------------------------------------------------------------------------
// A column of `len` tiles of step k's trailing block from tile (bx, by) down.
template <int W>
__device__ __forceinline__ void update64_column(const JobDev &J, int k, int bx, int by, int len, double2 *sm) {
  constexpr int R = dm::Tile<W, W>::kRows, C = dm::Tile<W, W>::kCols;
  const int N = J.N, ld = J.ld;
  const int kb = min(kNb, J.n - k);
  double2 *F = static_cast<double2 *>(J.F);
  const int col0 = k + kb + bx * C, row0 = k + kb + by * R;
  if (col0 >= N || row0 >= N) return;
  dm::zgemm_column<W, W, kSubtract>(F + (size_t)row0 + (size_t)k * ld, ld, F + (size_t)k + (size_t)col0 * ld, ld,
                                      F + (size_t)row0 + (size_t)col0 * ld, ld, min(len * R, N - row0),
                                      min(C, N - col0), kb, sm);
}

// Which tiles of the trailing block an update launch covers: all, the ones of its first 64 x 64
// (the next step's diagonal block), or the others.
enum { kAllTiles = 0, kFirstBlock = 1, kOtherTiles = 2 };

// Step k's update as the integer tensor cores take it (split8.cuh).
struct OpTrailing {
  __device__ bool operator()(const JobDev &J, int k, s8::View &g) const {
    if (k >= J.n || J.inactive) return false;
    const int kb = min(kNb, J.n - k), e = k + kb;
    double2 *F = static_cast<double2 *>(J.F);
    g.A = F + (size_t)e + (size_t)k * J.ld;
    g.B = F + (size_t)k + (size_t)e * J.ld;
    g.C = F + (size_t)e + (size_t)e * J.ld;
    g.lda = g.ldb = g.ldc = J.ld;
    g.m = g.n = J.N - e;
    g.K = kb;
    return g.m > 0;
  }
};

// W = D A12 overwrites its own operand, so a CTA takes all kb rows of its columns.
template <int WN>
__global__ void __launch_bounds__(dm::kThreads, 2) zgemm64_w_kernel(const JobDev *__restrict__ jobs, int k) {
  extern __shared__ __align__(16) double2 zsm64[];
  const JobDev &J = jobs[blockIdx.z];
  if (k >= J.n || J.inactive) return;
  const int ld = J.ld, kb = min(kNb, J.n - k);
  double2 *F = static_cast<double2 *>(J.F);
  const int col0 = k + kb + blockIdx.x * dm::Tile<4, WN>::kCols;
  if (col0 >= J.N) return;
  double2 *A12 = F + (size_t)k + (size_t)col0 * ld;
  dm::zgemm_column<4, WN, kOverwrite>(F + (size_t)k + (size_t)k * ld, ld, A12, ld, A12, ld, kb,
                                      min(dm::Tile<4, WN>::kCols, J.N - col0), kb, zsm64);
}

// Tiles of 16 W x 16 W in columns of `len`: tx columns of tiles, ty rows of columns.  W = 2, or 1 for the
// next diagonal block of a few jobs (a tile keeps its SM's FP64 pipe for 2.2 us with W = 2).  Four CTAs of four warps
// on an SM: 31 jobs of N = 2160 took 32.3 ms of updates with 64 x 64 tiles at two CTAs, 28.4 with
// 64 x 32 at three, 27.9 with these at four (48.2 -> 30.0 ms for the whole elimination, from DFMA tiles
// without look-ahead).
template <int W>
__global__ void __launch_bounds__(dm::kThreads, 4) zgemm64_update_kernel(const JobDev *__restrict__ jobs, int k, int tx,
                                                                         int ty, int nj, int part, int len, bool sparse, bool small) {
  extern __shared__ __align__(16) double2 zsm64[];
  using TL = dm::Tile<W, W>;
  if (!sparse) {  // grid (tx, ty, nj)
    const JobDev &J = jobs[blockIdx.z];
    const int bx = blockIdx.x;
    int by = blockIdx.y * len, l = len;
    if (k >= J.n || J.inactive) return;
    if (small) {  // only the jobs that the digit products leave
      const int m = J.N - k - min(kNb, J.n - k);
      if (split_pays(m, m, kSplitTrailing)) return;
    }
    if (part == kOtherTiles && bx * TL::kCols < kNb) {  // without the first 64 rows
      const int skip = max(0, min(l, kNb / TL::kRows - by));
      by += skip;
      l -= skip;
      if (l <= 0) return;
    }
    update64_column<W>(J, k, bx, by, l, zsm64);
    return;
  }
  // sparse: a 1-D grid, smaller than the tiles (the FP64 re-solve of a mixed wave, where most jobs are
  // inactive and a full grid would spend its time launching CTAs that exit at once): jobs one
  // after another (an inactive job costs one check), its columns spread over the CTAs
  for (int z = 0; z < nj; ++z) {
    const JobDev &J = jobs[z];
    if (J.inactive || k >= J.n) continue;
    for (int v = blockIdx.x; v < tx * ty; v += gridDim.x)
      update64_column<W>(J, k, v % tx, (v / tx) * len, len, zsm64);
  }
}

// out = tau00 (out_mode 1) or rotate(tau00 - t0) (out_mode 0), tau00 in A[r][b + c].
__device__ void write_out(const JobDev &J, double2 (*A)[2 * kMaxB + 1], int ns, int kkrsz) {
  const int tid = threadIdx.x;
  const int b = J.b;
  double2 *out = J.out;
  if (J.out_mode == 1) {
    for (int e = tid; e < b * b; e += blockDim.x) {
      const int c = e / b, r = e - c * b;
      out[e] = A[r][b + c];
    }
    return;
  }
  for (int e = tid; e < b * b; e += blockDim.x) {
    const int c = e / b, r = e - c * b;
    A[r][c] = csub(A[r][b + c], J.t0[r + (size_t)c * J.t0_ld]);
  }
  __syncthreads();
  if (ns == 1) {
    for (int e = tid; e < b * b; e += blockDim.x) {
      const int c = e / b, r = e - c * b;
      out[e] = A[r][c];
    }
  } else {
    // trgtol.f:3-110: ml(:,:,k) = (u d ud) spin block k, k column-major over the 2x2 spin matrix
    const int nr = kkrsz;
    for (int e = tid; e < 4 * nr * nr; e += blockDim.x) {
      const int kblk = e / (nr * nr);
      const int rem = e - kblk * nr * nr;
      const int c = rem / nr, r = rem - c * nr;
      const int ia = kblk & 1, jb = kblk >> 1;
      double2 s = make_double2(0.0, 0.0);
      for (int pp = 0; pp < 2; ++pp)
        for (int qq = 0; qq < 2; ++qq) {
          const double2 f = cmul(J.ubr[ia + 2 * pp], J.ubrd[qq + 2 * jb]);
          const double2 fg = cmul(f, A[pp * nr + r][qq * nr + c]);
          s.x += fg.x;
          s.y += fg.y;
        }
      out[e] = s;
    }
  }
}

// tau00 = S^-1 t0 from the Schur block in F (no refinement).
template <typename T>
__global__ void __launch_bounds__(256) finalize_direct_kernel(const JobDev *__restrict__ jobs, int ns,
                                                              int kkrsz, int *info) {
  const JobDev &J = jobs[blockIdx.x];
  const int b = J.b;
  __shared__ double2 A[kMaxB][2 * kMaxB + 1];
  const T *Sb = static_cast<const T *>(J.F) + (size_t)J.n + (size_t)J.n * J.ld;
  for (int e = threadIdx.x; e < b * b; e += blockDim.x) {
    const int c = e / b, r = e - c * b;
    A[r][c] = ldc(Sb + r + (size_t)c * J.ld);
    A[r][b + c] = J.t0[r + (size_t)c * J.t0_ld];
  }
  __syncthreads();
  if (gj_solve_smem(A, b) && threadIdx.x == 0) atomicCAS(&info[blockIdx.x], 0, -1);
  write_out(J, A, ns, kkrsz);
}

// out from X[n:N] (refined tau00).
__global__ void __launch_bounds__(256) finalize_from_x_kernel(const JobDev *__restrict__ jobs, int ns,
                                                              int kkrsz) {
  const JobDev &J = jobs[blockIdx.x];
  if (J.inactive) return;
  // a dataflow sweep whose bounded wait ran out aborted this job: report it in the error word
  if (threadIdx.x == 0 && J.conv != nullptr && J.err != nullptr && *J.conv == kAborted)
    atomicOr(J.err, kErrSweepWait);
  const int b = J.b;
  __shared__ double2 A[kMaxB][2 * kMaxB + 1];
  for (int e = threadIdx.x; e < b * b; e += blockDim.x) {
    const int c = e / b, r = e - c * b;
    A[r][b + c] = J.X[(size_t)(J.n + r) + (size_t)c * J.ld];
  }
  __syncthreads();
  write_out(J, A, ns, kkrsz);
}

// ---------------------------------------------------------------------------------------------
// Refinement pieces.  X, R, Y are N x b FP64 column-major with leading dimension ld.
// ---------------------------------------------------------------------------------------------

__device__ __forceinline__ bool converged(const JobDev &J) { return cx::converged(J.conv); }

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}

// R = B - M X with B = [0; t0] (rows n..N-1 hold t0), FP64.  The product is FP64 bound (b complex
// multiply-adds per 16-byte element of M) and runs on the FP64 tensor cores (mma.sync m8n8k4
// f64): as real products, [Rr | Ri] = Mr [Xr | Xi] + Mi [-Xi | Xr], four 8 x 8 x 4 MMAs per row
// tile and 8-column block per K step of 4, a few instructions per 1024 FMAs where DFMAs take 32.
// Each warp owns ROWS / 4 rows (8-row tiles) x BC columns of accumulators.  M and X stream
// through a three-stage cp.async ring in shared memory (kResK columns of M and rows of X per
// stage), so two stages of loads are in flight while one is multiplied.
// BC = 16 or 32 is the padded column count (b <= BC).
// A late refinement round has a few jobs left, 17 row blocks each at N = 2160: then a row block's K
// range is split over up to the 8 CTAs of a cluster, whose partial sums are added through
// distributed shared memory in rank order (a round on one job took 241 us with one CTA per row
// block, the latency of its 270 stages, and takes 51 us split in eight).
constexpr int kResK = 8;       // K per stage
constexpr int kResStages = 3;

constexpr int kResThreads = 128;  // four CTAs per SM, so a round on a few jobs still spans the GPU
template <int BC>
__host__ __device__ constexpr int residual_rows() {
  return kResThreads * 16 / BC;
}
constexpr int kResCluster = 8;  // CTAs per cluster, and the most that share a row block
// Row blocks x split the launch aims at: one full wave of four CTAs per SM.
constexpr int kResWave = 4 * 148;
// The rows of a stage are padded by two elements: a fragment load's eight lanes of a 128-byte phase (two
// rows or columns, four k) then hit eight different 16-byte banks, where unpadded rows put the four k
// of a row on the same one.
constexpr int kResPad = 2;
template <int BC>
__host__ __device__ constexpr int residual_smem_bytes() {
  return kResStages * kResK * (residual_rows<BC>() + BC + 2 * kResPad) * (int)sizeof(double2);
}

// The jobs of a wave still refining: list[0] = their number, list[1..] their indices in order.
// One warp.
__global__ void active_list_kernel(const JobDev *__restrict__ jobs, int njobs, int *list) {
  const int lane = threadIdx.x;
  int count = 0;
  for (int base = 0; base < njobs; base += 32) {
    const int w = base + lane;
    const bool a = w < njobs && !converged(jobs[w]) && !jobs[w].inactive;
    const unsigned mask = __ballot_sync(0xffffffffu, a);
    if (a) list[1 + count + __popc(mask & ((1u << lane) - 1u))] = w;
    count += __popc(mask);
  }
  if (lane == 0) list[0] = count;
}

// Work item i is row block i / count of the i % count-th job: of the jobs listed in `active`
// (active_list_kernel), so that the jobs still refining spread evenly over the SMs, or of all njobs.
// With few items, `split` CTAs of a cluster share one item, each over its share of K; `whole`: always all
// of them (FP64 factors, whose results then do not depend on how many jobs share the wave).
template <int BC>
__global__ void __cluster_dims__(kResCluster, 1, 1) __launch_bounds__(kResThreads, 4)
    residual_kernel(const JobDev *__restrict__ jobs, const int *__restrict__ active, int njobs, int rowblocks, bool whole) {
  constexpr int ROWS = residual_rows<BC>();  // rows per CTA
  constexpr int RT = ROWS / 32;              // 8-row tiles per warp (four warps)
  constexpr int NB = BC / 8;                 // 8-column blocks
  static_assert(kResThreads == 128 && RT * 32 == ROWS && NB * 8 == BC && kResK % 4 == 0, "residual layout");
  const int cnt = active != nullptr ? active[0] : njobs;
  int split = kResCluster;  // the same in every CTA
  while (!whole && split > 1 && cnt * rowblocks * split > kResWave) split >>= 1;
  const int item = blockIdx.x / split, slice = blockIdx.x % split;
  if ((int)(blockIdx.x / kResCluster) * (kResCluster / split) >= cnt * rowblocks) return;  // (the whole cluster)
  const bool valid = item < cnt * rowblocks;
  const int ji = valid ? item % cnt : 0, rb = valid ? item / cnt : 0;
  const JobDev &J = jobs[active != nullptr ? active[1 + ji] : ji];
  const int N = J.N, ld = J.ld, b = J.b;
  const int row0 = rb * ROWS;
  const bool live = valid && !converged(J) && !J.inactive && row0 < N;
  if ((split == 1 || split == kResCluster) && !live) return;  // (at kResCluster the whole cluster)
  extern __shared__ __align__(16) unsigned char rsm[];
  double2(*Ms)[kResK][ROWS + kResPad] = reinterpret_cast<double2(*)[kResK][ROWS + kResPad]>(rsm);
  double2(*Xs)[kResK][BC + kResPad] = reinterpret_cast<double2(*)[kResK][BC + kResPad]>(
      rsm + sizeof(double2) * kResStages * kResK * (ROWS + kResPad));
  const int tid = threadIdx.x;
  const int lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wrow = (tid >> 5) * (8 * RT);  // the warp's first row within the CTA's rows
  const double2 *__restrict__ M = J.M;
  const double2 *__restrict__ X = J.X;
  const double2 zero = make_double2(0.0, 0.0);
  // columns [k0, k0 + kResK) of M (rows of the CTA) and rows [k0, k0 + kResK) of X into stage st;
  // entries past N or b read as zero
  auto stage = [&](int k0, int st) {
    for (int e = tid; e < kResK * ROWS; e += kResThreads) {
      const int kk = e / ROWS, rr = e - kk * ROWS;
      const int gk = k0 + kk, grr = row0 + rr;
      if (gk < N && grr < N) cp_async16(&Ms[st][kk][rr], M + (size_t)grr + (size_t)gk * ld);
      else Ms[st][kk][rr] = zero;
    }
    for (int e = tid; e < kResK * BC; e += kResThreads) {
      const int kk = e % kResK, c = e / kResK;
      const int gk = k0 + kk;
      if (c < b && gk < N) cp_async16(&Xs[st][kk][c], X + (size_t)gk + (size_t)c * ld);
      else Xs[st][kk][c] = zero;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double ar[RT][NB][2], ai[RT][NB][2];  // M X, real and imaginary parts
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int j = 0; j < NB; ++j) ar[r][j][0] = ar[r][j][1] = ai[r][j][0] = ai[r][j][1] = 0.0;
  // this CTA's stages [q0, q0 + nst) of the K range
  const int stages = (N + kResK - 1) / kResK, per = (stages + split - 1) / split;
  const int q0 = slice * per, nst = live ? max(0, min(per, stages - q0)) : 0;
#pragma unroll
  for (int q = 0; q < kResStages - 1; ++q) {
    if (q < nst) stage((q0 + q) * kResK, q);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int q = 0; q < nst; ++q) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kResStages - 2) : "memory");
    __syncthreads();  // stage q landed for every thread; stage q - 1 is no longer read
    const int nq = q + kResStages - 1;
    if (nq < nst) stage((q0 + nq) * kResK, nq % kResStages);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const int st = q % kResStages;
#pragma unroll
    for (int ks = 0; ks < kResK; ks += 4) {
      double2 xv[NB];
#pragma unroll
      for (int j = 0; j < NB; ++j) xv[j] = Xs[st][ks + t][8 * j + g];
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const double2 mv = Ms[st][ks + t][wrow + 8 * r + g];
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          dm::mma_884(ar[r][j][0], ar[r][j][1], mv.x, xv[j].x);
          dm::mma_884(ar[r][j][0], ar[r][j][1], mv.y, -xv[j].y);
          dm::mma_884(ai[r][j][0], ai[r][j][1], mv.x, xv[j].y);
          dm::mma_884(ai[r][j][0], ai[r][j][1], mv.y, xv[j].x);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // with panel pivoting the factors are those of P M: row gr of R goes to its physical row
  const int *__restrict__ rowpos = J.piv != nullptr ? J.piv + ld : nullptr;
  // entry e = (r * NB + j) * 2 + i of this thread
  auto put = [&](int e, double2 v) {
    const int gr = row0 + wrow + 8 * (e / (2 * NB)) + g, c = 8 * ((e / 2) % NB) + 2 * t + (e & 1);
    if (gr >= N || c >= b) return;
    const int dst = rowpos != nullptr ? rowpos[gr] : gr;
    const double2 bv = (gr >= J.n) ? J.t0[(gr - J.n) + (size_t)c * J.t0_ld] : zero;
    J.R[(size_t)dst + (size_t)c * ld] = make_double2(bv.x - v.x, bv.y - v.y);
  };
  constexpr int E = RT * NB * 2;
  if (split == 1) {
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int j = 0; j < NB; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) put((r * NB + j) * 2 + i, make_double2(ar[r][j][i], ai[r][j][i]));
    return;
  }
  // partial sums to shared memory; CTA `slice` of the item adds up its share of the entries
  static_assert(E * kResThreads * (int)sizeof(double2) <= residual_smem_bytes<BC>(), "partial sums fit the ring");
  double2 *part = reinterpret_cast<double2 *>(rsm);
  __syncthreads();  // the ring is no longer read
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        part[((r * NB + j) * 2 + i) * kResThreads + tid] = make_double2(ar[r][j][i], ai[r][j][i]);
  cl::cluster_sync();
  if (live) {
    const int first = cl::cluster_rank() - slice;
    for (int e = slice * (E / split); e < (slice + 1) * (E / split); ++e) {
      double2 v = zero;
      for (int c = 0; c < split; ++c) {
        const double2 p = cl::ld_remote(cl::remote_u32(part + e * kResThreads + tid, first + c));
        v = make_double2(v.x + p.x, v.y + p.y);
      }
      put(e, v);
    }
  }
  cl::cluster_sync();  // no CTA leaves while another reads its partial sums
}

// Y[n:N] = S^-1 rhs with rhs = R[n:N] (mode 1) or t0 (mode 0, whose backward sweep takes Y[0:n] as 0).
template <typename T>
__global__ void __launch_bounds__(256) schur_solve_kernel(const JobDev *__restrict__ jobs, int mode,
                                                          int *info) {
  const JobDev &J = jobs[blockIdx.x];
  if ((mode == 1 && converged(J)) || J.inactive) return;
  const int b = J.b, n = J.n, ld = J.ld;
  __shared__ double2 A[kMaxB][2 * kMaxB + 1];
  const T *Sb = static_cast<const T *>(J.F) + (size_t)n + (size_t)n * ld;
  for (int e = threadIdx.x; e < b * b; e += blockDim.x) {
    const int c = e / b, r = e - c * b;
    A[r][c] = ldc(Sb + r + (size_t)c * ld);
    A[r][b + c] = mode == 0 ? J.t0[r + (size_t)c * J.t0_ld] : J.R[(size_t)(n + r) + (size_t)c * ld];
  }
  __syncthreads();
  if (gj_solve_smem(A, b) && threadIdx.x == 0) atomicCAS(&info[blockIdx.x], 0, -1);
  for (int e = threadIdx.x; e < b * b; e += blockDim.x) {
    const int c = e / b, r = e - c * b;
    J.Y[(size_t)(n + r) + (size_t)c * ld] = A[r][b + c];
  }
}

// CTAs of the looping trailing-update grid (two per SM)
constexpr int kSparseGrid = 2 * 148;

// Step k: W = D A12 (with W's operand pack) and A21's pack on s, then the update of the tile holding
// the next diagonal block; s2 waits for it and inverts that block while s updates the other tiles;
// s waits for the inverse before step k + 1.  Only the diagonal inverse moves off s, so the packs of step k + 1 are
// written after every tile of step k has read those of step k.
// With panel pivoting the first update covers the whole first tile column (the next step's panel,
// every row), the second stream also runs the next step's row selection and applies its row moves to
// the columns left of the other tiles, and the main stream applies them to the other columns once
// their update is done.
cudaError_t eliminate_lookahead(const JobDev *jobs, int njobs, int max_n, int max_N, int *info, cudaStream_t s,
                                long *launches, KernelTimer *timer, const TcMaps &tc, int *err, const Lookahead &la,
                                int smem_diag, int smem_gemm, bool panel) {
  cudaError_t e;
  const FactorKind fk = kFactorFP32;
  // SMs left to the second stream's work during the interior update.  The update is a persistent
  // kernel with a fixed share of tiles per CTA, so a CTA of it that cannot start (an inverse took
  // its SM) delays the whole launch: without panel pivoting the inverses, which the scheduler may
  // spread one per SM, get one SM per job.  With panel pivoting the row selection (one block per
  // SM) runs first on the second stream, in waves over the SMs left to it, and the inverses then
  // pack at their occupancy: one wave of those is enough, and the update keeps more SMs.
  int per_sm = 1;
  if (panel && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, diag_inverse_kernel<float2, 2>, kDiagThreads,
                                                               smem_diag) != cudaSuccess ||
                per_sm < 1)) {
    cudaGetLastError();
    per_sm = 1;
  }
  const int free_sms = std::min((njobs + per_sm - 1) / per_sm, tc_num_sms() / 2);
  if (panel) {
    if ((e = launch_pivot_init(jobs, njobs, s, launches)) != cudaSuccess) return e;
    if ((e = launch_panel_select(fk, jobs, njobs, 0, max_n, s, launches)) != cudaSuccess) return e;
    if ((e = launch_row_moves(fk, jobs, njobs, 0, 0, max_N, max_N, s, launches)) != cudaSuccess) return e;
  }
  launch_diag_inverse<float2>(panel, jobs, njobs, 0, info, smem_diag, s);
  if (launches) *launches += 1;
  for (int k = 0; k < max_n; k += kNb) {
    const int rest = max_N - k - 1;
    const int tiles = (rest + kTile - 1) / kTile;
    const bool next = k + kNb < max_n;
    const int k2 = k + kNb;
    // Paired steps k and k2: the update of the trailing block after k2 by both steps in one pass
    // (its FP32 read-modify-write, which bounds the update, once per two steps).  Step k's update
    // of the strips that step k2 needs first (block column k2, which holds the next diagonal
    // block, and block row k2) runs as SIMT tiles; the factors left in F are those of two
    // single steps.
    // With panel pivoting the pair keeps every row's pending update the same when step k2's rows
    // move: block column k2 is updated by step k (all rows) before step k2's selection, and block
    // row k2 only after its row moves, so that at the moves every row below step k still owes
    // step k's update right of block column k2 (done for all of them by the combined pass) and
    // the moves carry A21_k's rows with them.
    if (panel && la.pair_min_rest > 0 && k2 + kNb <= la.min_n && k2 + kNb < max_n &&
        max_N - k2 - kNb >= la.pair_min_rest) {
      const int tiles2 = (max_N - k2 - 1 + kTile - 1) / kTile;
      const int split2 = k2 + kNb + kTcTileCols;
      PackB pk0;  // W(k): its columns right of block column k2 -> K half 0 of the pair's B operand
      pk0.hi = tc.b_hi;
      pk0.lo = tc.b_lo;
      pk0.slot = tc.b_slot;
      pk0.shift_k = k2;
      zgemm_tile_kernel<kOverwrite><<<dim3(tiles, 1, njobs), 256, smem_gemm, s>>>(jobs, k, pk0, 0);
      // step k on block column k2, every row below step k (the diagonal block included)
      zgemm_tile_kernel<kSubtract><<<dim3(1, tiles, njobs), 256, smem_gemm, s>>>(jobs, k, PackB(), 0, 0);
      if ((e = launch_panel_select(fk, jobs, njobs, k2, max_n, s, launches)) != cudaSuccess) return e;
      if ((e = launch_row_moves(fk, jobs, njobs, k2, 0, max_N, max_N, s, launches)) != cudaSuccess) return e;
      // the inverse of the moved diagonal block beside step k's update of block row k2
      if ((e = cudaEventRecord(la.panel, s)) != cudaSuccess) return e;
      if ((e = cudaStreamWaitEvent(la.s2, la.panel, 0)) != cudaSuccess) return e;
      launch_diag_inverse<float2>(true, jobs, njobs, k2, info, smem_diag, la.s2);
      if ((e = cudaEventRecord(la.diag, la.s2)) != cudaSuccess) return e;
      if (tiles > 1)
        zgemm_tile_kernel<kSubtract><<<dim3(tiles - 1, 1, njobs), 256, smem_gemm, s>>>(jobs, k, PackB(), 1, 0);
      if ((e = cudaStreamWaitEvent(s, la.diag, 0)) != cudaSuccess) return e;
      PackB pk1;  // W(k2) -> K half 1
      pk1.hi = tc.b_hi;
      pk1.lo = tc.b_lo;
      pk1.slot = tc.b_slot;
      pk1.k_off = 2 * kNb;
      zgemm_tile_kernel<kOverwrite><<<dim3(tiles2, 1, njobs), 256, smem_gemm, s>>>(jobs, k2, pk1, 0);
      const bool timed = timer && timer->used + 2 <= timer->cap;
      if (timed) cudaEventRecord(timer->ev[timer->used++], s);
      if ((e = launch_tc_pack(tc, jobs, njobs, k, 2, k2, max_N, s, false)) != cudaSuccess) return e;
      if ((e = launch_tc_update(tc, jobs, njobs, k2, max_N, err, s, 3, 0, 2)) != cudaSuccess) return e;
      // the next step's selection, its moves left of the tiles still being updated, its inverse
      if ((e = cudaEventRecord(la.panel, s)) != cudaSuccess) return e;
      if ((e = cudaStreamWaitEvent(la.s2, la.panel, 0)) != cudaSuccess) return e;
      if ((e = launch_panel_select(fk, jobs, njobs, k2 + kNb, max_n, la.s2, launches)) != cudaSuccess) return e;
      if ((e = launch_row_moves(fk, jobs, njobs, k2 + kNb, 0, split2, max_N, la.s2, launches)) != cudaSuccess)
        return e;
      launch_diag_inverse<float2>(true, jobs, njobs, k2 + kNb, info, smem_diag, la.s2);
      if ((e = cudaEventRecord(la.diag, la.s2)) != cudaSuccess) return e;
      if ((e = launch_tc_update(tc, jobs, njobs, k2, max_N, err, s, 4, tc_num_sms() - free_sms, 2)) != cudaSuccess)
        return e;
      if (timed) cudaEventRecord(timer->ev[timer->used++], s);
      if ((e = cudaStreamWaitEvent(s, la.diag, 0)) != cudaSuccess) return e;
      if ((e = launch_row_moves(fk, jobs, njobs, k2 + kNb, split2, max_N, max_N, s, launches)) != cudaSuccess)
        return e;
      // W(k), the column strip, the row strip, k2's inverse, W(k2), the pack, the two update
      // launches, the next inverse (selections and moves count themselves)
      if (launches) *launches += 7 + (tiles > 1 ? 1 : 0);
      k = k2;  // the loop's increment moves past k2
      continue;
    }
    // (only where step k2 is a full block of every job: the strips below apply step k to 64 columns and
    // rows from k2 on, and the combined pass starts behind step k2's own block, so after a partial block of
    // kb2 the last 64 - kb2 of them would have step k subtracted twice)
    if (!panel && la.pair_min_rest > 0 && k2 + kNb <= la.min_n && k2 + kNb < max_n &&
        max_N - k2 - kNb >= la.pair_min_rest) {
      const int tiles2 = (max_N - k2 - 1 + kTile - 1) / kTile;
      const bool next2 = k2 + kNb < max_n;
      PackB pk0;  // W(k): its columns right of block column k2 -> K half 0 of the pair's B operand
      pk0.hi = tc.b_hi;
      pk0.lo = tc.b_lo;
      pk0.slot = tc.b_slot;
      pk0.shift_k = k2;
      zgemm_tile_kernel<kOverwrite><<<dim3(tiles, 1, njobs), 256, smem_gemm, s>>>(jobs, k, pk0, 0);
      // step k on block column k2 (all rows below step k) and on block row k2 (right of it): first
      // the diagonal block of k2, whose inverse then runs on the second stream beside the rest of
      // the two strips
      zgemm_tile_kernel<kSubtract><<<dim3(1, 1, njobs), 256, smem_gemm, s>>>(jobs, k, PackB(), 0, 0);
      if ((e = cudaEventRecord(la.panel, s)) != cudaSuccess) return e;
      if ((e = cudaStreamWaitEvent(la.s2, la.panel, 0)) != cudaSuccess) return e;
      launch_diag_inverse<float2>(false, jobs, njobs, k2, info, smem_diag, la.s2);
      if ((e = cudaEventRecord(la.diag, la.s2)) != cudaSuccess) return e;
      if (tiles > 1) zgemm_strips_kernel<<<dim3(2 * (tiles - 1), 1, njobs), 256, smem_gemm, s>>>(jobs, k, tiles - 1);
      if ((e = cudaStreamWaitEvent(s, la.diag, 0)) != cudaSuccess) return e;
      PackB pk1;  // W(k2) -> K half 1
      pk1.hi = tc.b_hi;
      pk1.lo = tc.b_lo;
      pk1.slot = tc.b_slot;
      pk1.k_off = 2 * kNb;
      zgemm_tile_kernel<kOverwrite><<<dim3(tiles2, 1, njobs), 256, smem_gemm, s>>>(jobs, k2, pk1, 0);
      const bool timed = timer && timer->used + 2 <= timer->cap;
      if (timed) cudaEventRecord(timer->ev[timer->used++], s);
      if ((e = launch_tc_pack(tc, jobs, njobs, k, 2, k2, max_N, s, false)) != cudaSuccess) return e;
      if ((e = launch_tc_update(tc, jobs, njobs, k2, max_N, err, s, 1, 0, 2)) != cudaSuccess) return e;
      if (next2) {
        if ((e = cudaEventRecord(la.panel, s)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(la.s2, la.panel, 0)) != cudaSuccess) return e;
        launch_diag_inverse<float2>(false, jobs, njobs, k2 + kNb, info, smem_diag, la.s2);
        if ((e = cudaEventRecord(la.diag, la.s2)) != cudaSuccess) return e;
      }
      if ((e = launch_tc_update(tc, jobs, njobs, k2, max_N, err, s, 2, next2 ? tc_num_sms() - free_sms : 0, 2)) !=
          cudaSuccess)
        return e;
      if (timed) cudaEventRecord(timer->ev[timer->used++], s);
      if (next2 && (e = cudaStreamWaitEvent(s, la.diag, 0)) != cudaSuccess) return e;
      // W(k), the diagonal block, its inverse, W(k2), the pack, the two update launches (+ the
      // two strips in one launch, + the next inverse)
      if (launches) *launches += 7 + (tiles > 1 ? 1 : 0) + (next2 ? 1 : 0);
      k = k2;  // the loop's increment moves past k2
      continue;
    }
    if (tiles > 0) {
      PackB pk;
      pk.hi = tc.b_hi;
      pk.lo = tc.b_lo;
      pk.slot = tc.b_slot;
      zgemm_tile_kernel<kOverwrite><<<dim3(tiles, 1, njobs), 256, smem_gemm, s>>>(jobs, k, pk, 0);
      const bool timed = timer && timer->used + 2 <= timer->cap;
      if (timed) cudaEventRecord(timer->ev[timer->used++], s);
      if ((e = launch_tc_pack(tc, jobs, njobs, k, 1, k, max_N, s, false)) != cudaSuccess) return e;
      if ((e = launch_tc_update(tc, jobs, njobs, k, max_N, err, s, panel ? 3 : 1, 0)) != cudaSuccess) return e;
      // the next step's columns left of the tiles still being updated: [0, k + 64 + one tile)
      const int split = k + kNb + kTcTileCols;
      if (next) {
        if ((e = cudaEventRecord(la.panel, s)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(la.s2, la.panel, 0)) != cudaSuccess) return e;
        if (panel) {
          if ((e = launch_panel_select(fk, jobs, njobs, k + kNb, max_n, la.s2, launches)) != cudaSuccess) return e;
          if ((e = launch_row_moves(fk, jobs, njobs, k + kNb, 0, split, max_N, la.s2, launches)) != cudaSuccess)
            return e;
        }
        launch_diag_inverse<float2>(panel, jobs, njobs, k + kNb, info, smem_diag, la.s2);
        if ((e = cudaEventRecord(la.diag, la.s2)) != cudaSuccess) return e;
      }
      if ((e = launch_tc_update(tc, jobs, njobs, k, max_N, err, s, panel ? 4 : 2,
                                next ? tc_num_sms() - free_sms : 0)) != cudaSuccess)
        return e;
      if (timed) cudaEventRecord(timer->ev[timer->used++], s);  // the update kernels only
      if (next && (e = cudaStreamWaitEvent(s, la.diag, 0)) != cudaSuccess) return e;
      if (next && panel && (e = launch_row_moves(fk, jobs, njobs, k + kNb, split, max_N, max_N, s, launches)) !=
                               cudaSuccess)
        return e;
      if (launches) *launches += next ? 5 : 4;
    } else if (next) {
      if (panel) {
        if ((e = launch_panel_select(fk, jobs, njobs, k + kNb, max_n, s, launches)) != cudaSuccess) return e;
        if ((e = launch_row_moves(fk, jobs, njobs, k + kNb, 0, max_N, max_N, s, launches)) != cudaSuccess) return e;
      }
      launch_diag_inverse<float2>(panel, jobs, njobs, k + kNb, info, smem_diag, s);
      if (launches) *launches += 1;
    }
  }
  if (panel && (e = launch_pivot_finish(jobs, njobs, s, launches)) != cudaSuccess) return e;
  return cudaGetLastError();
}

// FP32 factors.
cudaError_t eliminate32(const JobDev *jobs, int njobs, int max_n, int max_N, int *info, cudaStream_t s,
                        long *launches, KernelTimer *timer, const TcMaps *tc, int *err, const Lookahead *la,
                        bool panel) {
  const int smem_diag = kNb * (kNb + 1) * (int)sizeof(double2);
  const int smem_gemm = kTileSmem;
  cudaError_t e;
  if ((e = ensure_smem(diag_inverse_kernel<float2, 1>, smem_diag)) != cudaSuccess) return e;
  if ((e = ensure_smem(diag_inverse_kernel<float2, 2>, smem_diag)) != cudaSuccess) return e;
  if ((e = ensure_smem(zgemm_tile_kernel<kOverwrite>, smem_gemm)) != cudaSuccess) return e;
  if ((e = ensure_smem(zgemm_tile_kernel<kSubtract>, smem_gemm)) != cudaSuccess) return e;
  if ((e = ensure_smem(zgemm_strips_kernel, smem_gemm)) != cudaSuccess) return e;
  // Look-ahead (tensor-core path): the update of step k first covers the tile holding the next
  // step's diagonal block; the next diagonal inverse then runs on the second stream while the other
  // tiles are updated on SMs left free for it (the inverses take one SM per job).
  if (tc != nullptr && la != nullptr && la->s2 != nullptr)
    return eliminate_lookahead(jobs, njobs, max_n, max_N, info, s, launches, timer, *tc, err, *la, smem_diag,
                               smem_gemm, panel);
  if (panel && (e = launch_pivot_init(jobs, njobs, s, launches)) != cudaSuccess) return e;
  for (int k = 0; k < max_n; k += kNb) {
    if (panel) {
      if ((e = launch_panel_select(kFactorFP32, jobs, njobs, k, max_n, s, launches)) != cudaSuccess) return e;
      if ((e = launch_row_moves(kFactorFP32, jobs, njobs, k, 0, max_N, max_N, s, launches)) != cudaSuccess) return e;
    }
    launch_diag_inverse<float2>(panel, jobs, njobs, k, info, smem_diag, s);
    const int rest = max_N - k - 1;
    const int tiles = (rest + kTile - 1) / kTile;
    if (launches) *launches += 1;
    if (tiles > 0) {
      zgemm_tile_kernel<kOverwrite><<<dim3(tiles, 1, njobs), 256, smem_gemm, s>>>(jobs, k, PackB(), 0);
      const bool timed = timer && timer->used + 2 <= timer->cap;
      if (timed) cudaEventRecord(timer->ev[timer->used++], s);
      if (tc != nullptr) {
        if ((e = launch_tc_step(*tc, jobs, njobs, k, max_N, err, s)) != cudaSuccess) return e;
        if (launches) *launches += 1;  // pack + update
      } else {
        zgemm_tile_kernel<kSubtract><<<dim3(tiles, tiles, njobs), 256, smem_gemm, s>>>(jobs, k, PackB(), 0);
      }
      if (timed) cudaEventRecord(timer->ev[timer->used++], s);
      if (launches) *launches += 2;
    }
  }
  if (panel && (e = launch_pivot_finish(jobs, njobs, s, launches)) != cudaSuccess) return e;
  return cudaGetLastError();
}

template <int W>
void launch_update64_tiles(const JobDev *jobs, int njobs, int k, int max_N, int part, bool sparse, bool small,
                           cudaStream_t s) {
  using TL = dm::Tile<W, W>;
  const int rows = part == kFirstBlock ? kNb : small ? std::min(kSplitSide - 1, max_N - k - 1) : max_N - k - 1;
  const int tx = (rows + TL::kCols - 1) / TL::kCols, tr = (rows + TL::kRows - 1) / TL::kRows;
  const int len = sparse ? 1 : dm::column_tiles((long)tx * tr * njobs);
  const int ty = (tr + len - 1) / len;
  const dim3 grid = sparse ? dim3(std::min(tx * ty * njobs, kSparseGrid)) : dim3(tx, ty, njobs);
  zgemm64_update_kernel<W><<<grid, dm::kThreads, TL::kSmem, s>>>(jobs, k, tx, ty, njobs, part, len, sparse, small);
}

// `small`: only the jobs whose update split_pays leaves to these tiles.
void launch_update64(const JobDev *jobs, int njobs, int k, int max_N, int part, bool sparse, bool small, cudaStream_t s) {
  if (part == kFirstBlock && 16 * njobs <= 4 * 148)
    launch_update64_tiles<1>(jobs, njobs, k, max_N, part, sparse, small, s);
  else
    launch_update64_tiles<2>(jobs, njobs, k, max_N, part, sparse, small, s);
}

// FP64 factors.  With a second stream (and pivots inside the diagonal blocks) the update of step k
// first covers the next diagonal block, whose inverse (a chain of 64 dependent pivot steps on one
// SM per job) then runs on the second stream beside the rest of the update.
cudaError_t eliminate64(const JobDev *jobs, int njobs, int max_n, int max_N, int *info, cudaStream_t s,
                        long *launches, KernelTimer *timer, bool sparse, const Lookahead *la, bool panel,
                        const SplitBufs *split, int *err) {
  const int smem_diag = kNb * (kNb + 1) * (int)sizeof(double2);
  cudaError_t e;
  if ((e = ensure_smem(diag_inverse_kernel<double2, 1>, smem_diag)) != cudaSuccess) return e;
  if ((e = ensure_smem(diag_inverse_kernel<double2, 2>, smem_diag)) != cudaSuccess) return e;
  if ((e = ensure_smem(zgemm64_w_kernel<2>, dm::Tile<4, 2>::kSmem)) != cudaSuccess) return e;
  if ((e = ensure_smem(zgemm64_update_kernel<1>, dm::Tile<1, 1>::kSmem)) != cudaSuccess) return e;
  if ((e = ensure_smem(zgemm64_update_kernel<2>, dm::Tile<2, 2>::kSmem)) != cudaSuccess) return e;
  if ((e = ensure_smem(zgemm64_w_kernel<1>, dm::Tile<4, 1>::kSmem)) != cudaSuccess) return e;
  const bool ahead = la != nullptr && la->s2 != nullptr && !sparse && !panel;
  if (sparse) split = nullptr;
  // the smallest job's N (b is the same for all; 0: not known)
  const int min_N = la != nullptr ? la->min_n + max_N - max_n : 0;
  if (split && (e = cudaMemsetAsync(split->counters, 0, sizeof(int) * split->steps, s)) != cudaSuccess) return e;
  if (panel && (e = launch_pivot_init(jobs, njobs, s, launches)) != cudaSuccess) return e;
  for (int k = 0; k < max_n; k += kNb) {
    if (panel) {
      if ((e = launch_panel_select(kFactorFP64, jobs, njobs, k, max_n, s, launches)) != cudaSuccess) return e;
      if ((e = launch_row_moves(kFactorFP64, jobs, njobs, k, 0, max_N, max_N, s, launches)) != cudaSuccess) return e;
    }
    if (!ahead || k == 0) {
      launch_diag_inverse<double2>(panel, jobs, njobs, k, info, smem_diag, s);
      if (launches) *launches += 1;
    }
    const int rest = max_N - k - 1;
    if (rest <= 0) continue;
    const bool next = ahead && k + kNb < max_n;
    // 16 columns a CTA where that is at most a CTA an SM (half the time of a 32-column tile: 9 -> 7.9 us)
    if ((rest + 15) / 16 * njobs <= 148)
      zgemm64_w_kernel<1><<<dim3((rest + 15) / 16, 1, njobs), dm::kThreads, dm::Tile<4, 1>::kSmem, s>>>(jobs, k);
    else
      zgemm64_w_kernel<2><<<dim3((rest + 31) / 32, 1, njobs), dm::kThreads, dm::Tile<4, 2>::kSmem, s>>>(jobs, k);
    const bool timed = timer && timer->used + 2 <= timer->cap;
    if (timed) cudaEventRecord(timer->ev[timer->used++], s);
    if (next) {
      launch_update64(jobs, njobs, k, max_N, kFirstBlock, false, false, s);
      if ((e = cudaEventRecord(la->panel, s)) != cudaSuccess) return e;
      if ((e = cudaStreamWaitEvent(la->s2, la->panel, 0)) != cudaSuccess) return e;
      launch_diag_inverse<double2>(false, jobs, njobs, k + kNb, info, smem_diag, la->s2);
      if ((e = cudaEventRecord(la->diag, la->s2)) != cudaSuccess) return e;
    }
    // every job's update by digit products or on the FP64 tensor cores, as its own size asks (split_pays);
    // no launch for a side that no job takes
    const int most = max_N - k - kNb, least = min_N - k - kNb;
    const bool large = split && split_pays(most, most, kSplitTrailing);
    if (large) {
      const s8::Large<OpTrailing, kSplitTrailing> op;
      if ((e = s8::launch_split_pack(*split, jobs, njobs, k, most, most, s, op)) != cudaSuccess) return e;
      if ((e = s8::launch_split_update(*split, jobs, njobs, k, most, most, next, split->counters + k / kNb, err, s, op)) !=
          cudaSuccess)
        return e;
      if (launches) *launches += 4;
    }
    if (!large || !split_pays(least, least, kSplitTrailing)) {
      launch_update64(jobs, njobs, k, max_N, next ? kOtherTiles : kAllTiles, sparse, large, s);
      if (launches) *launches += 1;
    }
    if (timed) cudaEventRecord(timer->ev[timer->used++], s);
    if (next && (e = cudaStreamWaitEvent(s, la->diag, 0)) != cudaSuccess) return e;
    if (launches) *launches += next ? 3 : 1;
  }
  if (panel && (e = launch_pivot_finish(jobs, njobs, s, launches)) != cudaSuccess) return e;
  return cudaGetLastError();
}

template <typename T>
cudaError_t sweep_solve(const JobDev *jobs, int njobs, int b, int max_N, int mode, int *info, cudaStream_t s,
                        long *launches, bool fp32, const CUtensorMap *fmap, int active_hint = 0) {
  const FactorKind fk = sizeof(T) == sizeof(double2) ? kFactorFP64 : kFactorFP32;
  cudaError_t e;
  // forward (skipped for the initial solve: B is zero above the central block)
  if (mode == 1) {
    if ((e = launch_sweep(fk, jobs, njobs, b, max_N, true, mode, fp32, fmap, s, active_hint)) != cudaSuccess)
      return e;
    if (launches) *launches += 1;
  }
  schur_solve_kernel<T><<<njobs, 256, 0, s>>>(jobs, mode, info);
  if ((e = launch_sweep(fk, jobs, njobs, b, max_N, false, mode, fp32, fmap, s, active_hint)) != cudaSuccess)
    return e;
  if (launches) *launches += 2;
  return cudaSuccess;
}

// After a refinement round: c = max|correction| / max|tau00| on the tau00 block (NaN where an element of
// either is not finite, which refinement cannot mend), and what refine_state
// (refine_rule.h) makes of it and the two corrections before it.  A job that is kConverged or kDiverged is
// skipped from then on; every job that is not kConverged after the last round is re-solved by FP64 block LU.
__global__ void __launch_bounds__(256) converge_check_kernel(const JobDev *__restrict__ jobs, bool accelerated,
                                                             bool last) {
  const JobDev &J = jobs[blockIdx.x];
  if (J.conv == nullptr || converged(J) || J.inactive) return;
  const int b = J.b, n = J.n, ld = J.ld;
  double my = 0.0, mx = 0.0;
  int finite = 1;
  for (int e = threadIdx.x; e < b * b; e += blockDim.x) {
    const int r = e % b, c = e / b;
    const size_t idx = (size_t)(n + r) + (size_t)c * ld;
    const double y = cabs1(J.Y[idx]), x = cabs1(J.X[idx]);
    my = fmax(my, y);
    mx = fmax(mx, x);
    finite = finite && isfinite(y) && isfinite(x);  // (fmax passes over a NaN)
  }
  __shared__ double sy[256], sx[256];
  sy[threadIdx.x] = my;
  sx[threadIdx.x] = mx;
  finite = __syncthreads_and(finite);
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      sy[threadIdx.x] = fmax(sy[threadIdx.x], sy[threadIdx.x + o]);
      sx[threadIdx.x] = fmax(sx[threadIdx.x], sx[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double c = !finite ? nan("") : sx[0] > 0.0 ? sy[0] / sx[0] : 0.0;
    const double prev = J.cnorm ? J.cnorm[0] : 0.0, prev2 = J.cnorm ? J.cnorm[1] : 0.0;
    *J.conv = refine_state(c, prev, prev2, accelerated, last);
    if (J.cnorm) {
      J.cnorm[0] = c;
      J.cnorm[1] = prev;
    }
  }
}

// Anderson acceleration of the refinement (D. G. Anderson, J. ACM 12, 547 (1965), depth 2; for a linear
// system it is a truncated GMRES on F^-1 M), one column of one job per CTA.  Round i's
// sweeps took X_i to P_i = X_i + Y_i, Y_i = F^-1 (B - M X_i).  With the two earlier rounds' P and Y,
//   X_(i+1) = P_i - g1 (P_i - P_(i-1)) - g2 (P_(i-1) - P_(i-2)),
// g the least-squares coefficients of Y_i against (Y_i - Y_(i-1), Y_(i-1) - Y_(i-2)).  A job whose block
// factors are poor in a few directions (pivots kept inside the diagonal blocks) has those directions
// taken out instead of shrunk.  Rounds are a chain of two sweeps each, whose time hardly falls with the
// jobs left: 256 jobs of N = 688 to 2160, one point next to the real axis, 31.0 -> 21.5 ms of refinement
// (and no FP64 re-solve where there was one); 16 jobs of N = 4320, 32.5 -> 30.7 ms.  A round's step is
// accelerated before the convergence check, which takes a fifth of the plain rounds' tolerance and the larger
// of the last two contractions (refine_rule.h).
// hist: 0 the iterate X_i; 1, 2 P of odd and even rounds; 3, 4 Y of odd and even rounds.
constexpr int kAccThreads = 1024;
__global__ void __launch_bounds__(kAccThreads) accelerate_kernel(const JobDev *__restrict__ jobs, int round) {
  const JobDev &J = jobs[blockIdx.y];
  const int c = blockIdx.x;
  if (J.hist == nullptr || c >= J.b || J.inactive || (round > 0 && converged(J))) return;
  const int N = J.N, tid = threadIdx.x;
  const size_t vec = (size_t)J.ld * kMaxB, col = (size_t)c * J.ld;
  double2 *X = J.X + col, *X0 = J.hist + col;
  double2 *P1 = J.hist + (1 + ((round + 1) & 1)) * vec + col, *P2 = J.hist + (1 + (round & 1)) * vec + col;
  double2 *Y1 = J.hist + (3 + ((round + 1) & 1)) * vec + col, *Y2 = J.hist + (3 + (round & 1)) * vec + col;
  const int depth = round <= 1 ? 0 : round == 2 ? 1 : 2;
  // Gram matrix of d1 = Y - Y1 and d2 = Y1 - Y2 (a11, a22, a12) and right-hand sides <d1, Y>, <d2, Y>
  double s[8] = {};
  if (depth > 0)
    for (int r = tid; r < N; r += blockDim.x) {
      const double2 y = csub(X[r], X0[r]), y1 = Y1[r];
      const double2 d1 = csub(y, y1), d2 = depth > 1 ? csub(y1, Y2[r]) : make_double2(0.0, 0.0);
      s[0] += d1.x * d1.x + d1.y * d1.y;
      s[1] += d2.x * d2.x + d2.y * d2.y;
      s[2] += d1.x * d2.x + d1.y * d2.y;  // conj(d1) d2
      s[3] += d1.x * d2.y - d1.y * d2.x;
      s[4] += d1.x * y.x + d1.y * y.y;  // conj(d1) y
      s[5] += d1.x * y.y - d1.y * y.x;
      s[6] += d2.x * y.x + d2.y * y.y;
      s[7] += d2.x * y.y - d2.y * y.x;
    }
  __shared__ double part[8][kAccThreads / 32];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
    if ((tid & 31) == 0) part[i][tid >> 5] = s[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    s[i] = 0.0;
    for (int w = 0; w < (int)blockDim.x / 32; ++w) s[i] += part[i][w];
  }
  double2 g1 = make_double2(0.0, 0.0), g2 = g1;
  if (depth > 0) {
    const double2 a12 = make_double2(s[2], s[3]), r1 = make_double2(s[4], s[5]), r2 = make_double2(s[6], s[7]);
    const double det = s[0] * s[1] - (a12.x * a12.x + a12.y * a12.y);
    if (depth > 1 && det > 1e-10 * s[0] * s[1]) {
      const double2 t1 = cmul(a12, r2), t2 = cmul(make_double2(a12.x, -a12.y), r1);
      g1 = make_double2((s[1] * r1.x - t1.x) / det, (s[1] * r1.y - t1.y) / det);
      g2 = make_double2((s[0] * r2.x - t2.x) / det, (s[0] * r2.y - t2.y) / det);
    } else if (s[0] > 0.0) {  // one direction
      g1 = make_double2(r1.x / s[0], r1.y / s[0]);
    }
    if (!(fabs(g1.x) + fabs(g1.y) + fabs(g2.x) + fabs(g2.y) < 1e6)) g1 = g2 = make_double2(0.0, 0.0);
  }
  for (int r = tid; r < N; r += blockDim.x) {
    const double2 p = X[r];
    double2 x = p;
    if (round > 0) {
      const double2 y = csub(p, X0[r]);
      if (depth > 0) {
        const double2 p1 = P1[r];
        x = csub(x, cmul(g1, csub(p, p1)));
        if (depth > 1) x = csub(x, cmul(g2, csub(p1, P2[r])));
        X[r] = x;
      }
      P2[r] = p;  // (the slots of round i - 2 take round i)
      Y2[r] = y;
    }
    X0[r] = x;
  }
}

template <typename T>
__global__ void copy_to_factor_kernel(const double2 *__restrict__ M, T *__restrict__ F, int n, int ld) {
  const size_t total = (size_t)n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const size_t c = e / n, r = e - c * n;
    stc(F + r + c * ld, M[r + c * ld]);
  }
}

// The FP64 re-solve records of a mixed wave (launch_fallback_prepare).
__global__ void fallback_prepare_kernel(const JobDev *__restrict__ jobs, JobDev *__restrict__ out, int njobs,
                                        double2 *f64, size_t f64_stride, int *count, int panel) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= njobs) return;
  JobDev J = jobs[w];
  const bool conv = J.conv != nullptr && *J.conv == kConverged;
  if (conv) {
    J.inactive = 1;
  } else {
    J.F = f64 + (size_t)w * f64_stride;
    J.conv = nullptr;  // the FP64 rounds run unconditionally
    J.cnorm = nullptr;
    if (!panel) J.piv = nullptr;  // pivots inside the diagonal blocks: rows stay in place
    atomicAdd(count, 1);
  }
  out[w] = J;
}

// The re-solve gate of a mixed wave: the graph's conditional body (the FP64 re-solve) runs only
// when some record has not converged.
__global__ void fallback_gate_kernel(const JobDev *__restrict__ jobs, int njobs, cudaGraphConditionalHandle h) {
  int any = 0;
  for (int w = threadIdx.x; w < njobs; w += blockDim.x) {
    const int *c = jobs[w].conv;
    any |= (c == nullptr || *c != kConverged) ? 1 : 0;
  }
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) cudaGraphSetConditional(h, any ? 1u : 0u);
}

// F = M (FP64, N x N) for the active records; CTAs (blockIdx.x) stride over the columns of job
// blockIdx.y
__global__ void __launch_bounds__(256) copy_jobs_to_factor_kernel(const JobDev *__restrict__ jobs) {
  const JobDev &J = jobs[blockIdx.y];
  if (J.inactive) return;
  double2 *F = static_cast<double2 *>(J.F);
  for (int c = blockIdx.x; c < J.N; c += gridDim.x)
    for (int r = threadIdx.x; r < J.N; r += 256) F[(size_t)r + (size_t)c * J.ld] = J.M[(size_t)r + (size_t)c * J.ld];
}

}  // namespace

cudaError_t launch_fallback_prepare(const JobDev *jobs, JobDev *out, int njobs, double2 *f64, size_t f64_stride,
                                    int max_N, int *count, bool panel, cudaStream_t s, long *launches) {
  if (njobs <= 0) return cudaSuccess;
  fallback_prepare_kernel<<<(njobs + 63) / 64, 64, 0, s>>>(jobs, out, njobs, f64, f64_stride, count, panel ? 1 : 0);
  copy_jobs_to_factor_kernel<<<dim3(std::min(max_N, 64), njobs), 256, 0, s>>>(out);
  if (launches) *launches += 2;
  return cudaGetLastError();
}

cudaError_t add_fallback_gate_node(cudaGraph_t g, cudaGraphNode_t *node, const JobDev *jobs, int njobs,
                                   cudaGraphConditionalHandle h) {
  cudaKernelNodeParams kp = {};
  void *args[3] = {&jobs, &njobs, &h};
  kp.func = reinterpret_cast<void *>(fallback_gate_kernel);
  kp.gridDim = dim3(1);
  kp.blockDim = dim3(256);
  kp.sharedMemBytes = 0;
  kp.kernelParams = args;
  return cudaGraphAddKernelNode(node, g, nullptr, 0, &kp);
}

cudaError_t launch_copy_to_factor(FactorKind fk, const double2 *M, void *F, int n, int ld, cudaStream_t s) {
  const int blocks = 148 * 8;
  if (fk == kFactorFP64)
    copy_to_factor_kernel<double2><<<blocks, 256, 0, s>>>(M, static_cast<double2 *>(F), n, ld);
  else
    copy_to_factor_kernel<float2><<<blocks, 256, 0, s>>>(M, static_cast<float2 *>(F), n, ld);
  return cudaGetLastError();
}

cudaError_t launch_eliminate(FactorKind fk, const JobDev *jobs, int njobs, int max_n, int max_N, int *info,
                             cudaStream_t s, long *launches, KernelTimer *timer, const TcMaps *tc,
                             int *err, bool sparse_jobs, const Lookahead *la, bool panel, const SplitBufs *split) {
  if (fk == kFactorFP64)
    return eliminate64(jobs, njobs, max_n, max_N, info, s, launches, timer, sparse_jobs, la, panel, split, err);
  if (tc) {
    cudaError_t e = tc_prepare();
    if (e == cudaSuccess) e = launch_tc_counters_reset(*tc, s);
    if (e != cudaSuccess) return e;
  }
  return eliminate32(jobs, njobs, max_n, max_N, info, s, launches, timer, tc, err, la, panel);
}

cudaError_t launch_finalize_direct(FactorKind fk, const JobDev *jobs, int njobs, int ns, int kkrsz, int *info,
                                   cudaStream_t s, long *launches) {
  if (fk == kFactorFP64)
    finalize_direct_kernel<double2><<<njobs, 256, 0, s>>>(jobs, ns, kkrsz, info);
  else
    finalize_direct_kernel<float2><<<njobs, 256, 0, s>>>(jobs, ns, kkrsz, info);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_refine_begin(FactorKind fk, const JobDev *jobs, int njobs, int max_n, int max_N, int b,
                                int *info, cudaStream_t s, long *launches, bool fp32_sweep,
                                const CUtensorMap *fmap) {
  (void)max_n;
  const cudaError_t e = fk == kFactorFP64 ? sweep_solve<double2>(jobs, njobs, b, max_N, 0, info, s, launches, false, nullptr)
                                           : sweep_solve<float2>(jobs, njobs, b, max_N, 0, info, s, launches, fp32_sweep, fmap);
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <int BC>
cudaError_t launch_residual(const JobDev *jobs, int njobs, int max_N, int *active, bool whole, cudaStream_t s) {
  constexpr int sm = residual_smem_bytes<BC>();
  const cudaError_t e = ensure_smem(residual_kernel<BC>, sm);
  if (e != cudaSuccess) return e;
  const int rowblocks = (max_N + residual_rows<BC>() - 1) / residual_rows<BC>();
  if (active) active_list_kernel<<<1, 32, 0, s>>>(jobs, njobs, active);
  // room for every item alone, or for the split of the few items that are split
  int grid = whole ? njobs * rowblocks * kResCluster
                   : std::max(njobs * rowblocks, std::min(njobs * rowblocks * kResCluster, kResWave));
  grid = (grid + kResCluster - 1) / kResCluster * kResCluster;
  residual_kernel<BC><<<grid, kResThreads, sm, s>>>(jobs, active, njobs, rowblocks, whole);
  return cudaGetLastError();
}

cudaError_t launch_accelerate(const JobDev *jobs, int njobs, int b, int round, cudaStream_t s, long *launches) {
  // one column per SM: 1024 threads for the passes' latency; more columns: 256, four CTAs to an SM (1024
  // columns of N = 2160: 197 us over a solve's eleven launches, 398 us with 1024 threads)
  const int threads = b * njobs <= tc_num_sms() ? kAccThreads : 256;
  accelerate_kernel<<<dim3(b, njobs), threads, 0, s>>>(jobs, round);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_refine_round(FactorKind fk, const JobDev *jobs, int njobs, int max_n, int max_N, int b,
                                bool check, int *info, cudaStream_t s, long *launches, bool fp32_sweep,
                                const CUtensorMap *fmap, int active_hint, int *active, int accelerate, bool last) {
  (void)max_n;
  const cudaError_t e0 = b <= 16 ? launch_residual<16>(jobs, njobs, max_N, active, fk == kFactorFP64, s)
                                 : launch_residual<32>(jobs, njobs, max_N, active, fk == kFactorFP64, s);
  if (e0 != cudaSuccess) return e0;
  if (launches) *launches += active ? 2 : 1;
  const cudaError_t e = fk == kFactorFP64 ? sweep_solve<double2>(jobs, njobs, b, max_N, 1, info, s, launches, false, nullptr)
                                           : sweep_solve<float2>(jobs, njobs, b, max_N, 1, info, s, launches, fp32_sweep, fmap,
                                                                 active_hint);
  if (e != cudaSuccess) return e;
  if (accelerate > 0) {
    const cudaError_t ea = launch_accelerate(jobs, njobs, b, accelerate, s, launches);
    if (ea != cudaSuccess) return ea;
  }
  if (check) {
    converge_check_kernel<<<njobs, 256, 0, s>>>(jobs, accelerate > 0, last);
    if (launches) *launches += 1;
  }
  return cudaGetLastError();
}

cudaError_t launch_refine_end(const JobDev *jobs, int njobs, int ns, int kkrsz, cudaStream_t s, long *launches) {
  finalize_from_x_kernel<<<njobs, 256, 0, s>>>(jobs, ns, kkrsz);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_solve_refine(FactorKind fk, const JobDev *jobs, int njobs, int max_n, int max_N, int b,
                                int steps, int ns, int kkrsz, int *info, cudaStream_t s, long *launches,
                                bool fp32_sweep, const CUtensorMap *fmap) {
  cudaError_t e = launch_refine_begin(fk, jobs, njobs, max_n, max_N, b, info, s, launches, fp32_sweep, fmap);
  for (int it = 0; it < steps && e == cudaSuccess; ++it)
    e = launch_refine_round(fk, jobs, njobs, max_n, max_N, b, it + 1 < steps, info, s, launches, fp32_sweep,
                            fmap);
  if (e != cudaSuccess) return e;
  return launch_refine_end(jobs, njobs, ns, kkrsz, s, launches);
}

}  // namespace b200
