// Complex FP64 GEMM tile on the FP64 tensor cores (mma.sync m8n8k4 f64), shared by the block
// elimination and the inverse passes of the adjoint and the full tau.
//
// As real products C = A B is Cr = Ar Br - Ai Bi, Ci = Ar Bi + Ai Br: four 8 x 8 x 4 MMAs per 8 x 8
// complex block and K step of 4, each 256 FMAs in one instruction.  An SM does 64 FP64 FMAs a cycle by
// DFMA or by MMA; what bounds the DFMA form is everything around the FMAs (per 16 of them a thread
// issues 8 shared-memory loads of 16 bytes, which take as many cycles as the FMAs), and the MMA form
// needs 8 loads per 64 MMAs = 1024 cycles of the pipe.
#pragma once

#include <cuda_runtime.h>

namespace b200 {
namespace dm {

enum { kOverwrite = 0, kSubtract = 1 };

constexpr int kThreads = 128;  // four warps, 2 x 2 over the tile
constexpr int kMaxK = 64;      // largest inner dimension: one elimination step
constexpr int kKc = 8;         // K per stage of A's ring
constexpr int kStages = 4;

// D (8 x 8) += A (8 x 4) B (4 x 8) in FP64 on the tensor cores, per warp: lane l holds
// a = A[l / 4][l % 4], b = B[l % 4][l / 4] and D[l / 4][2 (l % 4) + i] in d_i.
__device__ __forceinline__ void mma_884(double &d0, double &d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// 16 bytes to shared memory, zeros (and no read) where `in` is false.
__device__ __forceinline__ void cp_async16_zfill(void *smem, const void *gmem, bool in) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int bytes = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}

// Shared memory of a tile of WM x WN 8 x 8 blocks per warp (16 WM rows, 16 WN columns): all K rows of
// B's columns, and a ring of K chunks of A.  A's rows are padded to a stride of 32 and B's columns to
// one of 64 modulo 128 bytes: the eight lanes of a 128-byte phase (two rows or columns, four k) then
// hit eight different 16-byte banks.
template <int WM, int WN>
struct Tile {
  static constexpr int kRows = 16 * WM, kCols = 16 * WN;
  static constexpr int kAs = kRows + 2;
  static constexpr int kBs = kMaxK + 4;
  static constexpr int kSmem = (kStages * kKc * kAs + kCols * kBs) * (int)sizeof(double2);
};

// A column of tiles: C (m x n) = A (m x K) B (K x n)  [kOverwrite; m within one tile; C may be B, whose
// reads all precede the last barrier before the first write of C] or C -= A B [kSubtract], column-major
// with leading dimensions, n up to the tile's columns, K <= kMaxK.  Called by all kThreads threads.
// B stays in shared memory while A streams through the ring, whose loads run three chunks ahead and
// across tile boundaries, so only the first tile waits for its operands.
template <int WM, int WN, int MODE>
__device__ __forceinline__ void zgemm_column(const double2 *__restrict__ A, int lda, const double2 *B, int ldb,
                                             double2 *C, int ldc, int m, int n, int K, double2 *sm) {
  using TL = Tile<WM, WN>;
  constexpr int R = TL::kRows, C0 = TL::kCols;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wr = (warp & 1) * 8 * WM, wc = (warp >> 1) * 8 * WN;
  const int nch = (K + kKc - 1) / kKc;
  const int total = nch * ((m + R - 1) / R);
  double2 *bs = sm, *ring = sm + C0 * TL::kBs;
  int lt = 0, lc = 0;  // tile and chunk of the next load
  auto load = [&](int q) {  // load number q of the sequence
    double2 *as = ring + (q % kStages) * (kKc * TL::kAs);
    const int k0 = lc * kKc, r0 = lt * R;
#pragma unroll
    for (int u = 0; u < kKc * R / kThreads; ++u) {
      const int e = tid + u * kThreads;
      const int r = e % R, kk = e / R;
      const bool in = r0 + r < m && k0 + kk < K;
      cp_async16_zfill(as + kk * TL::kAs + r, in ? A + (r0 + r) + (size_t)(k0 + kk) * lda : A, in);
    }
    if (lt == 0) {
#pragma unroll
      for (int u = 0; u < kKc * C0 / kThreads; ++u) {
        const int e = tid + u * kThreads;
        const int kk = e % kKc, c = e / kKc;
        const bool in = c < n && k0 + kk < K;
        cp_async16_zfill(bs + c * TL::kBs + k0 + kk, in ? B + (k0 + kk) + (size_t)c * ldb : B, in);
      }
    }
    if (++lc == nch) {
      lc = 0;
      ++lt;
    }
  };
  __syncthreads();  // (a caller that loops: the shared memory is free again)
#pragma unroll
  for (int q = 0; q < kStages - 1; ++q) {
    if (q < total) load(q);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  double re[WM][WN][2], im[WM][WN][2];
  int ch = 0, r0 = 0;
#pragma unroll 1
  for (int q = 0; q < total; ++q) {
    if (ch == 0) {
#pragma unroll
      for (int i = 0; i < WM; ++i)
#pragma unroll
        for (int j = 0; j < WN; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
      if (MODE == kSubtract)  // C's lines on their way to L2 while the product runs
        for (int e = tid; e < C0 * (R / 8); e += kThreads) {
          const int r = r0 + (e % (R / 8)) * 8, c = e / (R / 8);
          if (r < m && c < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + r + (size_t)c * ldc));
        }
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();  // load q has landed for every thread; the ring stage of q - 1 is no longer read
    if (q + kStages - 1 < total) load(q + kStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const double2 *as = ring + (q % kStages) * (kKc * TL::kAs);
    const double2 *bk = bs + ch * kKc;
#pragma unroll
    for (int ks = 0; ks < kKc; ks += 4) {
      double2 a[WM], b[WN];
#pragma unroll
      for (int i = 0; i < WM; ++i) a[i] = as[(ks + t) * TL::kAs + wr + 8 * i + g];
#pragma unroll
      for (int j = 0; j < WN; ++j) b[j] = bk[(wc + 8 * j + g) * TL::kBs + ks + t];
#pragma unroll
      for (int i = 0; i < WM; ++i)
#pragma unroll
        for (int j = 0; j < WN; ++j) {
          mma_884(re[i][j][0], re[i][j][1], a[i].x, b[j].x);
          mma_884(im[i][j][0], im[i][j][1], a[i].x, b[j].y);
        }
#pragma unroll
      for (int i = 0; i < WM; ++i)
#pragma unroll
        for (int j = 0; j < WN; ++j) {
          mma_884(re[i][j][0], re[i][j][1], -a[i].y, b[j].y);
          mma_884(im[i][j][0], im[i][j][1], a[i].y, b[j].x);
        }
    }
    if (++ch < nch) continue;
    ch = 0;
#pragma unroll
    for (int j = 0; j < WN; ++j) {
      double2 v[WM][2];
      if (MODE == kSubtract) {
#pragma unroll
        for (int i = 0; i < WM; ++i)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = r0 + wr + 8 * i + g, c = wc + 8 * j + 2 * t + h;
            v[i][h] = (r < m && c < n) ? C[r + (size_t)c * ldc] : make_double2(0.0, 0.0);
          }
      }
#pragma unroll
      for (int i = 0; i < WM; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = r0 + wr + 8 * i + g, c = wc + 8 * j + 2 * t + h;
          if (r >= m || c >= n) continue;
          C[r + (size_t)c * ldc] = MODE == kOverwrite
                                       ? make_double2(re[i][j][h], im[i][j][h])
                                       : make_double2(v[i][h].x - re[i][j][h], v[i][h].y - im[i][j][h]);
        }
    }
    r0 += R;
  }
}

// Tiles of a column that one CTA walks: as many as leave the launch about four waves of CTAs, at
// most 8.
inline int column_tiles(long tiles) {
  const long t = tiles / (4 * 4 * 148);
  return t < 1 ? 1 : t > 8 ? 8 : (int)t;
}

}  // namespace dm
}  // namespace b200
