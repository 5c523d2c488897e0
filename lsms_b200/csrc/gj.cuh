// Small dense solves in shared memory shared by the elimination and adjoint kernels.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"
#include "cplx.cuh"

namespace b200 {
namespace cx {

// Pivot search key of a row: |re| + |im| (non-negative doubles order as their bit patterns; NaN
// counts as 0) with its 6 low mantissa bits replaced by 63 - row, so that the largest key is the
// largest value, ties - and values within 2^-46 relative of each other - going to the lowest row.
__device__ __forceinline__ unsigned long long pivot_key(double v, int row) {
  v = (v == v) ? v : 0.0;
  return ((unsigned long long)__double_as_longlong(v) & ~63ull) | (unsigned long long)(63 - row);
}
// The largest of the lanes' keys, as the row it names: two warp max-reductions (high word, then the
// low word among the lanes holding the high max).
__device__ __forceinline__ int pivot_row(unsigned long long key) {
  const unsigned hi = (unsigned)(key >> 32);
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? (unsigned)key : 0u);
  return 63 - (int)(mlo & 63u);
}
// x - g u
__device__ __forceinline__ double2 cfnma(double2 x, double2 g, double2 u) {
  x.x = fma(-g.x, u.x, x.x);
  x.x = fma(g.y, u.y, x.x);
  x.y = fma(-g.x, u.y, x.y);
  x.y = fma(-g.y, u.x, x.y);
  return x;
}

// b x b solve by Gauss-Jordan on [A | rhs] in shared memory (FP64, partial pivoting on |re| + |im|, no
// row interchanges).  A is kMaxB x (2 kMaxB + 1); on return columns [b, 2b) hold A^-1 rhs.  Called by
// every thread of a 256-thread block.  Returns singular.
// Warp w holds columns 8w .. 8w + 7 and lane l row l, in registers.  Step p subtracts g u from every
// row, u = row pv and g_r = A[r][p] / d (g_pv = 1 - 1/d), which leaves row pv divided by d.  The update
// writes each column one place down, so the column to search is always the first, and the warp that
// holds column p + 1 searches it and publishes step p + 1's g before it updates its other columns: one
// block barrier per step: 17 us at b = 16 (26 us with the matrix in shared memory and six barriers a
// step).
__device__ inline bool gj_solve_smem(double2 (*A)[2 * kMaxB + 1], int b) {
  __shared__ double2 s_g[2][32];
  __shared__ double2 s_row[8][8];
  __shared__ int s_pv[2], s_inv[32], s_hi[8], s_sing;
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  double2 a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = (l < b && 8 * w + j < 2 * b) ? A[l][8 * w + j] : make_double2(0.0, 0.0);
  if (tid < 32) s_inv[tid] = tid;
  if (tid == 0) s_sing = 0;
  // A is taken times a power of two that brings its largest element to 1 .. 2: 1 - 1/d would lose the digits
  // of a large d
  int hi = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (8 * w + j < b) hi = max(hi, max(__double2hiint(a[j].x) & 0x7fffffff, __double2hiint(a[j].y) & 0x7fffffff));
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (l == 0) s_hi[w] = hi;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) hi = max(hi, s_hi[i]);
  const int e2 = hi >> 20;  // (0x7ff: an element is not finite)
  const double scale = e2 == 0x7ff ? 1.0 : __hiloint2double(max(1, 2046 - e2) << 20, 0);
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (8 * w + j < b) a[j] = make_double2(a[j].x * scale, a[j].y * scale);
  bool used = l >= b;
  auto search = [&](double2 x, int p) {
    const double v = cabs1(x);
    // 1/x of the lane's own row, scaled by a power of two against overflow, beside the reductions
    const bool zero = x.x == 0.0 && x.y == 0.0;
    const double m = fmax(fabs(x.x), fabs(x.y));
    const int ex = (__double2hiint(m) >> 20) & 0x7ff;
    const double sc = __hiloint2double(max(1, min(2045, 2046 - ex)) << 20, 0);
    const double xr = x.x * sc, xi = x.y * sc;
    const double rr = sc / (zero ? 1.0 : xr * xr + xi * xi);
    const double2 rl = make_double2(zero ? 0.0 : xr * rr, zero ? 0.0 : -xi * rr);
    const int pv = min(pivot_row(used ? 0ull : pivot_key(v, l)), b - 1);
    double2 dinv;
    dinv.x = __shfl_sync(0xffffffffu, rl.x, pv);
    dinv.y = __shfl_sync(0xffffffffu, rl.y, pv);
    const bool sing = __shfl_sync(0xffffffffu, zero ? 1 : 0, pv) != 0;
    s_g[p & 1][l] = l == pv ? make_double2(1.0 - dinv.x, -dinv.y) : cmul(x, dinv);
    if (l == 0) {
      s_pv[p & 1] = pv;
      s_inv[pv] = p;
      if (sing) s_sing = 1;
    }
  };
  if (w == 0) search(a[0], 0);
  __syncthreads();
#pragma unroll 1
  for (int p = 0; p < b; ++p) {  // place j holds column 8w + ((p + j) & 7)
    const int pv = s_pv[p & 1];
    const double2 g = s_g[p & 1][l];
    if (l == pv) {
#pragma unroll
      for (int j = 0; j < 8; ++j) s_row[w][j] = a[j];
      used = true;
    }
    __syncwarp();
    const double2 o = a[0];
    a[0] = cfnma(a[1], g, s_row[w][1]);
    if (p + 1 < b && w == ((p + 1) >> 3)) search(a[0], p + 1);
#pragma unroll
    for (int j = 2; j < 8; ++j) a[j - 1] = cfnma(a[j], g, s_row[w][j]);
    a[7] = cfnma(o, g, s_row[w][0]);
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = 8 * w + ((j + b) & 7);
    if (l < b && c >= b && c < 2 * b) A[s_inv[l]][c] = make_double2(a[j].x * scale, a[j].y * scale);
  }
  __syncthreads();
  return s_sing != 0;
}

}  // namespace cx
}  // namespace b200
