// Panel pivoting of the block elimination: each 64-column step picks its diagonal-block rows from
// the whole remaining column, not from the 64 x 64 diagonal block alone.
//
// The reference's CPU solver pivots with LAPACK's zgetrf inside each of its nblk diagonal blocks
// of ~N/3 rows (zblock_lu_cpp.cpp:58, nblk = 3 at linearSolvers_CPU.cpp:270); its zgesv path
// (linearSolvers_CPU.cpp:76-96) pivots over the whole column.  Restricting the pivots of a 64-column
// step to its own diagonal block is enough for the collinear contour matrices, but the
// non-collinear N = 4320 matrices (condition numbers up to ~1e7) then lose most of the FP32
// factorisation's accuracy and the mixed refinement stalls.  Here step k's rows come from every
// candidate row [k, n), in two launches:
//   magnitudes  every row below the diagonal block gets max_j |re| + |im| over the panel columns
//               k..k+kb-1 (one thread per row, coalesced over the column-major panel);
//   selection   one CTA per job: the kPivCands - kb rows of largest magnitude (a radix select on
//               the float bits, compacted in row order, so the choice is deterministic) join the
//               kb rows of the diagonal block, and Gaussian elimination with partial pivoting
//               (GEPP) on these candidates' panel rows picks the kb pivot rows in pivot order.
// That is the node of communication-avoiding "tournament pivoting" with a magnitude filter in
// front: a row that is small in every panel column is not a candidate.  On the non-collinear
// N = 4320 matrices a numpy emulation of the whole mixed solve gives the first refinement round an
// error of 1.6e-3 .. 1e-2 with it, 1.6e-3 .. 5e-3 with a full tournament over all rows and
// 5e-3 .. 9e-2 with the pivots restricted to the diagonal block.
// The kb rows then move to positions k..k+kb-1 (the rows displaced from there take the vacated
// positions): a permutation of at most 2 kb rows, applied to every column of F, so the factor
// storage is that of LAPACK's P M = L U and the kernels of the elimination and of the sweeps run
// unchanged.  The permutation of the whole elimination is tracked per job (perm), and its inverse
// (rowpos) makes the refinement's residual land in the permuted row order.  Pivots come only from
// rows [k, n), never from the central site's rows, so the trailing b x b block still holds the
// Schur complement 1 - Delta.
//
// Selection arithmetic is FP32 on either factor type (it only ranks pivot magnitudes, |re| + |im|
// as izamax, ties to the earlier candidate); the factorisation itself is unchanged.

#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"

namespace b200 {
namespace {

constexpr int kSelThreads = 512;                   // two candidates, one 16-column group per thread
constexpr int kHalf = kPivCands / 2;               // a thread's candidates are r and r + kHalf
constexpr int kGroups = kSelThreads / kHalf;       // column groups of the panel
constexpr int kGroupCols = kNb / kGroups;          // 16
static_assert(kGroups * kGroupCols == kNb, "selection thread layout");

__device__ __forceinline__ float2 to_f2(double2 a) { return make_float2((float)a.x, (float)a.y); }
__device__ __forceinline__ float2 to_f2(float2 a) { return a; }
__device__ __forceinline__ float cabs1f(float2 a) { return fabsf(a.x) + fabsf(a.y); }

// Row magnitudes below the diagonal block of step k: mags[row] = max_j |F[row, k + j]|_1 over the
// kb panel columns, as float bits (a NaN ranks as zero).
template <typename T>
__global__ void __launch_bounds__(256) panel_mags_kernel(const JobDev *__restrict__ jobs, int k) {
  const JobDev &J = jobs[blockIdx.y];
  if (J.inactive || J.piv == nullptr || k >= J.n) return;
  const int kb = min(kNb, J.n - k);
  const int row = k + kb + blockIdx.x * 256 + threadIdx.x;
  if (row >= J.n) return;
  const T *__restrict__ F = static_cast<const T *>(J.F);
  float m = 0.f;
  for (int j = 0; j < kb; ++j) {
    const float v = cabs1f(to_f2(F[(size_t)row + (size_t)(k + j) * J.ld]));
    m = v > m ? v : m;  // (a NaN compares false)
  }
  J.piv[pivot_mags_offset(J.ld) + row] = __float_as_int(m);
}

// Block-wide exclusive prefix sum of one int per thread (kSelThreads threads); returns the total.
__device__ __forceinline__ int block_scan(int v, int *s_warp, int &excl) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = lane < kSelThreads / 32 ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < kSelThreads / 32) s_warp[lane] = w;  // inclusive over warps
  }
  __syncthreads();
  const int total = s_warp[kSelThreads / 32 - 1];
  excl = (warp > 0 ? s_warp[warp - 1] : 0) + x - v;
  __syncthreads();  // s_warp is reused by the next scan
  return total;
}

// Step k's selection, one CTA per job (see the file comment); the kb pivot rows in pivot order
// become the step's row moves, also applied to the job's permutation.
template <typename T>
__global__ void __launch_bounds__(kSelThreads) panel_select_kernel(const JobDev *__restrict__ jobs, int k) {
  const JobDev &J = jobs[blockIdx.x];
  if (J.inactive || J.piv == nullptr || k >= J.n) return;
  const int kb = min(kNb, J.n - k);
  const int n = J.n, ld = J.ld;
  int *__restrict__ piv = J.piv;
  const unsigned *__restrict__ mags = reinterpret_cast<const unsigned *>(piv + pivot_mags_offset(ld));
  __shared__ float2 s_col[2][kPivCands];  // the step's column, by step parity
  __shared__ __align__(16) float2 s_row[kNb];  // the pivot row's columns, in the threads' places
  __shared__ unsigned long long s_best[2][kHalf / 32];
  __shared__ int s_dst[2 * kNb], s_src[2 * kNb];
  __shared__ int s_vac[kNb];
  __shared__ unsigned s_in[2], s_moved[2], s_below[2];
  __shared__ int s_ok;
  __shared__ int s_cand[kPivCands];
  __shared__ int s_out[kNb];
  __shared__ int s_hist[256];
  __shared__ int s_warp[kSelThreads / 32];
  __shared__ unsigned s_prefix;
  __shared__ int s_remain;
  const int tid = threadIdx.x;

  // --- candidates: the diagonal block's rows, then the largest rows below it ---
  const int lo = k + kb, m2 = n - lo;  // rows below the diagonal block
  const int K2 = min(m2, kPivCands - kb);
  if (tid < kb) s_cand[tid] = k + tid;
  if (K2 == m2) {
    for (int i = tid; i < m2; i += kSelThreads) s_cand[kb + i] = lo + i;
  } else {
    // radix select (8 bits at a time, most significant first) of the K2-th largest key
    unsigned prefix = 0u, mask = 0u;
    int remain = K2;
    for (int shift = 24; shift >= 0; shift -= 8) {
      if (tid < 256) s_hist[tid] = 0;
      __syncthreads();
      for (int i = tid; i < m2; i += kSelThreads) {
        const unsigned key = mags[lo + i];
        if ((key & mask) == prefix) atomicAdd(&s_hist[(key >> shift) & 255u], 1);
      }
      __syncthreads();
      if (tid < 32) {  // the digit of the remain-th largest key: lane l has bins 255 - 8 l down
        int sum = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) sum += s_hist[255 - 8 * tid - i];
        int x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (tid >= o) x += y;
        }
        if (x >= remain && x - sum < remain) {  // (one lane: at least `remain` keys match the prefix)
          int cum = x - sum, d = 255 - 8 * tid;
          for (; d > 0 && cum + s_hist[d] < remain; --d) cum += s_hist[d];
          s_prefix = prefix | ((unsigned)d << shift);
          s_remain = remain - cum;
        }
      }
      __syncthreads();
      prefix = s_prefix;
      remain = s_remain;
      mask |= 255u << shift;
      __syncthreads();
    }
    // keys above the threshold, then `remain` of the keys equal to it, each in row order
    const int chunk = (m2 + kSelThreads - 1) / kSelThreads;
    const int r0 = min(m2, tid * chunk), r1 = min(m2, r0 + chunk);
    int ngt = 0, neq = 0;
    for (int i = r0; i < r1; ++i) {
      const unsigned key = mags[lo + i];
      ngt += key > prefix;
      neq += key == prefix;
    }
    int bgt = 0, beq = 0;
    const int tgt = block_scan(ngt, s_warp, bgt);
    block_scan(neq, s_warp, beq);
    for (int i = r0; i < r1; ++i) {
      const unsigned key = mags[lo + i];
      if (key > prefix) {
        s_cand[kb + bgt++] = lo + i;
      } else if (key == prefix) {
        if (beq < remain) s_cand[kb + tgt + beq] = lo + i;
        ++beq;
      }
    }
  }
  __syncthreads();
  const int R = kb + K2;  // candidates

  // --- GEPP on the candidates' panel rows ---
  if (R <= kb) {  // the last step: the block's own rows, in place
    if (tid < kb) s_out[tid] = k + tid;
    __syncthreads();
  } else {
    const T *__restrict__ F = static_cast<const T *>(J.F);
    // Thread (candidates r and r + kHalf, column group g) holds its 2 x 16 elements in registers.  What bounds
    // a step is the shared-memory reads of the pivot row, the same 128 bytes for every row of a group,
    // so a thread has two rows for them (a launch takes 100 us; 124 us with one row to each of 1024 threads, and
    // the moves and the radix digits found by one thread).  A step writes the columns of the group that
    // holds the step's column one place down, so that group's column to rank is always in place 0; the
    // others stay put.
    const int r = tid & (kHalf - 1), g = tid / kHalf, c0 = g * kGroupCols;
    int cand[2];
    float2 a[2][kGroupCols];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      cand[h] = r + h * kHalf < R ? s_cand[r + h * kHalf] : -1;
#pragma unroll
      for (int j = 0; j < kGroupCols; ++j)
        a[h][j] = (cand[h] >= 0 && c0 + j < kb) ? to_f2(F[(size_t)cand[h] + (size_t)(k + c0 + j) * ld])
                                                : make_float2(0.f, 0.f);
    }
    bool taken[2] = {false, false};
    for (int p = 0; p < kb; ++p) {
      const int par = p & 1;
      const bool mine = g == p / kGroupCols;  // (uniform over a warp)
      if (mine) {  // rank the rows: the largest |re| + |im| (its bits order as integers), ties low
        unsigned key[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float v = cabs1f(a[h][0]);
          if (!(v == v)) v = 0.f;  // a NaN ranks as zero, so a row in range is still chosen
          key[h] = cand[h] >= 0 && !taken[h] ? __float_as_uint(v) + 1u : 0u;
          s_col[par][r + h * kHalf] = a[h][0];
        }
        const unsigned hi = max(key[0], key[1]), row = key[0] >= key[1] ? r : r + kHalf;
        const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
        const unsigned lo = __reduce_max_sync(0xffffffffu, hi == mhi ? kPivCands - 1 - row : 0u);
        if ((tid & 31) == 0) s_best[par][r >> 5] = ((unsigned long long)mhi << 32) | lo;
      }
      __syncthreads();
      unsigned long long best = s_best[par][0];
#pragma unroll
      for (int w = 1; w < kHalf / 32; ++w) best = s_best[par][w] > best ? s_best[par][w] : best;
      // R > kb > p candidates remain untaken, each ranked above the taken ones: bi is one of them
      const int bi = kPivCands - 1 - (int)(unsigned)best;
      const float2 d = s_col[par][bi];
      const float dd = d.x * d.x + d.y * d.y;
      float2 f[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (r + h * kHalf == bi) {
          taken[h] = true;
#pragma unroll
          for (int j = 0; j < kGroupCols; j += 2)
            *reinterpret_cast<float4 *>(&s_row[c0 + j]) =
                make_float4(a[h][j].x, a[h][j].y, a[h][j + 1].x, a[h][j + 1].y);
        }
        const float2 x0 = s_col[par][r + h * kHalf];
        f[h] = make_float2(0.f, 0.f);
        if (dd > 0.f && !taken[h])
          f[h] = make_float2((x0.x * d.x + x0.y * d.y) / dd, (x0.y * d.x - x0.x * d.y) / dd);
      }
      if (tid == 0) s_out[p] = s_cand[bi];
      __syncthreads();
      auto sub = [&](int h, float2 x, float2 pj) {
        x.x -= f[h].x * pj.x - f[h].y * pj.y;
        x.y -= f[h].x * pj.y + f[h].y * pj.x;
        return x;
      };
      if (mine || p < c0) {
#pragma unroll
        for (int j = 0; j < kGroupCols; j += 2) {
          const float4 q = *reinterpret_cast<const float4 *>(&s_row[c0 + j]);
          const float2 q0 = make_float2(q.x, q.y), q1 = make_float2(q.z, q.w);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float2 v0 = sub(h, a[h][j], q0), v1 = sub(h, a[h][j + 1], q1);
            if (mine) {
              if (j > 0) a[h][j - 1] = v0;
              a[h][j] = v1;
            } else {
              a[h][j] = v0;
              a[h][j + 1] = v1;
            }
          }
        }
        if (mine) a[0][kGroupCols - 1] = a[1][kGroupCols - 1] = make_float2(0.f, 0.f);  // (not needed again)
      }
    }
    __syncthreads();
  }
  // the moves that bring the pivot rows to k..k+kb-1 (pivot order) and the displaced rows to the
  // vacated positions, the q-th displaced row to the q-th vacated position in pivot order; a permutation of
  // at most 2 kb positions, also applied to perm.  Thread i < 64: step i and position k + i.
  if (tid == 0) s_ok = 1;
  if (tid < 2) s_in[tid] = 0u;
  __syncthreads();
  const int out = tid < kb ? s_out[tid] : k + tid;
  if (tid < kNb) {
    // kb distinct rows in [k, n) by construction; anything else leaves the rows in place
    if (tid < kb && (out < k || out >= n)) s_ok = 0;
    if (tid < kb && out >= k && out - k < kb) atomicOr(&s_in[(out - k) >> 5], 1u << ((out - k) & 31));
    const unsigned mv = __ballot_sync(0xffffffffu, tid < kb && out != k + tid);
    const unsigned vac = __ballot_sync(0xffffffffu, tid < kb && out >= k + kb);
    if ((tid & 31) == 0) {
      s_moved[tid >> 5] = mv;
      s_below[tid >> 5] = vac;
    }
  }
  __syncthreads();
  const unsigned long long moved = (unsigned long long)s_moved[1] << 32 | s_moved[0];
  const unsigned long long vacated = (unsigned long long)s_below[1] << 32 | s_below[0];
  const unsigned long long stay = (unsigned long long)s_in[1] << 32 | s_in[0];
  const unsigned long long lower = tid < kNb ? (1ull << tid) - 1 : 0ull;
  const int nmv = __popcll(moved), nvac = __popcll(vacated);
  if (tid < kb) {
    if (moved >> tid & 1) {
      const int i = __popcll(moved & lower);
      s_dst[i] = k + tid;
      s_src[i] = out;
    }
    if (vacated >> tid & 1) s_vac[__popcll(vacated & lower)] = out;
  }
  __syncthreads();
  if (tid < kb && !(stay >> tid & 1)) {
    const int i = __popcll(~stay & lower);
    if (i < nvac) {  // (as many vacated positions as displaced rows)
      s_dst[nmv + i] = s_vac[i];
      s_src[nmv + i] = k + tid;
    }
  }
  __syncthreads();
  const int cnt = s_ok ? nmv + nvac : 0;
  int *mv = piv + pivot_moves_offset(ld);
  if (tid == 0) mv[0] = cnt;
  int old = 0;
  if (tid < cnt) {
    mv[1 + tid] = s_dst[tid];
    mv[1 + 2 * kNb + tid] = s_src[tid];
    old = piv[s_src[tid]];
  }
  __syncthreads();
  if (tid < cnt) piv[s_dst[tid]] = old;
}

// The step's row moves applied to columns [c0, c1) of F: one warp per column reads every moved
// element, then writes it at its destination.
template <typename T>
__global__ void __launch_bounds__(256) row_move_kernel(const JobDev *__restrict__ jobs, int k, int c0, int c1) {
  const JobDev &J = jobs[blockIdx.y];
  if (J.inactive || J.piv == nullptr || k >= J.n) return;
  const int *__restrict__ mv = J.piv + pivot_moves_offset(J.ld);
  const int cnt = mv[0];
  if (cnt == 0) return;
  const int hi = min(c1, J.N);
  T *__restrict__ F = static_cast<T *>(J.F);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  int dst[4], src[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = lane + 32 * q;
    dst[q] = i < cnt ? mv[1 + i] : -1;
    src[q] = i < cnt ? mv[1 + 2 * kNb + i] : -1;
  }
  for (int c = c0 + blockIdx.x * nw + warp; c < hi; c += gridDim.x * nw) {
    T *col = F + (size_t)c * J.ld;
    T v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (src[q] >= 0) v[q] = col[src[q]];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (dst[q] >= 0) col[dst[q]] = v[q];
    __syncwarp();
  }
}

__global__ void pivot_init_kernel(const JobDev *__restrict__ jobs) {
  const JobDev &J = jobs[blockIdx.x];
  if (J.inactive || J.piv == nullptr) return;
  for (int p = threadIdx.x; p < J.N; p += blockDim.x) J.piv[p] = p;
  if (threadIdx.x == 0) J.piv[pivot_moves_offset(J.ld)] = 0;
}

// rowpos: the physical row of every original row once the elimination is done.
__global__ void pivot_finish_kernel(const JobDev *__restrict__ jobs) {
  const JobDev &J = jobs[blockIdx.x];
  if (J.inactive || J.piv == nullptr) return;
  int *rowpos = J.piv + J.ld;
  for (int p = threadIdx.x; p < J.N; p += blockDim.x) rowpos[J.piv[p]] = p;
}

template <typename T>
cudaError_t select_impl(const JobDev *jobs, int njobs, int k, int max_n, cudaStream_t s, long *launches) {
  if (max_n - k <= 0) return cudaSuccess;
  const int m = max_n - k - kNb;  // rows below the diagonal block, at most
  if (m > kPivCands - kNb) {  // magnitudes are ranked only when the candidates must be filtered
    panel_mags_kernel<T><<<dim3((m + 255) / 256, njobs), 256, 0, s>>>(jobs, k);
    if (launches) *launches += 1;
  }
  panel_select_kernel<T><<<njobs, kSelThreads, 0, s>>>(jobs, k);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

template <typename T>
cudaError_t move_impl(const JobDev *jobs, int njobs, int k, int c0, int c1, int max_N, cudaStream_t s,
                      long *launches) {
  const int hi = std::min(c1, max_N);
  if (hi <= c0) return cudaSuccess;
  const int cols = hi - c0;
  const int per_cta = 8 * 4;  // 8 warps, 4 columns each
  const int grid = std::max(1, std::min((cols + per_cta - 1) / per_cta, 4 * 148 / std::max(1, njobs) + 1));
  row_move_kernel<T><<<dim3(grid, njobs), 256, 0, s>>>(jobs, k, c0, c1);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_pivot_init(const JobDev *jobs, int njobs, cudaStream_t s, long *launches) {
  pivot_init_kernel<<<njobs, 256, 0, s>>>(jobs);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_panel_select(FactorKind fk, const JobDev *jobs, int njobs, int k, int max_n, cudaStream_t s,
                                long *launches) {
  return fk == kFactorFP64 ? select_impl<double2>(jobs, njobs, k, max_n, s, launches)
                           : select_impl<float2>(jobs, njobs, k, max_n, s, launches);
}

cudaError_t launch_row_moves(FactorKind fk, const JobDev *jobs, int njobs, int k, int c0, int c1, int max_N,
                             cudaStream_t s, long *launches) {
  return fk == kFactorFP64 ? move_impl<double2>(jobs, njobs, k, c0, c1, max_N, s, launches)
                           : move_impl<float2>(jobs, njobs, k, c0, c1, max_N, s, launches);
}

cudaError_t launch_pivot_finish(const JobDev *jobs, int njobs, cudaStream_t s, long *launches) {
  pivot_finish_kernel<<<njobs, 256, 0, s>>>(jobs);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

}  // namespace b200
