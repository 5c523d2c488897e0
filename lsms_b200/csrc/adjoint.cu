// Reverse-mode derivatives of tau00 and of ln det M with respect to every LIZ site's t-matrix,
// from the FP64 block factors of the forward solve (no second factorisation).
//
// With M = 1 - T G (T = blockdiag(t_j), G the structure constants, G_jj = 0), X = M^-1 [0; t_0]
// (tau00 = X_0, positions with the central site last) and a cotangent taubar on tau00, the
// holomorphic pull-back (no conjugation: delta<taubar, tau00> = sum_j sum_ab tbar_j,ab dt_j,ab) is
//   Lambda = M^-T E_0 taubar,   Z = G X,
//   tbar_j = Lambda_j Z_j^T  (+ Lambda_0 for the central site, which also enters through t_0),
// and d ln det M = tr(M^-1 dM) = -sum_j tr(dt_j (G M^-1)_jj) gives
//   dlogdet_j = -((G M^-1)_jj)^T.
// The reference has no derivative code; these follow from dM = -dT G and d(M^-1) = -M^-1 dM M^-1.
//
// Work: V = M^-1 by the block factors applied to the identity (forward and backward passes of
// batched 64 x 64 FP64 GEMM tiles, ~(2/3) N^3 complex multiply-adds per job), G rebuilt into M's
// storage by the build kernel, then one CTA per (site, job) contracts its row block of G with X
// and with its column block of V (2 N b^2 multiply-adds) and forms the small products.

#include <cuda_runtime.h>

#include "common.cuh"
#include "cplx.cuh"
#include "dmma.cuh"
#include "gj.cuh"
#include "split8.cuh"

namespace b200 {
namespace {

using namespace cx;

using dm::kOverwrite;
using dm::kSubtract;

using GemmView = s8::View;

// C (m x n) = A B  [kOverwrite, C may alias B: one row of tiles, so a CTA reads all of its columns of
// B before it writes them]
// C (m x n) -= A B [kSubtract]
// Tiles of 16 WM x 16 WN on the FP64 tensor cores (dmma.cuh), in columns of `len`.
template <class Op, int WM, int WN, int MODE>
__global__ void __launch_bounds__(dm::kThreads, WM == 4 ? 3 : 4)
    zgemm_view_kernel(const JobDev *__restrict__ jobs, int k, Op op, int len, bool small) {
  extern __shared__ __align__(16) double2 vsm64[];
  using TL = dm::Tile<WM, WN>;
  const JobDev &J = jobs[blockIdx.z];
  GemmView g;
  if (!op(J, k, g) || (small && split_pays(g.m, g.n, kSplitInverse))) return;
  const int row0 = blockIdx.y * len * TL::kRows, col0 = blockIdx.x * TL::kCols;
  if (row0 >= g.m || col0 >= g.n) return;
  dm::zgemm_column<WM, WN, MODE>(g.A + row0, g.lda, g.B + (size_t)col0 * g.ldb, g.ldb,
                                 g.C + row0 + (size_t)col0 * g.ldc, g.ldc, min(len * TL::kRows, g.m - row0),
                                 min(TL::kCols, g.n - col0), g.K, vsm64);
}

// --- the passes of V = M^-1 = U^-1 S^-1 L^-1 over the block factors in F (positions order) ---
// forward step k:  V_k = D_k V_k  (columns [0, k + kb): L^-1 is lower triangular)
struct OpInvDiag {
  __device__ bool operator()(const JobDev &J, int k, GemmView &g) const {
    if (k >= J.n) return false;
    const int kb = min(kNb, J.n - k);
    const double2 *F = static_cast<const double2 *>(J.F);
    g.A = F + (size_t)k + (size_t)k * J.ld;
    g.B = J.V + k;
    g.C = J.V + k;
    g.lda = g.ldb = g.ldc = J.ld;
    g.m = kb;
    g.n = k + kb;
    g.K = kb;
    return true;
  }
};
// forward step k:  V[k+kb:N, 0:k+kb] -= A21_k V_k
struct OpInvLower {
  __device__ bool operator()(const JobDev &J, int k, GemmView &g) const {
    if (k >= J.n) return false;
    const int kb = min(kNb, J.n - k);
    const double2 *F = static_cast<const double2 *>(J.F);
    g.A = F + (size_t)(k + kb) + (size_t)k * J.ld;
    g.B = J.V + k;
    g.C = J.V + (k + kb);
    g.lda = g.ldb = g.ldc = J.ld;
    g.m = J.N - k - kb;
    g.n = k + kb;
    g.K = kb;
    return g.m > 0;
  }
};
// V_c = S^-1 V_c with S^-1 staged in the Y buffer (b x b, leading dimension ld)
struct OpSchurApply {
  __device__ bool operator()(const JobDev &J, int, GemmView &g) const {
    g.A = J.Y;
    g.B = J.V + J.n;
    g.C = J.V + J.n;
    g.lda = g.ldb = g.ldc = J.ld;
    g.m = J.b;
    g.n = J.N;
    g.K = J.b;
    return true;
  }
};
// backward, block at k (k < 0: the central block):  V[0:k, :] -= W[0:k, k:k+kb] V_k
struct OpInvUpper {
  __device__ bool operator()(const JobDev &J, int k, GemmView &g) const {
    int kb;
    if (k < 0) {
      k = J.n;
      kb = J.b;
    } else {
      if (k >= J.n) return false;
      kb = min(kNb, J.n - k);
    }
    if (k == 0) return false;
    const double2 *F = static_cast<const double2 *>(J.F);
    g.A = F + (size_t)k * J.ld;
    g.B = J.V + k;
    g.C = J.V;
    g.lda = g.ldb = g.ldc = J.ld;
    g.m = k;
    g.n = J.N;
    g.K = kb;
    return true;
  }
};

// V = identity (N x N); one CTA per column
__global__ void __launch_bounds__(256) identity_kernel(const JobDev *__restrict__ jobs) {
  const JobDev &J = jobs[blockIdx.y];
  const int c = blockIdx.x;
  if (c >= J.N) return;
  for (int r = threadIdx.x; r < J.N; r += 256)
    J.V[(size_t)r + (size_t)c * J.ld] = make_double2(r == c ? 1.0 : 0.0, 0.0);
}

// S^-1 (the trailing b x b block of F) into the Y buffer
__global__ void __launch_bounds__(256) schur_inverse_kernel(const JobDev *__restrict__ jobs) {
  const JobDev &J = jobs[blockIdx.x];
  const int b = J.b, n = J.n, ld = J.ld;
  __shared__ double2 A[kMaxB][2 * kMaxB + 1];
  const double2 *S = static_cast<const double2 *>(J.F) + (size_t)n + (size_t)n * ld;
  for (int e = threadIdx.x; e < b * b; e += blockDim.x) {
    const int c = e / b, r = e - c * b;
    A[r][c] = S[r + (size_t)c * ld];
    A[r][b + c] = make_double2(r == c ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  gj_solve_smem(A, b);  // a singular S was already reported by the forward solve
  for (int e = threadIdx.x; e < b * b; e += blockDim.x) {
    const int c = e / b, r = e - c * b;
    J.Y[(size_t)r + (size_t)c * ld] = A[r][b + c];
  }
}

template <class Op, int WM, int WN, int MODE>
cudaError_t gemm_launch_tile(const JobDev *jobs, int njobs, int k, int max_m, int max_n, bool small, cudaStream_t s) {
  using TL = dm::Tile<WM, WN>;
  const cudaError_t e = ensure_smem(zgemm_view_kernel<Op, WM, WN, MODE>, TL::kSmem);
  if (e != cudaSuccess) return e;
  const int tx = (max_n + TL::kCols - 1) / TL::kCols, ty = (max_m + TL::kRows - 1) / TL::kRows;
  const int len = dm::column_tiles((long)tx * ty * njobs);
  zgemm_view_kernel<Op, WM, WN, MODE>
      <<<dim3(tx, (ty + len - 1) / len, njobs), dm::kThreads, TL::kSmem, s>>>(jobs, k, Op(), len, small);
  return cudaGetLastError();
}

// kOverwrite: at most 64 rows, one row of 64 x 32 tiles.  kSubtract: 32 x 32 tiles, as in the
// elimination's update.
template <class Op, int MODE>
cudaError_t gemm_launch(const JobDev *jobs, int njobs, int k, int max_m, int max_n, cudaStream_t s,
                        long *launches, bool small = false) {
  if (max_m <= 0 || max_n <= 0) return cudaSuccess;
  if (launches) *launches += 1;
  return gemm_launch_tile<Op, MODE == kOverwrite ? 4 : 2, 2, MODE>(jobs, njobs, k, max_m, max_n, small, s);
}

// A pass's update at step k, m x n of at most max_m x max_n and, for every job, at least min_m x min_n: on
// the integer tensor cores for the jobs whose own is large enough (split_pays).
template <class Op>
cudaError_t subtract_launch(const JobDev *jobs, int njobs, int k, int min_m, int min_n, int max_m, int max_n,
                            const SplitBufs *split, int pass, int *err, cudaStream_t s, long *launches) {
  const bool large = split && split_pays(max_m, max_n, kSplitInverse);
  if (large) {
    const s8::Large<Op, kSplitInverse> op;
    cudaError_t e = s8::launch_split_pack(*split, jobs, njobs, k, max_m, max_n, s, op);
    if (e == cudaSuccess)
      e = s8::launch_split_update(*split, jobs, njobs, k, max_m, max_n, false,
                                  split->counters + pass * split->steps + k / kNb, err, s, op);
    if (e != cudaSuccess) return e;
    if (launches) *launches += 4;
    if (split_pays(min_m, min_n, kSplitInverse)) return cudaSuccess;
  }
  return gemm_launch<Op, kSubtract>(jobs, njobs, k, max_m, max_n, s, launches, large);
}

// One CTA per (LIZ position p, job): with G in M's storage, X refined and V = M^-1,
//   Z = G[p, :] X (bp x b),  H = G[p, :] V[:, p] (bp x bp),  Lambda = V[c, p]^T taubar (bp x b),
//   tbar_site = Lambda Z^T (+ Lambda for the central site),  dlogdet_site = -H^T,
// written as b x b blocks in the t-matrix store layout (row s kkrsz + lm for the site's lm < kk,
// zero elsewhere).  bp = ns kk <= kMaxB.
//
// The two contractions run on the FP64 tensor cores: warps 0 - 3 take Z, 4 - 7 H, each every fourth K
// step of 4, with the MMA fragments loaded straight from global memory (a G fragment is eight rows of
// four columns, an X or V fragment four rows of eight columns: whole 32-byte sectors); the four partial
// results are added in shared memory in warp order.  NB = 2 or 4 blocks of eight a side (bp, b <= 8 NB).
// 16 jobs of 87 sites (N = 1392) take 402 us; the DFMA form took 1180 us.
constexpr int kVjpSmem = (int)sizeof(double2) * 3 * kMaxB * (kMaxB + 1);

template <int NB>
__global__ void __launch_bounds__(256) vjp_assemble_kernel(const JobDev *__restrict__ jobs, int kkrsz, int ns) {
  const JobDev &J = jobs[blockIdx.y];
  const int p = blockIdx.x;
  if (p >= J.L) return;
  const int off = J.off[p], bp = J.off[p + 1] - off;
  const int site = J.perm[p];
  const int kk = bp / ns;
  const int N = J.N, n = J.n, b = J.b, ld = J.ld;
  extern __shared__ __align__(16) unsigned char vsm[];
  double2(*Zs)[kMaxB + 1] = reinterpret_cast<double2(*)[kMaxB + 1]>(vsm);
  double2(*Hs)[kMaxB + 1] = Zs + kMaxB;
  double2(*Ls)[kMaxB + 1] = Hs + kMaxB;  // Lambda
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  {
    const bool z = warp < 4;  // Z = G X, else H = G V[:, p]
    const double2 *__restrict__ Gp = J.M + off + g;
    const double2 *__restrict__ Bp = z ? J.X : J.V + (size_t)off * ld;
    const int nc = z ? b : bp;
    const double2 zero = make_double2(0.0, 0.0);
    double re[NB][NB][2], im[NB][NB][2];
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
#pragma unroll 2
    for (int k0 = 4 * (warp & 3); k0 < N; k0 += 16) {
      const int k = k0 + t;
      double2 a[NB], x[NB];
#pragma unroll
      for (int i = 0; i < NB; ++i) a[i] = k < N && 8 * i + g < bp ? Gp[8 * i + (size_t)k * ld] : zero;
#pragma unroll
      for (int j = 0; j < NB; ++j) x[j] = k < N && 8 * j + g < nc ? Bp[k + (size_t)(8 * j + g) * ld] : zero;
#pragma unroll
      for (int i = 0; i < NB; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          dm::mma_884(re[i][j][0], re[i][j][1], a[i].x, x[j].x);
          dm::mma_884(im[i][j][0], im[i][j][1], a[i].x, x[j].y);
        }
#pragma unroll
      for (int i = 0; i < NB; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          dm::mma_884(re[i][j][0], re[i][j][1], -a[i].y, x[j].y);
          dm::mma_884(im[i][j][0], im[i][j][1], a[i].y, x[j].x);
        }
    }
    double2(*D)[kMaxB + 1] = z ? Zs : Hs;
    for (int w = 0; w < 4; ++w) {
      if ((warp & 3) == w)
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
          for (int j = 0; j < NB; ++j)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              double2 &d = D[8 * i + g][8 * j + 2 * t + q];
              d = w == 0 ? make_double2(re[i][j][q], im[i][j][q])
                         : make_double2(d.x + re[i][j][q], d.y + im[i][j][q]);
            }
      __syncthreads();
    }
  }
  // Lambda[i][c] = sum_r V[n + r][off + i] taubar[r][c]
  for (int e = tid; e < bp * b; e += 256) {
    const int i = e % bp, c = e / bp;
    double2 s = make_double2(0.0, 0.0);
    for (int r = 0; r < b; ++r)
      s = cfma(J.V[(size_t)(n + r) + (size_t)(off + i) * ld], J.taubar[r + (size_t)c * b], s);
    Ls[i][c] = s;
  }
  __syncthreads();
  double2 *tb = J.tbar + (size_t)site * b * b;
  double2 *dl = J.dlogdet ? J.dlogdet + (size_t)site * b * b : nullptr;
  for (int e = tid; e < b * b; e += 256) {
    const int R = e % b, C = e / b;  // store layout row and column
    const int sr = R / kkrsz, lr = R - sr * kkrsz, sc = C / kkrsz, lc = C - sc * kkrsz;
    double2 tv = make_double2(0.0, 0.0), dv = make_double2(0.0, 0.0);
    if (lr < kk && lc < kk) {
      const int i = sr * kk + lr, j = sc * kk + lc;  // local indices in the site block
      for (int c = 0; c < b; ++c) tv = cfma(Ls[i][c], Zs[j][c], tv);
      if (site == 0) tv = make_double2(tv.x + Ls[i][j].x, tv.y + Ls[i][j].y);
      dv = make_double2(-Hs[j][i].x, -Hs[j][i].y);
    }
    tb[e] = tv;
    if (dl) dl[e] = dv;
  }
}

// Full tau = M^-1 T (T = blockdiag of the sites' t-matrices), N x N without padding into M's storage,
// column-major or (`rows`) row-major, in the reference's site order (the central site, last in positions
// order, first), so that the caller gets it by one contiguous copy: one CTA per (256 rows, position p,
// job), one row per thread; a thread reads the bp elements of its row in the position's column block of
// M^-1 and writes the bp products with t_p.  With panel pivoting V holds (P M)^-1, and column j of M^-1
// is column rowpos[j] of V.  N = 880: the call took 7.7 ms with a padded tau, copied in four
// pieces and transposed on the host, and takes 3.1 ms.
__global__ void __launch_bounds__(256) tau_full_kernel(const JobDev *__restrict__ jobs, TmatView tv, bool rows) {
  const JobDev &J = jobs[blockIdx.z];
  const int p = blockIdx.y;
  if (p >= J.L || J.inactive) return;
  const int off = J.off[p], bp = J.off[p + 1] - off;
  const int site = J.perm[p];
  const int kk = bp / tv.ns;  // (lmax + 1)^2 of the site
  __shared__ double2 ts[kMaxB][kMaxB + 1];
  // the site's t block, rows / columns s kk + l for the site's own l < kk (the build's gather)
  const double2 *tb = tv.tmat + (long)J.store[site] * tv.tmat_ld + (long)J.iie * tv.blk + tv.jsm(J.ispin);
  for (int e = threadIdx.x; e < bp * bp; e += 256) {
    const int r = e % bp, c = e / bp;
    const int sr = r / kk, lr = r - sr * kk, sc = c / kk, lc = c - sc * kk;
    ts[r][c] = tb[(sr * tv.kkrsz + lr) + (long)(sc * tv.kkrsz + lc) * tv.bstore];
  }
  __syncthreads();
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r >= J.N) return;
  const int *__restrict__ rowpos = J.piv != nullptr ? J.piv + J.ld : nullptr;
  double2 v[kMaxB];
#pragma unroll
  for (int k = 0; k < kMaxB; ++k) {
    const int j = off + k;
    const int col = k < bp ? (rowpos != nullptr ? rowpos[j] : j) : 0;
    v[k] = k < bp ? J.V[(size_t)r + (size_t)col * J.ld] : make_double2(0.0, 0.0);
  }
  const auto place = [&](int x) { return x < J.n ? x + J.b : x - J.n; };  // in the reference's order
  const int pr = place(r), pc = place(off);
  double2 *out = J.M + (rows ? (size_t)pr * J.N + pc : (size_t)pr + (size_t)pc * J.N);
  const size_t step = rows ? 1 : J.N;
  for (int c = 0; c < bp; ++c) {
    double2 acc = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < kMaxB; ++k)
      if (k < bp) acc = cfma(v[k], ts[k][c], acc);
    out[c * step] = acc;
  }
}

}  // namespace

cudaError_t launch_tau_full(const JobDev *jobs, int njobs, int max_L, int max_N, const TmatView &tv, bool rows,
                            cudaStream_t s, long *launches) {
  if (njobs <= 0) return cudaSuccess;
  tau_full_kernel<<<dim3((max_N + 255) / 256, max_L, njobs), 256, 0, s>>>(jobs, tv, rows);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_inverse(const JobDev *jobs, int njobs, int min_n, int max_n, int max_N, const SplitBufs *split,
                           int *err, cudaStream_t s, long *launches) {
  if (njobs <= 0) return cudaSuccess;
  cudaError_t e;
  const int min_N = min_n + max_N - max_n;
  if (split && (e = cudaMemsetAsync(split->counters + split->steps, 0, 2 * sizeof(int) * split->steps, s)) != cudaSuccess)
    return e;
  identity_kernel<<<dim3(max_N, njobs), 256, 0, s>>>(jobs);
  if (launches) *launches += 1;
  for (int k = 0; k < max_n; k += kNb) {
    if ((e = gemm_launch<OpInvDiag, kOverwrite>(jobs, njobs, k, kNb, k + kNb, s, launches)) != cudaSuccess) return e;
    if ((e = subtract_launch<OpInvLower>(jobs, njobs, k, min_N - k - kNb, k + kNb, max_N - k - 1, k + kNb, split, 1, err,
                                         s, launches)) != cudaSuccess)
      return e;
  }
  schur_inverse_kernel<<<njobs, 256, 0, s>>>(jobs);
  if (launches) *launches += 1;
  if ((e = gemm_launch<OpSchurApply, kOverwrite>(jobs, njobs, 0, kMaxB, max_N, s, launches)) != cudaSuccess) return e;
  if ((e = gemm_launch<OpInvUpper, kSubtract>(jobs, njobs, -1, max_n, max_N, s, launches)) != cudaSuccess) return e;
  for (int k = ((max_n - 1) / kNb) * kNb; k >= 0 && max_n > 0; k -= kNb)
    if ((e = subtract_launch<OpInvUpper>(jobs, njobs, k, k < min_n ? k : 0, min_N, k, max_N, split, 2, err, s, launches)) !=
        cudaSuccess)
      return e;
  return cudaGetLastError();
}

cudaError_t launch_vjp_assemble(const JobDev *jobs, int njobs, int max_L, int kkrsz, int ns, cudaStream_t s,
                                long *launches) {
  if (njobs <= 0) return cudaSuccess;
  const int nb = ns * kkrsz <= 16 ? 2 : 4;
  const cudaError_t e = nb == 2 ? ensure_smem(vjp_assemble_kernel<2>, kVjpSmem) : ensure_smem(vjp_assemble_kernel<4>, kVjpSmem);
  if (e != cudaSuccess) return e;
  const dim3 grid(max_L, njobs);
  if (nb == 2) vjp_assemble_kernel<2><<<grid, 256, kVjpSmem, s>>>(jobs, kkrsz, ns);
  else vjp_assemble_kernel<4><<<grid, 256, kVjpSmem, s>>>(jobs, kkrsz, ns);
  if (launches) *launches += 1;
  return cudaGetLastError();
}

}  // namespace b200
