// Block sweeps of the correction solve in FP64 arithmetic, on the FP64 tensor cores.
//
// Same contract as the sweeps of sweep.cu (forward: Y_k = D_k R_k, R[k+kb:N] -= A21_k Y_k; backward:
// X_k (+)= Y_k, Y[0:k] -= W[0:k, k] Y_k, i.e. zgetrs on the block LU factors, zblock_lu_cpp.cpp:60-86),
// for 16 columns of the right-hand side and factors stored in FP64 or FP32.
//
// What bounds a sweep of one job is the chain of blocks: block k + 1 is final only after block k's
// product with one 64 x 64 block, 2.1 us of an SM's FP64 rate (64 FMAs a cycle), and in the forward
// sweep D_(k+1)'s product after it.  So rows are dealt out in tiles of 16: the four tiles of a block
// belong to four CTAs of the job's cluster, which share the chain's products (0.5 us each), and a
// finished block goes to every CTA of the cluster through distributed shared memory.  One cluster
// barrier per block (two in the forward sweep, whose D product needs all 64 rows) orders the steps;
// the updates of the rows further away run between a CTA's arrival and its wait, so they overlap the
// chain.  A tile of R or Y is only ever touched by the same thread, in place, and its operand panels
// (16 rows x 64 columns) stream through a three-stage cp.async ring.
// At N = 2160, against DFMA products of 64-row tiles with one owner each: forward 768 -> 351 us and
// backward 635 -> 231 us for one job, 1270 -> 627 and 910 -> 528 us for 31.  (Requesting a tile's R or Y
// one tile ahead changed nothing: 357 and 270 us.)

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

#include "cluster.cuh"
#include "common.cuh"
#include "cplx.cuh"
#include "dmma.cuh"

namespace b200 {
namespace {

using namespace cx;
using namespace cl;

constexpr int kRows = 16;       // rows per tile
constexpr int kCols = 16;       // right-hand-side columns per launch slice
constexpr int kThreads = 128;   // four warps, one 8 x 8 block of a tile's product each
constexpr int kRing = 3;        // operand units in flight
constexpr int kStride = kRows + 2;  // elements between columns (rows of a slot) in shared memory: 32
                                    // bytes modulo 128, so a fragment load has no bank conflicts
constexpr int kUnit = 64 * kStride;
constexpr int kMaxCluster = 16;

// Shared memory: the operand ring, then three 64 x 16 slots (forward: two of Y, one of R).
template <typename T>
constexpr int smem_bytes() {
  return kRing * kUnit * (int)sizeof(T) + 3 * kUnit * (int)sizeof(double2);
}

__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();  // (the barrier is the warp's)
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_remote_c(unsigned addr, double2 v) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}

// First tile at or after lo that belongs to rank q of cs (a power of two).
__device__ __forceinline__ int first_own(int lo, int q, int cs) { return lo + ((q - lo) & (cs - 1)); }
__device__ __forceinline__ int block_rows(int n, int k) { return min(64, n - 64 * k); }

// The units of one CTA in the order it consumes them: per step the tiles on the chain (phase 0), in
// the forward sweep their D products (phase 1), then the other tiles (phase 2).
struct FwdUnits {
  int n, N, cs, q, nsteps;
  int k, ph, r, end;
  bool fin;
  __device__ int tiles() const { return (N + kRows - 1) / kRows; }
  // end of the chain tiles of step k: the tiles with rows of block k + 1
  __device__ int chain_end() const { return (64 * (k + 1) + block_rows(n, k + 1) + kRows - 1) / kRows; }
  __device__ void range() {  // [first own tile, end) of the current phase
    const bool next = k + 1 < nsteps;
    int lo;
    if (ph < 2) {
      lo = 4 * (k + 1);
      end = next && (k >= 0 || ph == 1) ? chain_end() : lo;
    } else {
      lo = next ? chain_end() : (64 * k + block_rows(n, k)) / kRows;
      end = k >= 0 ? tiles() : lo;
    }
    r = first_own(lo, q, cs);
  }
  __device__ void seek() {
    while (r >= end) {
      if (++ph == 3) {
        ph = 0;
        if (++k >= nsteps) {
          fin = true;
          return;
        }
      }
      range();
    }
  }
  __device__ void begin() {
    k = -1;
    ph = 0;
    fin = false;
    range();
    seek();
  }
  __device__ void next() {
    r += cs;
    seek();
  }
  __device__ bool at(int kk, int p) const { return !fin && k == kk && ph == p; }
  __device__ int row0() const { return kRows * r; }
  __device__ int col0() const { return ph == 1 ? 64 * (k + 1) : 64 * k; }
  __device__ int ncol() const { return block_rows(n, ph == 1 ? k + 1 : k); }
};

// Step s: 0 the central block (column n, b wide), s >= 1 block last - (s - 1).
struct BwdUnits {
  int n, b, cs, q, nblk;
  int s, ph, r, end;
  bool fin;
  __device__ int blk() const { return nblk - s; }  // block of step s >= 1; the one of step s + 1 is blk() - 1
  __device__ void range() {
    const int nb = nblk - s - 1;  // the next block
    int lo = 0;
    if (ph == 0) {
      lo = 4 * nb;
      end = nb >= 0 ? (64 * nb + block_rows(n, nb) + kRows - 1) / kRows : lo;
    } else {
      end = nb >= 0 ? 4 * nb : 0;
    }
    r = first_own(lo, q, cs);
  }
  __device__ void seek() {
    while (r >= end) {
      if (++ph == 2) {
        ph = 0;
        if (++s > nblk) {
          fin = true;
          return;
        }
      }
      range();
    }
  }
  __device__ void begin() {
    s = 0;
    ph = 0;
    fin = false;
    range();
    seek();
  }
  __device__ void next() {
    r += cs;
    seek();
  }
  __device__ bool at(int ss, int p) const { return !fin && s == ss && ph == p; }
  __device__ int row0() const { return kRows * r; }
  __device__ int col0() const { return s == 0 ? n : 64 * blk(); }
  __device__ int ncol() const { return s == 0 ? b : block_rows(n, blk()); }
};

// Requests a unit: rows row0 .. + 15 of columns col0 .. + ncol - 1 of F, zeros up to the next multiple
// of four columns.
template <typename T, class Units>
__device__ __forceinline__ void request(T *dst, const T *F, int ld, const Units &u) {
  constexpr int kPer = 16 / (int)sizeof(T);     // elements per 16-byte copy
  constexpr int kCopies = kRows / kPer;         // copies per column
  const int nc = u.ncol();
  const T *src = F + (size_t)u.row0() + (size_t)u.col0() * ld;
#pragma unroll
  for (int i = 0; i < 64 * kCopies / kThreads; ++i) {
    const int e = threadIdx.x + i * kThreads;
    const int c = e / kCopies, part = (e % kCopies) * kPer;
    if (c < ((nc + 3) & ~3))
      dm::cp_async16_zfill(dst + c * kStride + part, c < nc ? src + part + (size_t)c * ld : src, c < nc);
  }
}

// This thread's part of a unit's product with a slot, entries (row, col) and (row, col + 1) of the
// warp's 8 x 8 block: row = 8 (warp % 2) + lane / 4, col = 8 (warp / 2) + 2 (lane % 4).
template <typename T>
__device__ __forceinline__ void product(double2 (&v)[2], const T *As, const double2 *Ys, int ncol) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const T *a0 = As + t * kStride + 8 * (warp & 1) + g;
  const double2 *y0 = Ys + t * kStride + 8 * (warp >> 1) + g;
  double rr[2] = {0.0, 0.0}, ii[2] = {0.0, 0.0}, ri[2] = {0.0, 0.0}, ir[2] = {0.0, 0.0};
#pragma unroll 4
  for (int ks = 0; ks < ncol; ks += 4) {
    const double2 a = to_v<double2>(a0[ks * kStride]), y = y0[ks * kStride];
    dm::mma_884(rr[0], rr[1], a.x, y.x);
    dm::mma_884(ii[0], ii[1], a.y, y.y);
    dm::mma_884(ri[0], ri[1], a.x, y.y);
    dm::mma_884(ir[0], ir[1], a.y, y.x);
  }
  v[0] = make_double2(rr[0] - ii[0], ri[0] + ir[0]);
  v[1] = make_double2(rr[1] - ii[1], ri[1] + ir[1]);
}

// Operand stream of a CTA: three units requested ahead, one consumed at a time.
template <typename T, class Units>
struct Stream {
  T *ring;
  const T *F;
  int ld;
  Units pf;
  int issued = 0, used = 0;
  __device__ void fetch() {
    if (!pf.fin) {
      request(ring + (issued % kRing) * kUnit, F, ld, pf);
      pf.next();
      ++issued;
    }
    cp_async_commit();
  }
  __device__ void begin() {
    for (int i = 0; i < kRing - 1; ++i) fetch();
  }
  // The next unit, landed for every thread (a block barrier, which also separates the last reads of
  // the stage that is requested anew).
  __device__ const T *take() {
    cp_async_wait<kRing - 2>();
    __syncthreads();
    fetch();
    return ring + (used++ % kRing) * kUnit;
  }
};

// Stores entries (row, col), (row, col + 1) of a 64 x 16 slot in the CTAs [0, cs) whose bit is set in
// `mask`.
__device__ __forceinline__ void publish(const double2 *slot, int row, int col, const double2 (&v)[2], int cs,
                                        unsigned mask) {
  const double2 *p = slot + row * kStride + col;
  for (int c = 0; c < cs; ++c)
    if ((mask >> c) & 1u) {
      const unsigned a = remote_u32(p, c);
      st_remote_c(a, v[0]);
      st_remote_c(a + 16, v[1]);
    }
}

// Grid (cs, njobs, slices of 16 columns), cluster (cs, 1, 1).  Refinement rounds only: the initial
// solve has B = 0 above the central block, so its forward sweep is the identity.
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) forward_sweep64_kernel(const JobDev *__restrict__ jobs) {
  const JobDev &J = jobs[blockIdx.y];
  const int col0 = kCols * blockIdx.z;
  // uniform over the cluster: the flag changes only between launches
  if (converged(J.conv) || J.n == 0 || J.inactive || col0 >= J.b) return;
  const int q = cluster_rank(), cs = cluster_size();
  const int n = J.n, N = J.N, ld = J.ld, b = min(kCols, J.b - col0);
  extern __shared__ __align__(128) unsigned char sm[];
  double2 *Ysl = reinterpret_cast<double2 *>(sm + kRing * kUnit * sizeof(T));  // two slots of Y
  double2 *Rsl = Ysl + 2 * kUnit;
  double2 *const Rg = J.R + (size_t)col0 * ld, *const Yg = J.Y + (size_t)col0 * ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row = 8 * (warp & 1) + (lane >> 2), col = 8 * (warp >> 1) + 2 * (lane & 3);
  const int nsteps = (n + 63) / 64;
  const unsigned all = cs >= 32 ? 0xffffffffu : (1u << cs) - 1u;

  FwdUnits it{n, N, cs, q, nsteps};
  it.begin();
  Stream<T, FwdUnits> st{reinterpret_cast<T *>(sm), static_cast<const T *>(J.F), ld, it};
  st.begin();
  if (it.at(-1, 1)) {  // R_0 for the D_0 products
    const int kb = block_rows(n, 0);
    for (int e = tid; e < 64 * kCols; e += kThreads) {
      const int rr = e & 63, c = e >> 6;
      Rsl[rr * kStride + c] = (rr < kb && c < b) ? Rg[(size_t)rr + (size_t)c * ld] : make_double2(0.0, 0.0);
    }
  }
  cluster_sync();  // every CTA is running before the first remote store

  // One tile of R minus its product: prefetched R entries, then either back to R (rows past the
  // block) or to the R slot of the CTAs that hold the next block's tiles.
  auto tile = [&](int k, bool chain, unsigned owners) {
    const int gr = it.row0() + row;
    double2 rv[2], v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
      rv[h] = (gr < N && col + h < b) ? Rg[(size_t)gr + (size_t)(col + h) * ld] : make_double2(0.0, 0.0);
    const int nc = it.ncol();
    const T *As = st.take();
    product(v, As, Ysl + (k & 1) * kUnit, nc);
    const int lo = 64 * k + block_rows(n, k);  // first row below the block
    v[0] = csub(rv[0], v[0]);
    v[1] = csub(rv[1], v[1]);
    const int kn = 64 * (k + 1), in = chain ? kn + block_rows(n, k + 1) : lo;  // rows [lo, in) go to the slot
    if (gr >= in && gr < N) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (col + h < b) Rg[(size_t)gr + (size_t)(col + h) * ld] = v[h];
    }
    if (chain) {
      if (gr >= in) v[0] = v[1] = make_double2(0.0, 0.0);
      publish(Rsl, gr - kn, col, v, cs, owners);
    }
    it.next();
  };

  for (int k = -1; k < nsteps; ++k) {
    // ranks that hold tiles of block k + 1
    unsigned owners = 0;
    if (k + 1 < nsteps)
      for (int i = 0; i < 4; ++i) owners |= 1u << ((4 * (k + 1) + i) & (cs - 1));
    while (it.at(k, 0)) tile(k, true, owners);
    if (k >= 0 && k + 1 < nsteps) {
      cluster_arrive();
      if (!it.at(k, 1) && it.at(k, 2)) tile(k, false, 0);
      cluster_wait();  // R_(k+1) is complete in its CTAs; Y_(k-1) is no longer read anywhere
    }
    while (it.at(k, 1)) {  // Y_(k+1) = D_(k+1) R_(k+1), to every CTA and to Y
      double2 v[2];
      const int rr = it.row0() - 64 * (k + 1) + row, nc = it.ncol(), gr = it.row0() + row;
      const T *As = st.take();
      product(v, As, Rsl, nc);
      if (rr >= nc) v[0] = v[1] = make_double2(0.0, 0.0);
      publish(Ysl + ((k + 1) & 1) * kUnit, rr, col, v, cs, all);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (rr < nc && col + h < b) Yg[(size_t)gr + (size_t)(col + h) * ld] = v[h];
      it.next();
    }
    cluster_arrive();
    while (it.at(k, 2)) tile(k, false, 0);
    cluster_wait();  // Y_(k+1) is in every CTA
  }
  cp_async_wait<0>();
}

// Grid and cluster as above.  mode 0 sets X = Y, mode 1 adds X += Y (and skips converged jobs).
template <typename T>
__global__ void __launch_bounds__(kThreads, 2) backward_sweep64_kernel(const JobDev *__restrict__ jobs, int mode) {
  const JobDev &J = jobs[blockIdx.y];
  const int col0 = kCols * blockIdx.z;
  if ((mode == 1 && converged(J.conv)) || J.inactive || col0 >= J.b) return;
  const int q = cluster_rank(), cs = cluster_size();
  const int n = J.n, ld = J.ld, bc = J.b, b = min(kCols, J.b - col0);
  extern __shared__ __align__(128) unsigned char sm[];
  double2 *Ysl = reinterpret_cast<double2 *>(sm + kRing * kUnit * sizeof(T));  // three slots
  double2 *const Yg = J.Y + (size_t)col0 * ld, *const Xg = J.X + (size_t)col0 * ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row = 8 * (warp & 1) + (lane >> 2), col = 8 * (warp >> 1) + 2 * (lane & 3);
  const int nblk = (n + 63) / 64;
  const unsigned all = cs >= 32 ? 0xffffffffu : (1u << cs) - 1u;

  BwdUnits it{n, bc, cs, q, nblk};
  it.begin();
  Stream<T, BwdUnits> st{reinterpret_cast<T *>(sm), static_cast<const T *>(J.F), ld, it};
  st.begin();
  // step 0, the central block from the Schur solve: every CTA fills its own slot 0
  for (int e = tid; e < 64 * kCols; e += kThreads) {
    const int rr = e & 63, c = e >> 6;
    const bool in = rr < bc && c < b;
    const double2 y = in ? Yg[(size_t)(n + rr) + (size_t)c * ld] : make_double2(0.0, 0.0);
    Ysl[rr * kStride + c] = y;
    if (q == 0 && in) {  // X_c (+)= Y_c
      double2 *x = Xg + (size_t)(n + rr) + (size_t)c * ld;
      *x = mode == 0 ? y : make_double2(x->x + y.x, x->y + y.y);
    }
  }
  cluster_sync();  // every CTA is running before the first remote store

  for (int s = 0; s <= nblk; ++s) {
    // Y[tile] minus its product with block s; `chain`: the rows are those of the next block, final now
    auto tile = [&](bool chain) {
      const int gr = it.row0() + row, nb = nblk - s - 1;
      const bool in = gr < n;
      double2 yv[2], v[2], xv[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const size_t idx = (size_t)gr + (size_t)(col + h) * ld;
        // (the initial solve, mode 0, has Y = 0 above the central block, whose step is every tile's first)
        yv[h] = (in && col + h < b && (mode == 1 || s > 0)) ? Yg[idx] : make_double2(0.0, 0.0);
        xv[h] = (chain && mode == 1 && in && col + h < b) ? Xg[idx] : make_double2(0.0, 0.0);
      }
      const int nc = it.ncol();
      const T *As = st.take();
      product(v, As, Ysl + (s % 3) * kUnit, nc);
      v[0] = in ? csub(yv[0], v[0]) : make_double2(0.0, 0.0);
      v[1] = in ? csub(yv[1], v[1]) : make_double2(0.0, 0.0);
      if (chain) publish(Ysl + ((s + 1) % 3) * kUnit, gr - 64 * nb, col, v, cs, all);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!in || col + h >= b) continue;
        const size_t idx = (size_t)gr + (size_t)(col + h) * ld;
        if (chain) Xg[idx] = make_double2(xv[h].x + v[h].x, xv[h].y + v[h].y);
        else Yg[idx] = v[h];
      }
      it.next();
    };
    while (it.at(s, 0)) tile(true);
    cluster_arrive();
    while (it.at(s, 1)) tile(false);
    cluster_wait();  // block s + 1 is in every CTA
  }
  cp_async_wait<0>();
}

// Clusters of `kern` (cs CTAs, smem bytes each) resident at once, cached per (kernel, cs, device); 0
// when the query fails.
int resident(const void *kern, int cs, int smem) {
  struct Entry {
    const void *kern;
    int cs, dev, v;
  };
  static std::mutex mu;
  static std::vector<Entry> cache;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  for (const Entry &c : cache)
    if (c.kern == kern && c.cs == cs && c.dev == dev) return c.v;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int v = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&v, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    v = 0;
  }
  cache.push_back({kern, cs, dev, v});
  return v;
}

// The largest cluster whose clusters for `want` (job, column slice) pairs are resident at once: a
// larger cluster shortens every step of a job as long as all jobs run at the same time.
template <typename K>
int cluster_for(K *kern, int smem, int want) {
  for (int cs = kMaxCluster; cs > 1; cs >>= 1)
    if (resident(reinterpret_cast<const void *>(kern), cs, smem) >= want) return cs;
  return 1;
}

template <typename T>
cudaError_t sweep64_impl(const JobDev *jobs, int njobs, int b, bool forward, int mode, int want, cudaStream_t s) {
  constexpr int smem = smem_bytes<T>();
  const int slices = (b + kCols - 1) / kCols;
  cudaError_t e = forward ? ensure_smem(forward_sweep64_kernel<T>, smem) : ensure_smem(backward_sweep64_kernel<T>, smem);
  if (e != cudaSuccess) return e;
  const int cs = forward ? cluster_for(forward_sweep64_kernel<T>, smem, want * slices)
                         : cluster_for(backward_sweep64_kernel<T>, smem, want * slices);
  if (forward)
    return launch_cluster_grid(forward_sweep64_kernel<T>, cs, dim3(cs, njobs, slices), kThreads, smem, s, jobs);
  return launch_cluster_grid(backward_sweep64_kernel<T>, cs, dim3(cs, njobs, slices), kThreads, smem, s, jobs, mode);
}

}  // namespace

cudaError_t launch_sweep64(FactorKind fk, const JobDev *jobs, int njobs, int b, bool forward, int mode, int want,
                           cudaStream_t s) {
  return fk == kFactorFP64 ? sweep64_impl<double2>(jobs, njobs, b, forward, mode, want, s)
                           : sweep64_impl<float2>(jobs, njobs, b, forward, mode, want, s);
}

}  // namespace b200
