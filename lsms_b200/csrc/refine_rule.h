// When a job's refinement stops: plain C++, shared by the device check (block_lu.cu) and its host test.
#pragma once

#ifdef __CUDACC__
#define B200_HD __host__ __device__ __forceinline__
#else
#define B200_HD inline
#endif

namespace b200 {

// A refining job stops once its estimated remaining error on tau00 is below this fraction of
// max|tau00|: 100x below the mixed path's 1e-10 accuracy target.
constexpr double kRefineTol = 1e-12;
// Accelerated rounds: the estimate's limit as a fraction of kRefineTol, and the growth of a correction
// past which a job is given up (accelerated corrections do not shrink monotonically).
constexpr double kAccTol = 0.2;
constexpr double kAccGrow = 4.0;

// JobDev::conv values (0: still refining)
constexpr int kConverged = 1;
constexpr int kDiverged = 2;  // the corrections stopped shrinking (numerical)
constexpr int kAborted = 3;   // a bounded wait of a dataflow sweep ran out on this job

// State of a job after a round whose correction had the relative size c: 0, kConverged or kDiverged.
// prev and prev2 are the sizes of the two corrections before it (0: none).
//
// c is the error that the round found, so c times the contraction of the rounds estimates what is left.
// Plain rounds contract linearly: c / prev serves.  An accelerated round can take out one poor direction
// at once (c = 3.8e-9 after 1.1e-4) while the next ones contract as before, so the larger of the
// last two ratios is taken: of 1024 jobs of N = 4320 the worst result accepted by the last
// ratio alone was off by 4.7e-11, with both by 3e-12, at 2% more rounds in sum (16 jobs of N = 4320
// 67.0 -> 67.8 ms, 256 of N = 688 to 2160 42.0 -> 42.2 ms, runs of one side differing by 2.5%).
// A job that stops shrinking, or has had its last round, is at its rounding floor if the correction itself is
// below kRefineTol; any other is left to the FP64 re-solve.
B200_HD int refine_state(double c, double prev, double prev2, bool accelerated, bool last) {
  if (!(c <= 1e300)) return kDiverged;  // not finite
  const bool stalled = prev > 0.0 && c >= prev;
  double ratio = prev > 0.0 ? c / prev : 1.0;
  if (accelerated && prev2 > 0.0 && prev / prev2 > ratio) ratio = prev / prev2;
  const double est = ratio < 1.0 ? c * ratio : c;
  if (est <= (accelerated ? kAccTol * kRefineTol : kRefineTol)) return kConverged;
  if (accelerated && (stalled || last) && c <= kRefineTol) return kConverged;
  if (stalled && c >= (accelerated ? kAccGrow : 1.0) * prev) return kDiverged;
  return 0;
}

}  // namespace b200
