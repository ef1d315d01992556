// v3dm_ransac.cuh -- definitions shared by the RANSAC kernels (v3dm_ransac.cu) and the refining
// selection kernel (v3dm_ransac_refine.cu, built without fused multiply-adds).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace v3dm {

constexpr int kRsMaxSol = 10;        // solutions per sample
constexpr int kRsSlotDoubles = 18;   // E, F
constexpr int kRsRound = 128;        // samples per pair per round

// The loop's state per pair, carried from round to round.
struct RsState {
  double minError;  // best cost so far (1e30: none)
  int budget;       // nSamples, lowered by each accepted candidate
  int drawn;        // samples consumed
  int chosen;       // sample of the accepted candidate, -1: none
  int done;         // the loop has ended for this pair
};

// ransacNSamples(5, outlierRatio, 1 - 1e-9) (reconstruction_common.h:627-635).
__device__ __forceinline__ int rs_budget(double outlierRatio) {
  const double maxN = 1e8;
  if (outlierRatio >= 1.0) return (int)maxN;
  double N = log(1.0 - (1.0 - 10e-10)) / log(1.0 - pow(1.0 - outlierRatio, 5));
  N = fmax(0.0, fmin(maxN, N));
  return (int)N;
}

// The refined candidates of a round (v3dm_ransac_refine.cu).  Sixteen per pair: the prefix minima of
// 1280 costs in random order are 7.7 on average, and a full list only moves a refinement to the
// selecting kernel.
constexpr int kRsTasks = 16;
struct RsRefined {
  double EF[18], RT[12];  // refined E, F and R, T
  double cost;            // cost of the refined F
  int nIn, ok;            // its inlier count; 0: the sample does not agree on a pose
};
struct RsRefineWork {
  int32_t* taskIdx;     // nPairs x kRsTasks: candidate of each task, ascending
  int32_t* taskN;       // nPairs
  int2* tasks;          // nPairs x kRsTasks: (pair x kRsTasks + task, candidate), any order
  int* nTasks;
  RsRefined* refined;   // nPairs x kRsTasks, then one per CTA
  int32_t* lists;       // ctas x listRoom inlier indices
  long long listRoom;   // the largest correspondence count of a pair
  int ctas;             // persistent CTAs
};

// The round's selection with mode.iterativeRefinement (v3dm_ransac_refine.cu).
cudaError_t launch_rs_select_refine(const int32_t* offsets, int nPairs, int nDraw, int s0, int len, const int8_t* counts,
                                    const uint8_t* slotOk, const double* cost, const double* slots, RsState* st,
                                    double* bestEF, const float4* corrs, const double4* norm, const int32_t* samples,
                                    const double* invK, double thr, double thr2, double* bestRT, const RsRefineWork& w,
                                    cudaStream_t stream);

}  // namespace v3dm
