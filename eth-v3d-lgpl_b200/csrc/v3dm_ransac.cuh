// v3dm_ransac.cuh -- definitions shared by the RANSAC kernels (v3dm_ransac.cu) and the refining
// selection kernel (v3dm_ransac_refine.cu, built without fused multiply-adds).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace v3dm {

constexpr int kRsMaxSol = 10;        // solutions per sample
constexpr int kRsSlotDoubles = 18;   // E, F
constexpr int kRsRound = 128;        // samples per pair of the first round, and of a pair's share at least

// The loop's state per pair, carried from round to round.
struct RsState {
  double minError;  // best cost so far (1e30: none)
  int budget;       // nSamples, lowered by each accepted candidate
  int drawn;        // samples consumed
  int chosen;       // sample of the accepted candidate, -1: none
  int done;         // the loop has ended for this pair
};

// A round: pair p has samples drawn_p .. drawn_p + len[p] - 1 (of its state) in the sample slots
// start[p] ..; a sample slot has kRsMaxSol candidate slots.
struct RsRoundPlan {
  const int* start;  // nPairs + 1
  const int* len;    // nPairs, 0: no work
};

// The samples the loop draws of the next len: until one more than the budget has been drawn.
__device__ __forceinline__ int rs_used(const RsState& s, int len) {
  return len <= s.budget - s.drawn ? len : s.budget - s.drawn + 1;
}

// The costs of kRsRound samples from sample slot `slot` on in shared memory, in loop order: +inf where
// a candidate slot is empty, its pose flag is not set, or past `have` samples.
__device__ __forceinline__ void rs_stage_costs(double* sCost, long long slot, int have, const int8_t* __restrict__ counts,
                                               const uint8_t* __restrict__ slotOk, const double* __restrict__ cost) {
  for (int idx = threadIdx.x; idx < kRsRound * kRsMaxSol; idx += blockDim.x) {
    const int j = idx / kRsMaxSol, r = idx - j * kRsMaxSol;
    const bool in = j < have && r < counts[slot + j] && slotOk[slot * kRsMaxSol + idx];
    sCost[idx] = in ? cost[slot * kRsMaxSol + idx] : INFINITY;
  }
}

// The first candidate in [from, limit) whose cost is below minError, or limit.  Whole warps, the
// same result on every lane.
__device__ __forceinline__ int rs_next_below(const double* sCost, int from, int limit, double minError) {
  const int lane = threadIdx.x & 31;
  for (int i0 = from; i0 < limit; i0 += 32) {
    const unsigned m = __ballot_sync(0xffffffffu, i0 + lane < limit && sCost[i0 + lane] < minError);
    if (m) return i0 + __ffs(m) - 1;
  }
  return limit;
}

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
  int2* tasks;          // nPairs x kRsTasks: (pair x kRsTasks + task, candidate), long ones from the front, others from the end
  int* nTasks;          // long tasks, others, the next one to take
  RsRefined* refined;   // nPairs x kRsTasks, then one per CTA
  int32_t* lists;       // ctas x listRoom inlier indices
  long long listRoom;   // the largest correspondence count of a pair
  int ctas;             // persistent CTAs
};

// The round's selection with mode.iterativeRefinement (v3dm_ransac_refine.cu).
cudaError_t launch_rs_select_refine(const int32_t* offsets, int nPairs, int nDraw, RsRoundPlan plan, const int8_t* counts,
                                    const uint8_t* slotOk, const double* cost, const double* slots, RsState* st,
                                    double* bestEF, const float4* corrs, const double4* norm, const int32_t* samples,
                                    const double* invK, double thr, double thr2, double* bestRT, const RsRefineWork& w,
                                    cudaStream_t stream);

}  // namespace v3dm
