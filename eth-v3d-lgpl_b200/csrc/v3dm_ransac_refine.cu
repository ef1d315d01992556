// v3dm_ransac_refine.cu -- the RANSAC loop's selection with mode.iterativeRefinement
// (V3D/Apps/SfM/reconstruction_common.cpp:255-314): each accepted candidate's pose is refined by
// refineRelativePose (V3D/Geometry/v3d_poseutilities.cpp:1063-1101) on the inliers of the
// candidate's F, the refined F is scored over all correspondences, and the loop keeps
// min(cost, refined cost), the refined model and the refined inlier count for its budget.
//
// The refinement is a Levenberg-Marquardt loop whose accept/reject and stopping decisions can
// turn on the last bits of its sums, so this file reproduces the arithmetic of the reference's
// CPU code (ess::refine_pose restates it and matches it inside the loop on every tested pair):
//   - it is built without contraction into fused multiply-adds (the reference builds for plain
//     x86-64), see the Makefile;
//   - the sums over the inliers run in index order: seven warps compute the correspondences'
//     residuals and Jacobian rows, 224 at a time, into shared memory, and lane q of the eighth
//     accumulates quantity q (one of the 21 entries of J^T J, 6 of J^T e, the two |e|^2 below)
//     over the previous 224 in order -- every sum has the sequential order of the reference's loops;
//   - the rotation update's sin and cos are correctly rounded (ess::pose_update, device path).
//
// Which candidates are refined does not have to be known one at a time.  The loop accepts a
// candidate whose cost lies below every accepted one's min(cost, refined cost), so the candidates
// it can accept in a round are among the strict prefix minima of the round's raw costs (those
// below the incoming minimum, in loop order, pose flag set), about ln(candidates) of them.
//   k_rs_refine_tasks   one warp per pair lists them (kRsTasks per pair and round at most);
//   k_rs_refine         a persistent CTA per task refines and scores each, all in parallel;
//   k_rs_select_refine  walks the loop in order and picks up the results; a candidate that has
//                       none (the list was full, or an earlier one's pose failed the exact test)
//                       is refined there and then.
// What bounds k_rs_refine: the order of the sums.  An inlier costs the summing warp two
// shared-memory loads, a product and a dependent add; the other warps' divisions and square roots
// run beside it.  A step of the Levenberg-Marquardt loop takes one sweep over the inliers: the
// sweep that scores the step (weights of the old pose) also forms the normal equations the next
// step needs if it is accepted (weights of the new pose).
// On 256 pairs of 500 to 3000 correspondences these kernels take 5.5 ms of a 12.1 ms call: an inlier
// costs a sweep 22 cycles, a step 17,000 more in the solve, the update and their barriers.  One warp
// per pair that refined its candidates one after the other, two sweeps per step, took 178 ms;
// tasks dealt out in a fixed order 1.5 ms more than taken as CTAs become free.
#include <cuda_runtime.h>

#include "v3dm_essential.cuh"
#include "v3dm_internal.h"
#include "v3dm_ransac.cuh"

namespace v3dm {

namespace {

// F = (invK2^T E) invK1, the reference's product order (reconstruction_common.cpp:271).
__device__ void rs_fund(const double* invK1, const double* invK2t, const double* E, double* F) {
  double tmp[9];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double v = 0.0;
      for (int k = 0; k < 3; ++k) v += invK2t[3 * i + k] * E[3 * k + j];
      tmp[3 * i + j] = v;
    }
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double v = 0.0;
      for (int k = 0; k < 3; ++k) v += tmp[3 * i + k] * invK1[3 * k + j];
      F[3 * i + j] = v;
    }
}

constexpr int kRsRefineThreads = 256;           // warp 0 sums, warps 1..7 produce
constexpr int kRsRefineCtas = 2;                // per SM
constexpr int kRsProducers = kRsRefineThreads - 32;
constexpr int kRsQuant = 29;   // 21 entries of J^T J (upper triangle), 6 of J^T e, |e|^2 under the new and the old weights
constexpr int kRsEntry = 9;    // doubles per staged inlier: J (6), e (new weights), e (old weights), padding (odd: no bank conflicts)
constexpr int kRsRow = 8;      // values of an entry
static_assert(kRsRow < kRsEntry && kRsQuant <= 32, "entry layout");

struct RsShared {
  double sv[2][kRsProducers * kRsEntry];  // staged inliers, double-buffered
  double E[9], Fn[9], Fo[9], inner[9][6];  // the sweep's matrices: E and F at the pose, F of the old weights
  double R[9], T[3], Rs[9], Ts[3];
  double JtJ[36], Jte[6], sums[kRsQuant];
  int warpCnt[kRsRefineThreads / 32];
  int nIn, flag;
};

// One pass over the inliers list[0..nIn) at pose (s.R, s.T): the weighted residuals and, in s.sums,
// the normal equations (ess::pose_jacobian_row, weights from the pixel positions under s.Fn) and
// |e|^2, and |e|^2 with the weights under s.Fo.  The CTA enters and leaves together; s.E, s.Fn,
// s.Fo and s.inner are set.
__device__ void rs_sweep(RsShared& s, const float4* __restrict__ px, const double4* __restrict__ nm,
                         const int32_t* __restrict__ list, double thr) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the quantity lane `lane` of warp 0 owns
  int qa = 0, qb = 0;
  if (lane < 21) {
    int t = lane;
    while (t >= 6 - qa) {
      t -= 6 - qa;
      ++qa;
    }
    qb = qa + t;
  } else if (lane < 27) {
    qa = lane - 21;
    qb = 6;
  } else {
    qa = qb = lane == 28 ? 7 : 6;
  }
  const int nIn = s.nIn, chunks = (nIn + kRsProducers - 1) / kRsProducers;
  double acc = 0.0;
  for (int c = 0; c <= chunks; ++c) {
    if (warp > 0) {
      const int i = (int)threadIdx.x - 32, k = c * kRsProducers + i;
      if (c < chunks && k < nIn) {
        double* o = s.sv[c & 1] + i * kRsEntry;
        const int idx = list[k];
        const float4 p = px[idx];
        const double4 q = nm[idx];
        double a[3], b[2], J[6];
        const double en = ess::pose_residual(s.Fn, p.x, p.y, p.z, p.w, a, b);
        const double eo = ess::pose_residual(s.Fo, p.x, p.y, p.z, p.w, a, b);
        const double wn = (fabs(en) < thr) ? 1.0 : sqrt(thr / fabs(en));
        const double wo = (fabs(eo) < thr) ? 1.0 : sqrt(thr / fabs(eo));
        const double f = 0.0 - ess::pose_residual(s.E, q.x, q.y, q.z, q.w, a, b);
        ess::pose_jacobian_row(s.E, s.inner, q.x, q.y, q.z, q.w, J);
        for (int j = 0; j < 6; ++j) o[j] = J[j];
        o[6] = wn * f;
        o[7] = wo * f;
      }
    } else if (c > 0) {
      const double* v = s.sv[(c - 1) & 1];
      const int m = min(kRsProducers, nIn - (c - 1) * kRsProducers);
#pragma unroll 8
      for (int i = 0; i < m; ++i) acc += v[i * kRsEntry + qa] * v[i * kRsEntry + qb];
    }
    __syncthreads();
  }
  if (warp == 0 && lane < kRsQuant) s.sums[lane] = acc;
  __syncthreads();
}

// s.E, s.inner and s.Fn from the pose (s.R, s.T).
__device__ void rs_matrices(RsShared& s, const double* invK1, const double* invK2t) {
  if (threadIdx.x == 0) {
    double E[9], F[9];
    ess::pose_essential(s.R, s.T, E);
    rs_fund(invK1, invK2t, E, F);
    for (int k = 0; k < 9; ++k) {
      s.E[k] = E[k];
      s.Fn[k] = F[k];
    }
    ess::pose_inner(E, s.R, s.inner);
  }
  __syncthreads();
}

// refineRelativePose on the inliers of F0 (Sampson distance below thr2, in index order; their
// indices go to list, room for n): ess::refine_pose's Levenberg-Marquardt loop
// (SimpleLevenbergOptimizer's damping schedule and stopping rules) from the pose in (s.R, s.T).
__device__ void rs_refine_cta(RsShared& s, const float4* __restrict__ px, const double4* __restrict__ nm, int n,
                              const double* F0, double thr2, const double* invK1, const double* invK2t, double thr,
                              int32_t* __restrict__ list) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int base = 0;
  for (int k0 = 0; k0 < n; k0 += kRsRefineThreads) {
    const int k = k0 + (int)threadIdx.x;
    bool in = false;
    if (k < n) {
      const float4 c = px[k];
      in = ess::sampson(F0, c.x, c.y, c.z, c.w) < thr2;
    }
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (lane == 0) s.warpCnt[warp] = __popc(m);
    __syncthreads();
    int before = base, total = 0;
    for (int w = 0; w < kRsRefineThreads / 32; ++w) {
      if (w < warp) before += s.warpCnt[w];
      total += s.warpCnt[w];
    }
    if (in) list[before + __popc(m & ((1u << lane) - 1))] = k;
    base += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) s.nIn = base;
  rs_matrices(s, invK1, invK2t);
  if (threadIdx.x < 9) s.Fo[threadIdx.x] = s.Fn[threadIdx.x];
  __syncthreads();
  rs_sweep(s, px, nm, list, thr);
  // the loop's scalars live in thread 0
  double lambda = 1e-3, err = 0.0, delta[6];
  bool fresh = true;  // s.sums holds the normal equations at (s.R, s.T)
  for (int it = 0; it < 50; ++it) {
    if (threadIdx.x == 0) {
      if (fresh) {
        int t = 0;
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
          for (int j = i; j < 6; ++j, ++t) s.JtJ[6 * i + j] = s.JtJ[6 * j + i] = s.sums[t];
#pragma unroll
        for (int k = 0; k < 6; ++k) s.Jte[k] = s.sums[21 + k];
        err = s.sums[27];
      }
      bool go = true;
      double gmax = 0.0;
      for (int k = 0; k < 6; ++k) gmax = fmax(gmax, fabs(s.Jte[k]));
      if (gmax < 1e-8) go = false;
      if (go) {
        if (it == 0) {
          double maxEl = -1e30;
          for (int k = 0; k < 6; ++k) maxEl = fmax(maxEl, s.JtJ[7 * k]);
          lambda = 1e-3 * maxEl;
        }
        double N[36], g[6];
#pragma unroll
        for (int k = 0; k < 36; ++k) N[k] = s.JtJ[k];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          N[7 * k] += lambda;
          g[k] = s.Jte[k];
        }
        go = ess::cholesky_solve6(N, g, delta);
      }
      if (go) {
        double dl = 0.0;
        for (int k = 0; k < 6; ++k) dl += delta[k] * delta[k];
        dl = sqrt(dl);
        if (it >= 10 && dl < 1e-8 * (4.0 + 1e-8)) go = false;
      }
      if (go) {
        for (int k = 0; k < 9; ++k) s.Rs[k] = s.R[k];
        for (int k = 0; k < 3; ++k) s.Ts[k] = s.T[k];
        ess::pose_update(s.Rs, s.Ts, delta, s.R, s.T);
      }
      s.flag = go;
    }
    __syncthreads();
    if (!s.flag) return;  // uniform
    rs_matrices(s, invK1, invK2t);  // s.Fo stays: the weights of the pose before the step
    rs_sweep(s, px, nm, list, thr);
    if (threadIdx.x == 0) {
      const double errNew = s.sums[28];
      double rho = err - errNew;
      double d1 = 0.0, d2 = 0.0;
      for (int k = 0; k < 6; ++k) {
        d1 += delta[k] * delta[k];
        d2 += delta[k] * s.Jte[k];
      }
      rho = rho / (lambda * d1 + d2);
      fresh = rho > 0;
      if (fresh) {
        lambda = fmax(1e-10, lambda * 0.1);
        for (int k = 0; k < 9; ++k) s.Fo[k] = s.Fn[k];
      } else {
        for (int k = 0; k < 9; ++k) s.R[k] = s.Rs[k];
        for (int k = 0; k < 3; ++k) s.T[k] = s.Ts[k];
        lambda *= 10.0;
      }
    }
    // thread 0 alone reads s.sums, s.JtJ and the pose until the next barrier
  }
  __syncthreads();
}

// sum_i min(d_i, thr2) over all correspondences in index order (the loop's sum, as k_rs_score
// forms it) and the count of d_i < thr2; every thread gets both.
__device__ void rs_cost_in_order(RsShared& s, const float4* __restrict__ px, int n, const double* F, double thr2,
                                 double* cost, int* nIn) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = (n + kRsProducers - 1) / kRsProducers;
  double sum = 0.0;
  int cnt = 0;
  for (int c = 0; c <= chunks; ++c) {
    if (warp > 0) {
      const int i = (int)threadIdx.x - 32, k = c * kRsProducers + i;
      if (c < chunks && k < n) {
        const float4 p = px[k];
        bool in;
        s.sv[c & 1][i] = ess::sampson_truncated(F, (double)p.x, (double)p.y, (double)p.z, (double)p.w, thr2, in);
        cnt += in;
      }
    } else if (c > 0) {
      const double* v = s.sv[(c - 1) & 1];
      const int m = min(kRsProducers, n - (c - 1) * kRsProducers);
#pragma unroll 8
      for (int i = 0; i < m; ++i) sum = ess::dadd(sum, v[i]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if (lane == 0) s.warpCnt[warp] = cnt;
  if (threadIdx.x == 0) s.sums[0] = sum;
  __syncthreads();
  *cost = s.sums[0];
  int total = 0;
  for (int w = 0; w < kRsRefineThreads / 32; ++w) total += s.warpCnt[w];
  *nIn = total;
  __syncthreads();
}

// Candidate idx (sample j of the round, solution r) of pair p: its pose on the sample, the refinement on the
// inliers of its F, the refined model and its cost.  o.ok = 0 when the sample's correspondences
// do not agree on a pose (the loop skips the candidate).  The CTA enters and leaves together.
__device__ void rs_refine_candidate(RsShared& s, int p, int idx, const int32_t* __restrict__ offsets, int nDraw,
                                    RsRoundPlan plan, const RsState* st, const double* __restrict__ slots, const float4* __restrict__ corrs,
                                    const double4* __restrict__ norm, const int32_t* __restrict__ samples,
                                    const double* __restrict__ invK, double thr, double thr2,
                                    int32_t* __restrict__ list, RsRefined* __restrict__ o) {
  const int b = offsets[p], n = offsets[p + 1] - b;
  double invK1[9], invK2t[9];
  for (int k = 0; k < 9; ++k) invK1[k] = invK[(size_t)p * 18 + k];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) invK2t[3 * i + j] = invK[(size_t)p * 18 + 9 + 3 * j + i];
  const double* EF = slots + ((long long)plan.start[p] * kRsMaxSol + idx) * kRsSlotDoubles;
  if (threadIdx.x == 0) {
    const int32_t* smp = samples + ((long long)p * nDraw + st[p].drawn + idx / kRsMaxSol) * 5;
    double x1[5], y1[5], x2[5], y2[5], E[9], R[9], T[3];
    for (int k = 0; k < 5; ++k) {
      const double4 v = norm[b + smp[k]];
      x1[k] = v.x;
      y1[k] = v.y;
      x2[k] = v.z;
      y2[k] = v.w;
    }
    for (int k = 0; k < 9; ++k) E[k] = EF[k];
    s.flag = ess::essential_pose(E, 5, x1, y1, x2, y2, R, T);  // relativePoseFromEssential
    for (int k = 0; k < 9; ++k) s.R[k] = R[k];
    for (int k = 0; k < 3; ++k) s.T[k] = T[k];
  }
  __syncthreads();
  const int ok = s.flag;
  __syncthreads();
  if (!ok) {
    if (threadIdx.x == 0) o->ok = 0;
    return;
  }
  double F0[9];
  for (int k = 0; k < 9; ++k) F0[k] = EF[9 + k];
  rs_refine_cta(s, corrs + b, norm + b, n, F0, thr2, invK1, invK2t, thr, list);
  rs_matrices(s, invK1, invK2t);
  double F[9], cost;
  int nIn;
  for (int k = 0; k < 9; ++k) F[k] = s.Fn[k];
  rs_cost_in_order(s, corrs + b, n, F, thr2, &cost, &nIn);
  if (threadIdx.x < 9) {
    o->EF[threadIdx.x] = s.E[threadIdx.x];
    o->EF[9 + threadIdx.x] = s.Fn[threadIdx.x];
    o->RT[threadIdx.x] = s.R[threadIdx.x];
  } else if (threadIdx.x < 12) {
    o->RT[threadIdx.x] = s.T[threadIdx.x - 9];
  }
  if (threadIdx.x == 0) {
    o->cost = cost;
    o->nIn = nIn;
    o->ok = 1;
  }
  __syncthreads();
}

// One warp per pair: the strict prefix minima of the round's costs below the incoming minimum,
// in loop order, as tasks.
__global__ void __launch_bounds__(32)
k_rs_refine_tasks(RsRoundPlan plan, const int8_t* __restrict__ counts, const uint8_t* __restrict__ slotOk,
                  const double* __restrict__ cost, const RsState* __restrict__ st, int32_t* __restrict__ taskIdx,
                  int32_t* __restrict__ taskN, int2* __restrict__ tasks, int* __restrict__ nTasks) {
  const int p = blockIdx.x, lane = threadIdx.x;
  __shared__ double sCost[kRsRound * kRsMaxSol];
  const RsState s = st[p];
  const int len = plan.len[p], used = len > 0 ? rs_used(s, len) : 0;  // uniform over the warp
  double minError = s.minError;
  int n = 0;
  for (int w0 = 0; w0 < used && n < kRsTasks; w0 += kRsRound) {
    const int have = min(kRsRound, used - w0), limit = have * kRsMaxSol;
    __syncwarp();
    rs_stage_costs(sCost, (long long)plan.start[p] + w0, have, counts, slotOk, cost);
    __syncwarp();
    for (int idx = rs_next_below(sCost, 0, limit, minError); idx < limit && n < kRsTasks;
         idx = rs_next_below(sCost, idx + 1, limit, minError)) {
      minError = sCost[idx];
      if (lane == 0) taskIdx[p * kRsTasks + n] = w0 * kRsMaxSol + idx;
      ++n;
    }
  }
  __syncwarp();
  if (lane == 0) taskN[p] = n;
  if (lane < n) {
    const int2 task = make_int2(p * kRsTasks + lane, taskIdx[p * kRsTasks + lane]);
    // the last two have the lowest costs, so the most inliers to refine on: they start first
    if (lane >= n - 2) tasks[atomicAdd(&nTasks[0], 1)] = task;
    else tasks[gridDim.x * kRsTasks - 1 - atomicAdd(&nTasks[1], 1)] = task;
  }
}

// Persistent CTAs that take the next task when they are done (a refinement lasts from 4 to 50 steps
// on 10 to 1000s of inliers); listRoom ints of inlier indices per CTA.
__global__ void __launch_bounds__(kRsRefineThreads, kRsRefineCtas)
k_rs_refine(const int32_t* __restrict__ offsets, int nDraw, RsRoundPlan plan, const RsState* __restrict__ st,
            const double* __restrict__ slots, const float4* __restrict__ corrs, const double4* __restrict__ norm,
            const int32_t* __restrict__ samples, const double* __restrict__ invK, double thr, double thr2,
            const int2* __restrict__ tasks, int* __restrict__ nTasks, int cap, int32_t* __restrict__ lists,
            long long listRoom, RsRefined* __restrict__ refined) {
  __shared__ RsShared s;
  __shared__ int sNext;
  const int first = nTasks[0], n = first + nTasks[1];
  while (true) {
    __syncthreads();
    if (threadIdx.x == 0) sNext = atomicAdd(&nTasks[2], 1);
    __syncthreads();
    const int t = sNext;
    if (t >= n) break;
    const int2 task = tasks[t < first ? t : cap - 1 - (t - first)];
    rs_refine_candidate(s, task.x / kRsTasks, task.y, offsets, nDraw, plan, st, slots, corrs, norm, samples, invK, thr,
                        thr2, lists + (long long)blockIdx.x * listRoom, refined + task.x);
  }
}

// The loop over the round's candidates in order (reconstruction_common.cpp:177-335), a CTA per pair
// at a time; every warp walks the same decisions.
__global__ void __launch_bounds__(kRsRefineThreads, kRsRefineCtas)
k_rs_select_refine(const int32_t* __restrict__ offsets, int nPairs, int nDraw, RsRoundPlan plan,
                   const int8_t* __restrict__ counts, const uint8_t* __restrict__ slotOk,
                   const double* __restrict__ cost, const double* __restrict__ slots, RsState* __restrict__ st,
                   double* __restrict__ bestEF, const float4* __restrict__ corrs, const double4* __restrict__ norm,
                   const int32_t* __restrict__ samples, const double* __restrict__ invK, double thr, double thr2,
                   double* __restrict__ bestRT, const int32_t* __restrict__ taskIdx, const int32_t* __restrict__ taskN,
                   int32_t* __restrict__ lists, long long listRoom, RsRefined* __restrict__ refined) {
  __shared__ RsShared sh;
  __shared__ double sCost[kRsRound * kRsMaxSol];
  for (int p = blockIdx.x; p < nPairs; p += gridDim.x) {
    const int len = plan.len[p];
    if (len == 0) continue;  // uniform
    RsState s = st[p];
    const int n = offsets[p + 1] - offsets[p];
    const int nt = taskN[p];
    const int s0 = s.drawn;
    int t = 0, used = rs_used(s, len);
    for (int w0 = 0; w0 < used; w0 += kRsRound) {
      __syncthreads();  // sCost is free
      rs_stage_costs(sCost, (long long)plan.start[p] + w0, min(kRsRound, used - w0), counts, slotOk, cost);
      __syncthreads();
      auto limit = [&]() { return min(kRsRound, used - w0) * kRsMaxSol; };
      for (int idx = rs_next_below(sCost, 0, limit(), s.minError); idx < limit();
           idx = rs_next_below(sCost, idx + 1, limit(), s.minError)) {
        const int at = w0 * kRsMaxSol + idx;
        while (t < nt && taskIdx[p * kRsTasks + t] < at) ++t;
        const bool have = t < nt && taskIdx[p * kRsTasks + t] == at;
        RsRefined* o = refined + (have ? p * kRsTasks + t : nPairs * kRsTasks + (int)blockIdx.x);
        if (!have) {
          rs_refine_candidate(sh, p, at, offsets, nDraw, plan, st, slots, corrs, norm, samples, invK, thr, thr2,
                              lists + (long long)blockIdx.x * listRoom, o);
          __syncthreads();
        }
        if (!o->ok) continue;
        s.minError = fmin(sCost[idx], o->cost);
        const int j = at / kRsMaxSol;
        s.chosen = s0 + j;
        const float frac = (float)(o->nIn - 5) / (float)(n - 5);
        s.budget = min(s.budget, rs_budget(1.0 - (double)frac));
        used = max(j + 1, rs_used(s, len));
        if (threadIdx.x < kRsSlotDoubles) bestEF[(size_t)p * kRsSlotDoubles + threadIdx.x] = o->EF[threadIdx.x];
        if (threadIdx.x < 12) bestRT[(size_t)p * 12 + threadIdx.x] = o->RT[threadIdx.x];
        __syncthreads();
      }
    }
    __syncthreads();  // every thread is done with the state
    if (threadIdx.x == 0) {
      s.drawn += used;
      if (s.drawn > s.budget || s.drawn >= nDraw) s.done = 1;  // the next sample would end the loop
      st[p] = s;
    }
  }
}

}  // namespace

cudaError_t launch_rs_select_refine(const int32_t* offsets, int nPairs, int nDraw, RsRoundPlan plan, const int8_t* counts,
                                    const uint8_t* slotOk, const double* cost, const double* slots, RsState* st,
                                    double* bestEF, const float4* corrs, const double4* norm, const int32_t* samples,
                                    const double* invK, double thr, double thr2, double* bestRT, const RsRefineWork& w,
                                    cudaStream_t stream) {
  if (nPairs <= 0) return cudaSuccess;
  cudaError_t e = cudaMemsetAsync(w.nTasks, 0, 3 * sizeof(int), stream);
  if (e != cudaSuccess) return e;
  k_rs_refine_tasks<<<nPairs, 32, 0, stream>>>(plan, counts, slotOk, cost, st, w.taskIdx, w.taskN, w.tasks, w.nTasks);
  k_rs_refine<<<w.ctas, kRsRefineThreads, 0, stream>>>(offsets, nDraw, plan, st, slots, corrs, norm, samples, invK, thr,
                                                       thr2, w.tasks, w.nTasks, nPairs * kRsTasks, w.lists, w.listRoom,
                                                       w.refined);
  k_rs_select_refine<<<nPairs < w.ctas ? nPairs : w.ctas, kRsRefineThreads, 0, stream>>>(
      offsets, nPairs, nDraw, plan, counts, slotOk, cost, slots, st, bestEF, corrs, norm, samples, invK, thr, thr2,
      bestRT, w.taskIdx, w.taskN, w.lists, w.listRoom, w.refined);
  return cudaGetLastError();
}

}  // namespace v3dm
