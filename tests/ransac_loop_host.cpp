// The RANSAC loop of one pair on the host (V3D/Apps/SfM/reconstruction_common.cpp:173-335), with
// the library's solver, pose recovery and refinement (eth-v3d-lgpl_b200/csrc/v3dm_essential.cuh),
// one candidate after the other: what the GPU's rounds and parallel refinements must equal.
#include <algorithm>
#include <cmath>
#include <vector>

#include "v3dm_essential.cuh"

using namespace v3dm::ess;

static int budget_of(double outlierRatio) {
  const double maxN = 1e8;
  if (outlierRatio >= 1.0) return (int)maxN;
  const double N = std::log(1.0 - (1.0 - 10e-10)) / std::log(1.0 - std::pow(1.0 - outlierRatio, 5));
  return (int)std::fmax(0.0, std::fmin(maxN, N));
}

// corrs: n x 4 floats; norm: n x 4 doubles; invK: K1^-1 then K2^-1; out: E 9, F 9, R 9, T 3, error;
// returns the chosen sample (-1: none), *nIn the inliers of the model (flags[n]).
extern "C" int host_ransac(int n, const float* corrs, const double* norm, const double* invK, double thr, int nSamples,
                           int nDraw, const int* samples, int refine, double* out, int* nIn, unsigned char* flags) {
  const double thr2 = thr * thr;
  double iK2t[9];
  for (int a = 0; a < 3; ++a)
    for (int c = 0; c < 3; ++c) iK2t[3 * a + c] = invK[9 + 3 * c + a];
  auto cost_of = [&](const double* F, int* count) {
    double sum = 0.0;
    *count = 0;
    for (int i = 0; i < n; ++i) {
      bool in;
      sum += sampson_truncated(F, corrs[4 * i], corrs[4 * i + 1], corrs[4 * i + 2], corrs[4 * i + 3], thr2, in);
      *count += in;
    }
    return sum;
  };
  auto fund = [&](const double* E, double* F) {
    double tmp[9];
    mat3_mul(iK2t, E, tmp);
    mat3_mul(tmp, invK, F);
  };
  double minError = 1e30;
  int budget = nSamples, drawn = 0, chosen = -1;
  for (int j = 0; j < nDraw; ++j) {
    if (drawn > budget) break;
    ++drawn;
    double x1[5], y1[5], x2[5], y2[5], Es[10][9];
    for (int k = 0; k < 5; ++k) {
      const double* v = norm + 4 * samples[5 * j + k];
      x1[k] = v[0];
      y1[k] = v[1];
      x2[k] = v[2];
      y2[k] = v[3];
    }
    const int ns = five_point(x1, y1, x2, y2, Es);
    for (int r = 0; r < ns; ++r) {
      double F[9], R[9], T[3], E[9];
      int inl;
      fund(Es[r], F);
      double cost = cost_of(F, &inl);
      if (!(cost < minError)) continue;
      if (!essential_pose(Es[r], 5, x1, y1, x2, y2, R, T)) continue;
      std::copy(Es[r], Es[r] + 9, E);
      if (refine) {
        std::vector<PoseCorr> c;
        for (int i = 0; i < n; ++i)
          if (sampson(F, corrs[4 * i], corrs[4 * i + 1], corrs[4 * i + 2], corrs[4 * i + 3]) < thr2)
            c.push_back({norm[4 * i], norm[4 * i + 1], norm[4 * i + 2], norm[4 * i + 3], corrs[4 * i],
                         corrs[4 * i + 1], corrs[4 * i + 2], corrs[4 * i + 3]});
        std::vector<double> w(c.size() + 1), e(c.size() + 1);
        refine_pose(c.data(), (int)c.size(), invK, iK2t, thr, R, T, w.data(), e.data());
        pose_essential(R, T, E);
        fund(E, F);
        cost = std::fmin(cost, cost_of(F, &inl));
      }
      minError = cost;
      chosen = j;
      budget = std::min(budget, budget_of(1.0 - (double)((float)(inl - 5) / (float)(n - 5))));
      std::copy(E, E + 9, out);
      std::copy(F, F + 9, out + 9);
      std::copy(R, R + 9, out + 18);
      std::copy(T, T + 3, out + 27);
    }
  }
  out[30] = chosen < 0 ? -1.0 : minError / n;
  *nIn = 0;
  for (int i = 0; i < n; ++i) {
    flags[i] = chosen >= 0 &&
               sampson(out + 9, corrs[4 * i], corrs[4 * i + 1], corrs[4 * i + 2], corrs[4 * i + 3]) < thr2;
    *nIn += flags[i];
  }
  return chosen;
}
