// v3dm_match_f.cu -- float descriptors: scores from a BF16 hi/lo split on the tensor cores.
//
// The reference scores float descriptors with cublasSgemm (v3d_cudamatching.cu:529-530).  For
// descriptors that are not of the exact u/512 form (the integer path's domain), each value x is
// split into hi = bf16(x) and lo = bf16(x - hi), and
//   score(a, b) = hi_a . hi_b + lo_a . hi_b + hi_a . lo_b       (the lo . lo term is dropped)
// is one K = 384 GEMM with FP32 accumulation: A rows read as [hi | lo | hi], B rows as [hi | hi | lo]
// (tcgen05.mma.kind::f16, BF16 x BF16 -> F32 in TMEM).  A row is stored once, as four 128-byte planes
// (hi, hi, lo, lo of 64 values each), and the MMAs name the planes they need.  For u/512 inputs hi is
// exact and lo = 0, so the scores equal the integer path's exactly.
//
// Selection is exact for the float scores.  Tf, the float candidate threshold, is the smallest score
// a second value must reach to change any decision (scores below it never matter, see
// host_float_threshold).  A CTA scores a row, an A group of up to 256 descriptors against every
// 128-column tile of its B side (or a segment of them, below): each epilogue lane keeps its
// descriptor's best and second in registers and writes the decision itself; gates are tested only
// where a score could enter those two.  No chunk records and no re-score pass exist.
//   - A batch walks its row table.  A pair's rows are implicit, and since they are few (28 for 7000
//     lefts, three or four for a pass B) each is cut into segments of tiles for as many CTAs as there
//     are; the epilogue warp that finishes a row's last segment merges the segments' best and second.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "v3dm_device.cuh"
#include "v3dm_tcgen05.cuh"

namespace v3dm {

namespace {

constexpr int kFM = 128;            // rows per MMA (TMEM lanes)
constexpr int kFGroups = 2;         // MMA row blocks of an A group: a B tile serves 256 rows
constexpr int kFGM = kFM * kFGroups;
constexpr int kFN = 128;            // B rows per tile (one MMA is 128 x 128 x 16: narrower MMAs ran 30% slower)
constexpr int kFChunks = kFN / 32;  // 32-column TMEM loads per tile and lane quadrant
constexpr int kFPlanes = 4;         // 128-byte planes per row
constexpr int kFStageBytes = kFPlanes * kFM * 128;  // 64 KB: a B tile or one block of an A group
constexpr int kFStages = 3;
constexpr int kFSteps = 24;         // K = 16 per MMA
// TMEM: an accumulator of kFN columns per block, then the blocks' A planes.  An A block lands in a
// stage of the ring and is copied once (tcgen05.cp) into TMEM, so that shared memory serves the B
// tiles and all stages hold B tiles between groups.
constexpr int kFACols = kFPlanes * 32;  // 4 bytes per column
constexpr int kFABase = kFGroups * kFN;
constexpr int kFTmemCols = 512;
static_assert(kFABase + kFGroups * kFACols <= kFTmemCols, "accumulators and the A group fit in TMEM");
constexpr int kFEpiWarp0 = 2;
constexpr int kFThreads = (kFEpiWarp0 + 4 * kFGroups) * 32;

constexpr int kFWait = 16;  // guided: scores a lane keeps until their gates are tested together

struct SmemF {
  uint8_t b[kFStages][kFStageBytes];
  uint2 waiting[4 * kFGroups][kFWait][32];  // score and column, per epilogue warp, place and lane
  unsigned long long full[kFStages], empty[kFStages];
  unsigned long long accFull[kFGroups], accEmpty[kFGroups];
  unsigned long long mmaDone;
  uint32_t tmemBase;
  int abort;
};
static_assert(sizeof(SmemF) + 1024 <= 227 * 1024, "shared memory of one CTA");

// kind::f16, D = F32, A = B = BF16, both K-major, M = 128, N = kFN.
__device__ __forceinline__ constexpr uint32_t idesc_f16() {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kFN >> 3) << 17) | ((uint32_t)(kFM >> 4) << 24);
}

// A from TMEM (lane = row, K values packed two per column), B from shared memory.
__device__ __forceinline__ void mma_bf16_ts(uint32_t dtmem, uint32_t atmem, uint64_t bd, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(dtmem),
      "r"(atmem), "l"(bd), "r"(idesc_f16()), "r"(accumulate)
      : "memory");
}

// A 128-row x 32-byte slice, described as the MMA would read it from shared memory, into TMEM
// (row i to lane i, 8 columns); executes in issue order with the MMAs of the same thread.
__device__ __forceinline__ void tmem_cp_slice(uint32_t taddr, uint64_t sd) {
  asm volatile("tcgen05.cp.cta_group::1.128x256b [%0], %1;" ::"r"(taddr), "l"(sd) : "memory");
}

// The runs of one CTA, in the order every role walks them: an A group against tiles t0 .. t0 + nT - 1
// of its B side.  A row table (a.rows): rows blockIdx.x, + gridDim.x, ..., all tiles.  A pair (rows
// null): row r is A rows 256 r .. against all a.nB B rows, cut into nSeg segments; items (row,
// segment) are dealt out in that order.
struct FWalk {
  const BatchRow* rows;
  int w, nItems, pairA, nTiles, nSeg;
  // the current run
  int aRow, validRows, bRow0, nB, t0, nT, row, seg;
  long long state0;
  __device__ void load() {
    if (w >= nItems) return;
    if (rows) {
      const BatchRow b = rows[w];
      aRow = b.aRow;
      validRows = b.validRows;
      bRow0 = b.bRow0;
      nB = b.nB;
      t0 = 0;
      nT = b.nTiles;
      state0 = b.state0;
    } else {
      row = w / nSeg;
      seg = w - row * nSeg;
      aRow = row * kFGM;
      validRows = min(kFGM, pairA - aRow);
      t0 = (int)((long long)nTiles * seg / nSeg);
      nT = (int)((long long)nTiles * (seg + 1) / nSeg) - t0;
      state0 = aRow;
    }
  }
  __device__ explicit FWalk(const SideArgs& a) {
    rows = a.rows;
    w = blockIdx.x;
    nSeg = 1;
    row = seg = 0;
    if (rows) {
      nItems = a.nRowsPtr ? *a.nRowsPtr : a.nRows;
    } else {
      pairA = a.nAptr ? *a.nAptr : a.nA;
      nB = a.nB;
      bRow0 = 0;
      nTiles = (nB + kFN - 1) / kFN;
      const int nRows = nTiles > 0 ? (pairA + kFGM - 1) / kFGM : 0;
      if (nRows > 0) nSeg = max(1, min((int)gridDim.x / nRows, min(nTiles, kFMaxSegments)));
      nItems = nRows * nSeg;
    }
    load();
  }
  __device__ bool more() const { return w < nItems; }
  __device__ void next() {
    w += gridDim.x;
    load();
  }
  __device__ int groups() const { return validRows > kFM ? 2 : 1; }
};

// Largest of eight scores, NaN when one of them is (three-input max of sm_100).
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max8_nan(const uint32_t* v) {
  const float a = max3_nan(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2]));
  const float b = max3_nan(__uint_as_float(v[3]), __uint_as_float(v[4]), __uint_as_float(v[5]));
  return max3_nan(max3_nan(a, b, __uint_as_float(v[6])), __uint_as_float(v[7]), a);
}

// Running top two of one A row over the columns of a run, as ordered keys (f32_order): b1 the
// largest, c1 its first column, b2 the largest of the other columns; both start below every score
// that reaches Tf.
__device__ __forceinline__ void top2_push(uint32_t key, int col, uint32_t& b1, uint32_t& b2, int& c1) {
  b2 = max(b2, min(key, b1));
  c1 = key > b1 ? col : c1;
  b1 = max(b1, key);
}

// The gate of one lane's row in a guided batch (one gate per pair, the reference's expressions):
// its pair's matrix and thr^2, the positions of the B image's descriptors, the A descriptor's
// terms.
struct GateLane {
  const float* m;
  const float2* bPos;
  float4 aT;
  int type, aIsLeft;
};

// Whether the gate masks (A descriptor of the lane, column col of the B image).
__device__ __forceinline__ bool gate_rejects_col(GateLane gl, int col) {
  const float2 pb = gl.bPos[col];
  if (gl.aIsLeft) return gate_rejects_terms(gl.type, gl.m[9], gl.aT, gate_right_terms(gl.type, gl.m, pb));
  return gate_rejects_terms(gl.type, gl.m[9], gate_left_terms(gl.type, gl.m, pb), gl.aT);
}

// Whether any of the single-pair matcher's gates (compounding since the last putative call) masks
// (left l, right r).
__device__ __forceinline__ bool gates_reject(const GateParams* gates, int n, int l, int r) {
  for (int g = 0; g < n; ++g)
    if (gate_rejects(gates[g], l, r)) return true;
  return false;
}

// Side A against side B: the runs of FWalk, every A row's decision to a.decision[state].
//   warp 0      TMA producer: an A group's blocks and its B tiles through one ring of 64 KB stages;
//   warp 1      MMA issuer (the warp walks, one elected lane issues): the A blocks into TMEM, then per
//               tile 24 MMAs for each block;
//   warps 2-9   epilogue, four per block: one A row per lane.
// Bounded waits as in k_side; the rows of a CTA that gives up keep whatever a.decision held, which the
// kernels that read it allow for.  With 'dump' set (a small diagnostic call without gates) every score is
// also written to dump[state * nB + column].
// What bounds it: the tensor pipe, 24 x 64 = 1536 cycles per block and tile, of which it takes 1760.
// Before, with 128-row groups and the hi planes stored twice (96 KB of L2 reads per block and tile
// against 32), a lane-0 issuer (145 cycles per MMA) and a branch per score in the epilogue, it took
// 3480.  A call over 40 images of 1000 - 8000 descriptors went from 13.9 to 8.9 ms, a guided pair of
// 7013 x 6450 from the host from 1.14 to 0.90 ms (its rows, 55 before, now fill every SM; 0.78 with the
// guided epilogue's waiting scores).
template <bool kGated>
__global__ void __launch_bounds__(kFThreads, 1)
k_side_f(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, SideArgs a, float Tf,
         float* dump) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ uint8_t smemRaw[];
  SmemF& s = *reinterpret_cast<SmemF*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const FWalk start(a);
  if (!start.more()) return;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kFStages; ++i) {
      mbar_init(&s.full[i], 1);
      mbar_init(&s.empty[i], 1);
    }
    for (int i = 0; i < kFGroups; ++i) {
      mbar_init(&s.accFull[i], 1);
      mbar_init(&s.accEmpty[i], 4);
    }
    mbar_init(&s.mmaDone, 1);
    s.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmemBase)),
                 "r"(kFTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmemBase;

  // Ring uses are numbered from 0 in every role (u): stage u % kFStages; tiles of block g (i[g]) too.
  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      uint32_t u = 0;
      uint32_t skipped = 0xffffffffu;  // test hook: the use that was not loaded
      int bLoads = 0;
      bool ok = true;
      auto load = [&](const CUtensorMap* m, int r) {
        const uint32_t st = u % kFStages;
        if (!mbar_wait(&s.empty[st], ((u / kFStages) & 1u) ^ 1u, &s.abort, a.err)) return false;
        if (m == &tmB && ++bLoads == a.skipLoad && blockIdx.x == 0) {
          skipped = u;
        } else {
          mbar_expect_tx(&s.full[st], (uint32_t)kFStageBytes);
          tma_load_3d(s.b[st], m, &s.full[st], 0, r, 0);
        }
        ++u;
        return true;
      };
      for (FWalk wk = start; wk.more() && ok; wk.next()) {
        for (int g = 0; g < wk.groups() && ok; ++g) ok = load(&tmA, wk.aRow + g * kFM);
        for (int t = wk.t0; t < wk.t0 + wk.nT && ok; ++t) ok = load(&tmB, wk.bRow0 + t * kFN);
      }
      // Drain: every load this thread issued has landed before the CTA may exit.
      for (uint32_t k = u > (uint32_t)kFStages ? u - kFStages : 0u; k < u; ++k) {
        const long long t0c = clock64();
        while (k != skipped && !mbar_try(&s.full[k % kFStages], (k / kFStages) & 1u) && clock64() - t0c < kWaitCycles) {
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    const bool leader = elect_one();
    const uint32_t base = sdesc_lo(smem_u32(s.b[0]));
    uint32_t u = 0, i[kFGroups] = {};
    bool ok = true;
    const long long lim = a.waitLimit > 0 ? a.waitLimit : kWaitCycles;  // the other roles follow its abort
    auto wait = [&](unsigned long long* b, uint32_t par) { return mbar_wait_warp(b, par, &s.abort, a.err, lim); };
    for (FWalk wk = start; wk.more() && ok; wk.next()) {
      const int groups = wk.groups();
      // the group into TMEM (after the previous group's MMAs, which were issued first); a stage is
      // free once its copies are done
      for (int g = 0; g < groups && ok; ++g, ++u) {
        const uint32_t st = u % kFStages;
        ok = wait(&s.full[st], (u / kFStages) & 1u);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sd = base + st * (uint32_t)(kFStageBytes >> 4);
        const uint32_t at = tmem + (uint32_t)(kFABase + g * kFACols);
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < 4 * kFPlanes; ++kk)
            tmem_cp_slice(at + (uint32_t)(8 * kk),
                          sdesc_of(sd + (uint32_t)((kk >> 2) * (kFM * 128 >> 4) + 2 * (kk & 3))));
          mma_commit(&s.empty[st]);
        }
      }
      for (int t = 0; t < wk.nT && ok; ++t, ++u) {
        const uint32_t st = u % kFStages;
        ok = wait(&s.full[st], (u / kFStages) & 1u);
        if (!ok) break;
        const uint32_t sd = base + st * (uint32_t)(kFStageBytes >> 4);
#pragma unroll
        for (int g = 0; g < kFGroups; ++g) {
          if (g >= groups) break;
          ok = ok && wait(&s.accEmpty[g], (i[g] & 1u) ^ 1u);
          if (!ok) break;
          ++i[g];
          tc_fence_after();
          const uint32_t d = tmem + (uint32_t)(g * kFN), at = tmem + (uint32_t)(kFABase + g * kFACols);
          if (leader) {
#pragma unroll
            for (int k = 0; k < kFSteps; ++k) {  // A [hi | lo | hi], B [hi | hi | lo]: planes of 64 values
              const int p = k >> 2, ap = p < 4 ? p : p - 4, bp = p < 2 ? p : p - 2;
              mma_bf16_ts(d, at + (uint32_t)(32 * ap + 8 * (k & 3)),
                          sdesc_of(sd + (uint32_t)(bp * (kFN * 128 >> 4) + 2 * (k & 3))), k > 0 ? 1u : 0u);
            }
            mma_commit(&s.accFull[g]);
          }
        }
        if (leader) mma_commit(&s.empty[st]);
      }
    }
    // Every MMA this thread issued has completed before TMEM is released.
    if (leader) {
      mma_commit(&s.mmaDone);
      const long long t0c = clock64();
      while (!mbar_try(&s.mmaDone, 0) && clock64() - t0c < kWaitCycles) {
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue ----------------
    const int q = warp & 3, g = (warp - kFEpiWarp0) >> 2;
    uint2* const waiting = &s.waiting[warp - kFEpiWarp0][0][lane];
    uint32_t i = 0;
    bool ok = true;
    // Scores below Tf change no decision, so the top two start just below it (-0 ranks below +0 but
    // equals it), and a group of eight scores whose maximum is below every lane's second is passed
    // over: on SIFT-like data a lane enters 0.6% of the groups.  All groups' maxima come first and one
    // vote tells which to enter, so that no branch waits for another's outcome.  In a guided call a
    // score that could enter waits in shared memory until some lane has several: testing each gate when
    // its score came up cost 300 cycles for every score of a group in turn (7013 x 6450 with F: the
    // two guided passes 224 us, 111 now).
    const uint32_t floorKey = f32_order(Tf == 0.0f ? -0.0f : Tf) - 1u;
    GateLane gl{};
    for (FWalk wk = start; wk.more() && ok; wk.next()) {
      if (g >= wk.groups()) continue;
      const int row = g * kFM + q * 32 + lane;
      const long long st = row < wk.validRows ? (a.amap ? (long long)a.amap[wk.aRow + row] : wk.state0 + row) : -1;
      uint32_t b1 = st >= 0 ? floorKey : ~0u, b2 = b1;  // nothing enters a lane without a row
      float enter = st >= 0 ? f32_unorder(floorKey) : INFINITY;  // the second, as a float
      int c1 = 0;
      if (kGated && a.bg.on && st >= 0) {
        int pair = 0, aIdx = 0;
        bgate_resolve(a.bg, a.aIsLeft, st, &pair, &aIdx);
        const int2 lr = a.bg.pairLR[pair];
        const int aImg = a.aIsLeft ? lr.x : lr.y, bImg = a.aIsLeft ? lr.y : lr.x;
        gl.m = a.bg.gm + (size_t)pair * kBGateFloats;
        gl.type = a.bg.type;
        gl.aIsLeft = a.aIsLeft;
        const float2 pa = a.bg.pos[a.bg.posOff[aImg] + aIdx];
        gl.aT = a.aIsLeft ? gate_left_terms(gl.type, gl.m, pa) : gate_right_terms(gl.type, gl.m, pa);
        gl.bPos = a.bg.pos + a.bg.posOff[bImg];
      }
      const int nB = wk.nB;
      // Guided: the gates of every lane's waiting scores, in column order.  A masked score counts as none
      // (the reference's -1e20 is below Tf).
      int nWait = 0;
      auto test_waiting = [&]() {
        for (int k = 0; __any_sync(0xffffffffu, k < nWait); ++k) {
          if (k >= nWait) continue;
          const uint2 w = waiting[32 * k];
          const uint32_t key = f32_order(__uint_as_float(w.x));
          const int col = (int)w.y;
          if (key <= b2) continue;
          const bool masked = a.bg.on ? gate_rejects_col(gl, col)
                                      : gates_reject(a.gatesDev, a.nGates, a.aIsLeft ? (int)st : col,
                                                     a.aIsLeft ? col : (int)st);
          if (!masked) top2_push(key, col, b1, b2, c1);
        }
        nWait = 0;
        if (st >= 0) enter = f32_unorder(b2);
      };
      for (int t = 0; t < wk.nT; ++t, ++i) {
        ok = mbar_wait_warp(&s.accFull[g], i & 1u, &s.abort, a.err);
        if (!ok) break;
        tc_fence_after();
        const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(g * kFN);
        uint32_t v[kFChunks][32];
#pragma unroll
        for (int c = 0; c < kFChunks; ++c) tmem_ld32(tbase + (uint32_t)(32 * c), v[c]);
#pragma unroll
        for (int c = 0; c < kFChunks; ++c) tmem_wait(v[c]);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.accEmpty[g]);
        const int col0 = (wk.t0 + t) * kFN;
        if (!kGated && dump && st >= 0)
#pragma unroll
          for (int c = 0; c < kFChunks; ++c)
#pragma unroll
            for (int k = 0; k < 32; ++k)
              if (col0 + 32 * c + k < nB) dump[(size_t)st * nB + col0 + 32 * c + k] = __uint_as_float(v[c][k]);
        uint32_t mask = 0;  // groups of eight to look at (NaN goes on to the exact keys)
#pragma unroll
        for (int c = 0; c < kFChunks; ++c)
#pragma unroll
          for (int k = 0; k < 4; ++k) mask |= !(max8_nan(&v[c][8 * k]) < enter) ? 1u << (4 * c + k) : 0u;
        mask = __reduce_or_sync(0xffffffffu, mask);
#pragma unroll
        for (int c = 0; c < kFChunks; ++c)
#pragma unroll
          for (int k8 = 0; k8 < 4; ++k8) {
            if (!(mask & (1u << (4 * c + k8)))) continue;  // warp-uniform
            if (kGated && __any_sync(0xffffffffu, nWait > kFWait - 8)) test_waiting();
#pragma unroll
            for (int k = 8 * k8; k < 8 * k8 + 8; ++k) {
              const int col = col0 + 32 * c + k;
              if (kGated) {
                if (32 * c + k < nB - col0 && !(__uint_as_float(v[c][k]) < enter))
                  waiting[32 * nWait++] = make_uint2(v[c][k], (uint32_t)col);
              } else {
                const uint32_t key = 32 * c + k < nB - col0 ? f32_order(__uint_as_float(v[c][k])) : 0u;
                top2_push(key, col, b1, b2, c1);
              }
            }
          }
        if (st >= 0) enter = f32_unorder(b2);
      }
      if (!ok) break;
      if (kGated) test_waiting();
      bool decide = true;
      if (wk.nSeg > 1) {
        // a row in segments: this warp's 32 top twos to the row's place, and whichever warp comes last
        // merges them, in segment order (so that the first column wins ties)
        constexpr int kSeg = kFGroups * 4 * 96;  // words of a segment
        const int unit = (wk.row * kFGroups + g) * 4 + q;
        uint32_t* part = a.fPartial + ((size_t)wk.row * wk.nSeg) * kSeg + (g * 4 + q) * 96 + lane;
        part[wk.seg * kSeg] = b1;
        part[wk.seg * kSeg + 32] = b2;
        part[wk.seg * kSeg + 64] = (uint32_t)c1;
        __threadfence();
        __syncwarp();
        int seen = 0;
        if (lane == 0) seen = atomicAdd(&a.fCount[unit], 1);
        seen = __shfl_sync(0xffffffffu, seen, 0);
        decide = seen == wk.nSeg - 1;
        if (decide) {
          __threadfence();
          b1 = b2 = floorKey;
          c1 = 0;
          for (int k = 0; k < wk.nSeg; ++k) {
            const uint32_t p1 = __ldcg(part + k * kSeg), p2 = __ldcg(part + k * kSeg + 32);
            const int pc = (int)__ldcg(part + k * kSeg + 64);
            b2 = max(max(b2, p2), min(p1, b1));
            c1 = p1 > b1 ? pc : c1;
            b1 = max(b1, p1);
          }
          if (lane == 0) a.fCount[unit] = 0;  // for the next pass
        }
      }
      if (decide && st >= 0 && a.decision) {
        const float s1 = f32_unorder(b1), s2 = f32_unorder(b2);
        const unsigned long long bk = (b1 != floorKey && s1 >= Tf) ? best_key_f(s1, c1) : 0ull;
        const uint32_t so = (b2 != floorKey && s2 >= Tf) ? b2 : 0u;
        a.decision[st] = decide_f(bk, so, a.minScore, a.minRatio);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kFTmemCols)
                              : "memory");
}

// The layout of n descriptors: float values (or uint8 values u, read as u / 512) split into BF16 hi
// and lo, four planes of rowsCap rows x 128 bytes (hi of values 0..63, hi of 64..127, lo, lo).  A warp
// per descriptor.  Sets *err when a value is not finite.  With srcOff set, the n descriptors are the
// concatenation of nImages images (image i starts at descriptor srcOff[i], ascending) and image i's
// descriptors go to rows rowOff[i] onwards; otherwise descriptor d goes to row d.
__global__ void __launch_bounds__(256)
k_hilo(const float4* __restrict__ f, const uchar4* __restrict__ u, long long n, int rowsCap,
       uint2* __restrict__ planes, int* err, const long long* __restrict__ srcOff, const int* __restrict__ rowOff,
       int nImages) {
  const int lane = threadIdx.x & 31;
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long step = ((long long)gridDim.x * blockDim.x) >> 5;
  bool finite = true;
  for (long long src = w; src < n; src += step) {
    long long d = src;
    if (srcOff) {
      int lo = 0, hi = nImages - 1;  // last image whose first descriptor is <= src
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (srcOff[mid] <= src) lo = mid;
        else hi = mid - 1;
      }
      d = rowOff[lo] + (src - srcOff[lo]);
    }
    float x[4];
    if (f) {
      const float4 v = f[src * 32 + lane];
      x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
    } else {
      const uchar4 v = u[src * 32 + lane];
      x[0] = (float)v.x, x[1] = (float)v.y, x[2] = (float)v.z, x[3] = (float)v.w;
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] *= 1.0f / 512.0f;
    }
    __nv_bfloat16 h[4], l[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      finite = finite && isfinite(x[k]);
      h[k] = __float2bfloat16_rn(x[k]);
      l[k] = __float2bfloat16_rn(x[k] - __bfloat162float(h[k]));
    }
    auto pack = [](const __nv_bfloat16* b) {
      return make_uint2((uint32_t)__bfloat16_as_ushort(b[0]) | ((uint32_t)__bfloat16_as_ushort(b[1]) << 16),
                        (uint32_t)__bfloat16_as_ushort(b[2]) | ((uint32_t)__bfloat16_as_ushort(b[3]) << 16));
    };
    uint2* o = planes + ((size_t)(lane >> 4) * rowsCap + d) * 16 + (lane & 15);
    o[0] = pack(h);
    o[(size_t)2 * rowsCap * 16] = pack(l);
  }
  if (!finite) atomicOr(err, kErrNotU8);
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode_f() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &qr) == cudaSuccess &&
        qr == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

}  // namespace

// 3-D BF16 map over a planar layout (64 values of a K slice, row, plane), box (64, 128, 4), 128-byte
// swizzle: one load fills four swizzled [128][128 B] blocks.  A and B operands load alike.
cudaError_t f_map(CUtensorMap* map, const void* base, int rows) {
  if (rows < kFM) return cudaErrorInvalidValue;
  auto fn = get_encode_f();
  if (!fn) return cudaErrorNotSupported;
  cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)kFPlanes};
  cuuint64_t strides[2] = {128, (cuuint64_t)rows * 128};
  cuuint32_t box[3] = {64, (cuuint32_t)kFM, (cuuint32_t)kFPlanes};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t launch_side_f(const CUtensorMap& mA, const CUtensorMap& mB, const SideArgs& a, float Tf, float* dump,
                          int numSMs, cudaStream_t st) {
  const size_t smem = sizeof(SmemF) + 1024;
  static bool attrSet[128] = {};  // per device ordinal
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 128) return cudaErrorInvalidDevice;
  if (!attrSet[dev]) {
    e = cudaFuncSetAttribute(k_side_f<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_side_f<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attrSet[dev] = true;
  }
  int grid = numSMs;
  if (!a.rows) {  // one pair: its rows are implicit, in segments when they are few
    if (a.nA <= 0 || a.nB <= 0) return cudaSuccess;
    if (!a.fPartial || !a.fCount) return cudaErrorInvalidValue;
    grid = (int)std::min<long long>(grid, (long long)((a.nA + kFGM - 1) / kFGM) * ((a.nB + kFN - 1) / kFN));
  } else if (!a.nRowsPtr) {
    if (a.nRows <= 0) return cudaSuccess;
    grid = std::min(grid, a.nRows);
  }
  if (!a.decision && !dump) return cudaErrorInvalidValue;
  const bool gated = a.bg.on != 0 || a.nGates > 0;
  return launch_pdl(gated ? k_side_f<true> : k_side_f<false>, dim3(grid), dim3(kFThreads), smem, st, mA, mB, a, Tf,
                    dump);
}

int f_group_rows() { return kFGM; }
int f_tile_cols() { return kFN; }

// Places of the merges of rows in segments: at most numSMs segments, a counter per epilogue warp of a
// row.
size_t f_partial_words(int numSMs) { return (size_t)numSMs * kFGroups * 4 * 96; }
size_t f_count_words(int numSMs) { return (size_t)numSMs * kFGroups * 4; }

static cudaError_t launch_hilo_any(const float* f, const uint8_t* u, long long n, int rowsCap, void* planes, int* err,
                                   const long long* srcOff, const int* rowOff, int nImages, cudaStream_t s) {
  const long long blocks = (n + 7) / 8;  // eight warps
  k_hilo<<<(unsigned)std::min<long long>(blocks, 148 * 64), 256, 0, s>>>(
      reinterpret_cast<const float4*>(f), reinterpret_cast<const uchar4*>(u), n, rowsCap, static_cast<uint2*>(planes),
      err, srcOff, rowOff, nImages);
  return cudaGetLastError();
}

cudaError_t launch_hilo(const float* f, const uint8_t* u, int n, int rowsCap, void* planes, int* err, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (n > rowsCap) return cudaErrorInvalidValue;
  return launch_hilo_any(f, u, n, rowsCap, planes, err, nullptr, nullptr, 0, s);
}

cudaError_t launch_hilo_images(const float* f, long long n, const long long* srcOff, const int* rowOff, int nImages,
                               int rowsCap, void* planes, int* err, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (nImages <= 0 || !srcOff || !rowOff) return cudaErrorInvalidValue;
  return launch_hilo_any(f, nullptr, n, rowsCap, planes, err, srcOff, rowOff, nImages, s);
}

// Smallest float score a second value must reach to change any decision.  accept(s1, s2) is
// monotone: for a fixed s1 it can only turn false as s2 grows, for a fixed s2 only true as s1
// grows, so the boundary at s1 = the smallest float above minScore bounds every s1.  Without a
// ratio test (or when no second value can matter) only candidates above minScore are needed.
float host_float_threshold(float minScore, float minRatio) {
  const float s1min = std::nextafter(minScore, INFINITY);
  if (!(minRatio == minRatio) || minRatio < 0.0f || !(minScore == minScore)) return s1min;
  if (!accept_scores(s1min, kNone, minScore, minRatio)) return s1min;
  if (accept_scores(s1min, INFINITY, minScore, minRatio)) return s1min;
  // accept(s1min, unorder(lo)) is true, accept(s1min, unorder(hi)) false
  uint32_t lo = f32_order(kNone), hi = f32_order(INFINITY);
  while (hi - lo > 1) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (accept_scores(s1min, f32_unorder(mid), minScore, minRatio)) lo = mid;
    else hi = mid;
  }
  const float t = f32_unorder(hi);  // the smallest second value that can flip a decision
  return t < s1min ? t : s1min;
}

}  // namespace v3dm
