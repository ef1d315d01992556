// v3dm_voctree_f.cu -- tensor-core descent of float vocabulary trees (sm_100a).
//
// The leaf ids are those of the reference's CPU tree, VocabularyTree::findBestNodeIndex
// (V3D/Base/v3d_voctree.h:82-99): sequential FP32 dot products, the first child strictly above the
// running maximum.  k_voctree_f32 (v3dm_voctree.cu) scores every child of every key's path with FP32
// FMAs and is bound by reading 512-byte node rows per key and child through L1.  Here the keys are
// grouped by the node they have reached, as in the byte descent (v3dm_voctree_tc.cu), and a node's
// children are scored for 128 keys at a time on the tensor cores; what those scores cannot decide is
// replayed exactly.
//   - Every value is split into hi = bf16(x), lo = bf16(x - hi), and score = hi.hi' + lo.hi' + hi.lo'
//     (24 MMAs of 128 x N x 16, FP32 accumulators in TMEM).  Against the exact dot product the split
//     loses at most 3 * 2^-18 * sum|x_i y_i| (the lo.lo' term and the rounding of both lo) and 24
//     accumulations of 17 terms, every addition truncated to FP32, at most 408 * 2^-23 of it; the
//     sequential FP32 sum is within 128 * 2^-24.  So the two differ by at most 6.8e-5 * |x| |y| <
//     kTcRel * |x| |y|.  That the tensor core loses no more than those truncations when it aligns the terms
//     of an accumulation is an assumption, documented nowhere.  What it leaves: on unit descriptors the scores are
//     within 8.1e-6 * sum|x_i y_i| of the FP64 ones, and on inputs made to lose as much as they can (terms below the
//     last bit of a large sum, magnitudes over 24 binades) within 1.7e-5, of 6.0e-5 allowed
//     (test_gpu_split_scores.py asserts the 6.0e-5).
//   - A key's best child is decided when its score leads by more than twice that bound (with the
//     largest norm among the node's children); else the key goes to a list and k_vtf_resolve evaluates
//     the reference's sequential sums over all the children, one child per lane: 1 to 4% of the
//     key-levels on k-means trees of unit descriptors.
//   - Keys of a norm below kVtTinyNorm are listed at every level: their bound would be relative to a norm that
//     FP32 squares do not give.
//   - Keys whose norm times the largest node norm is not below 1e30 (NaN, infinities, overflow) are
//     listed and descend with k_voctree_f32 at the end, whatever the phases made of them.
// A phase descends one level (BF <= 128), or two where BF^2 grandchildren and BF children fit 128
// MMA columns (BF <= 10); between phases k_vt_scan / k_vt_scatter sort the keys by node.  The keys
// are split once (k_vtf_split): splitting them in the phases, in the producers' registers, made the
// phases issue-bound at 2.3 TB/s.
//
// Roles (one persistent CTA per SM, 9 warps): warps 0-3 gather the tile's split key rows (512 bytes
// each, through the permutation) with cp.async, 16 bytes a lane, into the MMA's swizzled planes, and
// their norms; warp 0 also loads an item's node rows with TMA (pre-split planes); warp 4 issues;
// warps 5-8 read the scores, one key per lane.  Every wait is bounded as in k_side; after one that
// runs out, the phases behind it do nothing (as in the byte descent).
//
// What bounds it: reading the keys once per phase (and writing them once).  300,007 keys on a BF 50,
// depth 3 tree (125,000 leaves): 184 us a call, 2166 with k_voctree_f32; the split 45 us (6.8 TB/s),
// the phases 37, 42 and 64 us (4.1 TB/s where the tiles are full; 120 keys per bucket in the last),
// the lists 17, 11 and 10 us, the two sorts 31 us.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include "v3dm_device.cuh"
#include "v3dm_tcgen05.cuh"

namespace v3dm {

namespace {

constexpr int kVfProducers = 4;
constexpr int kVfMmaWarp = kVfProducers;
constexpr int kVfEpiWarp0 = kVfProducers + 1;
constexpr int kVfThreads = (kVfEpiWarp0 + 4) * 32;
constexpr int kVfRows = 128;              // keys per tile
static_assert(kVfProducers * 32 == kVfRows, "a producer warp has 32 rows of a tile, one key index per lane");
constexpr int kVfPlanes = 4;              // 128-byte K planes per row: hi 0..63, hi 64..127, lo, lo
constexpr int kVfABytes = kVfPlanes * kVfRows * 128;
constexpr int kVfBBytes = 65536;          // node planes of up to two items
constexpr int kVfASlots = 2;
constexpr int kVfAcc = 4;                 // accumulator stages of 128 columns
constexpr int kVfNorms = 8;               // key norms of the last tiles (see the producer)
constexpr int kVfMaxBufs = 4;
constexpr int kVfLocalBins = 2048;        // next-phase histogram kept in shared memory up to this
constexpr float kTcRel = 7.0e-5f;

struct VtfSmem {
  uint8_t a[kVfASlots][kVfABytes];
  uint8_t b[kVfBBytes];
  float norm[kVfNorms][kVfRows];
  int hist[kVfLocalBins];
  unsigned long long fullA[kVfASlots], done[kVfAcc], accEmpty[kVfAcc], fullB[kVfMaxBufs], emptyB[kVfMaxBufs];
  unsigned long long mmaDone;
  uint32_t tmemBase;
  int abort;
};
static_assert(sizeof(VtfSmem) + 1024 <= 227 * 1024, "shared memory of one CTA");

// kind::f16, D = F32, A = B = BF16, both K-major, M = 128.
__device__ __forceinline__ void vtf_mma(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void vtf_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

// 16 (4) bytes to shared memory, asynchronously.
__device__ __forceinline__ void vtf_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void vtf_cp4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// Raises the mbarrier's pending count by one now and arrives once every cp.async this thread has
// issued so far has completed (so the phase cannot complete before the copies have landed).
__device__ __forceinline__ void vtf_cp_arrive(unsigned long long* bar) {
  asm volatile("cp.async.mbarrier.arrive.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Two values' hi parts and lo parts, packed (the first value in the low half).
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const __nv_bfloat162 l = __floats2bfloat162_rn(x - __low2float(h), y - __high2float(h));
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Running first-largest with the runner-up's score.
struct Top2 {
  float s1 = -INFINITY, s2 = -INFINITY;
  int c = 0;
  __device__ __forceinline__ void push(float s, int k) {
    s2 = fmaxf(s2, fminf(s, s1));
    c = s > s1 ? k : c;
    s1 = fmaxf(s1, s);
  }
  // whether the leader is certainly the sequential rule's choice, e bounding a score's error
  __device__ __forceinline__ bool decided(float e) const { return s1 - s2 > 2.0f * e && s1 - e > -1e30f; }
};

// A node's children are the rows from (node + 1) * BF (the root is node -1).  kBF2 > 0: two levels
// with BF = kBF2; 0: one level with a.bf children.
template <int kBF2>
__global__ void __launch_bounds__(kVfThreads, 1)
k_vtf(VtfArgs a, const __grid_constant__ CUtensorMap tmNodes) {
  extern __shared__ uint8_t vtfRaw[];
  VtfSmem& s = *reinterpret_cast<VtfSmem*>((reinterpret_cast<uintptr_t>(vtfRaw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long lim = a.waitLimit > 0 ? a.waitLimit : kWaitCycles;
  const int failed = a.singleN > 0 || threadIdx.x != 0 ? 0 : *a.err != 0;
  int nIt = a.singleN > 0 ? (a.singleN + a.itemKeys - 1) / a.itemKeys : *a.nItems;
  const bool localHist = !a.final && a.bins <= kVfLocalBins;
  // B rows: one level, the children (N = BF rounded up to 16); two, N2 = BF^2 rounded up to 16 rows
  // of grandchildren and then 16 of children
  constexpr int kN2 = kBF2 ? (kBF2 * kBF2 + 15) / 16 * 16 : 0;
  const int bf = kBF2 ? kBF2 : a.bf;
  const int N = kBF2 ? kN2 + 16 : (bf + 15) / 16 * 16;
  const int bufBytes = kVfPlanes * N * 128;
  const uint32_t nBufs = (uint32_t)min(kVfMaxBufs, kVfBBytes / bufBytes);
  auto item_at = [&](int it) -> int4 {
    if (a.singleN > 0) return make_int4(0, it * a.itemKeys, min(a.itemKeys, a.singleN - it * a.itemKeys), 0);
    return __ldg(a.items + it);
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < kVfASlots; ++i) mbar_init(&s.fullA[i], kVfProducers);
    for (int i = 0; i < kVfAcc; ++i) {
      mbar_init(&s.done[i], 1);
      mbar_init(&s.accEmpty[i], 4);
    }
    for (int i = 0; i < kVfMaxBufs; ++i) {
      mbar_init(&s.fullB[i], 1);
      mbar_init(&s.emptyB[i], 1);
    }
    mbar_init(&s.mmaDone, 1);
    s.abort = failed;  // an earlier phase gave up: there are no items
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (localHist)
    for (int i = threadIdx.x; i < a.bins; i += blockDim.x) s.hist[i] = 0;
  if (warp == kVfMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmemBase)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmemBase;
  const bool run = !s.abort;
  if (!run) nIt = 0;

  // Tiles are numbered from 0 in every role (i), items likewise (j): A slot i % 2, accumulator and
  // done barrier i % 4, norms i % 8, B buffer j % nBufs.
  if (warp < kVfProducers) {
    // ---------------- producers: 32 rows of every tile each ----------------
    const int row0 = warp * 32;
    const uint32_t skip = blockIdx.x == 0 ? (uint32_t)a.skipLoad - 1u : 0xffffffffu;
    uint32_t i = 0, j = 0;
    bool ok = run;
    for (int it = blockIdx.x; it < nIt && ok; it += gridDim.x, ++j) {
      const int4 item = item_at(it);
      if (warp == 0) {
        const uint32_t buf = j % nBufs;
        ok = mbar_wait_warp(&s.emptyB[buf], ((j / nBufs) & 1u) ^ 1u, &s.abort, a.err, lim);
        if (!ok) break;
        if (lane == 0 && j != skip) {
          const long long r = a.bucketBase < 0 ? -1 : a.bucketBase + item.x;
          const long long g1 = (r + 1) * bf, g2 = (g1 + 1) * bf;
          uint8_t* b = s.b + buf * bufBytes;
          mbar_expect_tx(&s.fullB[buf], (uint32_t)bufBytes);
          for (int p = 0; p < kVfPlanes; ++p) {
            uint8_t* bp = b + p * N * 128;
            for (int x = 0; x < kN2; x += 16) tma_load_3d(bp + x * 128, &tmNodes, &s.fullB[buf], 0, (int)g2 + x, p);
            for (int x = 0; x < N - kN2; x += 16)
              tma_load_3d(bp + (kN2 + x) * 128, &tmNodes, &s.fullB[buf], 0, (int)g1 + x, p);
          }
        }
        __syncwarp();
      }
      const int tiles = (item.z + kVfRows - 1) / kVfRows;
      // the lane's row of tile t: its key, -1 past the item's keys
      auto load_key = [&](int t) -> int {
        const int pos = t * kVfRows + row0 + lane;
        if (pos >= item.z) return -1;
        return a.perm ? __ldg(a.perm + item.y + pos) : item.y + pos;
      };
      int mine = load_key(0);
      for (int t = 0; t < tiles; ++t, ++i) {
        // the slot's previous tile, i - 2, has been multiplied.  Its norms' slot is free as well: the
        // MMAs of tile i - 2 followed the epilogue's hand-back of tile i - 6, and this tile overwrites
        // the norms of tile i - 8.
        if (i >= kVfASlots) {
          const uint32_t d = i - kVfASlots;
          ok = mbar_wait_warp(&s.done[d % kVfAcc], (d / kVfAcc) & 1u, &s.abort, a.err, lim);
          if (!ok) break;
        }
        const int next = t + 1 < tiles ? load_key(t + 1) : -1;
        const uint32_t slot = i % kVfASlots;
        // lane's 16 bytes of a row: plane lane / 8, chunk lane % 8
        const uint32_t base = smem_u32(s.a[slot]) + (uint32_t)(lane >> 3) * (kVfRows * 128) + (uint32_t)row0 * 128u;
        const uint32_t ch = (uint32_t)lane & 7u;
        const int have = min(32, max(0, item.z - t * kVfRows - row0));  // rows past the item keep what is there
#pragma unroll 8
        for (int r = 0; r < 32; ++r) {
          const int key = __shfl_sync(0xffffffffu, mine, r);
          if (r < have)
            vtf_cp16(base + (uint32_t)r * 128u + ((ch ^ (uint32_t)(r & 7)) << 4),
                     a.split + (size_t)key * kVtfRowBytes + 16 * lane);
        }
        if (lane < have) vtf_cp4(smem_u32(&s.norm[i % kVfNorms][row0 + lane]), a.keyNorm + mine);
        vtf_cp_arrive(&s.fullA[slot]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.fullA[slot]);
        mine = next;
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // an item's node planes have landed before the CTA may exit (their bytes are waited for by the
    // issuer, except after an abort)
    if (warp == 0 && lane == 0)
      for (uint32_t k = j > nBufs ? j - nBufs : 0u; k < j; ++k) {
        const long long t0 = clock64();
        while (k != skip && !mbar_try(&s.fullB[k % nBufs], (k / nBufs) & 1u) && clock64() - t0 < kWaitCycles) {
        }
      }
  } else if (warp == kVfMmaWarp) {
    // ---------------- MMA issuer (the warp walks, one elected lane issues) ----------------
    const bool leader = elect_one();
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kVfRows >> 4) << 24);
    const uint32_t aBase = sdesc_lo(smem_u32(s.a[0])), bBase = sdesc_lo(smem_u32(s.b));
    const uint32_t bPlane = (uint32_t)(N * 128) >> 4;
    uint32_t i = 0, j = 0;
    bool ok = run;
    for (int it = blockIdx.x; it < nIt && ok; it += gridDim.x, ++j) {
      const int4 item = item_at(it);
      const uint32_t buf = j % nBufs;
      ok = mbar_wait_warp(&s.fullB[buf], (j / nBufs) & 1u, &s.abort, a.err, lim);
      const uint32_t bd = bBase + buf * ((uint32_t)bufBytes >> 4);
      const uint32_t iEnd = i + (uint32_t)((item.z + kVfRows - 1) / kVfRows);
      for (; i < iEnd && ok; ++i) {
        ok = mbar_wait_warp(&s.fullA[i % kVfASlots], (i / kVfASlots) & 1u, &s.abort, a.err, lim) &&
             mbar_wait_warp(&s.accEmpty[i % kVfAcc], ((i / kVfAcc) & 1u) ^ 1u, &s.abort, a.err, lim);
        if (!ok) break;
        tc_fence_after();
        const uint32_t ad = aBase + (i % kVfASlots) * (uint32_t)(kVfABytes >> 4);
        const uint32_t d = tmem + (i % kVfAcc) * 128u;
        if (leader) {
          // the rows were written by cp.async (generic proxy); the tensor core reads them through the
          // async proxy
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
#pragma unroll
          for (int k = 0; k < 24; ++k) {  // hi.hi', lo.hi', hi.lo', eight K steps of 16 values each
            const int prod = k >> 3, half = (k >> 2) & 1, step = k & 3;
            const uint32_t ap = (uint32_t)(prod == 1 ? 2 + half : half), bp = (uint32_t)(prod == 2 ? 2 + half : half);
            vtf_mma(d, sdesc_of(ad + ap * (uint32_t)(kVfRows * 128 >> 4) + (uint32_t)(2 * step)),
                    sdesc_of(bd + bp * bPlane + (uint32_t)(2 * step)), idesc, k > 0 ? 1u : 0u);
          }
          mma_commit(&s.done[i % kVfAcc]);
        }
      }
      if (leader) mma_commit(&s.emptyB[buf]);
    }
    if (leader) {  // every MMA issued has completed before TMEM is released
      mma_commit(&s.mmaDone);
      const long long t0 = clock64();
      while (!mbar_try(&s.mmaDone, 0) && clock64() - t0 < kWaitCycles) {
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue: one key per lane ----------------
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const float maxNorm = *a.maxNorm;
    uint32_t i = 0;
    bool ok = run;
    for (int it = blockIdx.x; it < nIt && ok; it += gridDim.x) {
      const int4 item = item_at(it);
      const long long r = a.bucketBase < 0 ? -1 : a.bucketBase + item.x;
      const long long g1 = (r + 1) * bf;
      const float childNorm = __ldg(a.childNorm + r + 1);
      const int tiles = (item.z + kVfRows - 1) / kVfRows;
      for (int t = 0; t < tiles; ++t, ++i) {
        const int pos = t * kVfRows + row;
        const int key = pos < item.z ? (a.perm ? __ldg(a.perm + item.y + pos) : item.y + pos) : -1;
        ok = mbar_wait_warp(&s.done[i % kVfAcc], (i / kVfAcc) & 1u, &s.abort, a.err, lim);
        if (!ok) break;
        tc_fence_after();
        const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (i % kVfAcc) * 128u;
        const float kn = s.norm[i % kVfNorms][row] * 1.00001f;
        Top2 ta, tc;  // the children; the chosen child's children
        if constexpr (kBF2 > 0) {
          uint32_t v1[16];
          vtf_ld16(tb + (uint32_t)kN2, v1);
          tmem_wait(v1);
#pragma unroll
          for (int k = 0; k < kBF2; ++k) ta.push(__uint_as_float(v1[k]), k);
          float g[kBF2];
#pragma unroll
          for (int k = 0; k < kBF2; ++k) g[k] = 0.0f;
#pragma unroll
          for (int c0 = 0; c0 < kBF2 * kBF2; c0 += 32) {
            uint32_t v[32];
            tmem_ld32(tb + (uint32_t)c0, v);
            tmem_wait(v);
#pragma unroll
            for (int k = 0; k < 32; ++k)
              if (c0 + k < kBF2 * kBF2)
                g[(c0 + k) % kBF2] = ta.c == (c0 + k) / kBF2 ? __uint_as_float(v[k]) : g[(c0 + k) % kBF2];
          }
#pragma unroll
          for (int k = 0; k < kBF2; ++k) tc.push(g[k], k);
        } else {
          for (int c0 = 0; c0 < bf; c0 += 32) {
            uint32_t v[32];
            tmem_ld32(tb + (uint32_t)c0, v);
            tmem_wait(v);
            if (c0 + 32 <= bf) {
#pragma unroll
              for (int k = 0; k < 32; ++k) ta.push(__uint_as_float(v[k]), c0 + k);
            } else {
#pragma unroll
              for (int k = 0; k < 32; ++k)
                if (c0 + k < bf) ta.push(__uint_as_float(v[k]), c0 + k);
            }
          }
        }
        const float tiny = 1e-30f * (1.0f + kn + maxNorm);  // underflow
        const float e1 = kn >= kVtTinyNorm ? kTcRel * kn * childNorm + tiny : INFINITY;
        const bool weird = !(kn * maxNorm < 1e30f);
        long long node = g1 + ta.c;
        int undecided = 0;  // levels left to the replay, from node `from` down
        long long from = r;
        if (key >= 0 && !weird) {
          if (!ta.decided(e1)) {
            undecided = kBF2 ? 2 : 1;
          } else if (kBF2 && !tc.decided(kTcRel * kn * __ldg(a.childNorm + node + 1) + tiny)) {
            undecided = 1;
            from = node;
          }
        }
        // one level: the children whose scores come within twice the bound of the first, the only
        // ones the sequential rule can choose
        uint32_t mask[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
        if constexpr (kBF2 == 0) {
          if (__any_sync(0xffffffffu, undecided)) {
            const float lead = ta.s1 - 2.0f * e1;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              if (32 * c >= bf) break;
              uint32_t v[32];
              tmem_ld32(tb + (uint32_t)(32 * c), v);
              tmem_wait(v);
              uint32_t m = 0;
#pragma unroll
              for (int k = 0; k < 32; ++k) m |= __uint_as_float(v[k]) >= lead ? 1u << k : 0u;
              mask[c] = m;
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.accEmpty[i % kVfAcc]);
        if (key < 0) continue;
        if (weird && a.weird) a.weird[atomicAdd(a.nWeird, 1)] = key;  // first phase: descends by itself at the end
        if (kBF2) node = (node + 1) * bf + tc.c;
        if (undecided) {
          const int at = atomicAdd(a.nFlagged, 1);
          a.flagged[2 * at] = make_int4(key, (int)from, undecided, 0);
          a.flagged[2 * at + 1] = make_int4((int)mask[0], (int)mask[1], (int)mask[2], (int)mask[3]);
          continue;
        }
        if (a.final) {
          a.out[key] = (int32_t)(a.idMode == V3DM_LEAF_LOCAL ? node - a.leafBase : node);
        } else {
          const int bkt = (int)(node - a.nextBase);
          a.next[key] = bkt;
          // one update per distinct bucket of the warp
          const unsigned peers = __match_any_sync(__activemask(), bkt);
          if (lane == __ffs(peers) - 1) atomicAdd(localHist ? &s.hist[bkt] : &a.hist[bkt], __popc(peers));
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (localHist)
    for (int i = threadIdx.x; i < a.bins; i += blockDim.x)
      if (s.hist[i]) atomicAdd(&a.hist[i], s.hist[i]);
  if (warp == kVfMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// The listed keys' levels in the reference's arithmetic: a warp per key, a candidate child per lane
// (the first level's come as a mask).  A level is the latency of a lane's 512-byte row and of 128 additions in
// order: with 16 of the 32 loads ahead, 4000 keys of a BF 5, depth 4 tree whose undecided ones are all listed
// took 24.8 us, with eight 29.0.
__global__ void __launch_bounds__(256)
k_vtf_resolve(VtfArgs a, const float* __restrict__ nodes, unsigned long long* __restrict__ exactCount) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int n = *a.nFlagged;
  const int bf = a.bf;
  unsigned long long levels = 0;
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n; w += (gridDim.x * blockDim.x) >> 5) {
    const int4 f = a.flagged[2 * w], fm = a.flagged[2 * w + 1];
    const float4* krow = reinterpret_cast<const float4*>(a.keys + (size_t)f.x * kDescBytes);
    long long node = f.y;
    for (int l = 0; l < f.z; ++l) {
      const long long base = (node + 1) * bf;
      uint32_t m[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t in = bf >= 32 * (c + 1) ? 0xffffffffu : bf > 32 * c ? (1u << (bf - 32 * c)) - 1u : 0u;
        m[c] = l == 0 ? in & (uint32_t)(c == 0 ? fm.x : c == 1 ? fm.y : c == 2 ? fm.z : fm.w) : in;
      }
      const int total = __popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3]);
      float best = -1e30f;
      int bi = -1;
      for (int c0 = lane; c0 < total; c0 += 32) {
        int k = c0, word = 0;  // the k-th candidate of the word
        while (k >= __popc(m[word])) k -= __popc(m[word++]);
        const int c = 32 * word + (int)__fns(m[word], 0, k + 1);
        const float4* nrow = reinterpret_cast<const float4*>(nodes + (size_t)(base + c) * kDescBytes);
        float sc = 0.0f;
#pragma unroll 16
        for (int q = 0; q < kDescBytes / 4; ++q) {
          const float4 x = __ldg(krow + q), y = __ldg(nrow + q);
          sc = __fadd_rn(sc, __fmul_rn(x.x, y.x));
          sc = __fadd_rn(sc, __fmul_rn(x.y, y.y));
          sc = __fadd_rn(sc, __fmul_rn(x.z, y.z));
          sc = __fadd_rn(sc, __fmul_rn(x.w, y.w));
        }
        if (sc > best) {
          best = sc;
          bi = c;
        }
      }
      __syncwarp();
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {  // the largest score, its first child
        const float so = __shfl_xor_sync(0xffffffffu, best, o);
        const int io = __shfl_xor_sync(0xffffffffu, bi, o);
        if (io >= 0 && (bi < 0 || so > best || (so == best && io < bi))) {
          best = so;
          bi = io;
        }
      }
      if (bi < 0) {  // cannot happen for the finite keys and nodes that are listed
        if (lane == 0) atomicOr(a.err, kErrBadTree);
        bi = 0;
      }
      node = base + bi;
    }
    levels += (unsigned long long)f.z;
    if (lane == 0) {
      if (a.final) {
        a.out[f.x] = (int32_t)(a.idMode == V3DM_LEAF_LOCAL ? node - a.leafBase : node);
      } else {
        const int bkt = (int)(node - a.nextBase);
        a.next[f.x] = bkt;
        atomicAdd(&a.hist[bkt], 1);
      }
    }
  }
  if (lane == 0 && levels) atomicAdd(exactCount, levels);
  if (a.ticket) {
    __syncthreads();  // the block has read the count
    if (threadIdx.x == 0 && atomicAdd(a.ticket, 1) == (int)gridDim.x - 1) *a.nFlagged = *a.ticket = 0;
  }
}

// Keys split: per key 512 bytes, BF16 hi of the 128 values and then lo, and the key's norm.  A warp
// per key.
__global__ void __launch_bounds__(256)
k_vtf_split(const float4* __restrict__ keys, int n, uint2* __restrict__ split, float* __restrict__ norm) {
  const int lane = threadIdx.x & 31;
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, step = (gridDim.x * blockDim.x) >> 5;
  for (int k0 = 4 * w; k0 < n; k0 += 4 * step) {
    float4 x[4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
      x[r] = k0 + r < n ? __ldg(keys + (size_t)(k0 + r) * 32 + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      uint2 hi, lo;
      split2(x[r].x, x[r].y, hi.x, lo.x);
      split2(x[r].z, x[r].w, hi.y, lo.y);
      float ss = fmaf(x[r].x, x[r].x, fmaf(x[r].y, x[r].y, fmaf(x[r].z, x[r].z, x[r].w * x[r].w)));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (k0 + r < n) {
        split[(size_t)(k0 + r) * 64 + lane] = hi;
        split[(size_t)(k0 + r) * 64 + 32 + lane] = lo;
        if (lane == 0) norm[k0 + r] = sqrtf(ss);
      }
    }
  }
}

// Node rows as four planes of `rows` x 128 bytes: BF16 hi 0..63, hi 64..127, lo 0..63, lo 64..127.
__global__ void k_vtf_nodes(const float4* __restrict__ nodes, long long rows, uint2* __restrict__ planes) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // row * 32 + quad
  if (t >= rows * 32) return;
  const float4 x = nodes[t];
  const long long row = t >> 5;
  const int quad = (int)(t & 31);
  uint2 hi, lo;
  split2(x.x, x.y, hi.x, lo.x);
  split2(x.z, x.w, hi.y, lo.y);
  const long long at = ((long long)(quad >> 4) * rows + row) * 16 + (quad & 15);
  planes[at] = hi;
  planes[at + 2 * rows * 16] = lo;
}

// The largest norm among every parent's children (entry r + 1 for node r, entry 0 the root's), and
// over all of them, as floats' bits (norms are not negative; NaN is above infinity).
__global__ void k_vtf_max_norm(const float* __restrict__ norm, long long parents, int bf, unsigned int* __restrict__ out,
                               unsigned int* __restrict__ all) {
  unsigned m = 0;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < parents;
       p += (long long)gridDim.x * blockDim.x) {
    unsigned c = 0;
    for (int k = 0; k < bf; ++k) c = max(c, __float_as_uint(norm[p * bf + k]) & 0x7fffffffu);
    out[p] = c;
    m = max(m, c);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(all, m);
}

template <int kBF2>
cudaError_t launch_bf2(const VtfArgs& a, const CUtensorMap& m, int grid, cudaStream_t st) {
  const size_t smem = sizeof(VtfSmem) + 1024;
  cudaError_t e = cudaFuncSetAttribute(k_vtf<kBF2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_vtf<kBF2><<<grid, kVfThreads, smem, st>>>(a, m);
  return cudaGetLastError();
}

}  // namespace

// One level per phase up to 128 children; two where BF^2 (rounded up to 16) + 16 columns fit 128.
int vtf_levels(int bf) { return bf < 2 || bf > 128 ? 0 : bf <= 10 ? 2 : 1; }

cudaError_t vtf_prepare(const float* nodes, const float* norm, long long rows, int bf, void* planes, float* childNorm,
                        float* maxNorm, CUtensorMap* map, cudaStream_t st) {
  void* fp = nullptr;
  cudaDriverEntryPointQueryResult qr;
  cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fp, 12000, cudaEnableDefault, &qr);
  if (e != cudaSuccess) return e;
  if (qr != cudaDriverEntryPointSuccess) return cudaErrorNotSupported;
  cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)kVfPlanes};
  cuuint64_t strides[2] = {128, (cuuint64_t)rows * 128};
  cuuint32_t box[3] = {64, 16, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  if (reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fp)(
          map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, planes, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) !=
      CUDA_SUCCESS)
    return cudaErrorInvalidValue;
  k_vtf_nodes<<<(unsigned)((rows * 32 + 255) / 256), 256, 0, st>>>(reinterpret_cast<const float4*>(nodes), rows,
                                                                  static_cast<uint2*>(planes));
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(maxNorm, 0, sizeof(float), st)) != cudaSuccess) return e;
  k_vtf_max_norm<<<kB200SMs, 256, 0, st>>>(norm, rows / bf, bf, reinterpret_cast<unsigned int*>(childNorm),
                                      reinterpret_cast<unsigned int*>(maxNorm));
  return cudaGetLastError();
}

cudaError_t launch_vtf_split(const float* keys, int n, void* split, float* norm, int numSMs, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int blocks = (n + 31) / 32;  // four keys per warp, eight warps
  k_vtf_split<<<blocks < 16 * numSMs ? blocks : 16 * numSMs, 256, 0, st>>>(reinterpret_cast<const float4*>(keys), n,
                                                                        static_cast<uint2*>(split), norm);
  return cudaGetLastError();
}

cudaError_t launch_vtf(const VtfArgs& a, const CUtensorMap& m, const float* nodes, unsigned long long* exactCount,
                       int grid, cudaStream_t st) {
  cudaError_t e;
  switch (a.levels == 2 ? a.bf : 0) {
    case 2: e = launch_bf2<2>(a, m, grid, st); break;
    case 3: e = launch_bf2<3>(a, m, grid, st); break;
    case 4: e = launch_bf2<4>(a, m, grid, st); break;
    case 5: e = launch_bf2<5>(a, m, grid, st); break;
    case 6: e = launch_bf2<6>(a, m, grid, st); break;
    case 7: e = launch_bf2<7>(a, m, grid, st); break;
    case 8: e = launch_bf2<8>(a, m, grid, st); break;
    case 9: e = launch_bf2<9>(a, m, grid, st); break;
    case 10: e = launch_bf2<10>(a, m, grid, st); break;
    default: e = launch_bf2<0>(a, m, grid, st); break;
  }
  if (e != cudaSuccess) return e;
  k_vtf_resolve<<<8 * grid, 256, 0, st>>>(a, nodes, exactCount);
  return cudaGetLastError();
}

cudaError_t launch_vtf_resolve(const VtfArgs& a, const float* nodes, unsigned long long* exactCount, int blocks,
                               cudaStream_t st) {
  return launch_pdl(k_vtf_resolve, dim3(blocks), dim3(256), 0, st, a, nodes, exactCount);
}

}  // namespace v3dm
