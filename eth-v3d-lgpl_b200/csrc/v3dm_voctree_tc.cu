// v3dm_voctree_tc.cu -- tensor-core descent of uint8 vocabulary trees (sm_100a).
//
// The reference descends one key per 32-thread block, level by level, with a dot product per
// child (V3D/CUDA/v3d_cudamatching.cu:745-792).  Here the keys are grouped so that the child
// rows they score are shared, and the scoring is a tcgen05 int8 GEMM:
//   - a phase descends up to two levels below a bucket node r (the root for the first phase):
//     level a scores r's BF children, level b all BF^2 grandchildren (children of node
//     (r + 1) BF + c are the BF rows from ((r + 1) BF + c + 1) BF, so the grandchildren are one
//     contiguous block of BF^2 rows, BFS order);
//   - the CTA stages that subtree (BF + BF^2 rows) in shared memory once per work item and
//     multiplies tiles of 128 keys of the bucket by it in one MMA chain (K = 128, u8 x u8 ->
//     s32 in TMEM, N = BF^2 rounded up to 16, plus 16): its first columns are D2 = keys x
//     grandchildren, its last 16 D1 = keys x children (the B rows are laid out that way);
//   - the epilogue (one key per thread, its row of D1 and D2 read with tcgen05.ld) takes the
//     first child with the largest D1 score (strict '>', .cu:781), then the BF scores of that
//     child's children out of D2 (a select network over the chosen child) and again the first
//     largest.  Scoring all BF^2 grandchildren costs BF times the MMA work of the BF needed,
//     which the tensor core absorbs; no dp4a is left.
// Between phases the keys are sorted by the node they reached (k_vt_scan / k_vt_scatter in
// v3dm_voctree.cu), so every bucket's keys come as consecutive positions of a permutation.  The
// dot products are exact integers (at most 255 * 255 * 128 < 2^23), so the leaf ids are the
// reference's whatever the summation order; ties keep the first child.
//
// Roles (one persistent CTA per SM, 13 warps):
//   warps 0-3   producers: the first phase's keys are consecutive and come as one TMA tile (128 rows,
//               128-byte swizzle) that warp 0 loads; later phases gather their rows through the
//               permutation with cp.async, 32 rows of a tile per warp (16-byte chunks into the same
//               swizzle, eight lanes per row), each lane's copies completing on the slot's mbarrier
//               (cp.async.mbarrier.arrive).  Warp 0 also loads every item's subtree rows with TMA
//               (boxes of 16 rows) into a ring of B buffers; the rows past the BF children and BF^2
//               grandchildren that a box brings along only fill columns the epilogue never reads;
//   warp 4      allocates 512 TMEM columns and issues the MMAs of a tile into one of
//               512 / (N2 + 16) accumulator stages (the warp walks, one elected lane issues);
//   warps 5-12  epilogue, two warps per TMEM lane quadrant taking alternate tiles.
// Every mbarrier wait is bounded (kWaitCycles); on timeout the CTA records kErrWaitTimeout,
// drains its own copies and MMAs, frees TMEM and returns.  Its keys then have no bucket, so the
// phases behind it, whose items and permutation would be made of them, do nothing.
#include <cuda.h>

#include <algorithm>

#include "v3dm_device.cuh"
#include "v3dm_tcgen05.cuh"

namespace v3dm {

namespace {

constexpr int kVtcProducers = 4;                // producer warps, 32 rows of a tile each
constexpr int kVtcMmaWarp = kVtcProducers;      // the MMA issuer's warp
constexpr int kVtcEpiWarp0 = kVtcProducers + 1; // first epilogue warp
constexpr int kVtcEpiHalves = 2;                // epilogue warps per TMEM lane quadrant
constexpr int kVtcThreads = (kVtcEpiWarp0 + 4 * kVtcEpiHalves) * 32;
constexpr int kVtcRows = 128;                   // keys per tile (TMEM lanes)
static_assert(kVtcProducers * 32 == kVtcRows, "a producer warp has 32 rows of a tile, one key index per lane");
constexpr int kVtcASlots = 8;                   // key-tile ring depth
constexpr int kVtcTmemCols = 512;
constexpr int kVtcLocalBins = 4096;             // next-phase histogram kept in shared memory up to this
constexpr int kVtcItemKeys = 2048;              // keys per implicit item of a single-bucket phase

template <int BF>
struct VtcShape {
  static constexpr int N2 = (BF * BF + 15) / 16 * 16;   // grandchildren columns (MMA N)
  static constexpr int N1 = 16;                         // children columns
  static constexpr int kRowsB = N2 + N1;                // B rows: grandchildren, then children
  static constexpr int kAccCols = N2 + N1;
  // accumulator stages (narrow trees would fit 10 or 16; see the assertion)
  static constexpr int kAcc = std::min(kVtcTmemCols / kAccCols, kVtcASlots);
  static constexpr int kABytes = kVtcRows * kDescBytes;
  static constexpr int kBBytes = kRowsB * kDescBytes;
  static constexpr int kBBufs = kBBytes <= 16384 ? 4 : 2;  // subtree ring depth
  static_assert(BF >= 2 && BF <= 15, "branching factor");
  static_assert(kAcc >= 2, "two accumulator stages");
  // The epilogue takes tile i when done[i % kVtcASlots] completes for it, so tile i + kVtcASlots must not
  // complete before every epilogue warp has seen tile i.  The issuer goes in order and waits for tile i's
  // hand-back before tile i + kAcc; with more stages than slots it could pass tile i + kVtcASlots first,
  // and a late warp would wait for a phase that needs its own hand-back.
  static_assert(kVtcASlots >= kAcc, "the done ring is at least as deep as the accumulator ring");
};

template <int BF>
struct VtcSmem {
  using S = VtcShape<BF>;
  uint8_t a[kVtcASlots][S::kABytes];
  uint8_t b[S::kBBufs][S::kBBytes];
  int hist[kVtcLocalBins];
  unsigned long long fullA[kVtcASlots], done[kVtcASlots];  // a tile's keys have landed; its MMAs have completed
  unsigned long long fullB[S::kBBufs], emptyB[S::kBBufs], accEmpty[S::kAcc], mmaDone;
  uint32_t tmemBase;
  int abort;
};

// Instruction descriptor: kind::i8, D = s32, A = B = unsigned 8-bit, both K-major, M = 128.
template <int N>
__device__ __forceinline__ constexpr uint32_t vtc_idesc() {
  return (2u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kVtcRows >> 4) << 24);
}

template <int N>
__device__ __forceinline__ void vtc_mma(uint32_t dtmem, uint64_t ad, uint64_t bd, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
      "l"(ad), "l"(bd), "r"(vtc_idesc<N>()), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void vtc_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// Raises the mbarrier's pending count by one now and arrives once every cp.async this thread has
// issued so far has completed (so the phase cannot complete before the copies have landed).
__device__ __forceinline__ void vtc_cp_arrive(unsigned long long* bar) {
  asm volatile("cp.async.mbarrier.arrive.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void vtc_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// 16 TMEM columns of this warp's 32 lanes; valid after tmem_wait.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

// First index of the largest of v[0..BF-1] (strict '>': the first wins ties).
template <int BF>
__device__ __forceinline__ int vtc_argmax(const uint32_t* v) {
  uint32_t best = v[0];
  int bi = 0;
#pragma unroll
  for (int k = 1; k < BF; ++k)
    if (v[k] > best) {
      best = v[k];
      bi = k;
    }
  return bi;
}

template <int BF>
__global__ void __launch_bounds__(kVtcThreads, 1)
    k_vtc(VtcArgs a, const __grid_constant__ CUtensorMap tmNodes, const __grid_constant__ CUtensorMap tmKeys) {
  using S = VtcShape<BF>;
  extern __shared__ uint8_t vtcRaw[];
  VtcSmem<BF>& s = *reinterpret_cast<VtcSmem<BF>*>((reinterpret_cast<uintptr_t>(vtcRaw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long lim = a.waitLimit > 0 ? a.waitLimit : kWaitCycles;
  const int failed = a.singleN > 0 || threadIdx.x != 0 ? 0 : *a.err != 0;
  int nIt = a.singleN > 0 ? (a.singleN + kVtcItemKeys - 1) / kVtcItemKeys : *a.nItems;
  const bool localHist = !a.final && a.bins <= kVtcLocalBins;
  const bool gathered = a.perm != nullptr;
  // item `it`: (bucket, first position, keys)
  auto item_at = [&](int it) -> int4 {
    if (a.singleN > 0) return make_int4(0, it * kVtcItemKeys, min(kVtcItemKeys, a.singleN - it * kVtcItemKeys), 0);
    return __ldg(a.items + it);
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < kVtcASlots; ++i) {
      mbar_init(&s.fullA[i], gathered ? kVtcProducers : 1);  // with a TMA's bytes, or every lane's copies
      mbar_init(&s.done[i], 1);
    }
    for (int i = 0; i < S::kBBufs; ++i) {
      mbar_init(&s.fullB[i], 1);
      mbar_init(&s.emptyB[i], 1);
    }
    for (int i = 0; i < S::kAcc; ++i) mbar_init(&s.accEmpty[i], 4);  // the four warps of the half that takes the tile
    mbar_init(&s.mmaDone, 1);
    s.abort = failed;  // an earlier phase gave up: there are no items
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (localHist)
    for (int i = threadIdx.x; i < a.bins; i += blockDim.x) s.hist[i] = 0;
  if (warp == kVtcMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmemBase)),
                 "r"(kVtcTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmemBase;
  if ((tmem & 0xFFFFu) != 0 && threadIdx.x == 0) {  // 512 columns start at column 0
    atomicOr(a.err, kErrTmem);
    s.abort = 1;
  }
  __syncthreads();
  const bool run = !s.abort;
  if (!run) nIt = 0;

  // Tiles are numbered from 0 in every role (i), items likewise (j): A slot and done barrier
  // i % kVtcASlots, accumulator i % kAcc, epilogue half i % 2, B buffer j % kBBufs.  (The walk was a
  // cursor advanced at every tile, with two producers and a lane-0 issuer: the waits, branches and
  // operand moves of one tile took longer than its 16 KB of keys.  2M keys on the BF 10, depth 6 tree:
  // 358 us a call then, 313 after; the streamed phase 54 us, 4.7 TB/s, the gathered ones 103 and 157, and with
  // the next items loaded ahead 81 and 133: 273 us a call.)
  // Every role loads its next item while it works on one (with two tiles to an item, as in a last phase,
  // the item's load and then its keys' indices were waited for each time).
  const int4 none = make_int4(0, 0, 0, 0);
  auto next_item = [&](int it) { return it + (int)gridDim.x < nIt ? item_at(it + (int)gridDim.x) : none; };
  const int4 first = (int)blockIdx.x < nIt ? item_at(blockIdx.x) : none;
  if (warp < kVtcProducers) {
    // ---------------- producers ----------------
    const int row0 = warp * 32;
    const uint32_t skip = blockIdx.x == 0 ? (uint32_t)a.skipLoad - 1u : 0xffffffffu;
    uint32_t i = 0, j = 0;
    bool ok = run;
    // the lane's row of tile t of an item: its key
    auto load_key = [&](const int4& item, int t) -> int {
      const int pos = t * kVtcRows + row0 + lane;
      return pos < item.z ? __ldg(a.perm + item.y + pos) : 0;
    };
    int4 item = first, after;
    int mine = gathered ? load_key(item, 0) : 0;
    for (int it = blockIdx.x; it < nIt && ok; it += gridDim.x, ++j, item = after) {
      after = next_item(it);
      if (warp == 0) {
        const uint32_t buf = j % S::kBBufs;
        ok = mbar_wait_warp(&s.emptyB[buf], ((j / S::kBBufs) & 1u) ^ 1u, &s.abort, a.err, lim);
        if (!ok) break;
        if (lane == 0 && j != skip) {
          // subtree of the item's bucket node r: children from g1 (buffer rows N2 ..), and
          // grandchildren from g2 (buffer rows 0 .. N2 - 1)
          const long long r = a.bucketBase < 0 ? -1 : a.bucketBase + item.x;
          const long long g1 = (r + 1) * BF, g2 = (g1 + 1) * BF;
          const int boxes = a.levels == 2 ? S::N2 / kVtcBoxRows : 0;
          mbar_expect_tx(&s.fullB[buf], (uint32_t)((boxes + 1) * kVtcBoxRows * kDescBytes));
          tma_load_2d(s.b[buf] + S::N2 * kDescBytes, &tmNodes, &s.fullB[buf], 0, (int)g1);
          for (int x = 0; x < boxes; ++x)
            tma_load_2d(s.b[buf] + x * kVtcBoxRows * kDescBytes, &tmNodes, &s.fullB[buf], 0,
                        (int)(g2 + x * kVtcBoxRows));
        }
        __syncwarp();
      }
      const int tiles = (item.z + kVtcRows - 1) / kVtcRows;
      if (!gathered) {
        if (warp == 0)  // consecutive keys: one TMA tile (rows past the last key read as zero)
          for (int t = 0; t < tiles; ++t, ++i) {
            const uint32_t slot = i % kVtcASlots;
            ok = mbar_wait_warp(&s.done[slot], ((i / kVtcASlots) & 1u) ^ 1u, &s.abort, a.err, lim);
            if (!ok) break;
            if (lane == 0) {
              mbar_expect_tx(&s.fullA[slot], (uint32_t)S::kABytes);
              tma_load_2d(s.a[slot], &tmKeys, &s.fullA[slot], 0, item.y + t * kVtcRows);
            }
            __syncwarp();
          }
        continue;
      }
      for (int t = 0; t < tiles; ++t, ++i) {
        const uint32_t slot = i % kVtcASlots;
        const int next = t + 1 < tiles ? load_key(item, t + 1) : load_key(after, 0);
        ok = mbar_wait_warp(&s.done[slot], ((i / kVtcASlots) & 1u) ^ 1u, &s.abort, a.err, lim);
        if (!ok) break;
        // eight lanes per 128-byte row, four rows per instruction; rows past the item keep what is there
        const int have = item.z - t * kVtcRows - row0;
        const uint32_t base = smem_u32(s.a[slot]) + (uint32_t)row0 * 128u;
        const int ch = lane & 7;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int rr = 4 * k + (lane >> 3);
          const int key = __shfl_sync(0xffffffffu, mine, rr);
          if (rr < have)
            vtc_cp16(base + (uint32_t)rr * 128u + (uint32_t)((ch ^ (rr & 7)) << 4),
                     a.keys + (size_t)key * kDescBytes + 16 * ch);
        }
        vtc_cp_arrive(&s.fullA[slot]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.fullA[slot]);
        mine = next;
      }
    }
    vtc_wait_all();
    // after an abort, the TMA loads still in flight land before the CTA exits
    if (warp == 0 && lane == 0) {
      for (uint32_t k = j > (uint32_t)S::kBBufs ? j - S::kBBufs : 0u; k < j; ++k) {
        const long long t0 = clock64();
        while (k != skip && !mbar_try(&s.fullB[k % S::kBBufs], (k / S::kBBufs) & 1u) &&
               clock64() - t0 < kWaitCycles) {
        }
      }
      for (uint32_t k = i > (uint32_t)kVtcASlots ? i - kVtcASlots : 0u; !gathered && k < i; ++k) {
        const long long t0 = clock64();
        while (!mbar_try(&s.fullA[k % kVtcASlots], (k / kVtcASlots) & 1u) && clock64() - t0 < kWaitCycles) {
        }
      }
    }
  } else if (warp == kVtcMmaWarp) {
    // ---------------- MMA issuer ----------------
    const bool leader = elect_one();
    const uint32_t aBase = sdesc_lo(smem_u32(s.a[0])), bBase = sdesc_lo(smem_u32(s.b[0]));
    uint32_t i = 0, j = 0;
    bool ok = run;
    int4 item = first, after;
    for (int it = blockIdx.x; it < nIt && ok; it += gridDim.x, ++j, item = after) {
      after = next_item(it);
      const uint32_t buf = j % S::kBBufs;
      ok = mbar_wait_warp(&s.fullB[buf], (j / S::kBBufs) & 1u, &s.abort, a.err, lim);
      const uint32_t bd = bBase + buf * (uint32_t)(S::kBBytes >> 4);
      const uint32_t iEnd = i + (uint32_t)((item.z + kVtcRows - 1) / kVtcRows);
      for (; i < iEnd && ok; ++i) {
        const uint32_t slot = i % kVtcASlots, acc = i % S::kAcc;
        ok = mbar_wait_warp(&s.fullA[slot], (i / kVtcASlots) & 1u, &s.abort, a.err, lim) &&
             mbar_wait_warp(&s.accEmpty[acc], ((i / S::kAcc) & 1u) ^ 1u, &s.abort, a.err, lim);
        if (!ok) break;
        tc_fence_after();
        const uint32_t ad = aBase + slot * (uint32_t)(S::kABytes >> 4);
        const uint32_t d2 = tmem + acc * (uint32_t)S::kAccCols;
        if (leader) {
          // the gathered key rows were written by cp.async (generic proxy); the tensor core reads
          // them through the async proxy
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
#pragma unroll
          for (int k = 0; k < kDescBytes / 32; ++k) {
            if (a.levels == 2)  // grandchildren and children: one chain over all kRowsB rows
              vtc_mma<S::kRowsB>(d2, sdesc_of(ad + 2u * k), sdesc_of(bd + 2u * k), k > 0 ? 1u : 0u);
            else
              vtc_mma<S::N1>(d2 + S::N2, sdesc_of(ad + 2u * k),
                             sdesc_of(bd + (uint32_t)(S::N2 * kDescBytes >> 4) + 2u * k), k > 0 ? 1u : 0u);
          }
          mma_commit(&s.done[slot]);
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
    // ---------------- epilogue: one key per thread ----------------
    const int q = warp & 3;                  // TMEM lane quadrant this warp may access
    const uint32_t half = (uint32_t)(warp - kVtcEpiWarp0) >> 2;  // the tiles it takes: every other one
    const int row = q * 32 + lane;
    uint32_t i0 = 0;                         // the item's first tile
    bool ok = run;
    int4 item = first, after;
    for (int it = blockIdx.x; it < nIt && ok; it += gridDim.x, item = after) {
      after = next_item(it);
      const int tiles = (item.z + kVtcRows - 1) / kVtcRows;
      const long long r = a.bucketBase < 0 ? -1 : a.bucketBase + item.x;
      const long long g1 = (r + 1) * BF;
      for (int t = (int)((i0 ^ half) & 1u); t < tiles; t += 2) {
        const uint32_t i = i0 + (uint32_t)t, acc = i % S::kAcc;
        // this row's key index, loaded before the wait for the accumulator
        const int pos = t * kVtcRows + row;
        const int key = pos < item.z ? (gathered ? __ldg(a.perm + item.y + pos) : item.y + pos) : -1;
        ok = mbar_wait_warp(&s.done[i % kVtcASlots], (i / kVtcASlots) & 1u, &s.abort, a.err, lim);
        if (!ok) break;
        tc_fence_after();
        const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * S::kAccCols);
        // D2 in columns 0 .. N2 - 1, D1 in N2 .. N2 + 15
        uint32_t d1[16];
        tmem_ld16(tb + S::N2, d1);
        tmem_wait(d1);
        const int c1 = vtc_argmax<BF>(d1);
        uint32_t g[BF];  // the chosen child's BF children: columns BF c1 .. BF c1 + BF - 1 of D2
        if (a.levels == 2) {
#pragma unroll
          for (int k = 0; k < BF; ++k) g[k] = 0u;
#pragma unroll
          for (int c0 = 0; c0 < BF * BF; c0 += 64) {
            uint32_t v[64];
            tmem_ld32(tb + (uint32_t)c0, v);
            if (c0 + 32 < BF * BF) tmem_ld32(tb + (uint32_t)(c0 + 32), v + 32);
            tmem_wait(v);
#pragma unroll
            for (int k = 0; k < 64; ++k)
              if (c0 + k < BF * BF) g[(c0 + k) % BF] = c1 == (c0 + k) / BF ? v[k] : g[(c0 + k) % BF];
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.accEmpty[acc]);
        if (key < 0) continue;
        const long long node = a.levels == 2 ? (g1 + 1) * BF + (long long)BF * c1 + vtc_argmax<BF>(g) : g1 + c1;
        if (a.final) {
          a.out[key] = (int32_t)(a.idMode == V3DM_LEAF_LOCAL ? node - a.leafBase : node);
        } else {
          const int bkt = (int)(node - a.nextBase);
          a.next[key] = bkt;
          // one update per distinct bucket of the warp (keys of a tile often share buckets)
          const unsigned peers = __match_any_sync(__activemask(), bkt);
          if (lane == __ffs(peers) - 1) atomicAdd(localHist ? &s.hist[bkt] : &a.hist[bkt], __popc(peers));
        }
      }
      i0 += (uint32_t)tiles;
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (localHist)
    for (int i = threadIdx.x; i < a.bins; i += blockDim.x)
      if (s.hist[i]) atomicAdd(&a.hist[i], s.hist[i]);
  if (warp == kVtcMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kVtcTmemCols) : "memory");
}

template <int BF>
cudaError_t launch_bf(const VtcArgs& a, const CUtensorMap& m, const CUtensorMap& mk, int grid, cudaStream_t st) {
  const size_t smem = sizeof(VtcSmem<BF>) + 1024;
  static_assert(sizeof(VtcSmem<BF>) + 1024 <= 227 * 1024, "shared memory");
  cudaError_t e = cudaFuncSetAttribute(k_vtc<BF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_vtc<BF><<<grid, kVtcThreads, smem, st>>>(a, m, mk);
  return cudaGetLastError();
}

}  // namespace

bool vtc_supported(int bf) { return bf >= 2 && bf <= 15; }

cudaError_t launch_vtc(const VtcArgs& a, const CUtensorMap& m, const CUtensorMap& mk, int grid, cudaStream_t st) {
  switch (a.bf) {
    case 2: return launch_bf<2>(a, m, mk, grid, st);
    case 3: return launch_bf<3>(a, m, mk, grid, st);
    case 4: return launch_bf<4>(a, m, mk, grid, st);
    case 5: return launch_bf<5>(a, m, mk, grid, st);
    case 6: return launch_bf<6>(a, m, mk, grid, st);
    case 7: return launch_bf<7>(a, m, mk, grid, st);
    case 8: return launch_bf<8>(a, m, mk, grid, st);
    case 9: return launch_bf<9>(a, m, mk, grid, st);
    case 10: return launch_bf<10>(a, m, mk, grid, st);
    case 11: return launch_bf<11>(a, m, mk, grid, st);
    case 12: return launch_bf<12>(a, m, mk, grid, st);
    case 13: return launch_bf<13>(a, m, mk, grid, st);
    case 14: return launch_bf<14>(a, m, mk, grid, st);
    case 15: return launch_bf<15>(a, m, mk, grid, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace v3dm
