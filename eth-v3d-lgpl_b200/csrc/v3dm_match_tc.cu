// v3dm_match_tc.cu -- tcgen05 side kernel for sm_100a: one persistent launch scores one side
// of a pair against the other and keeps, for every descriptor of the A side, its best
// candidate and an upper bound of its second-best score.  Two launches (lefts x rights,
// then the chosen rights x lefts) replace cublasSgemm + the four maxima kernels of the
// reference (v3d_cudamatching.cu:529-545); no score leaves the SM.
//
//   warp 0      TMA producer: an A group (NB blocks of 128 descriptors x 128 bytes) whenever
//               the group changes, B tiles (BN x 128 bytes) through a ring of shared-memory
//               stages, 128-byte swizzle;
//   warps 1-2   (warp 1 allocates 512 TMEM columns) issue tcgen05.mma.kind::i8 (u8 x u8 -> s32,
//               M=128, N=BN, four K=32 steps per block) into 512/(NB*BN) accumulator stages,
//               alternate tiles each;
//   warps 3-18  epilogue, four per TMEM lane quadrant.  Lane i of a warp owns A descriptor
//               'row' and reads its scores with tcgen05.ld (32 columns per chunk), hands the
//               stage back, and per chunk does one of two things:
//                 - all scores below Smin (the smallest score that can pass the min-score
//                   test): W = max(W, chunk maximum);
//                 - some score >= Smin (true matches, ~1e-6 of unrelated pairs): the lane
//                   writes a record (descriptor, first column, its 32 scores) to its warp's
//                   segment; k_records (v3dm_pair.cu) does the exact work on it: guided
//                   gates for every score >= Smin, chunk best (largest score, first index on
//                   ties, the reference's argMax rule, v3d_cudamatching.cu:145), maximum of
//                   the other scores.
//               At the end of a work unit the lane's W + 1 goes to sec[] (atomicMax).  W starts
//               as a negative float's bits (below every score) and takes the spare input of the
//               chunk's maximum tree: C = max(W, chunk); C >= Smin exactly when the chunk
//               reaches Smin (W < Smin always), else W = C.
// Resulting per-descriptor values (after the list pass in v3dm_pair.cu): best = the exact
// best over scores >= Smin that pass the gates; sec = the exact second-best score without
// gates, an upper bound of it with gates (masked scores are counted).  The decision
// accept(best, s2) is monotone in s2, so when accept(best, sec) == accept(best, none) the
// decision is exact; otherwise the descriptor is re-scored exactly (rare).
// The tile shape (NB, BN) and the stage counts are template parameters chosen at run time
// (TcConfig).  NB=2 keeps 256 A rows resident and halves the B bytes per MMA compared with one
// 128-row block; more TMEM stages hide the MMA -> epilogue -> MMA hand-off latency.
// The work is the flattened sequence (A group, B tile); each CTA takes one contiguous range
// of it.  Every role walks the same range; mbarriers order the hand-offs.
// What bounds the kernel is each role's own instruction latency per tile, not a pipe: a tile is 512
// tensor cycles, and a warp's wait, commit or branch is 50 to 100.  So the walk is two loops, an
// outer one over runs of tiles that share their A group and an inner one over a run's tiles, in
// which ring slots and parities come from one tile counter; one commit per tile tells the producer
// and the epilogue; and two issuers share the tiles.  Measured per tile and issuer before: 510
// cycles in a cursor that was advanced at every tile, 180 in two commits, 120 in each wait, 70 in
// the MMAs.  32768^2 went from 140 to 97 us (2833 TOPS, 85% of twice the bf16 burst), pass A of 120
// images (1000 to 12000 features) from 39.1 to 29.3 ms; without the epilogue's filtering a tile takes
// 523 of its 512 cycles, with it 710, so the epilogue's maxima are what is left.  On 200 images the
// 1 kW limit holds the SM clock at about 1600 MHz.  Pairs of CTAs on one 256 x 256 tile
// (cta_group::2) took 190 us for 32768^2, and epilogue groups on alternate tiles 102.  Every mbarrier wait
// is bounded: on timeout the CTA raises kErrWaitTimeout, drains its own TMA loads and MMAs,
// frees TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <new>
#include <type_traits>

#include "v3dm_device.cuh"
#include "v3dm_tcgen05.cuh"

namespace v3dm {

namespace {

constexpr int BM = 128;          // rows per MMA block (TMEM lanes)
constexpr int kEpiWarps = 16;    // four per TMEM lane quadrant
constexpr int kIssuers = 2;      // MMA issuer warps, taking alternate tiles
constexpr int kEpiWarp0 = 1 + kIssuers;
constexpr int kThreads = (kEpiWarp0 + kEpiWarps) * 32;
constexpr int kTmemCols = 512;

template <int NB_, int BN_, int STAGES_, int ASLOTS_ = 2, int PIPE_ = 0>
struct TcCfg {
  static constexpr int NB = NB_;                 // 128-row MMA blocks per left group
  static constexpr int BN = BN_;                 // rights per tile
  static constexpr int kStages = STAGES_;        // right-tile ring depth
  static constexpr int kASlots = ASLOTS_;        // left-group buffers (more: short rows prefetch further)
  // kPipe = 1: the epilogue loads its second chunk while it filters the first
  static constexpr int kPipe = PIPE_;
  static constexpr int GM = BM * NB;             // left rows per group
  static constexpr int kABytes = GM * kDescBytes;
  static constexpr int kBBytes = BN * kDescBytes;
  static constexpr int kAccCols = NB * BN;       // TMEM columns per accumulator stage
  static constexpr int kAcc = kTmemCols / kAccCols;  // accumulator stages
  // Epilogue split: the four warps of a lane quadrant own (block, column quarter or half) of a
  // stage: with NB == 2 a warp owns one block and half of the columns, with NB == 1 a quarter.
  static constexpr int kWarpCols = NB == 2 ? BN / 2 : BN / 4;
  static constexpr int kChunks = kWarpCols / 32;
  static_assert(NB == 1 || NB == 2, "one or two blocks per group");
  static_assert(kWarpCols >= 32 && kWarpCols % 32 == 0 && kChunks <= 2 && BN <= 256, "1..2 chunks per warp");
  static_assert(kPipe == 0 || kChunks == 2, "pipelined loads need two chunks");
  static_assert(kAcc >= 2, "at least two accumulator stages");
  // done[] serves the producer and the epilogue: a stage's next tile must not complete before
  // every epilogue warp has seen this one, which its accumulator's hand-back ensures
  static_assert(kStages >= kAcc, "the B ring is at least as deep as the accumulator ring");
};

template <class C>
struct Smem {
  uint8_t a[C::kASlots][C::kABytes];
  uint8_t b[C::kStages][C::kBBytes];
  unsigned long long fullB[C::kStages], done[C::kStages];  // a tile has landed; its MMAs have completed
  unsigned long long fullA[C::kASlots], emptyA[C::kASlots];
  unsigned long long accEmpty[C::kAcc];
  unsigned long long mmaDone;
  unsigned long long runFull[32];  // batched pass: the ring of runs (kRunRing)
  int4 runs[2 * 32];
  uint32_t tmemBase;
  int abort;
};

struct TcShape {
  int nGroups, nTiles;  // left groups, right tiles
  long long nWork;      // nGroups * nTiles
};

// Instruction descriptor: kind::i8, D = s32, A = B = unsigned 8-bit, both K-major, N, M = 128.
template <int N>
__device__ __forceinline__ constexpr uint32_t idesc() {
  return (2u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

template <int N>
__device__ __forceinline__ void mma_i8(uint32_t dtmem, uint64_t ad, uint64_t bd, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
      "l"(ad), "l"(bd), "r"(idesc<N>()), "r"(accumulate)
      : "memory");
}

static_assert(kMaxScore < (1 << 23), "scores are zero or subnormal as floats");

// Maximum of three scores in one instruction: the three-input max.f32 of sm_100 applied to the
// scores' bit patterns.  Scores are integers in [0, 255^2 * 128] < 2^23, i.e. zero or subnormal
// floats, whose float order is their integer order; max.f32 without .ftz keeps subnormals.
__device__ __forceinline__ uint32_t max3_bits(uint32_t a, uint32_t b, uint32_t c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(__uint_as_float(a)), "f"(__uint_as_float(b)), "f"(__uint_as_float(c)));
  return __float_as_uint(r);
}

// max(x, the 32 scores of v): a tree of three-input maxima, 16 instructions (a two-input tree
// takes 31 for the scores alone; the epilogue's filtering is what limits the side kernel).  x
// takes the spare input of the last one.
__device__ __forceinline__ uint32_t max32_bits(const uint32_t* v, uint32_t x) {
  uint32_t m[12];
#pragma unroll
  for (int i = 0; i < 10; ++i) m[i] = max3_bits(v[3 * i], v[3 * i + 1], v[3 * i + 2]);
  m[10] = v[30];
  m[11] = v[31];
  uint32_t n[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) n[i] = max3_bits(m[3 * i], m[3 * i + 1], m[3 * i + 2]);
  return max3_bits(max3_bits(n[0], n[1], n[2]), n[3], x);
}

// Work range of this CTA in the flattened (group, tile) sequence.
__device__ __forceinline__ void cta_range(const TcShape& sh, long long& w0, long long& w1) {
  w0 = sh.nWork * blockIdx.x / gridDim.x;
  w1 = sh.nWork * (blockIdx.x + 1) / gridDim.x;
}

// Slot and parity of the i-th use of a ring of N.
template <int N>
__device__ __forceinline__ uint32_t ring_slot(uint32_t i) {
  return i % (uint32_t)N;
}
template <int N>
__device__ __forceinline__ uint32_t ring_parity(uint32_t i) {
  return (i / (uint32_t)N) & 1u;
}

// Single pair: the runs of a work range, a run being the tiles t0 .. t0 + nT - 1 of one group.
struct WorkCursor {
  int g, t0, nT, nTiles;
  int left;     // tiles from this run on
  static constexpr bool newA = true;  // the run's A block differs from the previous run's
  __device__ __forceinline__ WorkCursor(long long w0, long long w1, int nT_) : nTiles(nT_), left((int)(w1 - w0)) {
    g = (int)(w0 / nTiles);
    t0 = (int)(w0 - (long long)g * nTiles);
    nT = min(nTiles - t0, left);
  }
  __device__ __forceinline__ bool more() const { return left > 0; }
  __device__ __forceinline__ void next() {
    left -= nT;
    ++g;
    t0 = 0;
    nT = min(nTiles, left);
  }
};

// A row entry as loaded.  Nothing is computed from it before its turn: the loads take some 800 cycles
// and any use, were it only the lower limit of nTiles, would wait for them where they are issued.
struct RawRow {
  int4 x, y;
  __device__ __forceinline__ void load(const BatchRow* rows, int r) {
    const int4* p = reinterpret_cast<const int4*>(rows + r);
    x = __ldg(p);
    y = __ldg(p + 1);
  }
  __device__ __forceinline__ BatchRow row() const {
    BatchRow b;
    b.aRow = x.x;
    b.validRows = x.y;
    b.bRow0 = x.z;
    b.nB = x.w;
    b.nTiles = y.x;
    b.pad = y.y;
    b.state0 = (long long)(((unsigned long long)(uint32_t)y.w << 32) | (uint32_t)y.z);
    return b;
  }
};

constexpr int kChunkRows = 32;  // schedule 2: rows per chunk

// Batched pass: walks the rows of a row table, every tile of a row in order.  Schedule 0
// gives CTA b the rows b, b + grid, b + 2 grid, ...: the CTAs then work on neighbouring rows
// (the same B image) at the same time, so the B tiles are read from L2.  Schedule 1 gives
// each CTA one contiguous range of rows.  Schedule 2 deals out chunks of kChunkRows
// consecutive rows the way schedule 0 deals out rows: consecutive rows that share their A
// block (short rows of one left block against many right blocks) keep it in shared memory,
// and the CTAs still work on neighbouring rows.  The next row's entry is loaded a row ahead.
// newA says whether the current row's A block differs from the previous row's (a row's A block
// is identified by its first row aRow).
struct BatchCursor {
  const BatchRow* rows;
  int R, Rend, schedule;
  BatchRow cur;
  RawRow raw;  // the next row
  int nT;
  bool newA;
  __device__ __forceinline__ int step_from(int r) const {
    if (schedule == 0) return r + (int)gridDim.x;
    if (schedule == 1) return r + 1;
    ++r;
    return (r % kChunkRows) == 0 ? r + ((int)gridDim.x - 1) * kChunkRows : r;
  }
  __device__ __forceinline__ BatchCursor(const BatchRow* rows_, int nRows, int sch)
      : rows(rows_), schedule(sch), newA(true) {
    cur = BatchRow{};
    raw = RawRow{};
    if (schedule == 0) {
      R = blockIdx.x;
      Rend = nRows;
    } else if (schedule == 1) {
      R = (int)((long long)nRows * blockIdx.x / gridDim.x);
      Rend = (int)((long long)nRows * (blockIdx.x + 1) / gridDim.x);
    } else {
      R = blockIdx.x * kChunkRows;
      Rend = nRows;
    }
    if (R < Rend) raw.load(rows, R);
    take();
  }
  __device__ __forceinline__ void take() {
    cur = raw.row();
    nT = cur.nTiles = max(cur.nTiles, 1);  // every row advances the cursor by at least one tile
    const int R1 = step_from(R);
    if (R1 < Rend) raw.load(rows, R1);
  }
  __device__ __forceinline__ bool more() const { return R < Rend; }
  __device__ __forceinline__ void next() {
    R = step_from(R);
    newA = raw.x.x != cur.aRow;
    take();
  }
  // the next row, where there is one with another A block
  __device__ __forceinline__ bool next_new_a() const { return step_from(R) < Rend && raw.x.x != cur.aRow; }
  __device__ __forceinline__ int next_a_row() const { return raw.x.x; }
  __device__ __forceinline__ int next_valid_rows() const { return raw.x.y; }
};

// The other roles of a batched pass read each run from a ring in shared memory, where the producer
// puts its row (newA in the entry's last word) before the row's first load; a row of no tiles ends
// the walk.  Walking the table themselves cost every epilogue warp the table's loads or, loaded a
// row ahead, spills: 860 cycles per run, as much as a tile's filtering (runs of one or two tiles:
// the pass over a cell's rights of the candidate proposal; a proposal call over 60 images of 8000
// took 8.0 ms, 7.4 with the ring, and 200 images of 8192, whose runs are long, 89 and 84.5: the
// spills).  A slot is not written again before
// every role has read it: the producer's tiles are at most kStages + kAcc ahead of the slowest
// warp, and a run has a tile or more.
constexpr int kRunRing = 32;
struct RunCursor {
  const int4* ring;
  unsigned long long* full;
  uint32_t r = 0;
  BatchRow cur;
  static constexpr int t0 = 0;
  int nT;
  bool newA;
  int* abortFlag;
  int* err;
  long long lim;
  __device__ __forceinline__ RunCursor(const int4* ring_, unsigned long long* full_, int* abort_, int* err_,
                                       long long lim_)
      : ring(ring_), full(full_), abortFlag(abort_), err(err_), lim(lim_) {
    load();
  }
  __device__ __forceinline__ void load() {
    const uint32_t slot = r % kRunRing;
    if (!mbar_wait_warp(&full[slot], (r / kRunRing) & 1u, abortFlag, err, lim)) {
      nT = 0;
      return;
    }
    RawRow raw;
    raw.x = ring[2 * slot];
    raw.y = ring[2 * slot + 1];
    cur = raw.row();
    nT = cur.nTiles;
    newA = cur.pad != 0;
  }
  __device__ __forceinline__ bool more() const { return nT > 0; }
  __device__ __forceinline__ void next() {
    ++r;
    load();
  }
};
// The producer's side: the row of its r-th run, or the end (row null).
__device__ __forceinline__ void put_run(int4* ring, unsigned long long* full, uint32_t r, const BatchRow* row,
                                        bool newA) {
  const uint32_t slot = r % kRunRing;
  if (row) {
    ring[2 * slot] = make_int4(row->aRow, row->validRows, row->bRow0, row->nB);
    ring[2 * slot + 1] = make_int4(row->nTiles, newA ? 1 : 0, (int)(uint32_t)row->state0,
                                   (int)(uint32_t)((unsigned long long)row->state0 >> 32));
  } else {
    ring[2 * slot] = make_int4(0, 0, 0, 0);
    ring[2 * slot + 1] = make_int4(0, 0, 0, 0);
  }
  mbar_arrive(&full[slot]);
}

// Gathered A blocks (kGather): the producer warp copies each A row from a.aSrc (row
// a.aSrcRow[entry]) into the 128-byte-swizzled shared layout the TMA would write (16-byte
// chunk k of row r at r * 128 + ((k ^ (r & 7)) << 4)), rows past the block's valid count
// zero-filled.  The copies are cp.async (generic proxy): each lane waits for its own copies,
// fences them toward the async proxy the tensor core reads through, and lane 0 then arrives
// on the slot's full barrier.  kGatherDepth newer gathers may stay in flight while an older
// one is completed.
constexpr int kGatherDepth = 3;
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t srcBytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(srcBytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Best and second of one lane's row over the chunks of a run that hold a score >= Smin (kMerge).
struct LaneTop {
  uint32_t best = 0;  // largest score + 1, 0: none
  int col = 0;        // its first column
  uint32_t next = 0;  // largest other score + 1, 0: none
};

// The chunks of one lane's scores (columns col0 ..) one by one: a chunk with a score >= sminRow goes
// to the warp's segment as a record (k_records does its exact work) or, with kMerge, into the lane's
// top; otherwise its maximum is folded into lw.
template <int CHUNKS, bool kMerge>
__device__ __forceinline__ void filter_chunks(uint32_t (&v)[CHUNKS][32], int colBase, int nB, int bRow0, int orig,
                                           int32_t sminRow, uint32_t& lw, int& segN, uint4* segBase,
                                           long long segCap, LaneTop& top) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    const int col0 = colBase + 32 * c;
    if (col0 >= nB) break;  // chunks past the last B descriptor (warp-uniform)
    if (col0 + 32 > nB) {
      // The chunk holding the last B descriptor: the columns past it hold zero fill, zero
      // padding or the next block's descriptors; a 0 there is <= every real score, so the
      // chunk maximum stays the maximum of its real scores.
#pragma unroll
      for (int k = 0; k < 32; ++k)
        if (col0 + k >= nB) v[c][k] = 0u;
    }
    const uint32_t cm = max32_bits(v[c], lw);  // max(lw, chunk maximum)
    const bool trig = (int32_t)cm >= sminRow;
    if (!trig) lw = cm;
    const unsigned m = __ballot_sync(0xffffffffu, trig);
    if (m == 0u) continue;
    if constexpr (kMerge) {
      if (trig) {  // cm is the chunk's maximum: lw is below sminRow
        uint32_t eq = 0, w = 0;
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          eq |= v[c][k] == cm ? 1u << k : 0u;
          w = max(w, v[c][k] == cm ? 0u : v[c][k]);
        }
        if (eq & (eq - 1u)) w = cm;
        uint32_t next = nB - col0 > 1 ? w + 1u : 0u;  // the zeros past nB are no scores
        const bool first = cm + 1u > top.best;
        top.next = max(top.next, max(next, first ? top.best : cm + 1u));
        if (first) {
          top.best = cm + 1u;
          top.col = col0 + __ffs(eq) - 1;
        }
      }
      continue;
    }
    if (trig) {
      const int idx = segN + __popc(m & ((1u << lane) - 1u));
      if (idx < segCap) {
        uint4* rec = segBase + (long long)idx * kRecordQuads;
        rec[0] = make_uint4((uint32_t)orig, (uint32_t)col0, (uint32_t)nB, (uint32_t)bRow0);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          rec[1 + k] = make_uint4(v[c][4 * k], v[c][4 * k + 1], v[c][4 * k + 2], v[c][4 * k + 3]);
      }
    }
    segN += __popc(m);
  }
}

// kBatch = false: one pair, the flattened (group, tile) range of this CTA (WorkCursor).
// kBatch = true: rows of a.rows (BatchCursor); a row's state indices are state0 + row.
// kMerge = true (one pair, no gates): no records.  A lane keeps its row's best and second over a run
// and merges them into best[] and sec[] at its end, which saves a small pair the record kernel.
// kGather = true (batched pass only): A blocks gathered row by row from a.aSrc (tmA unused).
template <class C, bool kBatch, bool kGather = false, bool kMerge = false>
__global__ void __launch_bounds__(kThreads, 1)
k_side(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int nTiles, SideArgs a) {
  static_assert(!kGather || kBatch, "gathered A blocks only in the batched pass");
  const long long lim = a.waitLimit > 0 ? a.waitLimit : kWaitCycles;
  extern __shared__ uint8_t smemRaw[];
  Smem<C>& s = *reinterpret_cast<Smem<C>*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  static_assert(C::kStages + C::kAcc + 2 <= kRunRing, "the producer does not lap a reader of the ring of runs");
  using ProducerCursor = typename std::conditional<kBatch, BatchCursor, WorkCursor>::type;
  using Cursor = typename std::conditional<kBatch, RunCursor, WorkCursor>::type;
  // Barriers and TMEM do not depend on the kernel before: their set-up overlaps its end.
  int nA = 0, nRows = 0;
  TcShape sh{};
  long long w0 = 0, w1 = 0;
  auto producer_cursor = [&]() -> ProducerCursor {
    if constexpr (kBatch) return BatchCursor(a.rows, nRows, a.schedule);
    else return WorkCursor(w0, w1, sh.nTiles);
  };
  auto make_cursor = [&]() -> Cursor {
    if constexpr (kBatch) return RunCursor(s.runs, s.runFull, &s.abort, a.err, lim);
    else return WorkCursor(w0, w1, sh.nTiles);
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::kStages; ++i) {
      mbar_init(&s.fullB[i], 1);
      mbar_init(&s.done[i], 1);
    }
    for (int i = 0; i < C::kASlots; ++i) {
      mbar_init(&s.fullA[i], 1);
      mbar_init(&s.emptyA[i], kIssuers);
    }
    for (int i = 0; i < C::kAcc; ++i) mbar_init(&s.accEmpty[i], kEpiWarps);
    mbar_init(&s.mmaDone, kIssuers);
    if (kBatch)
      for (int i = 0; i < kRunRing; ++i) mbar_init(&s.runFull[i], 1);
    s.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmemBase)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmemBase;
  pdl_wait();
  pdl_launch_dependents();
  bool work;  // uniform over the block: something to score (a pass of the chosen rights may have none)
  if constexpr (kBatch) {
    nRows = a.nRowsPtr ? *a.nRowsPtr : a.nRows;
    work = nRows > 0;
  } else {
    nA = a.nAptr ? *a.nAptr : a.nA;
    sh.nGroups = (nA + C::GM - 1) / C::GM;
    sh.nTiles = nTiles;
    sh.nWork = (long long)sh.nGroups * nTiles;
    work = sh.nWork > 0;
    if (work) cta_range(sh, w0, w1);
  }
  if ((tmem & 0xFFFFu) != 0) {  // 512 columns must start at column 0
    if (threadIdx.x == 0) {
      atomicOr(a.err, kErrTmem);
      s.abort = 1;
    }
    __syncthreads();
  }

  // Ring uses are numbered from 0 in every role: tile i has B stage i % kStages and accumulator
  // i % kAcc, the run's A block number j slot j % kASlots.
  if (!work) {
    if (!kMerge && warp >= kEpiWarp0 && lane == 0) a.segCount[blockIdx.x * kEpiWarps + (warp - kEpiWarp0)] = 0;
  } else if (warp == 0) {
   if constexpr (kGather) {
    // ---------------- producer, gathered A: the whole warp ----------------
    if (!s.abort) {
      uint32_t i = 0, j = 0;             // tiles, A blocks
      int pend[kGatherDepth + 1] = {};  // slots whose gather still needs its arrive, oldest first
      int nPend = 0;
      auto arrive_oldest = [&]() {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.fullA[pend[0]]);
        for (int k = 1; k <= kGatherDepth; ++k)
          if (k < nPend) pend[k - 1] = pend[k];
        --nPend;
      };
      auto arrive_all = [&]() {
        cp_async_wait<0>();
        while (nPend > 0) arrive_oldest();
      };
      // blocking wait by lane 0 (after handing over every pending gather, so that the MMA
      // can drain what the wait depends on); the result is broadcast
      auto wait_slot = [&](unsigned long long* bar, uint32_t par) -> bool {
        if (__all_sync(0xffffffffu, mbar_try(bar, par))) return true;
        arrive_all();
        int okl = 1;
        if (lane == 0) okl = mbar_wait(bar, par, &s.abort, a.err, lim) ? 1 : 0;
        return __shfl_sync(0xffffffffu, okl, 0) != 0;
      };
      // The copies of A block j (rows aRow .. of the entry table) into its slot.
      auto gather = [&](int aRow, int nValid) -> bool {
        const uint32_t slot = ring_slot<C::kASlots>(j);
        if (!wait_slot(&s.emptyA[slot], ring_parity<C::kASlots>(j) ^ 1)) return false;
        ++j;
        int src[C::GM / 32];
#pragma unroll
        for (int k = 0; k < C::GM / 32; ++k) {
          const int rr = lane + 32 * k;
          src[k] = rr < nValid ? __ldg(a.aSrcRow + aRow + rr) : -1;
        }
        const uint32_t dst0 = smem_u32(s.a[slot]);
#pragma unroll
        for (int k = 0; k < C::GM / 32; ++k) {
          const int rr = lane + 32 * k;
          const uint8_t* g = a.aSrc + (src[k] >= 0 ? (size_t)src[k] * kDescBytes : (size_t)0);
          const uint32_t nb = src[k] >= 0 ? 16u : 0u;  // 0: zero fill
          const uint32_t d = dst0 + (uint32_t)rr * 128u;
#pragma unroll
          for (int ch = 0; ch < 8; ++ch) cp_async16(d + (uint32_t)((ch ^ (rr & 7)) << 4), g + 16 * ch, nb);
        }
        cp_async_commit();
        pend[nPend++] = (int)slot;
        if (nPend > kGatherDepth) {
          cp_async_wait<kGatherDepth>();
          arrive_oldest();
        }
        return true;
      };
      bool go = true;
      uint32_t r = 0;                    // runs
      for (ProducerCursor wc = producer_cursor(); wc.more() && go; wc.next()) {
        if (lane == 0) put_run(s.runs, s.runFull, r, &wc.cur, wc.newA);
        // A block by A block a run ahead: the copies of the next one run under this run's tiles (gathered
        // at its own turn, six tiles ahead, a block was waited for 8800 cycles, a fifth of the pass).
        if (r++ == 0) go = gather(wc.cur.aRow, wc.cur.validRows);
        if (go && wc.next_new_a()) go = gather(wc.next_a_row(), wc.next_valid_rows());
        if (!go) break;
        for (int t = 0; t < wc.nT; ++t, ++i) {
          const uint32_t st = ring_slot<C::kStages>(i);
          if (!wait_slot(&s.done[st], ring_parity<C::kStages>(i) ^ 1)) {
            go = false;
            break;
          }
          if (lane == 0) {
            mbar_expect_tx(&s.fullB[st], C::kBBytes);
            tma_load_2d(s.b[st], &tmB, &s.fullB[st], 0, wc.cur.bRow0 + t * C::BN);
          }
        }
      }
      if (lane == 0) put_run(s.runs, s.runFull, r, nullptr, false);
      // every gather has landed (and is handed over) and every load lane 0 issued has landed
      // before the CTA may exit
      arrive_all();
      if (lane == 0)
        for (uint32_t k = i > (uint32_t)C::kStages ? i - C::kStages : 0u; k < i; ++k) {
          long long t0c = clock64();
          while (!mbar_try(&s.fullB[ring_slot<C::kStages>(k)], ring_parity<C::kStages>(k)) &&
                 clock64() - t0c < kWaitCycles) {
          }
        }
    }
   } else {
    // ---------------- TMA producer ----------------
    if (lane == 0 && !s.abort) {
      uint32_t i = 0, j = 0;  // tiles, A blocks
      uint32_t skipped = 0xffffffffu;  // test hook: the tile that was not loaded
      bool go = true;
      uint32_t r = 0;  // runs
      for (ProducerCursor wc = producer_cursor(); wc.more() && go; wc.next()) {
        if constexpr (kBatch) put_run(s.runs, s.runFull, r++, &wc.cur, wc.newA);
        if (wc.newA) {
          const uint32_t slot = ring_slot<C::kASlots>(j);
          if (!mbar_wait(&s.emptyA[slot], ring_parity<C::kASlots>(j) ^ 1, &s.abort, a.err, lim)) break;
          mbar_expect_tx(&s.fullA[slot], C::kABytes);
          int aRow;
          if constexpr (kBatch) aRow = wc.cur.aRow;
          else aRow = wc.g * C::GM;
          tma_load_2d(s.a[slot], &tmA, &s.fullA[slot], 0, aRow);
          ++j;
        }
        int bRow;
        if constexpr (kBatch) bRow = wc.cur.bRow0;
        else bRow = wc.t0 * C::BN;
        for (int t = 0; t < wc.nT; ++t, ++i, bRow += C::BN) {
          const uint32_t st = ring_slot<C::kStages>(i);
          if (!mbar_wait(&s.done[st], ring_parity<C::kStages>(i) ^ 1, &s.abort, a.err, lim)) {
            go = false;
            break;
          }
          if (a.skipLoad > 0 && blockIdx.x == 0 && i + 1 == (uint32_t)a.skipLoad) {
            skipped = i;  // test hook: this tile never arrives; the MMA's bounded wait gives up
          } else {
            mbar_expect_tx(&s.fullB[st], C::kBBytes);
            tma_load_2d(s.b[st], &tmB, &s.fullB[st], 0, bRow);
          }
        }
      }
      if constexpr (kBatch) put_run(s.runs, s.runFull, r, nullptr, false);
      // Drain: every load this thread issued has landed before the CTA may exit.
      for (uint32_t k = i > (uint32_t)C::kStages ? i - C::kStages : 0u; k < i; ++k) {
        long long t0c = clock64();
        while (k != skipped && !mbar_try(&s.fullB[ring_slot<C::kStages>(k)], ring_parity<C::kStages>(k)) &&
               clock64() - t0c < kWaitCycles) {
        }
      }
      for (uint32_t k = j > (uint32_t)C::kASlots ? j - C::kASlots : 0u; k < j; ++k) {
        long long t0c = clock64();
        while (!mbar_try(&s.fullA[ring_slot<C::kASlots>(k)], ring_parity<C::kASlots>(k)) &&
               clock64() - t0c < kWaitCycles) {
        }
      }
    }
   }
  } else if (warp < kEpiWarp0) {
    // ---------------- MMA issuers ----------------
    // The whole warp walks the loop and one elected lane issues: with the loop's values uniform over
    // the warp the instruction's operands stay in uniform registers.  Issuer w takes the tiles with
    // i % kIssuers == w.
    auto wait = [&](unsigned long long* bar, uint32_t par) -> bool {
      return mbar_wait_warp(bar, par, &s.abort, a.err, lim);
    };
    if (!s.abort) {
      const uint32_t aBase = sdesc_lo(smem_u32(s.a[0])), bBase = sdesc_lo(smem_u32(s.b[0]));
      const bool leader = elect_one();
      uint32_t i0 = 0;              // the run's first tile
      uint32_t i = warp - 1;        // this issuer's next tile
      uint32_t j = 0;               // A blocks started
      bool go = true;
      for (Cursor wc = make_cursor(); wc.more() && go; wc.next()) {
        if (wc.newA) {
          // the block before is done with: each issuer says so once it has issued its MMAs of it.  The
          // wait comes first and whether or not this issuer has a tile in the run: it keeps an issuer
          // from counting twice on a slot's barrier before the other has counted once.
          if (!wait(&s.fullA[ring_slot<C::kASlots>(j)], ring_parity<C::kASlots>(j))) break;
          if (j > 0 && leader) mma_commit(&s.emptyA[ring_slot<C::kASlots>(j - 1)]);
          ++j;
        }
        i0 += (uint32_t)wc.nT;
        const uint32_t aSlot = ring_slot<C::kASlots>(j - 1);
        const uint32_t ad = aBase + aSlot * (uint32_t)(C::kABytes >> 4);
        for (; i < i0; i += kIssuers) {
          const uint32_t st = ring_slot<C::kStages>(i), acc = ring_slot<C::kAcc>(i);
          if (!wait(&s.fullB[st], ring_parity<C::kStages>(i)) ||
              !wait(&s.accEmpty[acc], ring_parity<C::kAcc>(i) ^ 1)) {
            go = false;
            break;
          }
          tc_fence_after();
          const uint32_t bd = bBase + st * (uint32_t)(C::kBBytes >> 4);
          const uint32_t d = tmem + acc * (uint32_t)C::kAccCols;
          if (leader) {
#pragma unroll
            for (int blk = 0; blk < C::NB; ++blk) {
#pragma unroll
              for (int k = 0; k < kDescBytes / 32; ++k)
                mma_i8<C::BN>(d + (uint32_t)(blk * C::BN),
                              sdesc_of(ad + (uint32_t)((blk * BM * kDescBytes + 32 * k) >> 4)),
                              sdesc_of(bd + (uint32_t)(2 * k)), k > 0 ? 1u : 0u);
            }
            mma_commit(&s.done[st]);
          }
        }
      }
      // Every MMA the elected lane issued has completed before TMEM is released.
      if (leader) {
        if (j > 0) mma_commit(&s.emptyA[ring_slot<C::kASlots>(j - 1)]);
        mma_commit(&s.mmaDone);
        long long t0c = clock64();
        while (!mbar_try(&s.mmaDone, 0) && clock64() - t0c < kWaitCycles) {
        }
      }
      __syncwarp();
    }
  } else {
    // ---------------- epilogue ----------------
    const int e = warp - kEpiWarp0;
    const int q = warp & 3;                              // TMEM lane quadrant this warp may access
    const int sub = e >> 2;                              // 0..3 within the quadrant
    const int blk = C::NB == 2 ? (sub & 1) : 0;          // A block of the group
    const int colOff = (C::NB == 2 ? (sub >> 1) : sub) * C::kWarpCols;  // first tile column of this warp
    const int rowInGroup = blk * BM + q * 32 + lane;
    const uint32_t tbase0 = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(blk * C::BN + colOff);
    uint4* const segBase = a.records + (long long)(blockIdx.x * kEpiWarps + e) * a.segCap * kRecordQuads;
    int segN = 0;                                        // warp-uniform count of records written
    bool ok = !s.abort;
    bool rowValid = false;
    int orig = 0;
    int aLocal = 0;  // batched pass: index of this lane's A row within its image
    int nB = a.nB;
    int bRow0 = 0;
    // maximum of this lane's scores in the current run, chunks with a record excluded; kNoScore
    // (a negative float, below every score in the max.f32 order) while there is none
    constexpr uint32_t kNoScore = 0xbf800000u;
    uint32_t lw = kNoScore;
    LaneTop top;
    int32_t sminRow = 0x7fffffff;  // Smin for a valid row, above every score otherwise
    // a bound below Tsec cannot change the decision: no atomic for it
    auto flush = [&]() {
      uint32_t w = lw == kNoScore ? 0u : lw + 1u;  // sec[] holds second + 1
      if constexpr (kMerge) {
        if (rowValid && top.best) merge_chunk_best(&a.best[orig], &a.sec[orig], best_key((int32_t)top.best - 1, top.col));
        w = max(w, top.next);
        top = LaneTop{};
      }
      if (rowValid && w > (uint32_t)a.Tsec) atomicMax(&a.sec[orig], w);
    };
    uint32_t i = 0;
    for (Cursor wc = make_cursor(); wc.more() && ok; wc.next()) {
      if constexpr (kBatch) {
        rowValid = rowInGroup < wc.cur.validRows;
        if (wc.newA)  // the A block's index map is read once per block, not once per row
          aLocal = rowValid ? (a.amap ? __ldg(a.amap + wc.cur.aRow + rowInGroup) : rowInGroup) : 0;
        orig = rowValid ? (int)(wc.cur.state0 + aLocal) : 0;
        nB = wc.cur.nB;
        bRow0 = wc.cur.bRow0;
      } else {
        const int row = wc.g * C::GM + rowInGroup;
        rowValid = row < nA;
        orig = rowValid ? (a.amap ? a.amap[row] : row) : 0;
      }
      lw = kNoScore;
      sminRow = rowValid ? a.Smin : 0x7fffffff;
      int colBase = wc.t0 * C::BN + colOff;
      for (const uint32_t iEnd = i + (uint32_t)wc.nT; i < iEnd; ++i, colBase += C::BN) {
        const uint32_t acc = ring_slot<C::kAcc>(i);
        ok = mbar_wait_warp(&s.done[ring_slot<C::kStages>(i)], ring_parity<C::kStages>(i), &s.abort, a.err, lim);
        if (!ok) break;
        tc_fence_after();
        const uint32_t tbase = tbase0 + acc * (uint32_t)C::kAccCols;
        // All of this warp's scores into registers, then hand the stage back at once so the
        // MMA never waits for the filtering below (kPipe: the second chunk is loaded while the
        // first is filtered, and the stage handed back after it).
        uint32_t v[C::kChunks][32];
        uint32_t cm[C::kChunks];  // max(lw, chunk maximum)
        if constexpr (C::kPipe) {
          tmem_ld32(tbase, v[0]);
          tmem_wait(v[0]);
          tmem_ld32(tbase + 32u, v[1]);
          cm[0] = max32_bits(v[0], lw);
          tmem_wait(v[1]);
        } else {
#pragma unroll
          for (int c = 0; c < C::kChunks; ++c) tmem_ld32(tbase + (uint32_t)(c * 32), v[c]);
#pragma unroll
          for (int c = 0; c < C::kChunks; ++c) tmem_wait(v[c]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.accEmpty[acc]);
        // Whole chunks only (every tile but an image's last): straight-line code, the chunks' maxima
        // interleaved and one vote for both.  A test for the last B descriptor at every chunk, with
        // the code that clears the columns past it, cost as much as the filtering itself (32768^2
        // 137 us with it, 103 us without).
        if (colBase + C::kChunks * 32 <= nB) {  // warp-uniform
#pragma unroll
          for (int c = C::kPipe ? 1 : 0; c < C::kChunks; ++c) cm[c] = max32_bits(v[c], lw);
          const uint32_t tm = C::kChunks == 2 ? max3_bits(cm[0], cm[C::kChunks - 1], lw) : cm[0];
          // kNoScore is negative as an int32; an invalid row's lw is never flushed
          if (!__any_sync(0xffffffffu, (int32_t)tm >= sminRow)) {
            lw = tm;
            continue;
          }
        }
        filter_chunks<C::kChunks, kMerge>(v, colBase, nB, bRow0, orig, sminRow, lw, segN, segBase, a.segCap, top);
      }
      if (ok) flush();
    }
    if (!kMerge && lane == 0) a.segCount[blockIdx.x * kEpiWarps + e] = segN;
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols)
                              : "memory");
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// 2-D uint8 map over rows x 128 bytes with a box of boxRows x 128 and the 128-byte swizzle.
bool encode_rows(CUtensorMap* map, const uint8_t* base, int rows, int boxRows) {
  auto fn = get_encode();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)kDescBytes, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)kDescBytes};
  cuuint32_t box[2] = {(cuuint32_t)kDescBytes, (cuuint32_t)boxRows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}


// ---- configurations ------------------------------------------------------------------
// Each entry instantiates the kernel for one tile shape; shared memory per CTA is
// 2 * (NB*16 KB) for the left groups + stages * BN*128 bytes.
using Cfg0 = TcCfg<1, 256, 4>;   // 128 x 256 tiles, 2 accumulator stages, 4-deep ring
using Cfg1 = TcCfg<1, 128, 8>;   // 128 x 128 tiles, 4 accumulator stages
using Cfg2 = TcCfg<2, 128, 8>;   // 256 x 128 tiles, 2 accumulator stages
using Cfg3 = TcCfg<2, 64, 16>;   // 256 x 64 tiles, 4 accumulator stages
using Cfg4 = TcCfg<1, 256, 6>;   // 128 x 256 tiles, 2 accumulator stages, 6-deep ring
using Cfg5 = TcCfg<1, 256, 4, 4>;   // as Cfg0 with 4 left-group buffers (rows of few tiles)
using Cfg6 = TcCfg<1, 128, 6, 6>;   // 128 x 128 tiles, 6 left-group buffers
using Cfg7 = TcCfg<1, 256, 4, 3>;   // as Cfg5 with 3 left-group buffers
using Cfg8 = TcCfg<1, 256, 5, 2>;   // as Cfg0 with a 5-deep ring
using Cfg9 = TcCfg<1, 256, 4, 4, 1>;   // as Cfg5 with the epilogue's second chunk loaded while the first is filtered

template <class C, bool kBatch, bool kGather = false, bool kMerge = false>
cudaError_t launch_cfg(const CUtensorMap& mA, const CUtensorMap& mB, int nTiles, const SideArgs& a, int grid,
                       cudaStream_t st, bool& attrSet) {
  const size_t smem = sizeof(Smem<C>) + 1024;
  auto kernel = k_side<C, kBatch, kGather, kMerge>;
  if (!attrSet) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attrSet = true;
  }
  return launch_pdl(kernel, dim3(grid), dim3(kThreads), smem, st, mA, mB, nTiles, a);
}

constexpr int kNumCfg = 10;
constexpr int kCfgNB[kNumCfg] = {Cfg0::NB, Cfg1::NB, Cfg2::NB, Cfg3::NB, Cfg4::NB,
                                 Cfg5::NB, Cfg6::NB, Cfg7::NB, Cfg8::NB, Cfg9::NB};
constexpr int kCfgBN[kNumCfg] = {Cfg0::BN, Cfg1::BN, Cfg2::BN, Cfg3::BN, Cfg4::BN,
                                 Cfg5::BN, Cfg6::BN, Cfg7::BN, Cfg8::BN, Cfg9::BN};
constexpr int kDefaultCfg = 0;

}  // namespace

struct TcPlan {
  int device = 0;
  int numSMs = 148;
  int cfg = kDefaultCfg;
  bool attrSet[kNumCfg] = {};
  bool attrSetMerge[kNumCfg] = {};
  bool attrSetBatch[kNumCfg] = {};
  bool attrSetGather = false;
};

cudaError_t tc_plan_create(TcPlan** p, int device) {
  TcPlan* t = new (std::nothrow) TcPlan();
  if (!t) return cudaErrorMemoryAllocation;
  t->device = device;
  cudaError_t e = cudaDeviceGetAttribute(&t->numSMs, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) {
    delete t;
    return e;
  }
  *p = t;
  return cudaSuccess;
}

void tc_plan_destroy(TcPlan* p) { delete p; }

int tc_segments(TcPlan* p) { return p->numSMs * kEpiWarps; }

int tc_num_configs() { return kNumCfg; }

int tc_get_config(TcPlan* p) { return p->cfg; }

cudaError_t tc_set_config(TcPlan* p, int cfg) {
  if (cfg < 0 || cfg >= kNumCfg) return cudaErrorInvalidValue;
  p->cfg = cfg;
  return cudaSuccess;
}

void tc_config_shape(int cfg, int* rowsPerGroup, int* colsPerTile) {
  *rowsPerGroup = kCfgNB[cfg] * BM;
  *colsPerTile = kCfgBN[cfg];
}

cudaError_t tc_side_maps(TcPlan* p, TcMaps* m, const uint8_t* dA, int rowsA, const uint8_t* dB, int rowsB) {
  const int c = p->cfg;
  if (rowsA <= 0 || rowsB <= 0) return cudaErrorInvalidValue;
  if (!encode_rows(&m->a, dA, rowsA, kCfgNB[c] * BM) || !encode_rows(&m->b, dB, rowsB, kCfgBN[c]))
    return cudaErrorInvalidValue;
  m->cfg = c;
  return cudaSuccess;
}

namespace {

template <class C>
cudaError_t launch_pair(const TcMaps& m, int nTiles, const SideArgs& a, int grid, cudaStream_t st, bool& attrSet,
                        bool& attrSetMerge) {
  if (a.merge) return launch_cfg<C, false, false, true>(m.a, m.b, nTiles, a, grid, st, attrSetMerge);
  return launch_cfg<C, false>(m.a, m.b, nTiles, a, grid, st, attrSet);
}

}  // namespace

cudaError_t launch_side(TcPlan* p, const TcMaps& m, const SideArgs& a, cudaStream_t st) {
  const int c = m.cfg;
  const int bn = kCfgBN[c];
  const int nTiles = (a.nB + bn - 1) / bn;
  if (nTiles == 0) return cudaSuccess;
  // Persistent grid: one CTA per SM (or fewer when the work is known to be small).
  long long maxWork = (long long)((a.nA + kCfgNB[c] * BM - 1) / (kCfgNB[c] * BM)) * nTiles;
  int grid = (int)std::min<long long>(p->numSMs, std::max<long long>(1, maxWork));
  if (grid * kEpiWarps > a.nSeg) return cudaErrorInvalidValue;
  switch (c) {
    case 0: return launch_pair<Cfg0>(m, nTiles, a, grid, st, p->attrSet[0], p->attrSetMerge[0]);
    case 1: return launch_pair<Cfg1>(m, nTiles, a, grid, st, p->attrSet[1], p->attrSetMerge[1]);
    case 2: return launch_pair<Cfg2>(m, nTiles, a, grid, st, p->attrSet[2], p->attrSetMerge[2]);
    case 3: return launch_pair<Cfg3>(m, nTiles, a, grid, st, p->attrSet[3], p->attrSetMerge[3]);
    case 4: return launch_pair<Cfg4>(m, nTiles, a, grid, st, p->attrSet[4], p->attrSetMerge[4]);
    case 5: return launch_pair<Cfg5>(m, nTiles, a, grid, st, p->attrSet[5], p->attrSetMerge[5]);
    case 6: return launch_pair<Cfg6>(m, nTiles, a, grid, st, p->attrSet[6], p->attrSetMerge[6]);
    case 7: return launch_pair<Cfg7>(m, nTiles, a, grid, st, p->attrSet[7], p->attrSetMerge[7]);
    case 8: return launch_pair<Cfg8>(m, nTiles, a, grid, st, p->attrSet[8], p->attrSetMerge[8]);
    default: return launch_pair<Cfg9>(m, nTiles, a, grid, st, p->attrSet[9], p->attrSetMerge[9]);
  }
}

template <class C>
cudaError_t set_batch_attr(bool& attrSet) {
  if (attrSet) return cudaSuccess;
  const size_t smem = sizeof(Smem<C>) + 1024;
  cudaError_t e = cudaFuncSetAttribute(k_side<C, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) attrSet = true;
  return e;
}

cudaError_t tc_prepare_batch(TcPlan* p, int cfg) {
  switch (cfg) {
    case 0: return set_batch_attr<Cfg0>(p->attrSetBatch[0]);
    case 1: return set_batch_attr<Cfg1>(p->attrSetBatch[1]);
    case 2: return set_batch_attr<Cfg2>(p->attrSetBatch[2]);
    case 3: return set_batch_attr<Cfg3>(p->attrSetBatch[3]);
    case 4: return set_batch_attr<Cfg4>(p->attrSetBatch[4]);
    case 5: return set_batch_attr<Cfg5>(p->attrSetBatch[5]);
    case 6: return set_batch_attr<Cfg6>(p->attrSetBatch[6]);
    case 7: return set_batch_attr<Cfg7>(p->attrSetBatch[7]);
    case 8: return set_batch_attr<Cfg8>(p->attrSetBatch[8]);
    case 9: return set_batch_attr<Cfg9>(p->attrSetBatch[9]);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_side_batch(TcPlan* p, const TcMaps& m, const SideArgs& a, cudaStream_t st) {
  const int c = m.cfg;
  // Persistent grid: one CTA per SM (fewer when the row count is known to be small).
  int grid = p->numSMs;
  if (!a.nRowsPtr) {
    if (a.nRows <= 0) return cudaSuccess;
    grid = std::min(grid, a.nRows);
  }
  if (grid * kEpiWarps > a.nSeg || a.schedule < 0 || a.schedule > 2) return cudaErrorInvalidValue;
  switch (c) {
    case 0: return launch_cfg<Cfg0, true>(m.a, m.b, 0, a, grid, st, p->attrSetBatch[0]);
    case 1: return launch_cfg<Cfg1, true>(m.a, m.b, 0, a, grid, st, p->attrSetBatch[1]);
    case 2: return launch_cfg<Cfg2, true>(m.a, m.b, 0, a, grid, st, p->attrSetBatch[2]);
    case 3: return launch_cfg<Cfg3, true>(m.a, m.b, 0, a, grid, st, p->attrSetBatch[3]);
    case 4: return launch_cfg<Cfg4, true>(m.a, m.b, 0, a, grid, st, p->attrSetBatch[4]);
    case 5: return launch_cfg<Cfg5, true>(m.a, m.b, 0, a, grid, st, p->attrSetBatch[5]);
    case 6: return launch_cfg<Cfg6, true>(m.a, m.b, 0, a, grid, st, p->attrSetBatch[6]);
    case 7: return launch_cfg<Cfg7, true>(m.a, m.b, 0, a, grid, st, p->attrSetBatch[7]);
    case 8: return launch_cfg<Cfg8, true>(m.a, m.b, 0, a, grid, st, p->attrSetBatch[8]);
    default: return launch_cfg<Cfg9, true>(m.a, m.b, 0, a, grid, st, p->attrSetBatch[9]);
  }
}

// Gathered-A batched pass: one fixed configuration (128 x 128 tiles, six A slots, so that
// several gathers are in flight while short rows are scored).
using CfgG = Cfg6;

int tc_gather_rows() { return CfgG::GM; }
int tc_gather_cols() { return CfgG::BN; }

cudaError_t tc_rows_map(CUtensorMap* m, const uint8_t* base, int rows, int boxRows) {
  if (rows <= 0 || boxRows <= 0 || boxRows > 256) return cudaErrorInvalidValue;
  return encode_rows(m, base, rows, boxRows) ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t tc_gather_map(CUtensorMap* m, const uint8_t* dB, int rowsB) {
  if (rowsB <= 0) return cudaErrorInvalidValue;
  return encode_rows(m, dB, rowsB, CfgG::BN) ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t launch_side_gather(TcPlan* p, const CUtensorMap& mB, const SideArgs& a, cudaStream_t st) {
  int grid = p->numSMs;
  if (!a.nRowsPtr) {
    if (a.nRows <= 0) return cudaSuccess;
    grid = std::min(grid, a.nRows);
  }
  if (grid * kEpiWarps > a.nSeg || a.schedule < 0 || a.schedule > 2 || !a.aSrc || !a.aSrcRow)
    return cudaErrorInvalidValue;
  return launch_cfg<CfgG, true, true>(mB, mB, 0, a, grid, st, p->attrSetGather);
}

}  // namespace v3dm
