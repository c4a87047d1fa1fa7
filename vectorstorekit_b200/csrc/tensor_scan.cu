// Tensor-core search path for euclidean, cosine and dot-product over a flat fp32 index.
//
//   coarse   queries x rows contraction on the 5th-generation tensor cores (tcgen05.mma, fp16
//            operands, fp32 accumulators in tensor memory), operands staged by TMA into
//            128-byte-swizzled shared-memory tiles.  The epilogue turns each accumulator into a
//            coarse distance and appends only the rows at or below the query's running threshold
//            to that query's candidate list: the query x row matrix never reaches HBM.
//   bound    every operand is the fp16 rounding of a power-of-two scaled fp32 value, and the
//            rounding residuals are measured when the operands are made, so |coarse - exact| <= eps
//            holds with eps computed per query from measured norms (see prep kernels).
//   rerank   the few candidates per query that can still be in the true top-k are re-scored with
//            the reference's direct fp32 formulas (AccelerateOptimizer.swift:251-383) and sorted.
//   proof    a query's result is accepted only if  c_k + 2 eps < t,  where c_k is the k-th smallest
//            coarse value kept and t the threshold below which no row was ever dropped; then every
//            true top-k row is among the re-scored candidates.  Otherwise the query is re-run on
//            the fp32 scan.
//
// Kernel structure (one CTA per SM, persistent over 128-query x 256-row tiles, query tile fastest
// so that concurrently running CTAs share the same rows in L2):
//   warp 0      TMA producer: 4-stage ring of {128 x 64 query, 256 x 64 row} fp16 tiles
//   warp 1      tensor-memory allocation; one lane issues tcgen05.mma (M128 N256 K16 x 4 per stage)
//   warps 2..   epilogue (8 warps for long contractions and with a per-row term, 16 up to four K blocks without one):
//               tcgen05.ld of the thread's accumulator row (one query per thread; the warps of a lane quarter split the
//               tile's columns), threshold filter on the maxima of eight columns, hits queued in shared memory and
//               appended under the next tile's loads; double-buffered accumulators (2 x 256 columns)
// The same kernel scans the probed lists of an IVF index (tile-table mode: an explicit list of tiles over a
// query operand gathered per (query, list) pair) and assigns rows to centroids for k-means (argmin mode and a
// threshold mode whose tiles walk the centroids for a fixed block of rows).
// Every mbarrier wait is bounded: on expiry the kernel raises an error word, stops issuing work,
// drains its copies and frees tensor memory, and the host call returns VSK_ERR_TIMEOUT.
#include <cuda.h>
#include <math_constants.h>

#include <climits>
#include <cmath>

#include "block_select.cuh"
#include "common.cuh"
#include "tensor_scan.cuh"
#include "tc_ptx.cuh"

namespace vsk {
namespace {

using namespace tc;   // tile geometry and the tcgen05 / TMA / mbarrier wrappers (tc_ptx.cuh)
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int STAGES = 4;              // operand ring: 4 stages of 48 KB
constexpr int RING_BYTES = STAGES * STAGE_BYTES;
// (A variant on pairs of CTAs - tcgen05.mma.cta_group::2, a 256-query tile, each CTA staging half of the rows -
// was built and measured 2 - 3 % slower on the headline workload: the kernel is bound by the power cap, not by
// operand traffic from L2.  It was removed.)
// Warp 0 is the TMA producer, warp 1 the MMA issuer, then EW epilogue warps: EW / 4 per tensor-memory lane quarter,
// each taking one of EW / 4 equal parts of the tile's columns.  EW = 8 for long contractions (the epilogue hides
// behind the MMAs, and fewer warps cost less issue and power) and with a per-row term (tc_epilogue_warps); EW = 16 for
// short ones (d <= 256), where a tile's MMAs take about a microsecond and the epilogue warps' serial chain of
// tensor-memory loads sets the pace.
template <int EW> struct Epi {
  static constexpr int WARPS = EW;
  static constexpr int PARTS = EW / 4;
  static constexpr int COLS = TN / PARTS;      // columns per epilogue warp
  static constexpr int GROUPS = COLS / 32;
  static constexpr int THREADS = 64 + 32 * EW;
};

// A launch that lists every row (tile-table mode, no thresholds yet); beside the modes of ScanMode.
constexpr int SCAN_ALL = 4;

constexpr int kTcQueue = 8;   // hits a lane can hold before they go to its query's list

template <int EW, bool HAS_BETA>
struct TcSmemT {
  // stage buffers first: each must start on a 1024-byte boundary for the 128B swizzle
  uint8_t ring[RING_BYTES];
  float beta[HAS_BETA ? 2 : 1][HAS_BETA ? EW : 1][Epi<EW>::COLS];   // per accumulator buffer and epilogue warp: its columns' per-row terms
  uint2 queue[EW][kTcQueue][32];   // per epilogue lane: its hits {value, column}; the dense mode's keys on their way out
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint64_t drain;
  uint32_t tmem_base;
  volatile int abort_flag;
};
template <int EW, bool HAS_BETA> constexpr size_t tc_smem_bytes() { return sizeof(TcSmemT<EW, HAS_BETA>) + 1024; }   // + alignment slack

// The tiles of a unit, one after the other, without a division per tile.  (All counts of tiles are below 2^31.)
struct TcTiles {
  int mode;                           // 0: query tile fastest, 1: row tile fastest (a unit owns whole query tiles), 2: tile table
  uint32_t qtiles, ntiles, units, dq, dn;   // (tile table: ntiles is the table's length)
};
struct TcWalk {
  uint32_t qt, nt;   // query tile and row tile (tile table: nt is the tile's index in it)
  __device__ __forceinline__ void start(const TcTiles& t, uint32_t unit) {
    nt = t.mode == 2 ? unit : t.mode == 1 ? 0u : unit / t.qtiles;
    qt = t.mode == 2 ? 0u : t.mode == 1 ? unit : unit - nt * t.qtiles;
  }
  __device__ __forceinline__ bool valid(const TcTiles& t) const { return nt < t.ntiles && qt < t.qtiles; }
  __device__ __forceinline__ void advance(const TcTiles& t) {
    if (t.mode == 2) {
      nt += t.units;
    } else if (t.mode == 1) {
      if (++nt == t.ntiles) { nt = 0u; qt += t.units; }
    } else {
      nt += t.dn;
      qt += t.dq;
      if (qt >= t.qtiles) { qt -= t.qtiles; ++nt; }
    }
  }
};

struct TcArgs {
  int64_t nq;                 // queries (list positions)
  int64_t row_begin, row_end; // rows of this launch
  int32_t kblocks;            // dim16 / 64
  int32_t k16_last;           // K16 steps of the last K block that hold operand columns (the rest is padding); 0 = all 4
  int32_t stage_kblocks;      // K blocks per ring stage: 1 (four stages of 48 KB) or 2 (two stages of 96 KB: half the
                              // hand-overs between producer, MMA issuer and ring)
  int mode;                   // SCAN_DENSE or SCAN_THRESHOLD
  const float* alpha;         // value = alpha * acc + beta[row]: device scalar ...
  int32_t alpha_per_query;    // ... or [nq] by list position
  const float* beta;          // [n] or null (treated as 0)
  CandLists cand;
  int32_t cap;                // keys per candidate list (SCAN_THRESHOLD)
  unsigned long long* best;   // SCAN_ARGMIN: [nq] smallest (value, row) key, pre-set to all ones
  int32_t row_tile_fastest;   // tile order: 0 = query tile fastest (rows are the operand streamed once),
                              //             1 = row tile fastest (the "queries" are the operand streamed once)
  int32_t* err;               // device error word
  // Tile-table mode (IVF list scan): the launch walks an explicit list of tiles instead of the full
  // (query tile) x (row tile) grid, and the "query" operand holds one row per (query, probed list) pair, grouped
  // by list.  tiles[t] = {first pair, first row, valid rows | in-pilot-window << 30, valid pairs};
  // pair_info[p] = list position of the pair's query | remainder item << 31 (the rest of a query's nearest list
  // after the pilot window: such a pair skips the tiles inside the window).
  const int4* tiles;          // or null
  int64_t num_tiles;
  const uint32_t* pair_info;
  const float* pair_thr;      // [pairs] coarse threshold of the pair's query for this launch
  // Filter (HAS_MASK kernels): operand row r may be appended for query q iff (row_masks[r] & q_masks[q]) != 0.
  const uint64_t* row_masks;  // [rows of the row operand]
  const uint64_t* q_masks;    // [nq] by list position
  // Bounded waits: polls before a wait gives up (0 = WAIT_LIMIT).  stall_kblock >= 0 (testing only): the producer of
  // CTA 0 leaves out the copies of that k-block of its first tile, so that the consumer's wait for them runs out and
  // the time-out path (error word, abort flag, drain, tensor-memory release, VSK_ERR_TIMEOUT) can be exercised.
  uint32_t wait_limit;
  int32_t stall_kblock;
};


// The accumulator a value must reach to be a hit: alpha * acc <= thr with alpha < 0 holds for every acc >= thr / alpha;
// thr * (1 / alpha) and the product alpha * acc each differ from the exact quotient by a few units in the last place,
// so the bar is lowered by 2^-20 of its size (and a denormal's worth): no hit of the product form is lost.
__device__ __forceinline__ float as_bar(float thr, float inv_alpha) {
  const float b = thr * inv_alpha;
  return b - fabsf(b) * 9.5367431640625e-7f - 1e-37f;
}

// I8 (threshold mode, plain grid): both operands are 8-bit integers, 128 to a K block, and the accumulators exact 32-bit
// integers.  cand.thr then holds, as integer bits, the accumulator a row must reach; a listed key carries the row only
// (its value is formed by the re-scoring).
template <int MODE, bool HAS_BETA, bool HAS_MASK, int EW, bool I8 = false>
__global__ void __launch_bounds__(Epi<EW>::THREADS, 1)
tc_scan_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_x, TcArgs a) {
  extern __shared__ uint8_t smem_raw[];
  using TcSmem = TcSmemT<EW, HAS_BETA>;
  constexpr int EPI_WARPS = EW, EPI_COLS = Epi<EW>::COLS, EPI_GROUPS = Epi<EW>::GROUPS, EPI_PARTS = Epi<EW>::PARTS;
  TcSmem* sm = reinterpret_cast<TcSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t unit = blockIdx.x;
  const int64_t units = gridDim.x;
  constexpr int QT = TM;  // queries per tile
  constexpr int KCOLS = I8 ? 2 * TK : TK;   // operand columns of a K block (128 bytes)
  static_assert(!I8 || (MODE == SCAN_THRESHOLD && !HAS_BETA && !HAS_MASK), "integer operands: plain threshold scans only");
  const uint32_t wait_limit = a.wait_limit ? a.wait_limit : WAIT_LIMIT;
  const int kps = a.stage_kblocks == 2 ? 2 : 1;   // K blocks per ring stage
  const int nstages = STAGES / kps;

  const int64_t qtiles = (a.nq + QT - 1) / QT;
  const int64_t ntiles = (a.row_end - a.row_begin + TN - 1) / TN;
  const int64_t tiles = qtiles * ntiles;
  // The tiles of this unit.  Query-tile-fastest order interleaves units over the tile list (units that run
  // together read the same rows).  In row-tile-fastest order a unit OWNS whole query tiles and walks all their
  // row tiles in turn, so a query's running state (slot count, best key) stays in its thread's registers.
  TcTiles walk;
  walk.mode = a.tiles ? 2 : (a.row_tile_fastest ? 1 : 0);
  walk.units = (uint32_t)units;
  walk.qtiles = a.tiles ? 1u : (uint32_t)qtiles;
  walk.ntiles = a.tiles ? (uint32_t)a.num_tiles : (uint32_t)ntiles;
  walk.dn = walk.units / walk.qtiles;
  walk.dq = walk.units - walk.dn * walk.qtiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sm->full[s], 1);
      mbar_init(&sm->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm->tmem_full[b], 1);
      mbar_init(&sm->tmem_empty[b], EPI_WARPS);
    }
    mbar_init(&sm->drain, 1);
    sm->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sm->tmem_base;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      uint32_t issued = 0;       // bit s: a copy into stage s was issued ...
      uint32_t issued_ph = 0;    // ... with this full-barrier parity
      bool ok = true;
      // tile-table mode: the entry of the next tile is loaded while this tile's copies are issued, so that the
      // table look-up (a global load) is not on the producer's critical path
      int4 entry_next = make_int4(0, 0, 0, 0);
      if (a.tiles && unit < a.num_tiles) entry_next = __ldg(&a.tiles[unit]);
      TcWalk w;
      w.start(walk, blockIdx.x);
      for (bool first = true; ok && w.valid(walk); w.advance(walk), first = false) {
        const int64_t qt = w.qt, nt = w.nt;
        const int4 entry = entry_next;
        if (a.tiles && nt + units < a.num_tiles) entry_next = __ldg(&a.tiles[nt + units]);
        const int32_t qrow = a.tiles ? entry.x : (int32_t)(qt * QT);
        const int32_t xrow = a.tiles ? entry.y : (int32_t)(a.row_begin + nt * TN);
        for (int kb = 0; kb < a.kblocks; kb += kps) {
          if (!mbar_wait(&sm->empty[s], ph ^ 1, &sm->abort_flag, a.err, 1, wait_limit)) { ok = false; break; }
          uint8_t* st = sm->ring + s * kps * STAGE_BYTES;
          const int nkb = min(kps, a.kblocks - kb);
          if (a.stall_kblock >= 0 && unit == 0 && first && kb == a.stall_kblock) {
            // testing only: this stage is never filled, the consumer's bounded wait for it runs out
          } else {
            mbar_expect_tx(&sm->full[s], (uint32_t)(nkb * STAGE_BYTES));
            for (int j = 0; j < nkb; ++j) {
              tma_load_2d(st + j * STAGE_BYTES, &map_q, &sm->full[s], (kb + j) * KCOLS, qrow);
              tma_load_2d(st + j * STAGE_BYTES + A_BYTES, &map_x, &sm->full[s], (kb + j) * KCOLS, xrow);
            }
            issued |= 1u << s;
            issued_ph = (issued_ph & ~(1u << s)) | (ph << s);
          }
          if (++s == nstages) { s = 0; ph ^= 1; }
        }
      }
      // copies still in flight must land before the CTA's shared memory is released
      for (int i = 0; i < STAGES; ++i)
        if (issued & (1u << i)) {
          for (uint32_t it = 0; it < wait_limit; ++it) {
            if (mbar_try_wait(&sm->full[i], (issued_ph >> i) & 1)) break;
            __nanosleep(64);
          }
        }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // One lane, loop state in 32-bit registers, the number of tiles worked out once (the tile's coordinates, which
    // cost a 64-bit division per tile, are of no use to this role).  A converged warp with an elected lane and a
    // look-ahead at the next stage's barriers was measured 2 - 3 % slower here and is not used.
    if (lane == 0) {
      int64_t count;
      if (a.tiles) count = unit < a.num_tiles ? (a.num_tiles - unit + units - 1) / units : 0;
      else if (a.row_tile_fastest) count = unit < qtiles ? ((qtiles - unit + units - 1) / units) * ntiles : 0;
      else count = unit < tiles ? (tiles - unit + units - 1) / units : 0;
      const uint32_t ring_lo = desc_lo(smem_u32(sm->ring));
      const uint32_t full0 = smem_u32(&sm->full[0]), empty0 = smem_u32(&sm->empty[0]), tfull0 = smem_u32(&sm->tmem_full[0]);
      const int last_nk4 = a.k16_last > 0 ? a.k16_last : TK / 16;
      uint32_t s = 0, ph = 0, acc = 0, aph = 0;
      bool ok = true;
      for (int64_t left = count; ok && left > 0; --left) {
        if (!mbar_wait(&sm->tmem_empty[acc], aph ^ 1, &sm->abort_flag, a.err, 2, wait_limit)) { ok = false; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * (uint32_t)TN;
        for (int kb0 = 0; kb0 < a.kblocks; kb0 += kps) {
          if (!mbar_wait(&sm->full[s], ph, &sm->abort_flag, a.err, 3, wait_limit)) { ok = false; break; }
          tc_fence_after();
          const int nkb = min(kps, a.kblocks - kb0);
          for (int j = 0; j < nkb; ++j) {
            const int kb = kb0 + j;
            const uint32_t a_lo = ring_lo + (uint32_t)((s * kps + j) * (STAGE_BYTES >> 4));
            const uint32_t b_lo = a_lo + (uint32_t)(A_BYTES >> 4);
            const int nk4 = kb == a.kblocks - 1 ? last_nk4 : TK / 16;
#pragma unroll
            for (int k4 = 0; k4 < TK / 16; ++k4) {
              // 16 fp16 (32 int8) = 32 bytes further along K inside the swizzle atom: +2 in 16-byte units
              if (I8 && k4 < nk4)
                tc_mma_i8(tmem_d, desc_pack(a_lo + (uint32_t)(k4 * 2), kDescHi), desc_pack(b_lo + (uint32_t)(k4 * 2), kDescHi), kIdescI8,
                          (kb | k4) ? 1u : 0u);
              else if (k4 < nk4)
                tc_mma(tmem_d, desc_pack(a_lo + (uint32_t)(k4 * 2), kDescHi), desc_pack(b_lo + (uint32_t)(k4 * 2), kDescHi), kIdesc,
                       (kb | k4) ? 1u : 0u);
            }
          }
          tc_commit_a(empty0 + s * 8u);   // the stage is free once these MMAs have read it
          if (++s == (uint32_t)nstages) { s = 0; ph ^= 1u; }
        }
        if (ok) tc_commit_a(tfull0 + acc * 8u);
        aph = acc ? aph ^ 1u : aph;
        acc ^= 1u;
      }
      // all issued MMAs must retire before tensor memory is freed
      tc_commit(&sm->drain);
      for (uint32_t it = 0; it < wait_limit; ++it) {
        if (mbar_try_wait(&sm->drain, 0)) break;
        __nanosleep(64);
      }
    }
  } else {
    // ---------------- epilogue: one query per thread, a part of the tile's columns per warp ----------------
    const int quarter = warp & 3;                 // tensor-memory lanes this warp may read
    const int et = quarter * 32 + lane;           // row of the tile owned by this thread
    const int ew = warp - 2;                      // epilogue warp 0..
    const int part = ew >> 2;                     // which part of the tile's columns this warp takes
    const int c0 = part * EPI_GROUPS;             // first 32-column group of that part
    const float alpha0 = a.alpha_per_query ? -1.0f : __ldg(a.alpha);
    const bool owned = a.row_tile_fastest != 0;
    const int32_t row_begin = (int32_t)a.row_begin, row_end_all = (int32_t)a.row_end;   // (an index holds fewer than 2^31 rows)
    bool ok = true;
    int run_cnt = 0;                 // row-tile-fastest order: keys this thread has stored for its query so far
    float run_bv = CUDART_INF_F;     // ... and its best value / row so far (SCAN_ARGMIN)
    int64_t run_bn = 0;
    // What a lane needs to know of a tile before it can look at its values - the tile's entry and the pair behind it in
    // tile-table mode, the query's threshold and coefficient - are dependent global loads.  They are pipelined over the
    // tiles: the entry is loaded two tiles ahead, the rest one tile ahead, so that none is waited for (with short
    // contractions the epilogue, not the MMA, sets the pace).  pair_info / pair_thr are padded by one tile, so the loads
    // need no bounds test.
    struct Ahead {
      int4 e;
      uint32_t info;
      float thr, alpha;
      bool qok;
    };
    TcWalk w, wn;   // this tile and the next
    w.start(walk, blockIdx.x);
    wn = w;
    auto entry_of = [&](const TcWalk& t) { return (a.tiles && t.valid(walk)) ? __ldg(&a.tiles[t.nt]) : make_int4(0, 0, 0, 0); };
    auto look_ahead = [&](const TcWalk& t, const int4& e) {
      Ahead h{e, 0u, -CUDART_INF_F, alpha0, false};
      if (a.tiles) {
        h.info = __ldg(a.pair_info + e.x + et);
        if (MODE == SCAN_THRESHOLD || MODE == SCAN_ALL) h.thr = __ldg(a.pair_thr + e.x + et);
        h.qok = et < e.w;
      } else if (t.valid(walk)) {
        const int64_t q = (int64_t)t.qt * QT + et;
        h.qok = q < a.nq;
        if (MODE == SCAN_THRESHOLD && h.qok) h.thr = __ldg(a.cand.thr + q);
        if (a.alpha_per_query && h.qok) h.alpha = __ldg(a.alpha + q);
      }
      return h;
    };
    Ahead ahead = look_ahead(w, entry_of(w));
    wn.advance(walk);
    int4 entry_next = entry_of(wn);
    // Hits wait in the lane's queue while their slots are reserved (the atomic's round trip is not waited for): they go to
    // the lists when the next tile's values are on their way from tensor memory, or when a queue is full.
    constexpr int QCAP = kTcQueue;
    uint2(*queue)[32] = sm->queue[ew];
    int pend_cnt = 0, pend_base = 0;
    int32_t pend_q = 0;
    uint32_t pend_row = 0u;
    float pend_alpha = alpha0;
    const int cap_here = owned ? a.cap / EPI_PARTS : a.cap;
    auto flush = [&]() {
      if (MODE != SCAN_THRESHOLD || !__any_sync(0xffffffffu, pend_cnt != 0)) return;
      uint64_t* dst = a.cand.keys + (int64_t)pend_q * a.cap + (owned ? part * cap_here : 0) + pend_base;
      const int n = min(pend_cnt, cap_here - pend_base);
      for (int e = 0; __any_sync(0xffffffffu, e < pend_cnt); ++e) {
        const uint2 h = queue[e][lane];
        const float x = __uint_as_float(h.x);
        if (e < n) *VSK_CHK_W(dst + e) = make_key(I8 ? 0.f : HAS_BETA ? -x : x * pend_alpha, pend_row + h.y);
      }
      __syncwarp();
      pend_cnt = 0;
    };
    uint32_t local = 0;
    for (; ok && w.valid(walk); w = wn, wn.advance(walk), ++local) {
      const int acc = (int)(local & 1);
      const uint32_t aph = (local >> 1) & 1u;
      const Ahead cur = ahead;
      ahead = look_ahead(wn, entry_next);
      if (a.tiles) {
        TcWalk w2 = wn;
        w2.advance(walk);
        entry_next = entry_of(w2);
      }
      int32_t q = (int32_t)(w.qt * (uint32_t)QT) + et;
      if (owned && w.nt == 0u) { run_cnt = 0; run_bv = CUDART_INF_F; run_bn = 0; }
      int32_t n0 = row_begin + (int32_t)(w.nt * (uint32_t)TN);
      int32_t row_end = row_end_all;
      const bool qok = cur.qok;
      const float alpha = cur.alpha;
      float thr = cur.thr;
      if (a.tiles) {
        n0 = cur.e.y;
        row_end = cur.e.y + (cur.e.z & 0x3fffffff);
        q = (int32_t)(cur.info & 0x7fffffffu);
        // a remainder item (the rest of a query's nearest list) skips the tiles inside the pilot window
        if ((cur.info >> 31) != 0u && ((cur.e.z >> 30) & 1) != 0) thr = -CUDART_INF_F;
      }
      // The tile's per-row terms; each warp stages its own copy, so no CTA-wide barrier is needed.  The first tile
      // loads them directly; after that they are fetched one tile ahead into registers (the loads fly while this
      // tile is processed) and stored to the other buffer at the end of the iteration.
      float beta_next[EPI_COLS / 32];
      if (HAS_BETA) {
        if (local == 0) {
          for (int i = lane; i < EPI_COLS; i += 32)
            sm->beta[HAS_BETA ? acc : 0][HAS_BETA ? ew : 0][i] = (n0 + c0 * 32 + i < row_end) ? __ldg(a.beta + n0 + c0 * 32 + i) : 0.f;
          __syncwarp();
        }
        int32_t nn0 = 0, nrow_end = 0;
        if (wn.valid(walk)) {
          if (a.tiles) { nn0 = ahead.e.y; nrow_end = ahead.e.y + (ahead.e.z & 0x3fffffff); }
          else { nn0 = row_begin + (int32_t)(wn.nt * (uint32_t)TN); nrow_end = row_end_all; }
        }
#pragma unroll
        for (int i = 0; i < EPI_COLS / 32; ++i) {
          const int32_t r = nn0 + c0 * 32 + lane + 32 * i;
          beta_next[i] = r < nrow_end ? __ldg(a.beta + r) : 0.f;
        }
      }
      uint64_t qm = 0ull;   // this query's filter mask: a row is eligible iff (row mask & qm) != 0
      uint64_t rmask[EPI_GROUPS];   // the masks of the warp's columns lane, lane + 32, ..
      if (HAS_MASK) {
        if (qok) qm = __ldg(a.q_masks + q);
        if (MODE == SCAN_THRESHOLD || MODE == SCAN_ALL) {
#pragma unroll
          for (int g = 0; g < EPI_GROUPS; ++g) {
            const int32_t r = n0 + (c0 + g) * 32 + lane;
            rmask[g] = r < row_end ? __ldg(a.row_masks + r) : 0ull;
          }
        }
      }
      // SCAN_ALL: which columns are listed does not depend on their values, so their slots are asked for before the wait
      uint32_t all_bits[EPI_GROUPS];
      int all_base = 0;
      if constexpr (MODE == SCAN_ALL) {
        int n = 0;
#pragma unroll
        for (int g = 0; g < EPI_GROUPS; ++g) {
          const int left = row_end - (n0 + (c0 + g) * 32);
          uint32_t bits = left >= 32 ? 0xffffffffu : (left > 0 ? (1u << left) - 1u : 0u);
          if (!qok || !(thr > -CUDART_INF_F)) bits = 0u;
          if (HAS_MASK) {
            for (int j = 0; j < 32; ++j) {
              const uint64_t m = __shfl_sync(0xffffffffu, rmask[g], j);
              if ((m & qm) == 0ull) bits &= ~(1u << j);
            }
          }
          all_bits[g] = bits;
          n += __popc(bits);
        }
        if (n) all_base = atomicAdd(&a.cand.count[q], n);
      }
      // every lane of the warp must take part in the wait result
      bool got = mbar_wait(&sm->tmem_full[acc], aph, &sm->abort_flag, a.err, 4, wait_limit);
      got = __all_sync(0xffffffffu, got);
      if (!got) { ok = false; break; }
      tc_fence_after();
      const uint32_t trow = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * TN);
      if (MODE == SCAN_DENSE) {
        // Eight columns at a time through shared memory: stored by their own lanes, the keys of 32 queries would go to 32
        // different lines per instruction, which bound this epilogue; turned around, eight lanes store 64 bytes of one query.
        uint64_t* buf = reinterpret_cast<uint64_t*>(&queue[0][0]);
        constexpr int W = 8;   // columns per turn
        static_assert(QCAP * sizeof(uint2) >= W * sizeof(uint64_t), "room for the turned keys");
#pragma unroll 1
        for (int c = c0; c < c0 + EPI_GROUPS; ++c) {
          float v[32];
          tc_ld32(trow + (uint32_t)(c * 32), v);
          const int32_t nc = n0 + c * 32;
#pragma unroll
          for (int t = 0; t < 32 / W; ++t) {
#pragma unroll
            for (int j = 0; j < W; ++j) {
              const int col = t * W + j;
              const float val = HAS_BETA ? fmaf(v[col], alpha, sm->beta[HAS_BETA ? acc : 0][HAS_BETA ? ew : 0][(c - c0) * 32 + col]) : v[col] * alpha;
              uint64_t key = make_key(val, (uint32_t)(nc + col));
              // the same row mask for every lane (a broadcast load); an ineligible row leaves an empty slot
              if (HAS_MASK && nc + col < row_end && (__ldg(a.row_masks + nc + col) & qm) == 0ull) key = kEmptyKey;
              buf[lane * W + (j ^ (lane & (W - 1)))] = key;
            }
            __syncwarp();
#pragma unroll
            for (int r0 = 0; r0 < 32; r0 += 32 / W) {
              const int r = r0 + lane / W, j = lane & (W - 1);
              const int32_t qr = q - lane + r, row = nc + t * W + j;
              if (qr < a.nq && row < row_end)
                *VSK_CHK_W(a.cand.keys + (int64_t)qr * kCandCap + (row - row_begin)) = buf[r * W + (j ^ (r & (W - 1)))];
            }
            __syncwarp();
          }
        }
      } else if (MODE == SCAN_ARGMIN) {
        // smallest (value, row) key of this query over the tile's 256 rows, merged into best[q]
        float bv = CUDART_INF_F;
        int bj = 0;
#pragma unroll 1
        for (int c = c0; c < c0 + EPI_GROUPS; ++c) {
          float v[32];
          tc_ld32(trow + (uint32_t)(c * 32), v);
          const int left = row_end - (n0 + c * 32);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float val = HAS_BETA ? fmaf(v[j], alpha, sm->beta[HAS_BETA ? acc : 0][HAS_BETA ? ew : 0][(c - c0) * 32 + j]) : v[j] * alpha;
            if (j < left && val < bv) { bv = val; bj = c * 32 + j; }   // strict '<': the lowest row wins ties
          }
        }
        if (owned) {
          if (bv < run_bv) { run_bv = bv; run_bn = n0 + bj; }   // row tiles come in ascending order: '<' keeps the lowest row
          if (w.nt == walk.ntiles - 1u && qok && run_bv < CUDART_INF_F)
            atomicMin(a.best + q, (unsigned long long)make_key(run_bv, (uint32_t)run_bn));
        } else if (qok && bv < CUDART_INF_F) {
          atomicMin(a.best + q, (unsigned long long)make_key(bv, (uint32_t)(n0 + bj)));
        }
      } else {
        // alpha < 0 and a power of two (but for the per-row term): value <= threshold is accumulator >= threshold / alpha, so a
        // value that is not listed costs one instruction, the running maximum of its eight columns.  The accumulator goes back
        // as soon as its last columns are in registers.  Only eights in which some lane has a hit are looked at one by one.
        const float bar = I8 ? (qok ? thr : __int_as_float(0x7fffffff)) : !qok ? CUDART_INF_F : HAS_BETA ? -thr : as_bar(thr, 1.0f / alpha);
        auto reaches = [&](float v, float b) { return I8 ? __float_as_int(v) >= __float_as_int(b) : v >= b; };
        int cnt = 0;          // hits in the queue
        int tile_cnt = 0;     // ... and of the tile in all (owned order)
        const uint32_t row0 = (uint32_t)(n0 + c0 * 32);
        // the queue's hits: those the filter lets through stay, and their slots are asked for
        auto reserve = [&]() {
          if (HAS_MASK) {
            int kept = 0;
            for (int e = 0; __any_sync(0xffffffffu, e < cnt); ++e) {
              const uint2 h = queue[e][lane];
              uint64_t m = 0ull;
#pragma unroll
              for (int g = 0; g < EPI_GROUPS; ++g) {
                const uint64_t x = __shfl_sync(0xffffffffu, rmask[g], h.y & 31u);
                if ((h.y >> 5) == (uint32_t)g) m = x;
              }
              if (e < cnt && (m & qm) != 0ull) queue[kept++][lane] = h;
            }
            cnt = kept;
          }
          pend_cnt = cnt;
          pend_q = q;
          pend_row = row0;
          pend_alpha = alpha;
          pend_base = owned ? run_cnt + tile_cnt : (cnt ? atomicAdd(&a.cand.count[q], cnt) : 0);
          tile_cnt += cnt;
          cnt = 0;
        };
        if constexpr (MODE == SCAN_ALL) {
          // the keys turned around as in the dense mode
          constexpr int W = 8;
          uint64_t* buf = reinterpret_cast<uint64_t*>(&queue[0][0]);
          int base = all_base;
#pragma unroll
          for (int h = 0; h < EPI_GROUPS; ++h) {
            const uint32_t bits = all_bits[h];
            const uint32_t who = __ballot_sync(0xffffffffu, bits != 0u);   // (lists are short of a tile's 128 pairs as a rule)
            if (who == 0u) continue;
            float v[32];
            tc_ld32(trow + (uint32_t)((c0 + h) * 32), v);
#pragma unroll
            for (int t = 0; t < 32 / W; ++t) {
#pragma unroll
              for (int j = 0; j < W; ++j) {
                const int col = t * W + j;
                const float val = HAS_BETA ? fmaf(v[col], alpha, sm->beta[HAS_BETA ? acc : 0][HAS_BETA ? ew : 0][h * 32 + col]) : v[col] * alpha;
                buf[lane * W + (j ^ (lane & (W - 1)))] = make_key(I8 ? 0.f : val, row0 + (uint32_t)(h * 32 + col));
              }
              __syncwarp();
#pragma unroll
              for (int r0 = 0; r0 < 32; r0 += 32 / W) {
                if (((who >> r0) & ((1u << (32 / W)) - 1u)) == 0u) continue;
                const int r = r0 + lane / W, j = lane & (W - 1), col = t * W + j;
                const uint32_t rb = __shfl_sync(0xffffffffu, bits, r);
                const int at = __shfl_sync(0xffffffffu, base, r) + __popc(rb & ((1u << col) - 1u));
                const int32_t qr = __shfl_sync(0xffffffffu, q, r);
                if (((rb >> col) & 1u) != 0u && at < a.cap) *VSK_CHK_W(a.cand.keys + (int64_t)qr * a.cap + at) = buf[r * W + (j ^ (r & (W - 1)))];
              }
              __syncwarp();
            }
            base += __popc(bits);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm->tmem_empty[acc]);
        } else {
#pragma unroll 1
        for (int h = 0; h < EPI_GROUPS; ++h) {   // 32 columns at a time
          float v[32];
          tc_ld32_issue(trow + (uint32_t)((c0 + h) * 32), v);
          if (h == 0) flush();   // the last tile's hits
          tc_ld_wait();
          if (h + 1 == EPI_GROUPS) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm->tmem_empty[acc]);
          }
          if (HAS_BETA) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = -fmaf(v[j], alpha, sm->beta[HAS_BETA ? acc : 0][HAS_BETA ? ew : 0][h * 32 + j]);
          }
          const int left = row_end - (n0 + (c0 + h) * 32);   // columns inside the launch (tile)
          float top[4];
#pragma unroll
          for (int o = 0; o < 4; ++o) {
            const float* x = &v[o * 8];
            if constexpr (I8) {
              int t = __float_as_int(x[0]);
#pragma unroll
              for (int j = 1; j < 8; ++j) t = max(t, __float_as_int(x[j]));
              top[o] = __int_as_float(t);
            } else {
              top[o] = max3(x[6], x[7], fmaxf(max3(x[0], x[1], x[2]), max3(x[3], x[4], x[5])));
            }
          }
          if (!__any_sync(0xffffffffu, reaches(top[0], bar) || reaches(top[1], bar) || reaches(top[2], bar) || reaches(top[3], bar))) continue;
          uint32_t todo = 0u;   // fours of columns to be looked at, the same in every lane
#pragma unroll
          for (int o = 0; o < 4; ++o) todo |= __any_sync(0xffffffffu, reaches(top[o], bar)) ? 3u << (2 * o) : 0u;
          const uint32_t col0 = (uint32_t)(h * 32);
          while (todo != 0u) {
            bool full = false;
#pragma unroll
            for (int f = 0; f < 8; ++f) {
              if (((todo >> f) & 1u) == 0u || full) continue;
              full = __any_sync(0xffffffffu, cnt > QCAP - 4);
              if (full) continue;
              todo &= ~(1u << f);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float x = v[f * 4 + j];
                if (reaches(x, bar) && f * 4 + j < left) {
                  queue[cnt][lane] = make_uint2(__float_as_uint(x), col0 + (uint32_t)(f * 4 + j));
                  ++cnt;
                }
              }
            }
            if (full) {   // a queue without room: the hits so far go to their lists first
              __syncwarp();
              reserve();
              flush();
            }
          }
        }
        __syncwarp();
        reserve();
        }
        if (MODE == SCAN_THRESHOLD && owned) {
          run_cnt += tile_cnt;
          if (w.nt == walk.ntiles - 1u && qok)
            reinterpret_cast<unsigned char*>(a.cand.count)[(int64_t)q * 4 + part] = (unsigned char)min(run_cnt, 255);
        }
      }
      if (HAS_BETA) {
#pragma unroll
        for (int i = 0; i < EPI_COLS / 32; ++i) sm->beta[HAS_BETA ? acc ^ 1 : 0][HAS_BETA ? ew : 0][lane + 32 * i] = beta_next[i];
      }
      if (MODE == SCAN_DENSE || MODE == SCAN_ARGMIN) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm->tmem_empty[acc]);
      } else if (HAS_BETA) {
        __syncwarp();
      }
    }
    flush();
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ---- nearest-centroid assignment with a STATIONARY centroid block ---------------------------------------
// k-means assignment is a contraction of 10^7 data rows against a few thousand centroids with a short inner
// dimension (d = 128: two or three 64-wide k-blocks).  In the general kernel every 128 x 256 tile re-fetches both
// operands from L2 - 96 KB for 8 Mflop - and at that ratio the L2 -> shared-memory fill, not the tensor pipe, sets the
// pace (measured: 1.44 us per tile against 0.53 us of MMAs).  Here a CTA keeps one block of 256 centroids (all its
// k-blocks, up to 128 KB) resident in shared memory and streams 128-row data tiles past it: 16 KB per k-block and
// tile, a third of the traffic (a sixth with the row term folded in), so the MMAs set the pace again.
//   grid      blocks of 256 centroids x groups of CTAs; CTA (b, g) holds centroid block b and takes data tiles
//             g, g + groups, ...  (more blocks than SMs: a CTA takes several blocks in turn)
//   warp 0    TMA producer: the centroid block once, then the data tiles through a ring whose stage holds a whole
//             data tile (a K block where a tile is too large for two such stages); fold columns that begin a K block
//             of their own travel as a 16-column tile
//   warp 1    tcgen05.mma issuer: per data tile M128 N256 K16 x 4 per k-block against the resident block; it looks at
//             the next tile's barriers while this tile's last MMAs are still to be issued
//   warps 2.. epilogue (16 warps): the centroid's |c|^2 / 2 rides inside the contraction (fold columns), so a value
//             is alpha * accumulator and "no hit in these eight columns" is their largest accumulator against a bar.
//             Threshold mode: a hit (rare: the threshold is the row's previous assignment plus the error band)
//             is logged as {row, centroid} in the CTA's own stretch of a log, its slot taken from a shared-memory
//             counter; arg-min mode (first iteration): one atomicMin per row, centroid block and column part.
// Every mbarrier wait is bounded like the general kernel's.
constexpr int AS_EW = 16;
constexpr int AS_THREADS = 64 + 32 * AS_EW;
constexpr int AS_MAX_KB = 4;                       // k-blocks of the resident block (d + 16 fold columns <= 256)
constexpr int AS_RING_BYTES = 216 * 1024;          // resident block + data-tile stages
constexpr int AS_MAX_STAGES = 8;
// The 16-column fold tile is only loaded and issued in whole-tile stages: two such stages must fit beside the largest
// resident block that has one (the condition is tightest at the largest number of K blocks).
static_assert(2 * ((AS_MAX_KB - 1) * A_BYTES + A_NARROW_BYTES) <= AS_RING_BYTES - ((AS_MAX_KB - 1) * B_BYTES + B_NARROW_BYTES),
              "a 16-column fold tile implies whole-tile stages");

struct AsSmem {
  uint8_t ring[AS_RING_BYTES];   // [kblocks x 32 KB centroid block][stages x 16 KB data k-blocks]
  uint64_t a_full[AS_MAX_STAGES];
  uint64_t a_empty[AS_MAX_STAGES];
  uint64_t b_full, b_empty;
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint64_t drain;
  uint32_t tmem_base;
  volatile int abort_flag;
  int log_n;                     // hits this CTA has logged so far
};
constexpr size_t kAsSmemBytes = sizeof(AsSmem) + 1024;

struct AsArgs {
  int64_t n;                  // data rows
  int32_t k;                  // centroids
  int32_t kblocks;            // dim16 / 64, <= AS_MAX_KB
  int32_t k16_last;           // K16 steps of the last K block that hold operand columns; 0 = all 4
  int32_t max_stages;         // measurement: cap on the data-tile stages (0 = as many as fit)
  int32_t narrow_ok;          // the two 16-column tensor maps are valid (see `narrow` in the kernel)
  int32_t groups;             // CTAs per centroid block (1 when there are more blocks than CTAs)
  const float* alpha;         // value = alpha * accumulator = |c|^2 - 2 x.c
  const float* thr;           // [n] SCAN_THRESHOLD: a centroid is listed for a row iff value <= thr[row]
  // SCAN_THRESHOLD: every hit is logged as {row, centroid} in this CTA's own stretch of the log; the slot comes from a
  // shared-memory counter, so an append never waits for a round trip to L2 (with 32 rows x 64 columns per warp and
  // step, half of the steps hold a hit somewhere: a global atomic per hit made the epilogue wait out its latency)
  uint2* log;                 // [gridDim.x][log_cap]
  int32_t* log_count;         // [gridDim.x] entries written (capped); a CTA that ran out of room raises err = 9
  int64_t log_cap;            // entries per CTA = log_total / gridDim.x (set at launch)
  int64_t log_total;
  unsigned* best_value;       // [n] SCAN_ARGMIN: smallest value (float_to_ordered), pre-set to all ones
  int32_t* err;
  uint32_t wait_limit;
};

template <int MODE>
__global__ void __launch_bounds__(AS_THREADS, 1)
assign_scan_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_c,
                   const __grid_constant__ CUtensorMap map_xn, const __grid_constant__ CUtensorMap map_cn, AsArgs a) {
  extern __shared__ uint8_t smem_raw[];
  AsSmem* sm = reinterpret_cast<AsSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t wait_limit = a.wait_limit ? a.wait_limit : WAIT_LIMIT;
  const int nb = (a.k + TN - 1) / TN;                       // centroid blocks
  const int64_t qtiles = (a.n + TM - 1) / TM;               // data tiles
  // When only the first K16 step of the last K block holds operand columns (d a multiple of 64: the 16 fold columns
  // start a block of their own), that block is fetched and kept as a 16-column tile (32-byte swizzle: 4 KB of a data
  // tile, 8 KB of the centroid block) instead of 64 columns of which 48 are zeros: a quarter less to fetch per data
  // tile at d = 128, and room for four whole-tile stages instead of two.
  const bool narrow = a.narrow_ok != 0 && a.max_stages == 0 && a.k16_last == 1 && a.kblocks >= 2;
  const int nfull = narrow ? a.kblocks - 1 : a.kblocks;   // K blocks held as 64-column tiles
  const int bres_bytes = nfull * B_BYTES + (narrow ? B_NARROW_BYTES : 0);
  const int tile_bytes = nfull * A_BYTES + (narrow ? A_NARROW_BYTES : 0);
  // A stage of the data ring holds ALL K blocks of a data tile when two such stages fit (one wait, one batch of MMAs
  // and one commit per tile instead of per K block); otherwise, or when max_stages asks for it, one K block.
  const int skb = (a.max_stages == 0 && 2 * tile_bytes <= AS_RING_BYTES - bres_bytes) ? a.kblocks : 1;
  const int stage_bytes = skb == a.kblocks ? tile_bytes : A_BYTES;
  int stages = min(AS_MAX_STAGES, (AS_RING_BYTES - bres_bytes) / stage_bytes);
  if (a.max_stages > 0) stages = max(2, min(stages, a.max_stages));
  // this CTA's centroid blocks and its share of the data tiles
  const bool one_block = a.groups >= 1 && nb <= (int)gridDim.x;
  const int b_first = one_block ? (int)(blockIdx.x % nb) : (int)blockIdx.x;
  const int b_step = one_block ? (1 << 30) : (int)gridDim.x;
  const int64_t t_first = one_block ? (int64_t)(blockIdx.x / nb) : 0;
  const int64_t t_step = one_block ? a.groups : 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < AS_MAX_STAGES; ++s) {
      mbar_init(&sm->a_full[s], 1);
      mbar_init(&sm->a_empty[s], 1);
    }
    mbar_init(&sm->b_full, 1);
    mbar_init(&sm->b_empty, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm->tmem_full[b], 1);
      mbar_init(&sm->tmem_empty[b], AS_EW);
    }
    mbar_init(&sm->drain, 1);
    sm->abort_flag = 0;
    sm->log_n = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sm->tmem_base;
  uint8_t* a_ring = sm->ring + bres_bytes;
  uint2* my_log = MODE == SCAN_THRESHOLD ? a.log + (int64_t)blockIdx.x * a.log_cap : nullptr;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0, bph = 0;
      uint32_t issued = 0, issued_ph = 0;
      bool b_issued = false;
      uint32_t b_issued_ph = 0;
      bool ok = true;
      for (int b = b_first; ok && b < nb; b += b_step) {
        // the resident block may be replaced once every MMA that read the previous one has retired
        if (!mbar_wait(&sm->b_empty, bph ^ 1, &sm->abort_flag, a.err, 5, wait_limit)) { ok = false; break; }
        mbar_expect_tx(&sm->b_full, (uint32_t)bres_bytes);
        for (int kb = 0; kb < nfull; ++kb) tma_load_2d(sm->ring + kb * B_BYTES, &map_c, &sm->b_full, kb * TK, b * TN);
        if (narrow) tma_load_2d(sm->ring + nfull * B_BYTES, &map_cn, &sm->b_full, nfull * TK, b * TN);
        b_issued = true;
        b_issued_ph = bph;
        bph ^= 1;
        for (int64_t t = t_first; ok && t < qtiles; t += t_step) {
          for (int kb = 0; kb < a.kblocks; kb += skb) {
            if (!mbar_wait(&sm->a_empty[s], ph ^ 1, &sm->abort_flag, a.err, 1, wait_limit)) { ok = false; break; }
            mbar_expect_tx(&sm->a_full[s], (uint32_t)stage_bytes);
            const int nj = skb == a.kblocks ? nfull : 1;
            for (int j = 0; j < nj; ++j)
              tma_load_2d(a_ring + s * stage_bytes + j * A_BYTES, &map_x, &sm->a_full[s], (kb + j) * TK, (int32_t)(t * TM));
            if (narrow) tma_load_2d(a_ring + s * stage_bytes + nfull * A_BYTES, &map_xn, &sm->a_full[s], nfull * TK, (int32_t)(t * TM));
            issued |= 1u << s;
            issued_ph = (issued_ph & ~(1u << s)) | (ph << s);
            if (++s == stages) { s = 0; ph ^= 1; }
          }
        }
      }
      // copies still in flight must land before the CTA's shared memory is released
      if (b_issued)
        for (uint32_t it = 0; it < wait_limit; ++it) {
          if (mbar_try_wait(&sm->b_full, b_issued_ph)) break;
          __nanosleep(64);
        }
      for (int i = 0; i < stages; ++i)
        if (issued & (1u << i))
          for (uint32_t it = 0; it < wait_limit; ++it) {
            if (mbar_try_wait(&sm->a_full[i], (issued_ph >> i) & 1)) break;
            __nanosleep(64);
          }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // Measured with clock stamps in this warp: an M128 N256 K16 MMA executes in 128 cycles and the pipe queues only a
    // few, so the nine MMAs of a d = 128 tile are issued over about 1 250 cycles, and every cycle this warp then spends
    // before the next tile's first MMA (commits, loop, two barrier waits of 200 - 250 cycles each even when the barrier
    // has long completed) is a cycle the pipe idles: 2 130 cycles per tile at first, 1 152 of them MMA execution.
    if (skb == a.kblocks) {
      // A whole data tile per ring stage (the usual case): one lane, all loop state in 32-bit registers.  What this
      // thread executes between the last MMA of a tile and the first of the next is time the tensor pipe idles once
      // its short queue has drained, so the barriers of the next tile are looked at (one test, never a wait) while
      // this tile's last MMAs are still to be issued, and nothing is recomputed that can be carried along.
      if (lane == 0) {
        const uint32_t a_lo0 = desc_lo(smem_u32(a_ring)), stage_lo = (uint32_t)stage_bytes >> 4;
        uint32_t b_lo[AS_MAX_KB];
#pragma unroll
        for (int kb = 0; kb < AS_MAX_KB; ++kb) b_lo[kb] = desc_lo(smem_u32(sm->ring + kb * B_BYTES));
        const uint32_t bn_lo = desc_lo(smem_u32(sm->ring + nfull * B_BYTES));
        const uint32_t full0 = smem_u32(&sm->a_full[0]), empty0 = smem_u32(&sm->a_empty[0]);
        const uint32_t tfull0 = smem_u32(&sm->tmem_full[0]), tempty0 = smem_u32(&sm->tmem_empty[0]);
        const int last_nk4 = (!narrow && a.k16_last > 0) ? a.k16_last : TK / 16;   // MMAs of the last 64-column block
        const int32_t tiles_cta = t_first < qtiles ? (int32_t)((qtiles - t_first + t_step - 1) / t_step) : 0;
        uint32_t s = 0, ph = 0, bph = 0, acc = 0, aph = 0;
        bool ok = true, pre_acc = false, pre_stage = false;
        for (int b = b_first; ok && b < nb; b += b_step) {
          if (!mbar_wait(&sm->b_full, bph, &sm->abort_flag, a.err, 6, wait_limit)) { ok = false; break; }
          bph ^= 1;
          for (int32_t left = tiles_cta; left > 0; --left) {
            if (!pre_acc && !mbar_wait(&sm->tmem_empty[acc], aph ^ 1, &sm->abort_flag, a.err, 2, wait_limit)) { ok = false; break; }
            if (!pre_stage && !mbar_wait(&sm->a_full[s], ph, &sm->abort_flag, a.err, 3, wait_limit)) { ok = false; break; }
            tc_fence_after();
            const uint32_t tmem_d = tmem_base + acc * (uint32_t)TN;
            const uint32_t a_lo = a_lo0 + s * stage_lo;
            const uint32_t ns = s + 1 == (uint32_t)stages ? 0u : s + 1;
            const uint32_t nph = s + 1 == (uint32_t)stages ? ph ^ 1u : ph;
            const uint32_t naph = acc ? aph ^ 1u : aph;   // the other accumulator's use count flips parity every second tile
            const bool more = left > 1;                   // the next tile belongs to this centroid block
            pre_acc = false;
            pre_stage = false;
#pragma unroll
            for (int kb = 0; kb < AS_MAX_KB; ++kb) {
              if (kb < nfull) {
                if (kb == nfull - 1 && more) {
                  pre_stage = mbar_test_wait_a(full0 + ns * 8u, nph);
                  pre_acc = mbar_test_wait_a(tempty0 + (acc ^ 1u) * 8u, naph ^ 1u);
                }
                const int nk4 = kb == nfull - 1 ? last_nk4 : TK / 16;
#pragma unroll
                for (int k4 = 0; k4 < TK / 16; ++k4)
                  if (k4 < nk4)
                    tc_mma(tmem_d, desc_pack(a_lo + (uint32_t)(kb * (A_BYTES >> 4) + k4 * 2), kDescHi),
                           desc_pack(b_lo[kb] + (uint32_t)(k4 * 2), kDescHi), kIdesc, (kb | k4) ? 1u : 0u);
              }
            }
            if (narrow) {
              // a second look for what the first one came too early for
              if (more && !pre_stage) pre_stage = mbar_test_wait_a(full0 + ns * 8u, nph);
              if (more && !pre_acc) pre_acc = mbar_test_wait_a(tempty0 + (acc ^ 1u) * 8u, naph ^ 1u);
              tc_mma(tmem_d, desc_pack(a_lo + (uint32_t)(nfull * (A_BYTES >> 4)), kDescHiNarrow), desc_pack(bn_lo, kDescHiNarrow), kIdesc, 1u);
            }
            tc_commit_a(empty0 + s * 8u);
            tc_commit_a(tfull0 + acc * 8u);
            s = ns;
            ph = nph;
            aph = naph;
            acc ^= 1u;
          }
          if (ok) tc_commit(&sm->b_empty);   // arrives when every MMA issued so far (all readers of this block) has retired
        }
        tc_commit(&sm->drain);
        for (uint32_t it = 0; it < wait_limit; ++it) {
          if (mbar_try_wait(&sm->drain, 0)) break;
          __nanosleep(64);
        }
      }
      __syncwarp();
    } else {
      // One K block per ring stage (long rows, or a stage cap set for measurement): the whole warp runs the loop
      // converged and one elected lane issues; the same look-ahead, per stage.
      int s = 0;
      uint32_t ph = 0, bph = 0;
      int64_t local = 0;
      bool ok = true;
      bool pre_acc = false, pre_stage = false;
      for (int b = b_first; ok && b < nb; b += b_step) {
        if (!__all_sync(0xffffffffu, mbar_wait(&sm->b_full, bph, &sm->abort_flag, a.err, 6, wait_limit))) { ok = false; break; }
        bph ^= 1;
        tc_fence_after();
        for (int64_t t = t_first; ok && t < qtiles; t += t_step, ++local) {
          const int acc = (int)(local & 1);
          const uint32_t aph = (uint32_t)((local >> 1) & 1);
          if (!pre_acc && !__all_sync(0xffffffffu, mbar_wait(&sm->tmem_empty[acc], aph ^ 1, &sm->abort_flag, a.err, 2, wait_limit))) { ok = false; break; }
          pre_acc = false;
          const uint32_t tmem_d = tmem_base + (uint32_t)(acc * TN);
          for (int kb0 = 0; kb0 < a.kblocks; kb0 += skb) {
            if (!pre_stage && !__all_sync(0xffffffffu, mbar_wait(&sm->a_full[s], ph, &sm->abort_flag, a.err, 3, wait_limit))) { ok = false; break; }
            pre_stage = false;
            tc_fence_after();
            // The barriers of the NEXT step are looked at (one test, never a wait) before the last MMAs of this step are
            // issued, while the tensor pipe still has work queued: what is seen complete there is not waited for again,
            // so the next step's MMAs follow without the pipe running dry over two barrier waits.
            const bool tile_ends = kb0 + skb >= a.kblocks;
            const int ns = s + 1 == stages ? 0 : s + 1;
            const uint32_t nph = s + 1 == stages ? ph ^ 1 : ph;
            const bool more = !tile_ends || t + t_step < qtiles;   // the next step belongs to this centroid block
            const int nj = skb == a.kblocks ? nfull : 1;
            for (int j = 0; j < nj; ++j) {
              const int kb = kb0 + j;
              const uint64_t adesc = make_desc(smem_u32(a_ring + s * stage_bytes + j * A_BYTES));
              const uint64_t bdesc = make_desc(smem_u32(sm->ring + kb * B_BYTES));
              const int nk4 = (kb == a.kblocks - 1 && a.k16_last > 0) ? a.k16_last : TK / 16;
              if (j == nj - 1 && more) {
                pre_stage = __all_sync(0xffffffffu, mbar_test_wait(&sm->a_full[ns], nph));
                if (tile_ends)
                  pre_acc = __all_sync(0xffffffffu, mbar_test_wait(&sm->tmem_empty[acc ^ 1], (uint32_t)(((local + 1) >> 1) & 1) ^ 1u));
              }
              if (elect_one()) {
#pragma unroll
                for (int k4 = 0; k4 < TK / 16; ++k4)
                  if (k4 < nk4) tc_mma(tmem_d, adesc + (uint64_t)(k4 * 2), bdesc + (uint64_t)(k4 * 2), kIdesc, (kb | k4) ? 1u : 0u);
              }
              __syncwarp();
            }
            if (narrow) {
              const uint64_t adesc = make_desc_narrow(smem_u32(a_ring + s * stage_bytes + nfull * A_BYTES));
              const uint64_t bdesc = make_desc_narrow(smem_u32(sm->ring + nfull * B_BYTES));
              // a second look for what the first one came too early for (the other accumulator is handed back about
              // four MMAs after this tile's first)
              if (more && !pre_stage) pre_stage = __all_sync(0xffffffffu, mbar_test_wait(&sm->a_full[ns], nph));
              if (more && tile_ends && !pre_acc)
                pre_acc = __all_sync(0xffffffffu, mbar_test_wait(&sm->tmem_empty[acc ^ 1], (uint32_t)(((local + 1) >> 1) & 1) ^ 1u));
              if (elect_one()) tc_mma(tmem_d, adesc, bdesc, kIdesc, 1u);
              __syncwarp();
            }
            if (elect_one()) tc_commit(&sm->a_empty[s]);
            __syncwarp();
            s = ns;
            ph = nph;
          }
          if (ok && elect_one()) tc_commit(&sm->tmem_full[acc]);
          __syncwarp();
        }
        if (ok && elect_one()) tc_commit(&sm->b_empty);   // arrives when every MMA issued so far (all readers of this block) has retired
        __syncwarp();
      }
      if (lane == 0) {
        tc_commit(&sm->drain);
        for (uint32_t it = 0; it < wait_limit; ++it) {
          if (mbar_try_wait(&sm->drain, 0)) break;
          __nanosleep(64);
        }
      }
      __syncwarp();
    }
  } else {
    // ---------------- epilogue: one data row per thread, a quarter of the block's columns per warp ----------------
    constexpr int PARTS = AS_EW / 4, GROUPS = TN / PARTS / 32;
    const int quarter = warp & 3;
    const int et = quarter * 32 + lane;
    const int ew = warp - 2;
    const int part = ew >> 2;
    const int c0 = part * GROUPS;
    const float alpha = __ldg(a.alpha);
    const float inv_alpha = 1.0f / alpha;
    int64_t local = 0;
    bool ok = true;
    for (int b = b_first; ok && b < nb; b += b_step) {
      const int col_base = b * TN;
      float thr_next = CUDART_INF_F;
      if (MODE == SCAN_THRESHOLD && t_first < qtiles && t_first * TM + et < a.n) thr_next = __ldg(a.thr + t_first * TM + et);
      for (int64_t t = t_first; t < qtiles; t += t_step, ++local) {
        const int acc = (int)(local & 1);
        const uint32_t aph = (uint32_t)((local >> 1) & 1);
        const int64_t q = t * TM + et;
        const bool qok = q < a.n;
        const float thr = thr_next;
        const float bar = as_bar(thr, inv_alpha);
        if (MODE == SCAN_THRESHOLD) {   // the next tile's threshold is in flight while this tile is processed
          const int64_t qn = (t + t_step) * TM + et;
          thr_next = (t + t_step < qtiles && qn < a.n) ? __ldg(a.thr + qn) : CUDART_INF_F;
        }
        bool got = mbar_wait(&sm->tmem_full[acc], aph, &sm->abort_flag, a.err, 4, wait_limit);
        got = __all_sync(0xffffffffu, got);
        if (!got) { ok = false; break; }
        tc_fence_after();
        const uint32_t trow = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * TN);
        if (MODE == SCAN_THRESHOLD) {
          // Both 32-column groups of this warp are read at once and the accumulator is handed back BEFORE the values
          // are looked at: the next tile's MMAs never wait for the tests below (with a short contraction the
          // epilogue's own latency, not the MMAs and not the operand fill, sets the pace of this kernel).
          static_assert(GROUPS == 2, "two groups per warp");
          float v0[32], v1[32];
          tc_ld32_issue(trow + (uint32_t)(c0 * 32), v0);
          tc_ld32_issue(trow + (uint32_t)((c0 + 1) * 32), v1);
          tc_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm->tmem_empty[acc]);
          const int left0 = a.k - (col_base + c0 * 32), left1 = left0 - 32;
          // value = alpha * accumulator <= thr with alpha < 0 is accumulator >= bar (bar = thr / alpha, lowered by more
          // than the roundings of either form can differ: the hits are a superset, and every logged hit is evaluated
          // exactly afterwards).  Eight columns at a time: the largest of eight costs four instructions, and only a
          // set of eight that holds a hit is searched for its columns.
          const float m00 = max8<0>(v0), m01 = max8<8>(v0), m02 = max8<16>(v0), m03 = max8<24>(v0);
          const float m10 = max8<0>(v1), m11 = max8<8>(v1), m12 = max8<16>(v1), m13 = max8<24>(v1);
          const bool mine0 = qok && left0 > 0 && max3(m00, m01, fmaxf(m02, m03)) >= bar;
          const bool mine1 = qok && left1 > 0 && max3(m10, m11, fmaxf(m12, m13)) >= bar;
          if (!__any_sync(0xffffffffu, mine0 || mine1)) continue;
          auto log_hits = [&](uint32_t bits, int first_col) {   // one or two hits as a rule
            bits = (first_col + 8 <= a.k) ? bits : (first_col < a.k ? bits & ((1u << (a.k - first_col)) - 1u) : 0u);
            while (bits) {
              const int j = __ffs((int)bits) - 1;
              bits &= bits - 1u;
              const int slot = atomicAdd(&sm->log_n, 1);
              if (slot < a.log_cap) my_log[slot] = make_uint2((uint32_t)q, (uint32_t)(first_col + j));
            }
          };
          const int col0 = col_base + c0 * 32;
          if (mine0) {
            if (m00 >= bar) log_hits(ge_bits8<0>(v0, bar), col0);
            if (m01 >= bar) log_hits(ge_bits8<8>(v0, bar), col0 + 8);
            if (m02 >= bar) log_hits(ge_bits8<16>(v0, bar), col0 + 16);
            if (m03 >= bar) log_hits(ge_bits8<24>(v0, bar), col0 + 24);
          }
          if (mine1) {
            if (m10 >= bar) log_hits(ge_bits8<0>(v1, bar), col0 + 32);
            if (m11 >= bar) log_hits(ge_bits8<8>(v1, bar), col0 + 40);
            if (m12 >= bar) log_hits(ge_bits8<16>(v1, bar), col0 + 48);
            if (m13 >= bar) log_hits(ge_bits8<24>(v1, bar), col0 + 56);
          }
          continue;
        }
        // SCAN_ARGMIN: only the value is wanted (it becomes the row's threshold, and the pass that uses the threshold lists
        // the centroids), so it costs half an instruction per column, the accumulator goes back before the values are
        // looked at as above, and a warp's rows are one 128-byte atomic.  With the column and a 64-bit key per row the pass
        // took 21.7 ms over 10 million rows x 128 and 4 096 centroids, twice the threshold pass.
        float v0[32], v1[32];
        tc_ld32_issue(trow + (uint32_t)(c0 * 32), v0);
        tc_ld32_issue(trow + (uint32_t)((c0 + 1) * 32), v1);
        tc_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm->tmem_empty[acc]);
        const int left = a.k - (col_base + c0 * 32);   // valid centroids from this warp's first column on
        if (left < 64) {   // the last block only
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            v0[j] = j < left ? v0[j] : -CUDART_INF_F;
            v1[j] = j + 32 < left ? v1[j] : -CUDART_INF_F;
          }
        }
        // alpha < 0: the smallest value is alpha times the largest accumulator
        const float amax = fmaxf(max3(max8<0>(v0), max8<8>(v0), fmaxf(max8<16>(v0), max8<24>(v0))),
                                 max3(max8<0>(v1), max8<8>(v1), fmaxf(max8<16>(v1), max8<24>(v1))));
        if (qok && left > 0 && amax > -CUDART_INF_F) atomicMin(a.best_value + q, float_to_ordered(amax * alpha));
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (MODE == SCAN_THRESHOLD && threadIdx.x == 0) {
    const int logged = sm->log_n;
    a.log_count[blockIdx.x] = (int32_t)min((int64_t)logged, a.log_cap);
    if (logged > a.log_cap) atomicCAS(a.err, 0, 9);
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ---- row lists of a batch with a STATIONARY query block ---------------------------------------------------------
// The searches whose listed rows are re-scored after every chunk need one bit per (query, row) from the contraction: can the
// row still be among the query's best?  With a short inner dimension the general kernel is paced by its operands: a
// 128 x 256 tile of 144 fp16 columns fetches 144 KB for 1 152 cycles of MMAs through a ring that holds one tile and a half
// (10 000 queries x 10 million decoded rows: 38 ms, 1.8 us per tile).  Here, as in assign_scan_kernel, a block of 256
// queries stays in shared memory and 128-row tiles stream past it, a whole tile per ring stage (36 KB, four of them).
// The queries' thresholds ride inside the contraction as well, subtracted in columns (fp16) or in a K step (int8) of their
// own, so that "listed" is the sign of the accumulator: one instruction looks at three values, whatever their columns.
//   order     rows are walked in windows that stay in L2; inside a window every CTA takes an equal stretch of the
//             (query block, row tile) sequence, so it changes its block once or twice per window and no CTA is left over
//   fp16      fold columns: eight hold the row term (pieces p0 x2, p1 x2, p2 x4 of R / 16, queries: 8u x4, 4u x4), eight
//             the threshold (rows: the constant kLsBarConst, queries: pieces of minus the bar)
//   int8      a K32 step of a constant tile (all kLsBarByte) against the queries' 32 threshold bytes
// warp 0 TMA producer, warp 1 MMA issuer, 16 epilogue warps: a row per lane, 64 queries per warp.  A listed row goes to the
// CTA's stretch of a log, its slot from a shared-memory counter, and ls_scatter_kernel moves the log to the candidate lists:
// with an atomic on the list itself a warp sat out the round trip to L2, most tiles held such a warp, and the launch was no
// faster than the general kernel (1.8 us per tile).  A full log falls back to that atomic.  The query operand is padded to
// whole blocks with queries whose threshold nothing reaches, so the epilogue knows nothing of the last block's end (a test
// there made its CTAs twice as slow as the rest).  Every wait is bounded.
constexpr int LS_RING_BYTES = 224 * 1024;
constexpr int LS_MAX_STAGES = 8;
constexpr float kLsBarConst = 32768.f;
constexpr int kLsBarByte = 127;

struct LsSmem {
  uint8_t ring[LS_RING_BYTES];   // [resident query block][constant tile (int8)][stages x 128-row tiles]
  uint64_t full[LS_MAX_STAGES];
  uint64_t empty[LS_MAX_STAGES];
  uint64_t q_full, q_empty;
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint64_t drain;
  uint32_t tmem_base;
  volatile int abort_flag;
  int log_n;                     // rows this CTA has listed so far
};
constexpr size_t kLsSmemBytes = sizeof(LsSmem) + 1024;

struct LsArgs {
  int64_t rows;               // rows of the row operand
  int64_t nq;
  int64_t row_id0;            // id of operand row 0
  int32_t kblocks;            // 128-byte K blocks, the fold block included
  int32_t k16_last;           // 32-byte K steps of the last block that hold operand columns
  int32_t window;             // row tiles per window
  uint2* log;                 // [gridDim.x][log_cap] {row id, query}
  int32_t* log_count;         // [gridDim.x]
  int64_t log_cap;
  CandLists cand;
  int32_t* err;
  uint32_t wait_limit;
  int32_t stall;              // testing only: CTA 0 never fills its first row tile (see TcArgs::stall_kblock)
};

// Bytes of the resident block and of a row tile; false when two whole-tile stages do not fit beside the block.
struct LsLayout {
  int nfull, res_bytes, const_off, bar_off, tile_bytes, stages;
  bool narrow;
};
__host__ __device__ inline LsLayout ls_layout(int kblocks, int k16_last, bool i8) {
  LsLayout l;
  l.narrow = !i8 && k16_last == 1 && kblocks >= 2;   // the fold columns begin a block of their own: a 16-column tile
  l.nfull = l.narrow ? kblocks - 1 : kblocks;
  int at = l.nfull * B_BYTES + (l.narrow ? B_NARROW_BYTES : 0);
  l.bar_off = at;
  if (i8) at += B_NARROW_BYTES;
  l.const_off = at;
  if (i8) at += A_NARROW_BYTES;
  l.res_bytes = at;
  l.tile_bytes = l.nfull * A_BYTES + (l.narrow ? A_NARROW_BYTES : 0);
  l.stages = (LS_RING_BYTES - at) / l.tile_bytes;
  if (l.stages > LS_MAX_STAGES) l.stages = LS_MAX_STAGES;
  return l;
}

// The stretches of (query block, row tile) pairs a CTA takes, one after the other.
struct LsWalk {
  int64_t ntiles, w0;      // row tiles in all; first tile of the current window
  int nb, window;
  int64_t pos, end;        // the CTA's part of the window's sequence (block-major)
  int wt;                  // tiles of the window
  __device__ __forceinline__ void start(int64_t nt, int blocks, int win) {
    ntiles = nt;
    nb = blocks;
    window = win;
    w0 = -win;
    pos = end = 0;
  }
  // next stretch: block b, tiles [t, t + count)
  __device__ __forceinline__ bool next(int& b, int64_t& t, int& count) {
    while (pos >= end) {
      w0 += window;
      if (w0 >= ntiles) return false;
      wt = (int)min((int64_t)window, ntiles - w0);
      const int64_t all = (int64_t)wt * nb;
      pos = all * blockIdx.x / gridDim.x;
      end = all * (blockIdx.x + 1) / gridDim.x;
    }
    b = (int)(pos / wt);
    const int in = (int)(pos - (int64_t)b * wt);
    count = (int)min((int64_t)(wt - in), end - pos);
    t = w0 + in;
    pos += count;
    return true;
  }
};

template <bool I8>
__global__ void __launch_bounds__(AS_THREADS, 1)
list_scan_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_q,
                 const __grid_constant__ CUtensorMap map_xn, const __grid_constant__ CUtensorMap map_qn, LsArgs a) {
  extern __shared__ uint8_t smem_raw[];
  LsSmem* sm = reinterpret_cast<LsSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t wait_limit = a.wait_limit ? a.wait_limit : WAIT_LIMIT;
  const LsLayout l = ls_layout(a.kblocks, a.k16_last, I8);
  constexpr int KCOLS = I8 ? 2 * TK : TK;
  const int nb = (int)((a.nq + TN - 1) / TN);
  const int64_t ntiles = (a.rows + TM - 1) / TM;
  if (threadIdx.x == 0) {
    for (int s = 0; s < LS_MAX_STAGES; ++s) {
      mbar_init(&sm->full[s], 1);
      mbar_init(&sm->empty[s], 1);
    }
    mbar_init(&sm->q_full, 1);
    mbar_init(&sm->q_empty, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm->tmem_full[b], 1);
      mbar_init(&sm->tmem_empty[b], AS_EW);
    }
    mbar_init(&sm->drain, 1);
    sm->abort_flag = 0;
    sm->log_n = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (I8) {   // the constant tile: the same byte everywhere, so its swizzle does not matter
    for (int i = threadIdx.x; i < A_NARROW_BYTES / 4; i += AS_THREADS)
      reinterpret_cast<uint32_t*>(sm->ring + l.const_off)[i] = 0x01010101u * (uint32_t)kLsBarByte;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sm->tmem_base;
  uint8_t* ring = sm->ring + l.res_bytes;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0, qph = 0, issued = 0, issued_ph = 0, q_last = 0;
      bool ok = true, q_issued = false, stall = a.stall != 0 && blockIdx.x == 0;
      LsWalk w;
      w.start(ntiles, nb, a.window);
      int b, count;
      int64_t t;
      while (ok && w.next(b, t, count)) {
        // the block may be replaced once every MMA that read the previous one has retired
        if (!mbar_wait(&sm->q_empty, qph ^ 1, &sm->abort_flag, a.err, 5, wait_limit)) break;
        mbar_expect_tx(&sm->q_full, (uint32_t)(l.res_bytes - (I8 ? A_NARROW_BYTES : 0)));
        for (int kb = 0; kb < l.nfull; ++kb) tma_load_2d(sm->ring + kb * B_BYTES, &map_q, &sm->q_full, kb * KCOLS, b * TN);
        if (l.narrow) tma_load_2d(sm->ring + l.nfull * B_BYTES, &map_qn, &sm->q_full, l.nfull * KCOLS, b * TN);
        if (I8) tma_load_2d(sm->ring + l.bar_off, &map_qn, &sm->q_full, 0, b * TN);
        q_issued = true;
        q_last = qph;
        qph ^= 1;
        for (int i = 0; i < count; ++i, ++t) {
          if (!mbar_wait(&sm->empty[s], ph ^ 1, &sm->abort_flag, a.err, 1, wait_limit)) { ok = false; break; }
          uint8_t* st = ring + s * l.tile_bytes;
          if (stall) {
            stall = false;   // this stage is never filled, the consumer's bounded wait for it runs out
          } else {
            mbar_expect_tx(&sm->full[s], (uint32_t)l.tile_bytes);
            for (int kb = 0; kb < l.nfull; ++kb) tma_load_2d(st + kb * A_BYTES, &map_x, &sm->full[s], kb * KCOLS, (int32_t)(t * TM));
            if (l.narrow) tma_load_2d(st + l.nfull * A_BYTES, &map_xn, &sm->full[s], l.nfull * KCOLS, (int32_t)(t * TM));
            issued |= 1u << s;
            issued_ph = (issued_ph & ~(1u << s)) | (ph << s);
          }
          if (++s == l.stages) { s = 0; ph ^= 1; }
        }
      }
      // copies still in flight must land before the CTA's shared memory is released
      if (q_issued)
        for (uint32_t it = 0; it < wait_limit; ++it) {
          if (mbar_try_wait(&sm->q_full, q_last)) break;
          __nanosleep(64);
        }
      for (int i = 0; i < l.stages; ++i)
        if (issued & (1u << i))
          for (uint32_t it = 0; it < wait_limit; ++it) {
            if (mbar_try_wait(&sm->full[i], (issued_ph >> i) & 1)) break;
            __nanosleep(64);
          }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (see assign_scan_kernel for why it looks ahead) ----------------
    if (lane == 0) {
      const uint32_t a_lo0 = desc_lo(smem_u32(ring)), stage_lo = (uint32_t)l.tile_bytes >> 4;
      const uint32_t b_lo0 = desc_lo(smem_u32(sm->ring)), bn_lo = desc_lo(smem_u32(sm->ring + l.nfull * B_BYTES));
      const uint32_t bar_lo = desc_lo(smem_u32(sm->ring + l.bar_off)), const_lo = desc_lo(smem_u32(sm->ring + l.const_off));
      const uint32_t full0 = smem_u32(&sm->full[0]), empty0 = smem_u32(&sm->empty[0]);
      const uint32_t tfull0 = smem_u32(&sm->tmem_full[0]), tempty0 = smem_u32(&sm->tmem_empty[0]);
      const int last_nk4 = l.narrow ? 4 : a.k16_last;
      uint32_t s = 0, ph = 0, qph = 0, acc = 0, aph = 0;
      bool ok = true, pre_acc = false, pre_stage = false;
      LsWalk w;
      w.start(ntiles, nb, a.window);
      int b, count;
      int64_t t;
      while (ok && w.next(b, t, count)) {
        if (!mbar_wait(&sm->q_full, qph, &sm->abort_flag, a.err, 6, wait_limit)) break;
        qph ^= 1;
        for (int left = count; left > 0; --left) {
          if (!pre_acc && !mbar_wait(&sm->tmem_empty[acc], aph ^ 1, &sm->abort_flag, a.err, 2, wait_limit)) { ok = false; break; }
          if (!pre_stage && !mbar_wait(&sm->full[s], ph, &sm->abort_flag, a.err, 3, wait_limit)) { ok = false; break; }
          tc_fence_after();
          const uint32_t tmem_d = tmem_base + acc * (uint32_t)TN;
          const uint32_t a_lo = a_lo0 + s * stage_lo;
          const uint32_t ns = s + 1 == (uint32_t)l.stages ? 0u : s + 1;
          const uint32_t nph = s + 1 == (uint32_t)l.stages ? ph ^ 1u : ph;
          const uint32_t naph = acc ? aph ^ 1u : aph;
          const bool more = left > 1;
          pre_acc = false;
          pre_stage = false;
          if (I8)   // first, as it needs nothing of the row tile
            tc_mma_i8(tmem_d, desc_pack(const_lo, kDescHiNarrow), desc_pack(bar_lo, kDescHiNarrow), kIdescI8, 0u);
          for (int kb = 0; kb < l.nfull; ++kb) {
            if (kb == l.nfull - 1 && more) {
              pre_stage = mbar_test_wait_a(full0 + ns * 8u, nph);
              pre_acc = mbar_test_wait_a(tempty0 + (acc ^ 1u) * 8u, naph ^ 1u);
            }
            const int nk4 = kb == l.nfull - 1 ? last_nk4 : TK / 16;
#pragma unroll
            for (int k4 = 0; k4 < TK / 16; ++k4)
              if (k4 < nk4) {
                const uint64_t ad = desc_pack(a_lo + (uint32_t)(kb * (A_BYTES >> 4) + k4 * 2), kDescHi);
                const uint64_t bd = desc_pack(b_lo0 + (uint32_t)(kb * (B_BYTES >> 4) + k4 * 2), kDescHi);
                if (I8) tc_mma_i8(tmem_d, ad, bd, kIdescI8, 1u);
                else tc_mma(tmem_d, ad, bd, kIdesc, (kb | k4) ? 1u : 0u);
              }
          }
          if (l.narrow) {
            // a second look for what the first one came too early for
            if (more && !pre_stage) pre_stage = mbar_test_wait_a(full0 + ns * 8u, nph);
            if (more && !pre_acc) pre_acc = mbar_test_wait_a(tempty0 + (acc ^ 1u) * 8u, naph ^ 1u);
            tc_mma(tmem_d, desc_pack(a_lo + (uint32_t)(l.nfull * (A_BYTES >> 4)), kDescHiNarrow), desc_pack(bn_lo, kDescHiNarrow), kIdesc, 1u);
          }
          tc_commit_a(empty0 + s * 8u);
          tc_commit_a(tfull0 + acc * 8u);
          s = ns;
          ph = nph;
          aph = naph;
          acc ^= 1u;
        }
        if (ok) tc_commit(&sm->q_empty);
      }
      // all issued MMAs must retire before tensor memory is freed
      tc_commit(&sm->drain);
      for (uint32_t it = 0; it < wait_limit; ++it) {
        if (mbar_try_wait(&sm->drain, 0)) break;
        __nanosleep(64);
      }
    }
  } else {
    // ---------------- epilogue: one row per lane, 64 queries per warp ----------------
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    const int et = quarter * 32 + lane;
    bool ok = true;
    uint32_t acc = 0, aph = 0;
    LsWalk w;
    w.start(ntiles, nb, a.window);
    int b, count;
    int64_t t;
    uint2* my_log = a.log + (int64_t)blockIdx.x * a.log_cap;
    while (ok && w.next(b, t, count)) {
      const int64_t col0 = (int64_t)b * TN + part * 64;
      for (int i = 0; i < count; ++i, ++t) {
        bool got = mbar_wait(&sm->tmem_full[acc], aph, &sm->abort_flag, a.err, 4, wait_limit);
        got = __all_sync(0xffffffffu, got);
        if (!got) { ok = false; break; }
        tc_fence_after();
        const uint32_t trow = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * (uint32_t)TN + (uint32_t)(part * 64);
        float v0[32], v1[32];
        tc_ld32_issue(trow, v0);
        tc_ld32_issue(trow + 32u, v1);
        tc_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm->tmem_empty[acc]);   // the accumulator goes back before the values are looked at
        aph = acc ? aph ^ 1u : aph;
        acc ^= 1u;
        const int64_t row = t * TM + et;
        // the sign bits of eight values at a time: clear in the AND of the values' words iff one is not negative
        uint32_t neg[8];
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          neg[o] = 0xffffffffu;
          neg[o + 4] = 0xffffffffu;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            neg[o] &= __float_as_uint(v0[8 * o + j]);
            neg[o + 4] &= __float_as_uint(v1[8 * o + j]);
          }
        }
        const uint32_t all = neg[0] & neg[1] & neg[2] & neg[3] & neg[4] & neg[5] & neg[6] & neg[7];
        const bool mine = (int)all >= 0 && row < a.rows;
        if (!__any_sync(0xffffffffu, mine)) continue;
        if (!mine) continue;
        const uint32_t id = (uint32_t)(a.row_id0 + row);
        auto append = [&](uint32_t bits, int64_t first) {
          while (bits) {
            const int j = __ffs((int)bits) - 1;
            bits &= bits - 1u;
            const int64_t q = first + j;
            const int at = atomicAdd(&sm->log_n, 1);
            if (at < a.log_cap) {
              *VSK_CHK_W(my_log + at) = make_uint2(id, (uint32_t)q);
            } else {
              const int slot = atomicAdd(&a.cand.count[q], 1);
              if (slot < kCandCap) *VSK_CHK_W(a.cand.keys + q * kCandCap + slot) = make_key(0.f, id);
            }
          }
        };
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          if ((int)neg[o] >= 0) {
            uint32_t bits = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) bits |= (__float_as_uint(v0[8 * o + j]) >> 31) << j;
            append(bits ^ 0xffu, col0 + 8 * o);
          }
        }
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          if ((int)neg[o + 4] >= 0) {
            uint32_t bits = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) bits |= (__float_as_uint(v1[8 * o + j]) >> 31) << j;
            append(bits ^ 0xffu, col0 + 32 + 8 * o);
          }
        }
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) *VSK_CHK_W(a.log_count + blockIdx.x) = (int32_t)min((int64_t)sm->log_n, a.log_cap);
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// The logs of the CTAs (blockIdx.y) to the candidate lists; a key's value is formed by the re-scoring.
__global__ void __launch_bounds__(256) ls_scatter_kernel(const uint2* __restrict__ log, const int32_t* __restrict__ log_count, int64_t log_cap,
                                                         CandLists cand) {
  const int cnt = *VSK_CHK(log_count + blockIdx.y);
  const uint2* mine = log + (int64_t)blockIdx.y * log_cap;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < cnt; e += gridDim.x * blockDim.x) {
    const uint2 h = *VSK_CHK(mine + e);
    const int slot = atomicAdd(&cand.count[h.y], 1);
    if (slot < kCandCap) *VSK_CHK_W(cand.keys + (int64_t)h.y * kCandCap + slot) = make_key(0.f, h.x);
  }
}

// One warp per logged hit: the exact squared distance of the row to the listed centroid, direct fp32 formula, merged
// into best[row] - smallest (value, centroid), the reference's strict '<' scan (KMeansClustering.swift:283-288).
template <bool VEC>
__global__ void __launch_bounds__(256, 6) assign_log_exact_kernel(const float* __restrict__ x, int dim, const float* __restrict__ cent,
                                        const uint2* __restrict__ log, const int32_t* __restrict__ log_count, int64_t log_cap,
                                        unsigned long long* __restrict__ best) {
  const int cta = blockIdx.y;
  const int cnt = log_count[cta];
  const uint2* mine = log + (int64_t)cta * log_cap;
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (VEC) {
    // 16-byte loads (dim a multiple of 4, aligned rows), two hits per step: four independent loads in flight per lane
    const int nv = dim >> 2;
    for (int e = 2 * w; e < cnt; e += 2 * warps) {
      const bool two = e + 1 < cnt;
      const uint2 h0 = mine[e], h1 = two ? mine[e + 1] : h0;
      const float4* x0 = reinterpret_cast<const float4*>(x + (int64_t)h0.x * dim);
      const float4* c0 = reinterpret_cast<const float4*>(cent + (int64_t)h0.y * dim);
      const float4* x1 = reinterpret_cast<const float4*>(x + (int64_t)h1.x * dim);
      const float4* c1 = reinterpret_cast<const float4*>(cent + (int64_t)h1.y * dim);
      float s0 = 0.f, s1 = 0.f;
      for (int i = lane; i < nv; i += 32) {
        const float4 a0 = __ldg(x0 + i), b0 = __ldg(c0 + i), a1 = __ldg(x1 + i), b1 = __ldg(c1 + i);
        float d;
        d = a0.x - b0.x; s0 = fmaf(d, d, s0);
        d = a0.y - b0.y; s0 = fmaf(d, d, s0);
        d = a0.z - b0.z; s0 = fmaf(d, d, s0);
        d = a0.w - b0.w; s0 = fmaf(d, d, s0);
        d = a1.x - b1.x; s1 = fmaf(d, d, s1);
        d = a1.y - b1.y; s1 = fmaf(d, d, s1);
        d = a1.z - b1.z; s1 = fmaf(d, d, s1);
        d = a1.w - b1.w; s1 = fmaf(d, d, s1);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
      }
      if (lane == 0) {
        atomicMin(best + h0.x, (unsigned long long)make_key(s0, h0.y));
        if (two) atomicMin(best + h1.x, (unsigned long long)make_key(s1, h1.y));
      }
    }
    return;
  }
  for (int e = w; e < cnt; e += warps) {
    const uint2 h = mine[e];
    const float* xr = x + (int64_t)h.x * dim;
    const float* cr = cent + (int64_t)h.y * dim;
    float s = 0.f;
    for (int i = lane; i < dim; i += 32) {
      const float d = __ldg(xr + i) - __ldg(cr + i);
      s = fmaf(d, d, s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) atomicMin(best + h.x, (unsigned long long)make_key(s, h.y));
  }
}

// best[row] -> assignment and rooted distance; a row without any logged hit is handed to the exact scan
// (`err` given and raised: the scan's log is incomplete - nothing is written, so that the previous assignment and its
// distances survive for the repeat)
__global__ void assign_log_decode_kernel(const unsigned long long* __restrict__ best, int64_t n, int32_t* __restrict__ assign,
                                         float* __restrict__ dist, int32_t* __restrict__ bad_rows, int32_t* bad_count,
                                         const int32_t* __restrict__ err) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  if (err != nullptr && *err != 0) return;
  const unsigned long long b = best[r];
  if (b == ~0ull) {
    bad_rows[atomicAdd(bad_count, 1)] = (int32_t)r;
    return;
  }
  assign[r] = (int32_t)(uint32_t)b;
  if (dist) dist[r] = sqrtf(ordered_to_float((uint32_t)(b >> 32)));
}

// ---- operand preparation --------------------------------------------------------------------
// Statistics accumulated with atomics on order-preserving integer images of non-negative floats.
struct PrepStats {
  unsigned absmax;      // max |x_i|
  unsigned max_norm16;  // max over rows of |x'| (operand units)
  unsigned max_err16;   // max over rows of |s*x - x'|
  unsigned max_norm;    // max |x|
  unsigned min_norm_nz; // min nonzero |x| (initialised to +inf)
};

__global__ void absmax_kernel(const float* __restrict__ x, int64_t total, unsigned* out) {
  float m = 0.f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
    m = fmaxf(m, fabsf(__ldg(x + i)));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));  // non-negative floats order as uints
}

// scale = 2^e with 2^13 < absmax * scale <= 2^14 (1 when absmax is 0 or not finite); cosine: 2^14
// fold != 0 (queries against folded rows, see FoldArgs): the scale is also kept where the folded constant
// s 2^-exp is a normal fp16 number.
__device__ __forceinline__ float operand_scale(bool cosine, float absmax, bool fold, int fold_exp) {
  float s = 16384.f;
  if (!cosine) {
    s = 1.f;
    if (absmax > 0.f && absmax < CUDART_INF_F) {
      int e;
      frexpf(absmax, &e);          // absmax = f * 2^e, f in [0.5, 1)
      s = ldexpf(1.f, 14 - e);
    }
  }
  if (fold) s = fmaxf(fminf(s, ldexpf(1.f, fold_exp + 13)), ldexpf(1.f, fold_exp - 14));   // 4u <= 2^15, 2u normal
  return s;
}
__global__ void choose_scale_kernel(const unsigned* absmax, int cosine, float* scale, int fold = 0, int fold_exp = 0) {
  *scale = operand_scale(cosine != 0, __uint_as_float(*absmax), fold != 0, fold_exp);
}

// One warp per row: fp32 row -> fp16 operand row x' = fp16(s * x) (cosine: s * x/|x|), padded with
// zeros to dim16, and the measured quantities the error bound needs.
//   aux[row]   = |x|^2 (euclidean), unused otherwise
//   nrm16[row] = |x'|, err16[row] = |s*x^ - x'|   (optional per-row outputs, used for queries)
// Euclidean operands can carry the per-row term of the value inside the contraction.  Sixteen columns - one K16
// step of the MMA, placed right behind the data columns (fold_col0) - hold, on the row side, R = -(s_x |x|^2 / 2) 2^exp
// split into three fp16 pieces p0 + p1 + p2 = R / 16 (p0 in columns 0-3, p1 in 4-7, p2 in 8-15), and on the query
// side the constants 4u (columns 0-7) and 2u (columns 8-15), u = s_q 2^-exp a power of two: the sixteen products add
// up to 16 u (p0 + p1 + p2) = -s_q s_x |x|^2 / 2, so the accumulator is s_q s_x (q.x - |x|^2 / 2) and the value
// alpha * accumulator needs no per-row term in the epilogue.  Columns behind the sixteen are zero and the MMA issuer
// skips K16 steps that hold nothing but padding (kvalid), so the term costs one K16 step, not a K block.
constexpr int kFoldCols = 16;
__host__ __device__ inline int fold_col0(int dim) { return (dim + 15) / 16 * 16; }
// K16 steps of the last 64-column K block that hold operand columns, for `kvalid` columns in a width of dim16
inline int k16_last_of(int kvalid, int dim16) {
  const int steps = (kvalid + 15) / 16, before = 4 * (dim16 / 64 - 1);
  return std::max(1, std::min(4, steps - before));
}
struct FoldArgs {
  int side;   // 0: none, 1: rows (pieces of the term), 2: queries (the constants)
  int col0;   // first of the kFoldCols columns (fold_col0(dim))
  int exp;
  const int* exp_dev = nullptr;   // when given, the exponent is read from device memory instead
};

template <int METRIC>
__global__ void prep_rows_kernel(const float* __restrict__ x, int64_t n, int dim, int dim16, const float* scale_p,
                                 __half* __restrict__ out, float* __restrict__ aux, float* __restrict__ nrm16,
                                 float* __restrict__ err16, float* __restrict__ nrm, PrepStats* stats, FoldArgs fold) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  const int lane = threadIdx.x & 31;
  const float s = *scale_p;
  const float* p = x + row * dim;
  float ss = 0.f;
  for (int i = lane; i < dim; i += 32) {
    const float v = __ldg(p + i);
    ss = fmaf(v, v, ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float norm = sqrtf(ss);
  const float inv = (METRIC == VSK_METRIC_COSINE) ? (norm > 0.f ? 1.0f / norm : 0.f) : 1.0f;
  float n2 = 0.f, e2 = 0.f;
  for (int i = lane; i < dim16; i += 32) {
    float t = 0.f;
    if (i < dim) t = (METRIC == VSK_METRIC_COSINE) ? (__ldg(p + i) * inv) * s : __ldg(p + i) * s;
    const __half h = __float2half_rn(t);
    if (fold.side == 0 || i < fold.col0 || i >= fold.col0 + kFoldCols) out[row * dim16 + i] = h;
    const float back = __half2float(h);
    n2 = fmaf(back, back, n2);
    const float e = t - back;
    e2 = fmaf(e, e, e2);
  }
  const int fold_exp = fold.exp_dev ? *fold.exp_dev : fold.exp;
  if (fold.side == 1) {
    // pieces of R = s_x (|x|^2 / 2) 2^exp: p0 = fp16(R/16), then the same of what is left, twice (the remainders are
    // exact in fp32); what is left after three pieces is below 2^-33 R
    const float R = ldexpf(0.5f * ss * s, fold_exp);
    const __half p0 = __float2half_rn(R * 0.0625f);
    const float r1 = R - 16.0f * __half2float(p0);
    const __half p1 = __float2half_rn(r1 * 0.0625f);
    const float r2 = r1 - 16.0f * __half2float(p1);
    const __half p2 = __float2half_rn(r2 * 0.0625f);
    if (lane < kFoldCols) {
      const __half p = lane < 4 ? p0 : (lane < 8 ? p1 : p2);
      out[row * dim16 + fold.col0 + lane] = __hneg(p);
    }
  } else if (fold.side == 2) {
    // 4u against the four copies of p0 and of p1, 2u against the eight copies of p2
    if (lane < kFoldCols) out[row * dim16 + fold.col0 + lane] = __float2half_rn(ldexpf(s, (lane < 8 ? 2 : 1) - fold_exp));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    e2 += __shfl_xor_sync(0xffffffffu, e2, o);
  }
  if (lane == 0) {
    // round the measured norms up a little: they are used as upper bounds
    const float up = 1.0f + 1e-5f;
    const float a16 = sqrtf(n2) * up, r16 = sqrtf(e2) * up;
    if (aux && METRIC == VSK_METRIC_EUCLIDEAN) aux[row] = ss;
    if (nrm16) nrm16[row] = a16;
    if (err16) err16[row] = r16;
    if (nrm) nrm[row] = norm;
    if (stats) {
      atomicMax(&stats->max_norm16, __float_as_uint(a16));
      atomicMax(&stats->max_err16, __float_as_uint(r16));
      atomicMax(&stats->max_norm, __float_as_uint(norm));
      if (norm > 0.f) atomicMin(&stats->min_norm_nz, __float_as_uint(norm));
    }
  }
}

// The same for rows of at most 256 dimensions in 16-byte pieces (no fold, no metric of its own): a lane holds its pieces between
// the two passes, so the row is read once, and stores four halves at a time.  10 million x 128, 192 operand columns: 3.4 - 3.9 ms
// for the form above (its 64-byte stores), 2.1 here.
__global__ void __launch_bounds__(256) prep_rows_wide_kernel(const float* __restrict__ x, int64_t n, int dim, int dim16, const float* scale_p,
                                                             __half* __restrict__ out, float* __restrict__ nrm16, float* __restrict__ err16,
                                                             float* __restrict__ nrm) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  const int lane = threadIdx.x & 31, nv = dim >> 2;
  const float s = __ldg(scale_p);
  const float4* p = reinterpret_cast<const float4*>(x + row * dim);
  float4 v[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) v[c] = lane + 32 * c < nv ? __ldg(p + lane + 32 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
  float ss = 0.f, n2 = 0.f, e2 = 0.f;
  uint2* o = reinterpret_cast<uint2*>(out + row * dim16);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const float f[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
    __half2 h[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float t0 = f[2 * u] * s, t1 = f[2 * u + 1] * s;
      h[u] = __floats2half2_rn(t0, t1);
      const float2 b = __half22float2(h[u]);
      ss = fmaf(f[2 * u], f[2 * u], fmaf(f[2 * u + 1], f[2 * u + 1], ss));
      n2 = fmaf(b.x, b.x, fmaf(b.y, b.y, n2));
      e2 = fmaf(t0 - b.x, t0 - b.x, fmaf(t1 - b.y, t1 - b.y, e2));
    }
    if (lane + 32 * c < dim16 >> 2) *VSK_CHK_W(o + lane + 32 * c) = make_uint2(*reinterpret_cast<uint32_t*>(&h[0]), *reinterpret_cast<uint32_t*>(&h[1]));
  }
  for (int c = lane + 64; c < dim16 >> 2; c += 32) *VSK_CHK_W(o + c) = make_uint2(0u, 0u);
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) {
    ss += __shfl_xor_sync(0xffffffffu, ss, k);
    n2 += __shfl_xor_sync(0xffffffffu, n2, k);
    e2 += __shfl_xor_sync(0xffffffffu, e2, k);
  }
  if (lane == 0) {
    const float up = 1.0f + 1e-5f;   // the measured norms are used as upper bounds
    *VSK_CHK_W(nrm16 + row) = sqrtf(n2) * up;
    *VSK_CHK_W(err16 + row) = sqrtf(e2) * up;
    *VSK_CHK_W(nrm + row) = sqrtf(ss);
  }
}

struct BoundConsts {
  float scale_x;       // s_x
  float max_norm16;    // X' = max |x'|
  float max_err16;     // E' = max |s_x x - x'|
  float max_norm;      // max |x|
  float min_norm_nz;   // min nonzero |x|
  int dim16;
  float fold_bmax;     // folded rows: max |x|^2 / 2 (0 otherwise)
};

// eps[q]: |coarse - exact| <= eps for every row, in the units of the stored coarse value.
//   contraction error (operand units) <= |q'| E' + |e_q| X' + |e_q| E'      (Cauchy-Schwarz on the residuals)
//                                       + dim16 * 2^-22 * |q'| X'            (fp32 accumulation in the tensor core)
//   divided by s_q s_x; doubled for euclidean (value = |x|^2 - 2 q.x) plus the fp32 rounding of |x|^2;
//   cosine adds the effect of the reference's +1e-8 in the denominator and of normalising in fp32.
template <int METRIC>
__device__ __forceinline__ float query_eps(float a, float e, float qn, float inv, const BoundConsts& c) {
  float dot_err = (a * c.max_err16 + e * c.max_norm16 + e * c.max_err16) + (float)c.dim16 * 2.3841858e-7f * a * c.max_norm16;
  dot_err *= inv;
  // folded per-row term (true units): its products pass through the same fp32 accumulation, and three fp16 pieces
  // leave less than 2^-30 of it unrepresented
  dot_err += ((float)c.dim16 * 2.3841858e-7f + 9.3132257e-10f) * c.fold_bmax;
  float r;
  if (METRIC == VSK_METRIC_EUCLIDEAN) {
    // + fp32 rounding of the stored |x|^2 (a sum of dim squares) and of the final multiply-add
    r = 2.0f * dot_err + 4.0f * 5.9604645e-8f * (float)c.dim16 * c.max_norm * c.max_norm +
        2.0f * 5.9604645e-8f * (c.max_norm * c.max_norm + 2.0f * qn * c.max_norm);
  } else if (METRIC == VSK_METRIC_COSINE) {
    const float den = qn * c.min_norm_nz;
    r = dot_err + 1e-8f / (den + 1e-8f) + 4.0f * 5.9604645e-8f;
    if (!(den > 0.f)) r = dot_err + 4.0f * 5.9604645e-8f;  // zero query (or no nonzero row): every value is exactly 0
  } else {
    r = dot_err;
  }
  return r * 1.0001f + 1e-30f;
}

// Inverted lists and product-quantised rows (squared distances only), with one query scale for the batch; also writes alpha.
__global__ void bound_kernel(const float* __restrict__ qn16, const float* __restrict__ qe16,
                             const float* __restrict__ qnorm, int64_t nq, const float* scale_q, BoundConsts c,
                             float* __restrict__ eps, float* alpha) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const float inv = 1.0f / ((*scale_q) * c.scale_x);
  if (q == 0) *alpha = -2.0f * inv;
  if (q >= nq) return;
  eps[q] = query_eps<VSK_METRIC_EUCLIDEAN>(qn16[q], qe16[q], qnorm[q], inv, c);
}

// eps for int8-coded rows (operand residual of the rows is zero; the query operand is fp16(s_q q~), q~ = q / scale):
//   contraction   |e_q| C + dim16 2^-22 |q'| C, divided by s_q          (C = max |code row|)
//   formula       2^-22 (|q| max|x^| + |q~| C): fp32 rounding of x^ = (code - offset)/scale and of q~
// doubled for euclidean (value = |x^|^2 - 2 q.x^) plus the rounding of |x^|^2 and of the final multiply-add.
template <int METRIC>
__device__ __forceinline__ float query_eps_i8(float a, float e, float qt_norm, float q_norm, float inv, const BoundConsts& c) {
  float dot_err = (e * c.max_norm16 + (float)c.dim16 * 2.3841858e-7f * a * c.max_norm16) * inv;
  dot_err += 2.3841858e-7f * (q_norm * c.max_norm + qt_norm * c.max_norm16);
  float r = dot_err;
  if (METRIC == VSK_METRIC_EUCLIDEAN)
    r = 2.0f * dot_err + 4.0f * 5.9604645e-8f * (float)c.dim16 * c.max_norm * c.max_norm +
        2.0f * 5.9604645e-8f * (c.max_norm * c.max_norm + 2.0f * q_norm * c.max_norm);
  return r * 1.0001f + 1e-30f;
}

// All a flat search needs of its queries in one launch, a warp per query: a power-of-two scale of the query's own (as
// choose_scale_kernel picks the batch's), the fp16 operand row with its fold constants, |q|, the error bound, the coefficient of
// the values, and empty candidate lists.  With a scale for the whole batch this took a pass over the queries for it and five
// launches more, 30 of the 207 us of 1 000 queries over 100 000 x 128.
struct QueryPrep {
  const float* q;
  int64_t nq;
  int32_t dim, dim16;
  BoundConsts c;
  FoldArgs fold;            // side 2 or 0
  __half* out;
  float *alpha, *eps, *norm;
  CandLists cand;
  uint64_t* words;          // eight words to be zeroed (error word, counters)
  const float* sq_scale;    // I8: the codes are the row operand, the query's is made from q~ = q / scale per dimension:
                            // sum_i q_i x^_i = sum_i q~_i code_i - sum_i q_i offset_i / scale_i, whose second term is no row's own
};

template <int METRIC, bool I8 = false>
__global__ void __launch_bounds__(256) query_prep_kernel(QueryPrep a) {
  static_assert(!I8 || METRIC != VSK_METRIC_COSINE, "no cosine over codes");
  if (blockIdx.x == 0 && threadIdx.x < 8) *VSK_CHK_W(a.words + threadIdx.x) = 0ull;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= a.nq) return;
  const int lane = threadIdx.x & 31;
  const float* p = a.q + row * a.dim;
  auto value = [&](int i) { return I8 ? __fdiv_rn(__ldg(p + i), __ldg(a.sq_scale + i)) : __ldg(p + i); };
  float ss = 0.f, st = 0.f, top = 0.f;
  for (int i = lane; i < a.dim; i += 32) {
    const float v = __ldg(p + i), t = value(i);
    ss = fmaf(v, v, ss);
    if (I8) st = fmaf(t, t, st);
    top = fmaxf(top, fabsf(t));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (I8) st += __shfl_xor_sync(0xffffffffu, st, o);
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  }
  const float norm = sqrtf(ss);
  const float unit = (METRIC == VSK_METRIC_COSINE) ? (norm > 0.f ? 1.0f / norm : 0.f) : 1.0f;
  const float s = operand_scale(METRIC == VSK_METRIC_COSINE, top, a.fold.side != 0, a.fold.exp);
  float n2 = 0.f, e2 = 0.f;
  __half* out = a.out + row * a.dim16;
  for (int i = lane; i < a.dim16; i += 32) {
    float t = 0.f;
    if (i < a.dim) t = (METRIC == VSK_METRIC_COSINE) ? (__ldg(p + i) * unit) * s : value(i) * s;
    __half h = __float2half_rn(t);
    const float back = __half2float(h);
    n2 = fmaf(back, back, n2);
    const float e = t - back;
    e2 = fmaf(e, e, e2);
    const int f = i - a.fold.col0;   // 4u against the four copies of p0 and of p1, 2u against the eight copies of p2
    if (a.fold.side != 0 && f >= 0 && f < kFoldCols) h = __float2half_rn(ldexpf(s, (f < 8 ? 2 : 1) - a.fold.exp));
    *VSK_CHK_W(out + i) = h;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    e2 += __shfl_xor_sync(0xffffffffu, e2, o);
  }
  if (lane == 0) {
    const float up = 1.0f + 1e-5f, inv = 1.0f / (I8 ? s : s * a.c.scale_x);
    *VSK_CHK_W(a.alpha + row) = (METRIC == VSK_METRIC_EUCLIDEAN ? -2.0f : -1.0f) * inv;
    *VSK_CHK_W(a.eps + row) = I8 ? query_eps_i8<METRIC>(sqrtf(n2) * up, sqrtf(e2) * up, sqrtf(st), norm, inv, a.c)
                                 : query_eps<METRIC>(sqrtf(n2) * up, sqrtf(e2) * up, norm, inv, a.c);
    *VSK_CHK_W(a.norm + row) = norm;
    *VSK_CHK_W(a.cand.count + row) = 0;
    *VSK_CHK_W(a.cand.thr + row) = CUDART_INF_F;
    *VSK_CHK_W(a.cand.flags + row) = 0;
  }
}

// ---- int8-coded rows -----------------------------------------------------------------------
// One warp per row of int8 codes: the fp16 operand row is the code itself (exact: |code| <= 128), so the
// operand residual of the rows is zero.  aux = |x^|^2 of the dequantised row x^ = (code - offset)/scale
// (euclidean); stats: max |code row|, max |x^|.
__global__ void prep_codes_kernel(const int8_t* __restrict__ codes, int64_t n, int dim, int dim16,
                                  const float* __restrict__ scale, const float* __restrict__ offset,
                                  __half* __restrict__ out, float* __restrict__ aux, PrepStats* stats) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  const int lane = threadIdx.x & 31;
  const int8_t* p = codes + row * dim;
  float c2 = 0.f, x2 = 0.f;
  for (int i = lane; i < dim16; i += 32) {
    float c = 0.f;
    if (i < dim) {
      c = (float)p[i];
      const float xh = __fdiv_rn(__fsub_rn(c, __ldg(offset + i)), __ldg(scale + i));
      x2 = fmaf(xh, xh, x2);
    }
    out[row * dim16 + i] = __float2half_rn(c);
    c2 = fmaf(c, c, c2);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    c2 += __shfl_xor_sync(0xffffffffu, c2, o);
    x2 += __shfl_xor_sync(0xffffffffu, x2, o);
  }
  if (lane == 0) {
    const float up = 1.0f + 1e-5f;
    aux[row] = x2;
    atomicMax(&stats->max_norm16, __float_as_uint(sqrtf(c2) * up));
    atomicMax(&stats->max_norm, __float_as_uint(sqrtf(x2) * up));
  }
}

// a / b rounded once, with y = 1 / b rounded once: Markstein's correction (IBM J. Res. Dev. 34, 1990) - the remainder of the
// product a y is exact in a fused operation, and adding its share rounds correctly while nothing over- or underflows.
__device__ __forceinline__ float div_rn_by(float a, float b, float y) {
  const float q = a * y;
  return fmaf(fmaf(-q, b, a), y, q);
}
// The reciprocal for a dimension's codes, or NaN where the correction does not hold for all of them: a code less the offset is 0 or
// no smaller than the smaller of |offset| and one unit in the last place of it.
__device__ __forceinline__ float div_reciprocal(float scale, float offset) {
  const float s = fabsf(scale), o = fabsf(offset);
  const bool plain = s >= 1e-12f && s <= 1e12f && (o == 0.f || o >= 1e-15f) && o <= 1e14f;
  return plain ? __frcp_rn(scale) : CUDART_NAN_F;
}

// Sums of RR rows of codes against the query in shared memory (qs, and behind it the dimensions' reciprocals): the metric between
// the fp32 query and x^ = (code - offset)/scale, every operation of x^ rounded by itself (ScalarQuantizer.swift:576-578).  A lane's
// dimensions are lane, lane + 32, ..; the parameters of a dimension serve all rows, its reciprocal replaces the rows' divisions, and a
// code becomes a number by its place in a mantissa (8 388 608 + 128 + code; conversions run at an eighth of the rate).
template <int METRIC, int RR>
__device__ __forceinline__ void i8_row_sums(const float* qs, const int8_t* __restrict__ codes, int dim, const float* __restrict__ scale,
                                            const float* __restrict__ offset, const uint32_t (&id)[RR], int lane, float (&sum)[RR]) {
  const uint8_t* xr[RR];
#pragma unroll
  for (int r = 0; r < RR; ++r) {
    xr[r] = reinterpret_cast<const uint8_t*>(codes) + (int64_t)id[r] * dim;
    sum[r] = 0.f;
  }
#pragma unroll 2
  for (int i = lane; i < dim; i += 32) {
    uint32_t code[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) code[r] = __ldg(xr[r] + i);
    const float sc = __ldg(scale + i), of = __ldg(offset + i), qv = qs[i], y = qs[dim + i];
    float xv[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) xv[r] = __fsub_rn(__uint_as_float(code[r] ^ 0x4b000080u) - 8388736.0f, of);
    if (y == y) {
#pragma unroll
      for (int r = 0; r < RR; ++r) xv[r] = div_rn_by(xv[r], sc, y);
    } else {
#pragma unroll
      for (int r = 0; r < RR; ++r) xv[r] = __fdiv_rn(xv[r], sc);
    }
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      if (METRIC == VSK_METRIC_EUCLIDEAN) {
        const float d = qv - xv[r];
        sum[r] = fmaf(d, d, sum[r]);
      } else {
        sum[r] = fmaf(qv, xv[r], sum[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RR; ++r)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
}

// Exact re-scoring against dequantised rows, dot product (the integer contraction's lists).  Four rows per warp step share a
// dimension's parameters and reciprocal: a row at a time, each code divided by its scale, the seven launches of 10 000 queries over
// 6.25 million x 384 took 2.84 ms.
__global__ void __launch_bounds__(256) rerank_i8_kernel(const float* __restrict__ q, const int8_t* __restrict__ codes,
                                                        int dim, const float* __restrict__ scale,
                                                        const float* __restrict__ offset, CandLists cand,
                                                        unsigned long long* total) {
  extern __shared__ float qs[];
  const int64_t qi = blockIdx.x;
  const int cnt = min(cand.count[qi], kCandCap);
  uint64_t* keys = cand.keys + qi * kCandCap;
  for (int i = threadIdx.x; i < dim; i += blockDim.x) {
    qs[i] = q[qi * dim + i];
    qs[dim + i] = div_reciprocal(__ldg(scale + i), __ldg(offset + i));
  }
  if (threadIdx.x == 0) atomicAdd(total, (unsigned long long)cnt);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  constexpr int RR = 4;
  for (int c0 = warp * RR; c0 < cnt; c0 += nwarps * RR) {
    uint32_t id[RR];
    float sum[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) id[r] = (uint32_t)keys[min(c0 + r, cnt - 1)];
    i8_row_sums<VSK_METRIC_DOT_PRODUCT, RR>(qs, codes, dim, scale, offset, id, lane, sum);
#pragma unroll
    for (int r = 0; r < RR; ++r)
      if (lane == r && c0 + r < cnt) *VSK_CHK_W(keys + c0 + r) = make_key(-sum[r], id[r]);
  }
}

// Sums of RR fp32 rows against the query in shared memory (direct formulas; a lane's dimensions are lane, lane + 32, .., added in
// that order), four loads of every row in flight.  Bound by the gathered rows; with one load of each row in flight the re-scoring
// of the list search was bound by their latency (10 000 queries of 128 dimensions: 690 us in two launches, 468 with four).
template <int METRIC, int RR>
__device__ __forceinline__ void f32_row_sums(const float* qs, const float* __restrict__ x, int dim, const uint32_t (&id)[RR], int lane,
                                             float (&sum)[RR]) {
  constexpr int U = 4;
  const float* xr[RR];
#pragma unroll
  for (int r = 0; r < RR; ++r) {
    xr[r] = x + (int64_t)id[r] * dim;
    sum[r] = 0.f;
  }
  for (int i0 = lane; i0 < dim; i0 += 32 * U) {
    float xv[RR][U];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < RR; ++r) xv[r][u] = i0 + 32 * u < dim ? __ldg(xr[r] + i0 + 32 * u) : 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float qv = i0 + 32 * u < dim ? qs[i0 + 32 * u] : 0.f;
#pragma unroll
      for (int r = 0; r < RR; ++r) {
        if (METRIC == VSK_METRIC_EUCLIDEAN) {
          const float d = qv - xv[r][u];
          sum[r] = fmaf(d, d, sum[r]);
        } else {
          sum[r] = fmaf(qv, xv[r][u], sum[r]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RR; ++r)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
}

// ---- exact rerank -------------------------------------------------------------------------
// One CTA per query: replaces every kept candidate's coarse value with the reference's direct fp32 value:
//   euclidean sum (q-x)^2 (rooted at output), cosine 1 - q.x/(|q||x| + 1e-8), dotProduct -(q.x).
template <int METRIC>
__global__ void __launch_bounds__(256) rerank_kernel(const float* __restrict__ q, const float* __restrict__ x, int dim,
                                                     const float* __restrict__ qnorm, const float* __restrict__ xnorm,
                                                     CandLists cand, unsigned long long* total) {
  extern __shared__ float qs[];
  const int64_t qi = blockIdx.x;
  const int cnt = min(cand.count[qi], kCandCap);
  uint64_t* keys = cand.keys + qi * kCandCap;
  for (int i = threadIdx.x; i < dim; i += blockDim.x) qs[i] = q[qi * dim + i];
  if (threadIdx.x == 0) atomicAdd(total, (unsigned long long)cnt);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const float qn = (METRIC == VSK_METRIC_COSINE) ? qnorm[qi] : 0.f;
  // four candidate rows per warp step: their key loads and row loads are independent chains, which is what keeps
  // enough bytes in flight when a row is only a few hundred bytes
  constexpr int RR = 4;
  for (int c0 = warp * RR; c0 < cnt; c0 += nwarps * RR) {
    uint32_t id[RR];
    float s[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) id[r] = (uint32_t)keys[min(c0 + r, cnt - 1)];
    f32_row_sums<METRIC, RR>(qs, x, dim, id, lane, s);
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      if (lane == 0 && c0 + r < cnt) {
        float v;
        if (METRIC == VSK_METRIC_COSINE) v = 1.0f - s[r] / (qn * xnorm[id[r]] + 1e-8f);
        else if (METRIC == VSK_METRIC_DOT_PRODUCT) v = -s[r];
        else v = s[r];
        keys[c0 + r] = make_key(v, id[r]);
      }
    }
  }
}

// ---- the second half of a flat search in one launch -------------------------------------------
// One CTA per query: the last compaction with its certificate (select_kernel's, see there), the exact values of the rows it
// keeps (rerank_kernel's formulas, summed in its order), the final order, and the query's flags (low byte) with the number of
// re-scored rows to the host.  The kept keys never leave shared memory, the rows of one query are fetched while another one's
// list is ordered, and two launches, the copies of the flags and the gaps between them are gone.
struct FinishArgs {
  CandLists cand;
  int32_t dense_count;        // >= 0: the list holds exactly this many slots
  const float *q, *x, *qnorm, *xnorm;
  const int8_t* codes;        // I8: the rows, with ...
  const float *sq_scale, *sq_offset;
  int32_t dim, k;
  const float* eps;
  const float* ext_bound;     // or null (SelectArgs::ext_bound)
  float* out_dist;
  int64_t* out_ids;
  int64_t id_base;
  const int32_t* err;         // device error word of the scans
  int32_t* host_err;          // pinned host memory ...
  int32_t* host_flags;        // [nq]
};
template <int NT> constexpr int kFinishMinBlocks = NT == 128 ? 8 : 2;

template <int METRIC, int NT, bool I8 = false>
__global__ void __launch_bounds__(NT, kFinishMinBlocks<NT>) finish_kernel(FinishArgs a) {
  extern __shared__ __align__(16) uint64_t s_keys[];
  constexpr int CAPACITY = NT * SEL_ITEMS;
  float* qs = reinterpret_cast<float*>(s_keys + CAPACITY);
  __shared__ int hist[256];
  __shared__ int s_valid, s_bin, s_less, s_in_bin, s_out;
  const int64_t qi = blockIdx.x;
  const uint64_t* keys = a.cand.keys + qi * kCandCap;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int raw = a.dense_count >= 0 ? a.dense_count : *VSK_CHK(a.cand.count + qi);
  const int c = min(raw, CAPACITY);
  uint64_t key[SEL_ITEMS];
  int nvalid = 0;
#pragma unroll
  for (int i = 0; i < SEL_ITEMS; ++i) {
    const int idx = threadIdx.x + i * NT;
    key[i] = idx < c ? *VSK_CHK(keys + idx) : kEmptyKey;
    nvalid += key[i] != kEmptyKey;
  }
  for (int i = threadIdx.x; i < a.dim; i += NT) {
    qs[i] = *VSK_CHK(a.q + qi * a.dim + i);
    if (I8) qs[a.dim + i] = div_reciprocal(__ldg(a.sq_scale + i), __ldg(a.sq_offset + i));
  }
  if (threadIdx.x == 0) { s_valid = 0; s_out = 0; }
  __syncthreads();
  nvalid = __reduce_add_sync(0xffffffffu, nvalid);
  if (lane == 0) atomicAdd(&s_valid, nvalid);
  __syncthreads();
  // a row of the true top-k has coarse value <= c_k + 2 eps; the list is complete only below the threshold that filtered the scan
  float bound = CUDART_INF_F;
  bool have = false;
  if (s_valid >= a.k) {
    const uint64_t kth = block_radix_select(key, a.k, hist, &s_bin, &s_less, &s_in_bin);
    bound = ordered_to_float((uint32_t)(kth >> 32)) + 2.0f * *VSK_CHK(a.eps + qi);
    have = true;
  }
  if (a.ext_bound != nullptr && *VSK_CHK(a.ext_bound + qi) < CUDART_INF_F) {
    bound = fminf(bound, *VSK_CHK(a.ext_bound + qi) + *VSK_CHK(a.eps + qi));
    have = true;
  }
  uint64_t pivot = kEmptyKey - 1;
  if (have) {
    pivot = ((uint64_t)float_to_ordered(bound) << 32) | 0xffffffffull;
    if (pivot == kEmptyKey) pivot = kEmptyKey - 1;
  }
#pragma unroll
  for (int i = 0; i < SEL_ITEMS; ++i)
    if (key[i] <= pivot && key[i] != kEmptyKey) s_keys[atomicAdd(&s_out, 1)] = key[i];
  __syncthreads();
  const int cnt = s_out;
  if (threadIdx.x == 0) {
    int flags = *VSK_CHK(a.cand.flags + qi);
    if (raw > CAPACITY) flags |= 1;
    if (have && !(bound < *VSK_CHK(a.cand.thr + qi))) flags |= 2;
    *VSK_CHK_W(a.host_flags + qi) = flags | (cnt << 8);
    if (qi == 0) *VSK_CHK_W(a.host_err) = *VSK_CHK(a.err);
  }
  // exact values: four rows per warp step, four loads of each in flight
  const float qn = (METRIC == VSK_METRIC_COSINE) ? *VSK_CHK(a.qnorm + qi) : 0.f;
  constexpr int RR = 4;
  for (int c0 = warp * RR; c0 < cnt; c0 += (NT / 32) * RR) {
    if constexpr (I8) {
      uint32_t id[RR];
      float sum[RR];
#pragma unroll
      for (int r = 0; r < RR; ++r) id[r] = (uint32_t)s_keys[min(c0 + r, cnt - 1)];
      i8_row_sums<METRIC, RR>(qs, a.codes, a.dim, a.sq_scale, a.sq_offset, id, lane, sum);
      __syncwarp();
#pragma unroll
      for (int r = 0; r < RR; ++r)
        if (lane == r && c0 + r < cnt) s_keys[c0 + r] = make_key(METRIC == VSK_METRIC_EUCLIDEAN ? sum[r] : -sum[r], id[r]);
      continue;
    }
    uint32_t id[RR];
    float sum[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) id[r] = (uint32_t)s_keys[min(c0 + r, cnt - 1)];
    f32_row_sums<METRIC, RR>(qs, a.x, a.dim, id, lane, sum);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      if (lane == 0 && c0 + r < cnt) {
        float v;
        if (METRIC == VSK_METRIC_COSINE) v = 1.0f - sum[r] / (qn * __ldg(a.xnorm + id[r]) + 1e-8f);
        else if (METRIC == VSK_METRIC_DOT_PRODUCT) v = -sum[r];
        else v = sum[r];
        s_keys[c0 + r] = make_key(v, id[r]);
      }
    }
  }
  __syncthreads();
  auto put = [&](int j, uint64_t key1, bool has) {
    float d = has ? ordered_to_float((uint32_t)(key1 >> 32)) : CUDART_INF_F;
    if (has && METRIC == VSK_METRIC_EUCLIDEAN) d = sqrtf(d);
    *VSK_CHK_W(a.out_dist + qi * a.k + j) = d;
    *VSK_CHK_W(a.out_ids + qi * a.k + j) = has ? (int64_t)(uint32_t)key1 + a.id_base : -1;
  };
  if (cnt <= 2 * NT) {   // keys are distinct: a key's place is the number of smaller ones
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int at = threadIdx.x + h * NT;
      if (at >= cnt) continue;
      const uint64_t mine = s_keys[at];
      int below = 0;
      for (int j = 0; j < cnt; ++j) below += s_keys[j] < mine;
      if (below < a.k) put(below, mine, true);
    }
    for (int j = cnt + threadIdx.x; j < a.k; j += NT) put(j, 0ull, false);
    return;
  }
  const int P = next_pow2(cnt);
  for (int i = cnt + threadIdx.x; i < P; i += NT) s_keys[i] = kEmptyKey;
  __syncthreads();
  bitonic_sort(s_keys, P);
  for (int j = threadIdx.x; j < a.k; j += NT) put(j, j < cnt ? s_keys[j] : 0ull, j < cnt);
}

// ---- host side ------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
        qr == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// fp16 matrix [rows][dim16] row-major; box = 64 columns x box_rows, 128-byte swizzle, zero fill
int32_t make_map(Ctx* ctx, const __half* base, int64_t rows, int32_t dim16, int box_rows, CUtensorMap* map) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(ctx, VSK_ERR_EXECUTION_FAILED, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t gdim[2] = {(cuuint64_t)dim16, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)dim16 * 2};
  cuuint32_t box[2] = {(cuuint32_t)TK, (cuuint32_t)box_rows};
  cuuint32_t estride[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(base), gdim, gstride, box, estride,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(ctx, VSK_ERR_EXECUTION_FAILED, "cuTensorMapEncodeTiled failed with %d", (int)r);
  return VSK_OK;
}

// The same matrix seen through a box of 16 columns x box_rows with the 32-byte swizzle: one K16 step of a tile.
int32_t make_map_narrow(Ctx* ctx, const __half* base, int64_t rows, int32_t dim16, int box_rows, CUtensorMap* map) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(ctx, VSK_ERR_EXECUTION_FAILED, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t gdim[2] = {(cuuint64_t)dim16, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)dim16 * 2};
  cuuint32_t box[2] = {16u, (cuuint32_t)box_rows};
  cuuint32_t estride[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(base), gdim, gstride, box, estride,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(ctx, VSK_ERR_EXECUTION_FAILED, "cuTensorMapEncodeTiled (16-column box) failed with %d", (int)r);
  return VSK_OK;
}

// int8 matrix [rows][stride bytes], `cols` of them valid: box = 128 columns x box_rows, 128-byte swizzle; columns past
// `cols` and rows past `rows` read as zero.  stride must be a multiple of 16.
int32_t make_map_i8(Ctx* ctx, const int8_t* base, int64_t rows, int32_t cols, int32_t stride, int box_rows, CUtensorMap* map) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(ctx, VSK_ERR_EXECUTION_FAILED, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)stride};
  cuuint32_t box[2] = {(cuuint32_t)(2 * TK), (cuuint32_t)box_rows};
  cuuint32_t estride[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t*>(base), gdim, gstride, box, estride,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(ctx, VSK_ERR_EXECUTION_FAILED, "cuTensorMapEncodeTiled (int8) failed with %d", (int)r);
  return VSK_OK;
}

// bytes [rows][32], whole rows: box = 32 bytes x box_rows, 32-byte swizzle
int32_t make_map_bytes(Ctx* ctx, const int8_t* base, int64_t rows, int box_rows, CUtensorMap* map) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(ctx, VSK_ERR_EXECUTION_FAILED, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t gdim[2] = {32, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {32};
  cuuint32_t box[2] = {32u, (cuuint32_t)box_rows};
  cuuint32_t estride[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t*>(base), gdim, gstride, box, estride,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(ctx, VSK_ERR_EXECUTION_FAILED, "cuTensorMapEncodeTiled (bytes) failed with %d", (int)r);
  return VSK_OK;
}

template <int METRIC>
void launch_prep(Ctx* ctx, const float* x, int64_t n, int dim, int dim16, const float* scale, __half* out, float* aux,
                 float* nrm16, float* err16, float* nrm, PrepStats* stats, FoldArgs fold = FoldArgs{0, 0, 0}) {
  prep_rows_kernel<METRIC><<<(unsigned)ceil_div(n, 8), 256, 0, ctx->stream>>>(x, n, dim, dim16, scale, out, aux, nrm16,
                                                                               err16, nrm, stats, fold);
  ctx->stats.kernel_launches++;
}

// max over rows of |x|^2, summed as prep_rows_kernel sums it (one warp per row)
__global__ void max_sq_kernel(const float* __restrict__ x, int64_t n, int dim, unsigned* out) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  const int lane = threadIdx.x & 31;
  const float* p = x + row * dim;
  float ss = 0.f;
  for (int i = lane; i < dim; i += 32) {
    const float v = __ldg(p + i);
    ss = fmaf(v, v, ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (lane == 0) atomicMax(out, __float_as_uint(ss));
}

// fp16 operand copy of the index rows + the constants of the error bound (once per index state)
int32_t tensor_prepare(Index* ix) {
  Ctx* ctx = ix->ctx;
  if (ix->n16 == ix->n && ix->rows16) return VSK_OK;
  dev_free(ix->rows16);
  dev_free(ix->row_aux);
  ix->rows16 = nullptr;
  ix->row_aux = nullptr;
  ix->dim16 = (int32_t)(ceil_div(ix->dim, TK) * TK);
  // Folding the per-row term into the operands (FoldArgs) pays where the epilogue, not the MMAs, sets the pace
  // (up to four K blocks), and is free where the padding already has room for it.
  ix->fold16 = ctx->tuning.fold_row_term != 0 && ix->kind != INDEX_FLAT_I8 && ix->metric == VSK_METRIC_EUCLIDEAN &&
               (ix->dim16 / TK <= 4 || ix->dim16 - fold_col0(ix->dim) >= kFoldCols);
  if (ix->fold16 && ix->dim16 - fold_col0(ix->dim) < kFoldCols) ix->dim16 += TK;
  VSK_TRY(dev_alloc(ctx, (void**)&ix->rows16, (size_t)ix->n * ix->dim16 * sizeof(__half)));
  VSK_TRY(dev_alloc(ctx, (void**)&ix->row_aux, (size_t)ix->n * sizeof(float)));
  void* p;
  VSK_TRY(scratch(ctx, SLOT_TC_A, sizeof(PrepStats) + 32, &p));
  PrepStats* st = (PrepStats*)p;
  float* scale = (float*)((char*)p + sizeof(PrepStats));
  unsigned* max_sq = (unsigned*)((char*)p + sizeof(PrepStats) + 16);
  PrepStats init{0u, 0u, 0u, 0u, 0x7f800000u};
  VSK_CUDA(ctx, cudaMemcpyAsync(st, &init, sizeof(init), cudaMemcpyHostToDevice, ctx->stream));
  const bool cosine = ix->metric == VSK_METRIC_COSINE;
  if (ix->kind == INDEX_FLAT_I8) {
    const float one = 1.0f;
    VSK_CUDA(ctx, cudaMemcpyAsync(scale, &one, 4, cudaMemcpyHostToDevice, ctx->stream));
    prep_codes_kernel<<<(unsigned)ceil_div(ix->n, 8), 256, 0, ctx->stream>>>(ix->codes, ix->n, ix->dim, ix->dim16, ix->sq_scale,
                                                                            ix->sq_offset, ix->rows16, ix->row_aux, st);
    ctx->stats.kernel_launches++;
  } else {
  if (!cosine) {
    absmax_kernel<<<1184, 256, 0, ctx->stream>>>(ix->rows, ix->n * (int64_t)ix->dim, &st->absmax);
    ctx->stats.kernel_launches++;
  }
  choose_scale_kernel<<<1, 1, 0, ctx->stream>>>(&st->absmax, cosine ? 1 : 0, scale);
  ctx->stats.kernel_launches++;
  FoldArgs fold{0, 0, 0};
  ix->fold_exp = 0;
  ix->fold_bmax = 0.f;
  if (ix->fold16) {
    // the exponent that brings the largest piece, s_x (|x|^2 / 2) 2^exp / 16, just below 2^14
    VSK_CUDA(ctx, cudaMemsetAsync(max_sq, 0, 4, ctx->stream));
    max_sq_kernel<<<(unsigned)ceil_div(ix->n, 8), 256, 0, ctx->stream>>>(ix->rows, ix->n, ix->dim, max_sq);
    ctx->stats.kernel_launches++;
    float hmax = 0.f, hscale = 1.f;
    VSK_CUDA(ctx, cudaMemcpyAsync(&hmax, max_sq, 4, cudaMemcpyDeviceToHost, ctx->stream));
    VSK_CUDA(ctx, cudaMemcpyAsync(&hscale, scale, 4, cudaMemcpyDeviceToHost, ctx->stream));
    VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const double top = 0.5 * (double)hmax * (double)hscale / 16.0;
    int e = 0;
    if (top > 0.0 && std::isfinite(top)) e = 14 - (int)std::ceil(std::log2(top));
    ix->fold_exp = std::max(-100, std::min(100, e));
    ix->fold_bmax = 0.5f * hmax;
    if (!std::isfinite(top)) ix->fold16 = false;   // the plain form copes with what overflows here no better, but is the known path
    fold = FoldArgs{ix->fold16 ? 1 : 0, fold_col0(ix->dim), ix->fold_exp};
  }
  switch (ix->metric) {
    case VSK_METRIC_EUCLIDEAN:
      launch_prep<VSK_METRIC_EUCLIDEAN>(ctx, ix->rows, ix->n, ix->dim, ix->dim16, scale, ix->rows16, ix->row_aux, nullptr, nullptr, nullptr, st, fold);
      break;
    case VSK_METRIC_COSINE:
      launch_prep<VSK_METRIC_COSINE>(ctx, ix->rows, ix->n, ix->dim, ix->dim16, scale, ix->rows16, ix->row_aux, nullptr, nullptr, nullptr, st);
      break;
    default:
      launch_prep<VSK_METRIC_DOT_PRODUCT>(ctx, ix->rows, ix->n, ix->dim, ix->dim16, scale, ix->rows16, ix->row_aux, nullptr, nullptr, nullptr, st);
      break;
  }
  }
  VSK_CUDA(ctx, cudaGetLastError());
  PrepStats h;
  float hs;
  VSK_CUDA(ctx, cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(&hs, scale, 4, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  auto f = [](unsigned u) { float v; memcpy(&v, &u, 4); return v; };
  ix->scale16 = hs;
  ix->max_xnorm16 = f(h.max_norm16);
  ix->max_xerr16 = f(h.max_err16);
  ix->max_xnorm = f(h.max_norm);
  ix->min_xnorm_nz = h.min_norm_nz == 0x7f800000u ? 0.f : f(h.min_norm_nz);
  ix->n16 = ix->n;
  return VSK_OK;
}

// Launches the scan over tiles (persistent: one CTA per SM, or per tile when there are fewer tiles).
template <int MODE, int EW, bool I8 = false>
int32_t launch_tc_ew(Ctx* ctx, const CUtensorMap& mq, const CUtensorMap& mx, const TcArgs& a, bool has_beta) {
  const bool has_mask = MODE != SCAN_ARGMIN && a.row_masks != nullptr && a.q_masks != nullptr;
  void (*kern)(CUtensorMap, CUtensorMap, TcArgs);
  constexpr bool BETA = EW == 8 && !I8;   // (tc_epilogue_warps: a per-row term comes with eight warps)
  if constexpr (I8) {
    kern = tc_scan_kernel<MODE, false, false, EW, true>;
  } else if constexpr (MODE == SCAN_ARGMIN) {
    kern = has_beta ? tc_scan_kernel<MODE, BETA, false, EW> : tc_scan_kernel<MODE, false, false, EW>;
  } else {
    kern = has_mask ? (has_beta ? tc_scan_kernel<MODE, BETA, true, EW> : tc_scan_kernel<MODE, false, true, EW>)
                    : (has_beta ? tc_scan_kernel<MODE, BETA, false, EW> : tc_scan_kernel<MODE, false, false, EW>);
  }
  const size_t smem = has_beta ? tc_smem_bytes<EW, BETA>() : tc_smem_bytes<EW, false>();
  VSK_CUDA(ctx, opt_in_shared(ctx, kern, smem));
  const int64_t tiles = a.tiles ? a.num_tiles : ceil_div(a.nq, TM) * ceil_div(a.row_end - a.row_begin, TN);
  if (tiles <= 0) return VSK_OK;
  const int sms = ctx->prop.multiProcessorCount;
  const unsigned grid = (unsigned)std::min<int64_t>(tiles, sms);
  TcArgs la = a;
  la.wait_limit = ctx->tuning.wait_limit_log2 > 0 ? (1u << std::min(ctx->tuning.wait_limit_log2, 30)) : 0u;
  la.stall_kblock = -1;
  la.stage_kblocks = ctx->tuning.stage_kblocks == 2 ? 2 : 1;
  if (ctx->tuning.test_stall_scan > 0) {   // testing only, one shot
    la.stall_kblock = 0;
    ctx->tuning.test_stall_scan = 0;
  }
  prof_begin(ctx);
  kern<<<grid, Epi<EW>::THREADS, smem, ctx->stream>>>(mq, mx, la);
  prof_end(ctx);
  tl_mark(ctx, MODE == SCAN_DENSE ? "scan_dense" : (MODE == SCAN_ARGMIN ? "scan_argmin" : "scan"));
  ctx->stats.kernel_launches++;
  ctx->stats.tensor_tiles += tiles;
  VSK_CUDA(ctx, cudaGetLastError());
  return VSK_OK;
}

// Epilogue warps by contraction length (see Epi): 16 up to four K blocks (d <= 256), 8 beyond and with a per-row term, which needs more
// registers than sixteen warps have (2 000 queries over 500 000 x 200 int8 rows, euclidean: 0.76 ms with eight, 1.24 with sixteen).
inline int tc_epilogue_warps(int kblocks, bool has_beta) { return kblocks <= 4 && !has_beta ? 16 : 8; }

template <int MODE>
int32_t launch_tc(Ctx* ctx, const CUtensorMap& mq, const CUtensorMap& mx, const TcArgs& a, bool has_beta) {
  if (tc_epilogue_warps(a.kblocks, has_beta) == 16) return launch_tc_ew<MODE, 16>(ctx, mq, mx, a, false);
  return launch_tc_ew<MODE, 8>(ctx, mq, mx, a, has_beta);
}

// ---- k-means assignment on the tensor cores ----------------------------------------------------
// Data rows are the streamed operand (the "query" side of the tile), centroids the small one.
//   pass 1  coarse arg-min: best[row] = smallest coarse (|c|^2 - 2 x.c, centroid) key
//   pass 2  every centroid whose coarse value is within 2 eps(row) of that minimum is appended to the
//           row's short list (the true nearest centroid is among them: its exact value is <= the exact
//           value of the coarse winner <= coarse minimum + eps, so its coarse value <= minimum + 2 eps)
//   exact   the listed centroids are compared with the direct fp32 formula sum (x-c)^2; the smallest
//           (value, index) wins, as the reference's strict '<' scan does (KMeansClustering.swift:283-288)
// A row whose list overflows (more near-ties than a sub-list holds) is re-done by the fp32 tile.
constexpr int kAssignLogPerRow = 6;
constexpr int kAssignCap = 32;   // split into one sub-list per column part of a tile (2 parts of 16, or 4 of 8)

// eps per data row against the current centroids; stats of the centroid operand are read on the device.
__global__ void assign_bound_kernel(const float* __restrict__ xn16, const float* __restrict__ xe16,
                                    const float* __restrict__ xnorm, int64_t n, const float* scale_x,
                                    const float* scale_c, const PrepStats* cs, int dim16, float* __restrict__ eps,
                                    float* alpha, int folded) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const float inv = 1.0f / ((*scale_x) * (*scale_c));
  if (r == 0) *alpha = -2.0f * inv;
  if (r >= n) return;
  const float C16 = __uint_as_float(cs->max_norm16), E16 = __uint_as_float(cs->max_err16);
  const float Cn = __uint_as_float(cs->max_norm);
  const float a = xn16[r], e = xe16[r];
  float dot_err = ((a * E16 + e * C16 + e * E16) + (float)dim16 * 2.3841858e-7f * a * C16) * inv;
  // |c|^2 / 2 carried inside the contraction: its products pass through the same fp32 accumulation, and three fp16
  // pieces leave less than 2^-30 of it unrepresented
  if (folded) dot_err += ((float)dim16 * 2.3841858e-7f + 9.3132257e-10f) * 0.5f * Cn * Cn;
  const float v = 2.0f * dot_err + 4.0f * 5.9604645e-8f * (float)dim16 * Cn * Cn +
                  2.0f * 5.9604645e-8f * (Cn * Cn + 2.0f * xnorm[r] * Cn);
  eps[r] = v * 1.0001f + 1e-30f;
}

__global__ void assign_threshold_kernel(const unsigned long long* __restrict__ best, const float* __restrict__ eps,
                                        int64_t n, float* __restrict__ thr, int32_t* __restrict__ count) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  thr[r] = ordered_to_float((uint32_t)(best[r] >> 32)) + 2.0f * eps[r];
  count[r] = 0;
}
// ... from the stationary kernel's values
__global__ void assign_value_threshold_kernel(const unsigned* __restrict__ best, const float* __restrict__ eps, int64_t n,
                                              float* __restrict__ thr, int32_t* __restrict__ count) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  thr[r] = ordered_to_float(best[r]) + 2.0f * eps[r];
  count[r] = 0;
}

// Thresholds of the next scan from the previous assignment (Lloyd iterations after the first).  With u the exact value
// |c_p|^2 - 2 x.c_p = |x - c_p|^2 - |x|^2 of the centroid the row was assigned to last time, the nearest centroid c* has
// exact value <= u, hence coarse value <= u + eps; the threshold is u + 2 eps (the second eps covers the fp32 rounding
// of u itself).  Two ways to u, chosen per row:
//   exact   one read of the row: sum (x - c_p)^2 and sum x^2 in fp32 (a warp per row, four rows in flight);
//   bound   no read at all, when the centroid has moved by no more than `ratio` of the row's distance to it: the
//           triangle inequality, |x - c_new| <= |x - c_old| + |c_new - c_old|, with the distance the last iteration
//           left in `dist_old`, the shifts in `shift` and the row norms measured when the operand was made.  The bound
//           is looser than the exact value by at most (2 ratio + ratio^2) of the squared distance, which lists a few
//           more centroids for the exact decision and costs nothing in correctness.
// A lane takes one of 32 consecutive rows; the rows that need the exact form are then done by the whole warp.
template <bool VEC>
__global__ void __launch_bounds__(256) assign_prev_threshold_kernel(
    const float* __restrict__ x, int64_t n, int dim, const float* __restrict__ cent, const int32_t* __restrict__ prev,
    const float* __restrict__ eps, float* __restrict__ thr, int32_t* __restrict__ count, const float* __restrict__ dist_old,
    const float* __restrict__ shift, const float* __restrict__ xnorm, float ratio) {
  const int lane = threadIdx.x & 31;
  const int64_t row0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32;
  if (row0 >= n) return;
  const int64_t mine = row0 + lane;
  const bool have = mine < n;
  bool need = have;
  if (have && dist_old != nullptr) {
    const float d = dist_old[mine], sft = shift[prev[mine]];
    if (d > 0.f && d < CUDART_INF_F && sft <= ratio * d) {
      const float xn = xnorm[mine], x2 = xn * xn;
      const float ub = (d + sft) * (1.0f + 1e-5f);
      const float ub2 = ub * ub;
      thr[mine] = (ub2 - x2) + 2.0f * eps[mine] + 1e-5f * (ub2 + x2);
      count[mine] = 0;
      need = false;
    }
  }
  unsigned todo = __ballot_sync(0xffffffffu, need);
  while (todo) {
    // up to four rows per step, each read by the whole warp
    int64_t rr[4];
    int nr = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      rr[r] = row0;
      if (todo) {
        const int l = __ffs((int)todo) - 1;
        todo &= todo - 1u;
        rr[r] = row0 + l;
        nr = r + 1;
      }
    }
    float d2[4] = {0.f, 0.f, 0.f, 0.f}, x2[4] = {0.f, 0.f, 0.f, 0.f};
    if (VEC) {
      const int nv = dim >> 2;
      const float4* xr[4];
      const float4* cr[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        xr[r] = reinterpret_cast<const float4*>(x + rr[r] * dim);
        cr[r] = reinterpret_cast<const float4*>(cent + (int64_t)prev[rr[r]] * dim);
      }
      for (int i = lane; i < nv; i += 32) {
        float4 a[4], b[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) { a[r] = __ldg(xr[r] + i); b[r] = __ldg(cr[r] + i); }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          float d;
          d = a[r].x - b[r].x; d2[r] = fmaf(d, d, d2[r]); x2[r] = fmaf(a[r].x, a[r].x, x2[r]);
          d = a[r].y - b[r].y; d2[r] = fmaf(d, d, d2[r]); x2[r] = fmaf(a[r].y, a[r].y, x2[r]);
          d = a[r].z - b[r].z; d2[r] = fmaf(d, d, d2[r]); x2[r] = fmaf(a[r].z, a[r].z, x2[r]);
          d = a[r].w - b[r].w; d2[r] = fmaf(d, d, d2[r]); x2[r] = fmaf(a[r].w, a[r].w, x2[r]);
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float* xr = x + rr[r] * dim;
        const float* cr = cent + (int64_t)prev[rr[r]] * dim;
        for (int i = lane; i < dim; i += 32) {
          const float xv = __ldg(xr + i), d = xv - __ldg(cr + i);
          d2[r] = fmaf(d, d, d2[r]);
          x2[r] = fmaf(xv, xv, x2[r]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        d2[r] += __shfl_xor_sync(0xffffffffu, d2[r], o);
        x2[r] += __shfl_xor_sync(0xffffffffu, x2[r], o);
      }
      if (lane == 0 && r < nr) {
        thr[rr[r]] = (d2[r] - x2[r]) + 2.0f * eps[rr[r]] + 4.0f * 5.9604645e-8f * (d2[r] + x2[r]);
        count[rr[r]] = 0;
      }
    }
  }
}

// |c_new - c_old| per centroid (one warp each), a hair above its fp32 value
__global__ void assign_shift_kernel(const float* __restrict__ cent, const float* __restrict__ old, int k, int dim,
                                    float* __restrict__ shift) {
  const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (c >= k) return;
  const int lane = threadIdx.x & 31;
  float s = 0.f;
  for (int i = lane; i < dim; i += 32) {
    const float d = cent[(int64_t)c * dim + i] - old[(int64_t)c * dim + i];
    s = fmaf(d, d, s);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) shift[c] = sqrtf(s) * (1.0f + 1e-5f);
}

// launches the vector form when the rows allow 16-byte loads; dist_old == nullptr: every row takes the exact form
static void launch_prev_threshold(Ctx* ctx, const float* rows, int64_t n, int dim, const float* centroids, const int32_t* assign,
                                  const float* eps, float* thr, int32_t* count, const float* dist_old, const float* shift,
                                  const float* xnorm, float ratio) {
  const bool vec = dim % 4 == 0 && ((uintptr_t)rows & 15) == 0 && ((uintptr_t)centroids & 15) == 0;
  const unsigned grid = (unsigned)ceil_div(n, 256);
  if (vec)
    assign_prev_threshold_kernel<true><<<grid, 256, 0, ctx->stream>>>(rows, n, dim, centroids, assign, eps, thr, count, dist_old, shift, xnorm, ratio);
  else
    assign_prev_threshold_kernel<false><<<grid, 256, 0, ctx->stream>>>(rows, n, dim, centroids, assign, eps, thr, count, dist_old, shift, xnorm, ratio);
}

// one warp per data row: exact squared distances to the listed centroids
__global__ void assign_exact_kernel(const float* __restrict__ x, int64_t n, int dim, const float* __restrict__ cent,
                                    const uint64_t* __restrict__ keys, const int32_t* __restrict__ count,
                                    int32_t* __restrict__ assign, float* __restrict__ dist, int32_t* __restrict__ bad_rows,
                                    int32_t* bad_count, int parts) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  const int lane = threadIdx.x & 31;
  // one 8-bit count per sub-list; the scan's column parts (2 or 4) each wrote one sub-list of kAssignCap / parts keys
  // parts == 0: one list of up to kAssignCap keys with a plain count (the stationary-block kernel)
  unsigned packed = (unsigned)count[row];
  int sub = kAssignCap;
  int total = 0;
  bool over = false;
  if (parts == 0) {
    total = (int)packed;
    over = total > kAssignCap;
    packed = (unsigned)min(total, 255);
    parts = 1;
  } else {
    sub = kAssignCap / parts;
    for (int p = 0; p < parts; ++p) {
      const int c = (int)((packed >> (8 * p)) & 0xffu);
      over |= c > sub;
      total += c;
    }
  }
  if (over || total <= 0) {
    if (lane == 0) bad_rows[atomicAdd(bad_count, 1)] = (int32_t)row;
    return;
  }
  const float* xr = x + row * dim;
  uint64_t bestk = kEmptyKey;
  for (int p = 0; p < parts; ++p)
  for (int c = 0; c < (int)((packed >> (8 * p)) & 0xffu); ++c) {
    const uint32_t id = (uint32_t)keys[row * kAssignCap + p * sub + c];
    const float* cr = cent + (int64_t)id * dim;
    float s = 0.f;
    for (int i = lane; i < dim; i += 32) {
      const float d = __ldg(xr + i) - __ldg(cr + i);
      s = fmaf(d, d, s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    bestk = min(bestk, make_key(s, id));
  }
  if (lane == 0) {
    assign[row] = (int32_t)(uint32_t)bestk;
    if (dist) dist[row] = sqrtf(ordered_to_float((uint32_t)(bestk >> 32)));
  }
}

__global__ void scatter_best_kernel(const unsigned long long* __restrict__ best, const int32_t* __restrict__ rows,
                                    int64_t m, int32_t* __restrict__ assign, float* __restrict__ dist) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const unsigned long long b = best[i];
  assign[rows[i]] = (int32_t)(uint32_t)b;
  if (dist) dist[rows[i]] = sqrtf(ordered_to_float((uint32_t)(b >> 32)));
}

// Scale of the centroid operand and exponent of the folded term for one Lloyd iteration (device-side, nothing is
// read back).  With M = max |c|^2 / 2: the largest of the three fp16 pieces of s_c M 2^e / 16 should sit just below
// 2^14, and the constants on the data side, 4u and 2u with u = s_x 2^-e, must be normal fp16 numbers: u <= 2^13.  When u
// would be too large the centroid scale is lowered by the excess (the pieces shrink, e grows, u shrinks); the error
// bound is computed from the measured residuals of whatever scale is used, so it stays valid.
__global__ void assign_fold_setup_kernel(const unsigned* max_sq, float* scale_c, const float* scale_x, int* exp_out, float* u_out) {
  const float M = 0.5f * __uint_as_float(*max_sq);
  float sc = *scale_c;
  const float sx = *scale_x;
  int e = 0;
  if (M > 0.f && M < CUDART_INF_F) {
    int m2;
    frexpf(sc * M * 0.0625f, &m2);   // sc M / 16 = f 2^m2, f in [0.5, 1)
    e = 14 - m2;                     // brings it to [2^13, 2^14)
    int ex;
    frexpf(sx, &ex);                 // sx = 2^(ex-1)
    const int lu = (ex - 1) - e;     // log2 of u
    if (lu > 13) {
      const int shift = lu - 13;
      sc = ldexpf(sc, -shift);
      e += shift;
    } else if (lu < -14) {
      e -= (-14 - lu);               // u up to the smallest normal; the pieces only get smaller
    }
  }
  *scale_c = sc;
  *exp_out = e;
  *u_out = ldexpf(sx, -e);
}

// the data operand's fold columns hold the constant u (one 16-byte store of eight copies per thread)
// (u_done: the constant the columns hold already - a Lloyd iteration whose exponent has not changed writes nothing)
__global__ void assign_fill_fold_kernel(__half* __restrict__ rows16, int64_t n, int dim16, int col0, const float* __restrict__ u,
                                        const float* __restrict__ u_done) {
  if (*u == *u_done) return;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int chunks = kFoldCols / 8;
  if (i >= n * chunks) return;
  const int64_t row = i / chunks;
  const int c = (int)(i - row * chunks);
  const __half h = __float2half_rn(*u * (c == 0 ? 4.0f : 2.0f));   // columns 0-7: 4u, columns 8-15: 2u
  const __half2 h2 = __halves2half2(h, h);
  uint4 v;
  v.x = v.y = v.z = v.w = *reinterpret_cast<const unsigned*>(&h2);
  *reinterpret_cast<uint4*>(rows16 + row * dim16 + col0 + c * 8) = v;
}

template <int MODE>
int32_t launch_assign_scan(Ctx* ctx, const CUtensorMap& mx, const CUtensorMap& mc, const CUtensorMap& mxn, const CUtensorMap& mcn,
                           AsArgs a, unsigned* grid_out = nullptr, int64_t* log_cap_out = nullptr) {
  VSK_CUDA(ctx, opt_in_shared(ctx, assign_scan_kernel<MODE>, kAsSmemBytes));
  const int sms = ctx->prop.multiProcessorCount;
  const int nb = (int)ceil_div(a.k, TN);
  const int64_t qtiles = ceil_div(a.n, TM);
  unsigned grid;
  if (nb <= sms) {
    a.groups = (int)std::max<int64_t>(1, std::min<int64_t>(sms / nb, qtiles));
    grid = (unsigned)(nb * a.groups);
  } else {
    a.groups = 1;
    grid = (unsigned)sms;
  }
  a.wait_limit = ctx->tuning.wait_limit_log2 > 0 ? (1u << std::min(ctx->tuning.wait_limit_log2, 30)) : 0u;
  a.log_cap = std::min<int64_t>(a.log_total / grid, 0x7fffffff);
  if (grid_out) *grid_out = grid;
  if (log_cap_out) *log_cap_out = a.log_cap;
  prof_begin(ctx);
  assign_scan_kernel<MODE><<<grid, AS_THREADS, kAsSmemBytes, ctx->stream>>>(mx, mc, mxn, mcn, a);
  prof_end(ctx);
  tl_mark(ctx, MODE == SCAN_ARGMIN ? "assign_argmin" : "assign_scan");
  ctx->stats.kernel_launches++;
  ctx->stats.tensor_tiles += (int64_t)nb * qtiles;
  VSK_CUDA(ctx, cudaGetLastError());
  return VSK_OK;
}

}  // namespace

void tensor_invalidate(Index* ix) {
  ix->n16 = -1;
  ix->n8 = -1;
  ix->i8_rest = PathRest{};
  ix->n_u8 = -1;
  ix->l1_work = 0.0;
  ix->l1_rest = PathRest{};
}
int32_t tensor_prepare_index(Index* ix) { return tensor_prepare(ix); }

int32_t make_map_rows_f32(Ctx* ctx, const float* base, int64_t rows, int32_t dim, int box_cols, int box_rows, CUtensorMap* map) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(ctx, VSK_ERR_EXECUTION_FAILED, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t gdim[2] = {(cuuint64_t)dim, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)dim * 4};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  cuuint32_t estride[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), gdim, gstride, box, estride,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(ctx, VSK_ERR_EXECUTION_FAILED, "cuTensorMapEncodeTiled (fp32 rows) failed with %d", (int)r);
  return VSK_OK;
}

// ---- query operands of a search -----------------------------------------------------------------------
// fp16 operand rows of the queries, their error bound eps[q], the output coefficient alpha, and the small words a
// search needs (device error word, re-scored row counter), all in the current lane's scratch.
struct QueryOperands {
  float* norm = nullptr;    // [nq] |q| (flat_query_operands)
  __half* q16 = nullptr;
  float* eps = nullptr;
  float* alpha = nullptr;
  float* scale = nullptr;   // device scalar s_q
  int32_t* err = nullptr;
  unsigned long long* rr_total = nullptr;
};

// Over product-quantised rows: one scale and coefficient for the batch, operand rows up to list_scan_kernel's whole blocks.
int32_t prepare_query_operands(Index* ix, const float* q, int64_t nq, QueryOperands* out) {
  VSK_TRACE("vsk:query_operands");
  Ctx* ctx = ix->ctx;
  prefer_shared_carveout(ctx, absmax_kernel, choose_scale_kernel, prep_rows_kernel<VSK_METRIC_EUCLIDEAN>, bound_kernel);
  const int dim = ix->dim, dim16 = ix->dim16;
  void* p;
  const int64_t nq_pad = ceil_div(nq, TN) * TN;
  VSK_TRY(scratch(ctx, SLOT_Q16, (size_t)nq_pad * dim16 * sizeof(__half), &p));
  __half* q16 = (__half*)p;
  if (nq_pad > nq) VSK_CUDA(ctx, cudaMemsetAsync(q16 + nq * dim16, 0, (size_t)(nq_pad - nq) * dim16 * sizeof(__half), ctx->stream));
  VSK_TRY(scratch(ctx, SLOT_QAUX, (size_t)nq * 4 * sizeof(float) + 64, &p));
  float* qn16 = (float*)p;
  float* qe16 = qn16 + nq;
  float* eps = qe16 + nq;
  float* qn_tmp = eps + nq;
  VSK_TRY(scratch(ctx, SLOT_TC_B, 64, &p));
  unsigned* q_absmax = (unsigned*)p;
  float* q_scale = (float*)p + 1;
  float* alpha = (float*)p + 2;
  int32_t* err = (int32_t*)p + 3;
  unsigned long long* rr_total = (unsigned long long*)((char*)p + 16);
  VSK_CUDA(ctx, cudaMemsetAsync(p, 0, 64, ctx->stream));
  absmax_kernel<<<296, 256, 0, ctx->stream>>>(q, nq * (int64_t)dim, q_absmax);
  const bool fold = ix->fold16;
  const FoldArgs qfold{fold ? 2 : 0, fold_col0(ix->dim), ix->fold_exp};
  // (list_scan_kernel may put twice the constants into the fold columns)
  choose_scale_kernel<<<1, 1, 0, ctx->stream>>>(q_absmax, 0, q_scale, fold ? 1 : 0, ix->fold_exp - 1);
  BoundConsts bc{ix->scale16, ix->max_xnorm16, ix->max_xerr16, ix->max_xnorm, ix->min_xnorm_nz, dim16, fold ? ix->fold_bmax : 0.f};
  launch_prep<VSK_METRIC_EUCLIDEAN>(ctx, q, nq, dim, dim16, q_scale, q16, nullptr, qn16, qe16, qn_tmp, nullptr, qfold);
  bound_kernel<<<(unsigned)ceil_div(nq, 256), 256, 0, ctx->stream>>>(qn16, qe16, qn_tmp, nq, q_scale, bc, eps, alpha);
  ctx->stats.kernel_launches += 3;
  VSK_CUDA(ctx, cudaGetLastError());
  tl_mark(ctx, "query_operands");
  out->q16 = q16;
  out->eps = eps;
  out->alpha = alpha;
  out->scale = q_scale;
  out->err = err;
  out->rr_total = rr_total;
  return VSK_OK;
}

// Over a flat index, fp32 rows or int8 codes: a scale and a coefficient per query (alpha is an array), and the lists emptied.
int32_t flat_query_operands(Index* ix, const float* q, int64_t nq, const CandLists& cand, QueryOperands* out) {
  VSK_TRACE("vsk:query_operands");
  Ctx* ctx = ix->ctx;
  prefer_shared_carveout(ctx, query_prep_kernel<VSK_METRIC_EUCLIDEAN>, query_prep_kernel<VSK_METRIC_COSINE>, query_prep_kernel<VSK_METRIC_DOT_PRODUCT>,
                         finish_kernel<VSK_METRIC_EUCLIDEAN, 128>, finish_kernel<VSK_METRIC_COSINE, 128>, finish_kernel<VSK_METRIC_DOT_PRODUCT, 128>,
                         finish_kernel<VSK_METRIC_EUCLIDEAN, 512>, finish_kernel<VSK_METRIC_COSINE, 512>, finish_kernel<VSK_METRIC_DOT_PRODUCT, 512>,
                         query_prep_kernel<VSK_METRIC_EUCLIDEAN, true>, query_prep_kernel<VSK_METRIC_DOT_PRODUCT, true>,
                         finish_kernel<VSK_METRIC_EUCLIDEAN, 128, true>, finish_kernel<VSK_METRIC_DOT_PRODUCT, 128, true>,
                         finish_kernel<VSK_METRIC_EUCLIDEAN, 512, true>, finish_kernel<VSK_METRIC_DOT_PRODUCT, 512, true>);
  const bool i8 = ix->kind == INDEX_FLAT_I8;
  if (i8 && ix->metric != VSK_METRIC_EUCLIDEAN && ix->metric != VSK_METRIC_DOT_PRODUCT)
    return fail(ctx, VSK_ERR_UNSUPPORTED_OPERATION, "the tensor path over int8 codes covers euclidean and dotProduct");
  QueryPrep a{};
  a.sq_scale = ix->sq_scale;
  void* p;
  VSK_TRY(scratch(ctx, SLOT_Q16, (size_t)nq * ix->dim16 * sizeof(__half), &p));
  a.out = (__half*)p;
  VSK_TRY(scratch(ctx, SLOT_QAUX, (size_t)nq * 4 * sizeof(float) + 64, &p));
  a.alpha = (float*)p;
  a.eps = a.alpha + nq;
  a.norm = a.eps + nq;
  VSK_TRY(scratch(ctx, SLOT_TC_B, 64, &p));
  a.words = (uint64_t*)p;
  a.q = q;
  a.nq = nq;
  a.dim = ix->dim;
  a.dim16 = ix->dim16;
  a.c = BoundConsts{ix->scale16, ix->max_xnorm16, ix->max_xerr16, ix->max_xnorm, ix->min_xnorm_nz, ix->dim16, ix->fold16 ? ix->fold_bmax : 0.f};
  a.fold = FoldArgs{ix->fold16 ? 2 : 0, fold_col0(ix->dim), ix->fold_exp};
  a.cand = cand;
  const unsigned grid = (unsigned)ceil_div(nq, 8);
  if (i8) {
    if (ix->metric == VSK_METRIC_EUCLIDEAN) query_prep_kernel<VSK_METRIC_EUCLIDEAN, true><<<grid, 256, 0, ctx->stream>>>(a);
    else query_prep_kernel<VSK_METRIC_DOT_PRODUCT, true><<<grid, 256, 0, ctx->stream>>>(a);
  } else
  switch (ix->metric) {
    case VSK_METRIC_EUCLIDEAN: query_prep_kernel<VSK_METRIC_EUCLIDEAN><<<grid, 256, 0, ctx->stream>>>(a); break;
    case VSK_METRIC_COSINE: query_prep_kernel<VSK_METRIC_COSINE><<<grid, 256, 0, ctx->stream>>>(a); break;
    default: query_prep_kernel<VSK_METRIC_DOT_PRODUCT><<<grid, 256, 0, ctx->stream>>>(a); break;
  }
  ctx->stats.kernel_launches++;
  VSK_CUDA(ctx, cudaGetLastError());
  tl_mark(ctx, "query_operands");
  out->q16 = a.out;
  out->eps = a.eps;
  out->alpha = a.alpha;
  out->norm = a.norm;
  out->err = (int32_t*)p;
  out->rr_total = (unsigned long long*)((char*)p + 16);
  return VSK_OK;
}

int32_t cand_lists(Ctx* ctx, int64_t nq, CandLists* cand) {
  void* p;
  VSK_TRY(scratch(ctx, SLOT_CAND_KEYS, (size_t)nq * kCandCap * sizeof(uint64_t), &p));
  cand->keys = (uint64_t*)p;
  VSK_TRY(scratch(ctx, SLOT_CAND_COUNT, (size_t)nq * 4, &p));
  cand->count = (int32_t*)p;
  VSK_TRY(scratch(ctx, SLOT_CAND_THR, (size_t)nq * 4, &p));
  cand->thr = (float*)p;
  VSK_TRY(scratch(ctx, SLOT_CAND_FLAGS, (size_t)nq * 4, &p));
  cand->flags = (int32_t*)p;
  cand->nq = nq;
  return VSK_OK;
}

// Whether a query row fits beside the largest list in finish_kernel's shared memory.
bool finish_applies(int dim) { return (size_t)dim * sizeof(float) <= 160 * 1024; }

template <int METRIC, int NT, bool I8>
int32_t launch_finish_as(Ctx* ctx, const FinishArgs& f, int64_t nq) {
  const size_t smem = (size_t)NT * SEL_ITEMS * sizeof(uint64_t) + (size_t)f.dim * sizeof(float) * (I8 ? 2 : 1);
  if (smem > 48 * 1024) VSK_CUDA(ctx, cudaFuncSetAttribute(finish_kernel<METRIC, NT, I8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  finish_kernel<METRIC, NT, I8><<<(unsigned)nq, NT, smem, ctx->stream>>>(f);
  tl_mark(ctx, "finish");
  ctx->stats.kernel_launches++;
  VSK_CUDA(ctx, cudaGetLastError());
  return VSK_OK;
}
// small: no list holds more than 1 024 keys
template <int METRIC, bool I8 = false>
int32_t launch_finish(Ctx* ctx, const FinishArgs& f, int64_t nq, bool small) {
  return small ? launch_finish_as<METRIC, 128, I8>(ctx, f, nq) : launch_finish_as<METRIC, 512, I8>(ctx, f, nq);
}

// The search in two halves.  `begin` runs the scan and its compactions; `finish` certifies, re-scores and orders.
// A plain search calls them back to back.  A shard of a row-sharded search passes `bound_out` (and the number of
// shards): the last compaction is then left to `finish`, and bound_out[q] gets a value that this shard's
// ceil(k / shards) best rows do not exceed; the host takes the maximum over the shards (at least k rows overall lie
// below it) and hands it to `finish`, which keeps only rows that can still reach the overall top-k.
// qmasks (or null): per-query filter masks; rows are then filtered in the contraction's epilogue.
int32_t tensor_search_begin(Index* ix, const float* q, int64_t nq, int32_t k, const float* qnorm, const uint64_t* qmasks,
                            int32_t shards, float* bound_out) {
  VSK_TRACE("vsk:scan");
  Ctx* ctx = ix->ctx;
  ctx->pending[ctx->lane] = ShardPending{};
  VSK_TRY(tensor_prepare(ix));
  const int metric = ix->metric;
  const int dim16 = ix->dim16;
  const int32_t keep = std::min<int32_t>(kCandCap / 2, k + std::max(8, k / 8));
  // The second half is one launch, the last compaction in it (finish_kernel); rows too wide for its shared memory keep the
  // separate ones.
  const bool fused = finish_applies(ix->dim);
  CandLists cand;
  VSK_TRY(cand_lists(ctx, nq, &cand));
  QueryOperands qo;
  VSK_TRY(flat_query_operands(ix, q, nq, cand, &qo));
  if (!qnorm) qnorm = qo.norm;
  const bool fold = ix->fold16;

  CUtensorMap mq, mx;
  VSK_TRY(make_map(ctx, qo.q16, nq, dim16, TM, &mq));
  VSK_TRY(make_map(ctx, ix->rows16, ix->n, dim16, TN, &mx));

  // ---- the chunk schedule ----
  TcArgs a{};
  a.alpha_per_query = 1;
  a.nq = nq;
  a.kblocks = dim16 / TK;
  a.k16_last = k16_last_of(fold ? fold_col0(ix->dim) + kFoldCols : ix->dim, dim16);
  a.alpha = qo.alpha;
  a.beta = (metric == VSK_METRIC_EUCLIDEAN && !fold) ? ix->row_aux : nullptr;
  a.cand = cand;
  a.cap = kCandCap;
  a.err = qo.err;
  if (qmasks && ix->has_masks) {
    a.row_masks = ix->masks;
    a.q_masks = qmasks;
  }
  const bool has_beta = a.beta != nullptr;
  SelectArgs sel{};
  sel.cand = cand;
  sel.nq = nq;
  sel.keep = keep;
  const int64_t n = ix->n;
  const int64_t room = kCandCap - keep;
  int64_t seen = std::min<int64_t>(n, schedule_dense_rows(ctx, keep));
  a.mode = SCAN_DENSE;
  a.row_begin = 0;
  a.row_end = seen;
  VSK_TRY(launch_tc<SCAN_DENSE>(ctx, mq, mx, a, has_beta));
  sel.dense_count = (int32_t)seen;
  sel.max_count = (int32_t)seen;
  sel.k = k;
  // the compaction after the last chunk keeps what the exact re-scoring needs and certifies the query; a shard
  // only measures its bound there and leaves that compaction to the second half
  bool skip_last = false;
  auto last_select = [&]() {
    if (bound_out == nullptr && fused) {
      skip_last = true;
    } else if (bound_out == nullptr) {
      sel.cert_eps = qo.eps;
    } else {
      sel.bound_out = bound_out;
      sel.bound_rank = (k + std::max(1, shards) - 1) / std::max(1, shards);
      sel.bound_eps = qo.eps;
    }
  };
  if (seen == n) last_select();
  if (!skip_last) VSK_TRY(launch_select(ctx, sel));
  // (a dense list that was only measured has had its count written)
  const int32_t dense_left = skip_last ? sel.dense_count : -1;
  sel.dense_count = -1;
  a.mode = SCAN_THRESHOLD;
  // A small batch is bound by its launches, not by its hits: fewer, faster-growing chunks (each still within what a
  // list can take, schedule_chunk) save a contraction and a compaction launch per step they skip.
  const int64_t growth = nq <= 2048 ? std::max(16, ctx->tuning.chunk_growth) : std::max(1, ctx->tuning.chunk_growth);
  while (seen < n) {
    // schedule_chunk bounds the chunk so that a list cannot plausibly overflow; below that bound chunks
    // grow geometrically (each no larger than three times the rows seen so far), which keeps the share of
    // rows scanned under a loose threshold small: the epilogue's append path costs far more than its filter.
    int64_t chunk = schedule_chunk(seen, keep, 0);
    chunk = std::min<int64_t>(chunk, std::max<int64_t>(growth >= 100 ? room : 1024, growth * seen));
    chunk = std::max<int64_t>(TN, chunk / TN * TN);   // whole row tiles
    chunk = std::min(chunk, n - seen);
    // The certificate compares the k-th value with the threshold of the last chunk, the keep-th value of the rows before it: were
    // that chunk a small remainder, the two would lie next to each other.  The last two chunks are of one ratio then.
    // 300 000 x 768, cosine, 1 000 queries, k = 100 (1 024, 16 384, 278 528 and 4 064 rows): 564 queries re-run, 8 290 us,
    // now none and 690 (lists of 3 k / 2 keys: 710, but 1 million x 128, dot product, 2 000 queries: 1 350 for 1 236).
    if (const int64_t rest = n - seen - chunk; rest > 0 && 2 * rest < seen + chunk)
      chunk = std::min(chunk, ceil_div((int64_t)std::sqrt((double)seen * (double)n) - seen, TN) * TN);
    a.row_begin = seen;
    a.row_end = seen + chunk;
    VSK_TRY(launch_tc<SCAN_THRESHOLD>(ctx, mq, mx, a, has_beta));
    sel.max_count = schedule_max_count(seen, chunk, keep);
    seen += chunk;
    if (seen == n) last_select();
    if (!skip_last) VSK_TRY(launch_select(ctx, sel));
  }
  ShardPending& pd = ctx->pending[ctx->lane];
  pd.active = true;
  pd.tensor = true;
  pd.ix = ix;
  pd.q = q;
  pd.nq = nq;
  pd.k = k;
  pd.qnorm = qnorm;
  pd.qmasks = a.q_masks;
  pd.cand = cand;
  pd.eps = qo.eps;
  pd.err = qo.err;
  pd.rr_total = qo.rr_total;
  pd.keep = keep;
  pd.max_count = sel.max_count;
  pd.need_cert = bound_out != nullptr;
  pd.fused = fused;
  pd.dense_count = dense_left;
  return VSK_OK;
}

// Second half, part one: everything that can be enqueued without looking at results - the certifying compaction
// (a shard's), the exact re-scoring, the final order, and the copy of the flag words to pinned host memory.
int32_t tensor_search_finish_issue(Index* ix, const float* ext_bound, float* out_dist, int64_t* out_ids) {
  VSK_TRACE("vsk:finish");
  Ctx* ctx = ix->ctx;
  ShardPending& pd = ctx->pending[ctx->lane];
  if (!pd.active || !pd.tensor || pd.ix != ix || pd.issued)
    return fail(ctx, VSK_ERR_INVALID_INPUT, "no search is waiting for its second half on this index");
  const float* q = pd.q;
  const float* qnorm = pd.qnorm;
  const int64_t nq = pd.nq;
  const int32_t k = pd.k, keep = pd.keep;
  const CandLists cand = pd.cand;
  const int metric = ix->metric;
  const int dim = ix->dim;
  const bool i8 = ix->kind == INDEX_FLAT_I8;
  if (i8 && dim > 12 * 1024) return fail(ctx, VSK_ERR_INVALID_BUFFER_SIZE, "dimension %d is too large for the int8 rerank kernel", dim);
  PinnedBuf& hb = ctx->host_flags[ctx->lane];
  VSK_TRY(pinned_reserve(ctx, &hb, (size_t)nq * 4 + 16));
  if (pd.fused) {
    FinishArgs f{};
    f.cand = cand;
    f.dense_count = pd.dense_count;
    f.q = q;
    f.x = ix->rows;
    f.qnorm = qnorm;
    f.xnorm = ix->row_norm;
    f.codes = ix->codes;
    f.sq_scale = ix->sq_scale;
    f.sq_offset = ix->sq_offset;
    f.dim = dim;
    f.k = k;
    f.eps = pd.eps;
    f.ext_bound = ext_bound;
    f.out_dist = out_dist;
    f.out_ids = out_ids;
    f.id_base = ix->id_base;
    f.err = pd.err;
    f.host_err = (int32_t*)hb.p;
    f.host_flags = (int32_t*)hb.p + 4;
    const bool small = pd.max_count <= 128 * SEL_ITEMS && pd.dense_count <= 128 * SEL_ITEMS;
    if (i8) {
      if (metric == VSK_METRIC_EUCLIDEAN) VSK_TRY((launch_finish<VSK_METRIC_EUCLIDEAN, true>(ctx, f, nq, small)));
      else VSK_TRY((launch_finish<VSK_METRIC_DOT_PRODUCT, true>(ctx, f, nq, small)));
    } else
    switch (metric) {
      case VSK_METRIC_EUCLIDEAN: VSK_TRY(launch_finish<VSK_METRIC_EUCLIDEAN>(ctx, f, nq, small)); break;
      case VSK_METRIC_COSINE: VSK_TRY(launch_finish<VSK_METRIC_COSINE>(ctx, f, nq, small)); break;
      default: VSK_TRY(launch_finish<VSK_METRIC_DOT_PRODUCT>(ctx, f, nq, small)); break;
    }
    pd.issued = true;
    pd.out_dist = out_dist;
    pd.out_ids = out_ids;
    return VSK_OK;
  }
  if (pd.need_cert) {
    SelectArgs sel{};
    sel.cand = cand;
    sel.nq = nq;
    sel.keep = keep;
    sel.dense_count = -1;
    sel.k = k;
    sel.cert_eps = pd.eps;
    sel.ext_bound = ext_bound;
    sel.max_count = pd.max_count;
    VSK_TRY(launch_select(ctx, sel));
  }

  // ---- exact rerank + final order ----
  const size_t qsm = (size_t)dim * sizeof(float);
  if (qsm > 200 * 1024) return fail(ctx, VSK_ERR_INVALID_BUFFER_SIZE, "dimension %d is too large for the rerank kernel", dim);
#define VSK_RERANK(M_)                                                                                          \
  do {                                                                                                          \
    if (qsm > 48 * 1024)                                                                                        \
      VSK_CUDA(ctx, cudaFuncSetAttribute(rerank_kernel<M_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)qsm)); \
    rerank_kernel<M_><<<(unsigned)nq, 256, qsm, ctx->stream>>>(q, ix->rows, dim, qnorm, ix->row_norm, cand, pd.rr_total); \
  } while (0)
  switch (metric) {
    case VSK_METRIC_EUCLIDEAN: VSK_RERANK(VSK_METRIC_EUCLIDEAN); break;
    case VSK_METRIC_COSINE: VSK_RERANK(VSK_METRIC_COSINE); break;
    default: VSK_RERANK(VSK_METRIC_DOT_PRODUCT); break;
  }
#undef VSK_RERANK
  tl_mark(ctx, "rerank");
  ctx->stats.kernel_launches++;
  VSK_CUDA(ctx, cudaGetLastError());
  SelectArgs fin{};
  fin.cand = cand;
  fin.nq = nq;
  fin.dense_count = -1;
  fin.keep = k;
  fin.out_dist = out_dist;
  fin.out_ids = out_ids;
  fin.k = k;
  fin.metric = metric;
  fin.id_base = ix->id_base;
  fin.final_sqrt = metric == VSK_METRIC_EUCLIDEAN;
  fin.max_count = keep;
  VSK_TRY(launch_select(ctx, fin));

  // ---- flag words to the host: bounded-wait expiry, overflowed lists, failed certificates ----
  char* h = (char*)hb.p;
  VSK_CUDA(ctx, cudaMemcpyAsync(h, pd.err, 4, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(h + 8, pd.rr_total, 8, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(h + 16, cand.flags, (size_t)nq * 4, cudaMemcpyDeviceToHost, ctx->stream));
  pd.issued = true;
  pd.out_dist = out_dist;
  pd.out_ids = out_ids;
  return VSK_OK;
}

// Second half, part two, after the stream of lane `from_lane` has drained: reads that lane's flag words and re-runs
// on the fp32 scan (on the CURRENT lane) the queries whose candidate list overflowed or whose result could not be
// certified.
int32_t tensor_search_finish_collect(Index* ix, int from_lane) {
  Ctx* ctx = ix->ctx;
  if (from_lane < 0) from_lane = ctx->lane;
  const ShardPending pd = ctx->pending[from_lane];
  ctx->pending[from_lane] = ShardPending{};
  if (!pd.active || !pd.issued || pd.ix != ix)
    return fail(ctx, VSK_ERR_INVALID_INPUT, "no search is waiting to be collected on this index");
  const char* h = (const char*)ctx->host_flags[from_lane].p;
  int32_t herr;
  unsigned long long hrr;
  memcpy(&herr, h, 4);
  memcpy(&hrr, h + 8, 8);
  const int32_t* flags = (const int32_t*)(h + 16);
  if (pd.fused) {   // the words of finish_kernel: flags in the low byte, re-scored rows above
    hrr = 0;
    for (int64_t i = 0; i < pd.nq; ++i) hrr += (unsigned)flags[i] >> 8;
  }
  ctx->stats.reranked_rows += (int64_t)hrr;
  if (herr != 0)
    return fail(ctx, VSK_ERR_TIMEOUT, "tensor-core scan: a bounded pipeline wait ran out (role %d)", herr);
  std::vector<int32_t> bad;
  for (int64_t i = 0; i < pd.nq; ++i)
    if (flags[i] & 0xff) bad.push_back((int32_t)i);
  if (!bad.empty()) VSK_TRY(fp32_search_subset(ix, pd.q, bad, pd.k, pd.qnorm, pd.qmasks, pd.out_dist, pd.out_ids));
  return VSK_OK;
}

int32_t tensor_search_finish(Index* ix, const float* ext_bound, float* out_dist, int64_t* out_ids) {
  Ctx* ctx = ix->ctx;
  VSK_TRY(tensor_search_finish_issue(ix, ext_bound, out_dist, out_ids));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return tensor_search_finish_collect(ix, -1);
}

// How a batch of nq queries is split over the two lanes: the first half's size (a whole number of query tiles), or 0
// for one lane.  Two lanes need enough queries that each half still fills the machine, and timing the scan kernels
// with events (vsk_profile) needs them alone on the device.
int64_t tensor_lane_split(const Ctx* ctx, int64_t nq) {
  const int64_t min_q = ctx->tuning.overlap_min_queries;
  if (min_q <= 0 || nq < min_q || nq < 4 * TM || ctx->profile) return 0;
  return ceil_div(ceil_div(nq, 2), TM) * TM;
}

int32_t tensor_search(Index* ix, const float* q, int64_t nq, int32_t k, const float* qnorm, const uint64_t* qmasks,
                      float* out_dist, int64_t* out_ids) {
  Ctx* ctx = ix->ctx;
  const int64_t na = ctx->lane == 0 ? tensor_lane_split(ctx, nq) : 0;
  if (na == 0) {
    VSK_TRY(tensor_search_begin(ix, q, nq, k, qnorm, qmasks, 1, nullptr));
    return tensor_search_finish(ix, nullptr, out_dist, out_ids);
  }
  // Two halves on two streams.  Each half is a complete search of its own queries (own candidate lists, own
  // operands); the device runs one half's compactions, re-scoring and final order while the other half's
  // contraction holds the tensor cores.
  VSK_TRY(tensor_prepare(ix));   // the shared operand copy is made before the lanes part
  const int64_t nb = nq - na;
  const float* qb = q + na * ix->dim;
  const float* qnb = qnorm ? qnorm + na : nullptr;
  const uint64_t* qmb = qmasks ? qmasks + na : nullptr;
  VSK_TRY(lanes_fork(ctx));
  int32_t st = VSK_OK;
  auto on_lane = [&](int lane, auto&& fn) {
    if (st != VSK_OK) return;
    LaneGuard g(ctx, lane);
    st = fn();
  };
  on_lane(0, [&] { return tensor_search_begin(ix, q, na, k, qnorm, qmasks, 1, nullptr); });
  on_lane(1, [&] { return tensor_search_begin(ix, qb, nb, k, qnb, qmb, 1, nullptr); });
  on_lane(0, [&] { return tensor_search_finish_issue(ix, nullptr, out_dist, out_ids); });
  on_lane(1, [&] { return tensor_search_finish_issue(ix, nullptr, out_dist + na * k, out_ids + na * k); });
  const int32_t jst = lanes_join(ctx);
  cudaStreamSynchronize(ctx->stream_main);   // lane 1 has joined: both halves are complete (or failed)
  if (st != VSK_OK || jst != VSK_OK) {
    cudaStreamSynchronize(ctx->stream_aux);
    ctx->pending[0] = ShardPending{};
    ctx->pending[1] = ShardPending{};
    return st != VSK_OK ? st : jst;
  }
  // flagged queries of either half are re-run on lane 0, whose own work is over
  const int32_t sa = tensor_search_finish_collect(ix, 0);
  const int32_t sb = tensor_search_finish_collect(ix, 1);
  return sa != VSK_OK ? sa : sb;
}

// keys of a dense chunk -> their values, row-major [nq][rows]
__global__ void keys_to_values_kernel(const uint64_t* __restrict__ keys, int64_t nq, int64_t rows, float* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq * rows) return;
  const int64_t q = i / rows, r = i - q * rows;
  out[i] = ordered_to_float((uint32_t)(keys[q * kCandCap + r] >> 32));
}

// The coarse values of the first `rows` rows (one dense chunk of the scan) and the bound the certificate assumes.
int32_t tensor_coarse_values(Index* ix, const float* q, int64_t nq, int64_t rows, float* coarse, float* eps_out) {
  Ctx* ctx = ix->ctx;
  if (rows <= 0 || rows > kCandCap || rows > ix->n)
    return fail(ctx, VSK_ERR_INVALID_BUFFER_SIZE, "rows must be in [1, min(%d, index size)]", kCandCap);
  VSK_TRY(tensor_prepare(ix));
  CandLists cand;
  VSK_TRY(cand_lists(ctx, nq, &cand));
  QueryOperands qo;
  VSK_TRY(flat_query_operands(ix, q, nq, cand, &qo));
  CUtensorMap mq, mx;
  VSK_TRY(make_map(ctx, qo.q16, nq, ix->dim16, TM, &mq));
  VSK_TRY(make_map(ctx, ix->rows16, ix->n, ix->dim16, TN, &mx));
  TcArgs a{};
  a.alpha_per_query = 1;
  a.nq = nq;
  a.kblocks = ix->dim16 / TK;
  a.k16_last = k16_last_of(ix->fold16 ? fold_col0(ix->dim) + kFoldCols : ix->dim, ix->dim16);
  a.alpha = qo.alpha;
  a.beta = (ix->metric == VSK_METRIC_EUCLIDEAN && !ix->fold16) ? ix->row_aux : nullptr;
  a.cand = cand;
  a.cap = kCandCap;
  a.err = qo.err;
  a.mode = SCAN_DENSE;
  a.row_begin = 0;
  a.row_end = rows;
  VSK_TRY(launch_tc<SCAN_DENSE>(ctx, mq, mx, a, a.beta != nullptr));
  keys_to_values_kernel<<<(unsigned)ceil_div(nq * rows, 256), 256, 0, ctx->stream>>>(cand.keys, nq, rows, coarse);
  ctx->stats.kernel_launches++;
  VSK_CUDA(ctx, cudaGetLastError());
  if (eps_out) VSK_CUDA(ctx, cudaMemcpyAsync(eps_out, qo.eps, (size_t)nq * 4, cudaMemcpyDeviceToDevice, ctx->stream));
  int32_t herr = 0;
  VSK_CUDA(ctx, cudaMemcpyAsync(&herr, qo.err, 4, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (herr != 0) return fail(ctx, VSK_ERR_TIMEOUT, "tensor-core scan: a bounded pipeline wait ran out (role %d)", herr);
  return VSK_OK;
}


// ---- IVF list scan on the tensor cores --------------------------------------------------------------
// The probed lists of a batch, scanned with the same contraction kernel as the flat search.  Every (query, probed
// list) pair is an item; items are grouped by (stage, list), and the fp16 query operand is gathered in that order,
// so the queries that probe a list are consecutive rows of the "query" operand and a tile is 128 of them against
// 256 rows of the list.  The tiles of a launch are listed list by list (a list's rows are read from HBM once).
// Three launches: a pilot over the first rows of every query's nearest list with no threshold, then the remaining
// probe ranks in two groups (the rest of the nearest list is an item of the first group).  The kernel filters on
// the flat path's coarse values (|x|^2 - 2 q.x from fp16 operands); after every launch all listed rows are
// re-scored exactly and the k best exact values are kept, so thresholds are exact and the filter only has to be
// loose by the coarse values' error bound: no certificate is needed and the only queries handed back are those
// whose list overflowed.
constexpr int kIvfPilotTiles = 4;   // 1 024 rows of the nearest list set the first threshold

// key of item (query, slot): stage * nlist + list, or null_key.  Slot p < nprobe is probe rank p (stage 0 for the
// nearest list, 1 for ranks below r1, 2 above); slot nprobe is the rest of the nearest list beyond the pilot window.
__global__ void ivf_item_keys_kernel(const int64_t* __restrict__ probes, int64_t nq, int nprobe, int nlist, int r1,
                                     const int64_t* __restrict__ list_off, int64_t pilot_rows, int null_key,
                                     int32_t* __restrict__ keys) {
  const int slots = nprobe + 1;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq * slots) return;
  const int64_t pos = i / slots;
  const int p = (int)(i - pos * slots);
  int key = null_key;
  if (p < nprobe) {
    const int64_t l = probes[pos * nprobe + p];
    if (l >= 0 && l < nlist) key = (p == 0 ? 0 : (p < r1 ? 1 : 2)) * nlist + (int)l;
  } else {
    const int64_t l = probes[pos * nprobe];
    if (l >= 0 && l < nlist && list_off[l + 1] - list_off[l] > pilot_rows) key = nlist + (int)l;
  }
  keys[i] = key;
}

// per grouped item: its query and whether it is a remainder item; and the item's row of the gathered fp16 operand
__global__ void ivf_gather_items_kernel(const int32_t* __restrict__ order, int64_t nitems, int slots,
                                        const __half* __restrict__ q16, int dim16, uint32_t* __restrict__ pair_info,
                                        __half* __restrict__ g16) {
  const int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= nitems) return;
  const int item = order[i];
  const int pos = item / slots;
  const int lane = threadIdx.x & 31;
  if (lane == 0) pair_info[i] = (uint32_t)pos | ((item - pos * slots) == slots - 1 ? 0x80000000u : 0u);
  const uint4* src = reinterpret_cast<const uint4*>(q16 + (int64_t)pos * dim16);
  uint4* dst = reinterpret_cast<uint4*>(g16 + i * dim16);
  for (int c = lane; c < dim16 / 8; c += 32) dst[c] = __ldg(src + c);
}

// tiles of (stage, list): ceil(pairs / 128) x row tiles (the pilot takes only the window)
__device__ __forceinline__ int ivf_row_tiles(int64_t len, int stage, int pilot_tiles) {
  const int t = (int)((len + TN - 1) / TN);
  return stage == 0 ? min(pilot_tiles, t) : t;
}

__global__ void ivf_tile_count_kernel(const int64_t* __restrict__ pair_off, int stage, int nlist,
                                      const int64_t* __restrict__ list_off, int64_t* __restrict__ counts,
                                      int pilot_tiles) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= nlist) return;
  const int64_t pairs = pair_off[(int64_t)stage * nlist + l + 1] - pair_off[(int64_t)stage * nlist + l];
  counts[l] = ((pairs + TM - 1) / TM) * ivf_row_tiles(list_off[l + 1] - list_off[l], stage, pilot_tiles);
}

__global__ void ivf_tile_fill_kernel(const int64_t* __restrict__ pair_off, int stage, int nlist,
                                     const int64_t* __restrict__ list_off, const int64_t* __restrict__ offsets,
                                     int4* __restrict__ tiles, int pilot_tiles) {
  const int l = blockIdx.x;
  const int64_t pbeg = pair_off[(int64_t)stage * nlist + l], pairs = pair_off[(int64_t)stage * nlist + l + 1] - pbeg;
  const int64_t beg = list_off[l], len = list_off[l + 1] - beg;
  const int ptiles = (int)((pairs + TM - 1) / TM), rtiles = ivf_row_tiles(len, stage, pilot_tiles);
  int4* out = tiles + offsets[l];
  for (int i = threadIdx.x; i < ptiles * rtiles; i += blockDim.x) {
    const int rt = i / ptiles, pt = i - rt * ptiles;
    const int64_t r0 = (int64_t)rt * TN;
    out[i] = make_int4((int)(pbeg + (int64_t)pt * TM), (int)(beg + r0),
                       (int)min((int64_t)TN, len - r0) | ((rt < pilot_tiles ? 1 : 0) << 30),
                       (int)min((int64_t)TM, pairs - (int64_t)pt * TM));
  }
}

// after the exact rerank: a key's row field goes from its storage position to the row's insertion index, so that
// the final order breaks ties the way the fp32 list scan does
__global__ void ivf_remap_keys_kernel(CandLists cand, int64_t nq, const int32_t* __restrict__ list_rows) {
  const int64_t qi = blockIdx.x;
  const int cnt = min(cand.count[qi], kCandCap);
  uint64_t* keys = cand.keys + qi * kCandCap;
  for (int c = threadIdx.x; c < cnt; c += blockDim.x) {
    const uint64_t key = keys[c];
    if (key != kEmptyKey) keys[c] = (key & 0xffffffff00000000ull) | (uint32_t)list_rows[(uint32_t)key];
  }
}

// Coarse-domain threshold of a query from its exact one.  A row's exact squared distance is |q|^2 + c with
// c = |x|^2 - 2 q.x, and its coarse value differs from c by at most eps, so every row with exact value <= T has
// coarse value <= T - |q|^2 + eps; the last term covers fp32 rounding of the quantities being compared.
// `dropped` (or null): the smallest coarse value the pilot's coarse pre-selection dropped for the query.  The pilot
// keeps only its best rows by coarse value before the exact re-scoring; that is safe iff everything it dropped lies
// above the coarse threshold, otherwise the query is flagged for the fp32 list scan.
__global__ void ivf_coarse_threshold_kernel(const float* __restrict__ thr_exact, const float* __restrict__ qnorm,
                                            const float* __restrict__ eps, float max_xnorm, int64_t nq,
                                            float* __restrict__ thr_coarse, const float* __restrict__ dropped,
                                            int32_t* __restrict__ flags) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  const float t = thr_exact[i];
  float tc = CUDART_INF_F;
  if (t < CUDART_INF_F) {
    const float qn2 = qnorm[i] * qnorm[i];
    tc = (t - qn2) + eps[i] + 2e-6f * (qn2 + max_xnorm * max_xnorm + t);
  }
  *VSK_CHK_W(thr_coarse + i) = tc;
  if (dropped && dropped[i] <= tc) atomicOr(&flags[i], 2);
}

// saved[i] = thr[i]; thr[i] = +inf (the next compaction works on exact values and must not inherit a coarse one)
__global__ void ivf_save_threshold_kernel(float* __restrict__ thr, float* __restrict__ saved, int64_t nq) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  saved[i] = thr[i];
  thr[i] = CUDART_INF_F;
}

// threshold of every item's query, so that the scan reads it with the item's index
__global__ void ivf_pair_threshold_kernel(const uint32_t* __restrict__ pair_info, int64_t nitems,
                                          const float* __restrict__ thr_coarse, float* __restrict__ pair_thr) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nitems) pair_thr[i] = thr_coarse[pair_info[i] & 0x7fffffffu];
}

bool ivf_tensor_applicable(const Index* ix, int64_t nq, int32_t nprobe, int32_t k) {
  return ix->kind == INDEX_IVF && nq >= 2 * TM && k <= kCandCap / 4 && ix->n >= 8 * TN &&
         (int64_t)nq * (nprobe + 1) < ((int64_t)1 << 30);
}

int32_t ivf_tensor_search(Index* ix, const float* q, int64_t nq, const int64_t* probes, int32_t nprobe, int32_t k,
                          const uint64_t* qmasks, float* out_dist, int64_t* out_ids, std::vector<int32_t>* flagged) {
  VSK_TRACE("vsk:ivf_list_scan");
  Ctx* ctx = ix->ctx;
  flagged->clear();
  VSK_TRY(tensor_prepare(ix));
  const int dim = ix->dim, dim16 = ix->dim16, nlist = ix->nlist;
  const int32_t keep = k;   // every compaction works on exact values, so no margin is needed
  void* p;

  // ---- query operands, bound, alpha (euclidean) ----
  VSK_TRY(scratch(ctx, SLOT_Q16, (size_t)nq * dim16 * sizeof(__half), &p));
  __half* q16 = (__half*)p;
  VSK_TRY(scratch(ctx, SLOT_QAUX, (size_t)nq * 4 * sizeof(float) + 64, &p));
  float* qn16 = (float*)p;
  float* qe16 = qn16 + nq;
  float* eps = qe16 + nq;
  float* qn_tmp = eps + nq;
  VSK_TRY(scratch(ctx, SLOT_TC_B, 64, &p));
  unsigned* q_absmax = (unsigned*)p;
  float* q_scale = (float*)p + 1;
  float* alpha = (float*)p + 2;
  int32_t* err = (int32_t*)p + 3;
  unsigned long long* rr_total = (unsigned long long*)((char*)p + 16);
  VSK_CUDA(ctx, cudaMemsetAsync(p, 0, 64, ctx->stream));
  absmax_kernel<<<296, 256, 0, ctx->stream>>>(q, nq * (int64_t)dim, q_absmax);
  const bool fold = ix->fold16;
  const FoldArgs qfold{fold ? 2 : 0, fold_col0(ix->dim), ix->fold_exp};
  choose_scale_kernel<<<1, 1, 0, ctx->stream>>>(q_absmax, 0, q_scale, fold ? 1 : 0, ix->fold_exp);
  ctx->stats.kernel_launches += 2;
  BoundConsts bc{ix->scale16, ix->max_xnorm16, ix->max_xerr16, ix->max_xnorm, ix->min_xnorm_nz, dim16, fold ? ix->fold_bmax : 0.f};
  launch_prep<VSK_METRIC_EUCLIDEAN>(ctx, q, nq, dim, dim16, q_scale, q16, nullptr, qn16, qe16, qn_tmp, nullptr, qfold);
  bound_kernel<<<(unsigned)ceil_div(nq, 256), 256, 0, ctx->stream>>>(qn16, qe16, qn_tmp, nq, q_scale, bc, eps, alpha);
  ctx->stats.kernel_launches++;
  VSK_CUDA(ctx, cudaGetLastError());

  // ---- stage plan: which probe ranks go with the remainder of the nearest list ----
  const double mean_len = std::max(1.0, (double)ix->n / (double)nlist);
  const int pilot_tiles = ctx->tuning.ivf_pilot_tiles > 0 ? ctx->tuning.ivf_pilot_tiles : kIvfPilotTiles;
  const int64_t pilot_rows = (int64_t)pilot_tiles * TN;
  // rows one launch may add after the pilot's rows without (plausibly) overflowing a list: the flat schedule's rule.
  // When all probed lists fit, one launch takes every remaining rank; otherwise the ranks are split in two groups.
  const double chunk = (double)schedule_chunk(pilot_rows, keep, 0);
  int r1 = mean_len * nprobe <= chunk ? (int)nprobe : (int)(chunk / 4.0 / mean_len);
  r1 = std::max(1, std::min(r1, (int)nprobe));
  const int nstages = r1 < nprobe ? 3 : 2;

  // ---- items grouped by (stage, list); the query operand gathered in that order ----
  const int slots = nprobe + 1;
  const int64_t nitems = nq * slots;
  const int nkeys = 3 * nlist + 1;
  VSK_TRY(scratch(ctx, SLOT_IVF_KEYS, (size_t)nitems * 4, &p));
  int32_t* keys = (int32_t*)p;
  VSK_TRY(scratch(ctx, SLOT_IVF_ORDER, (size_t)nitems * 4, &p));
  int32_t* order = (int32_t*)p;
  VSK_TRY(scratch(ctx, SLOT_IVF_PAIR_OFF, (size_t)(nkeys + 1) * 8, &p));
  int64_t* pair_off = (int64_t*)p;
  ivf_item_keys_kernel<<<(unsigned)ceil_div(nitems, 256), 256, 0, ctx->stream>>>(probes, nq, nprobe, nlist, r1, ix->list_offsets,
                                                                              pilot_rows, nkeys - 1, keys);
  ctx->stats.kernel_launches++;
  VSK_TRY(launch_stable_group(ctx, keys, nitems, nkeys, order, pair_off));
  VSK_TRY(scratch(ctx, SLOT_IVF_SUBSET, (size_t)(nitems + TM) * 8, &p));   // one tile of padding behind each array
  uint32_t* pair_info = (uint32_t*)p;
  float* pair_thr = (float*)(pair_info + nitems + TM);
  VSK_CUDA(ctx, cudaMemsetAsync(pair_info, 0, (size_t)(nitems + TM) * 8, ctx->stream));
  VSK_TRY(scratch(ctx, SLOT_IVF_STAGES, (size_t)(nitems + TM) * dim16 * sizeof(__half), &p));
  __half* g16 = (__half*)p;
  ivf_gather_items_kernel<<<(unsigned)ceil_div(nitems, 8), 256, 0, ctx->stream>>>(order, nitems, slots, q16, dim16, pair_info, g16);
  ctx->stats.kernel_launches++;

  CUtensorMap mq, mx;
  VSK_TRY(make_map(ctx, g16, nitems, dim16, TM, &mq));
  VSK_TRY(make_map(ctx, ix->rows16, ix->n, dim16, TN, &mx));

  CandLists cand;
  VSK_TRY(scratch(ctx, SLOT_CAND_KEYS, (size_t)nq * kCandCap * sizeof(uint64_t), &p));
  cand.keys = (uint64_t*)p;
  VSK_TRY(scratch(ctx, SLOT_CAND_COUNT, (size_t)nq * 4, &p));
  cand.count = (int32_t*)p;
  VSK_TRY(scratch(ctx, SLOT_CAND_THR, (size_t)nq * 4, &p));
  cand.thr = (float*)p;
  VSK_TRY(scratch(ctx, SLOT_CAND_FLAGS, (size_t)nq * 4, &p));
  cand.flags = (int32_t*)p;
  cand.nq = nq;
  VSK_TRY(launch_init_cand(ctx, cand, nq));

  // the kernel filters on coarse values: it sees the lists with a coarse threshold derived from the exact one
  VSK_TRY(scratch(ctx, SLOT_TC_D, (size_t)nq * sizeof(float), &p));
  float* thr_coarse = (float*)p;
  CandLists cand_coarse = cand;
  cand_coarse.thr = thr_coarse;
  VSK_TRY(scratch(ctx, SLOT_TC_C, (size_t)nq * sizeof(float), &p));
  float* pilot_dropped = (float*)p;
  const int32_t pilot_keep = std::min<int32_t>(1024, std::max(8 * k, 256));
  TcArgs a{};
  a.nq = nq;
  a.kblocks = dim16 / TK;
  a.k16_last = k16_last_of(fold ? fold_col0(ix->dim) + kFoldCols : ix->dim, dim16);
  a.mode = SCAN_THRESHOLD;
  a.alpha = alpha;
  a.beta = fold ? nullptr : ix->row_aux;
  a.cand = cand_coarse;
  a.cap = kCandCap;
  a.err = err;
  a.pair_info = pair_info;
  if (qmasks && ix->has_masks) {   // masks are kept in storage order, the order of the row operand
    a.row_masks = ix->masks;
    a.q_masks = qmasks;
  }
  SelectArgs sel{};
  sel.cand = cand;
  sel.nq = nq;
  sel.keep = keep;
  sel.dense_count = -1;
  sel.k = k;
  const size_t qsm = (size_t)dim * sizeof(float);
  if (qsm > 48 * 1024) return fail(ctx, VSK_ERR_INVALID_BUFFER_SIZE, "dimension %d is too large for the rerank kernel", dim);
  const unsigned qgrid = (unsigned)ceil_div(nq, 256);

  void *cnt_p, *off_p;
  VSK_TRY(scratch(ctx, SLOT_IVF_ITEM_CNT, (size_t)(nlist + 1) * 8, &cnt_p));
  VSK_TRY(scratch(ctx, SLOT_IVF_ITEM_OFF, (size_t)(nlist + 1) * 8, &off_p));
  for (int stage = 0; stage < nstages; ++stage) {
    ivf_tile_count_kernel<<<(unsigned)ceil_div(nlist, 256), 256, 0, ctx->stream>>>(pair_off, stage, nlist, ix->list_offsets, (int64_t*)cnt_p, pilot_tiles);
    VSK_TRY(launch_scan_i64(ctx, (const int64_t*)cnt_p, nlist, (int64_t*)off_p));
    int64_t total = 0;
    VSK_CUDA(ctx, cudaMemcpyAsync(&total, (int64_t*)off_p + nlist, 8, cudaMemcpyDeviceToHost, ctx->stream));
    VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    ctx->stats.kernel_launches += 2;
    if (total <= 0) continue;
    if (total > 0x7fffffffLL) return fail(ctx, VSK_ERR_INVALID_BUFFER_SIZE, "too many list tiles in one launch");
    VSK_TRY(scratch(ctx, SLOT_X_TMP, (size_t)total * sizeof(int4), &p));
    ivf_tile_fill_kernel<<<(unsigned)nlist, 128, 0, ctx->stream>>>(pair_off, stage, nlist, ix->list_offsets, (const int64_t*)off_p, (int4*)p, pilot_tiles);
    ivf_coarse_threshold_kernel<<<qgrid, 256, 0, ctx->stream>>>(cand.thr, qn_tmp, eps, ix->max_xnorm, nq, thr_coarse,
                                                                nullptr, cand.flags);
    ivf_pair_threshold_kernel<<<(unsigned)ceil_div(nitems, 256), 256, 0, ctx->stream>>>(pair_info, nitems, thr_coarse, pair_thr);
    ctx->stats.kernel_launches += 3;
    a.tiles = (const int4*)p;
    a.num_tiles = total;
    a.pair_thr = pair_thr;
    if (stage == 0) VSK_TRY(launch_tc<SCAN_ALL>(ctx, mq, mx, a, !fold));
    else VSK_TRY(launch_tc<SCAN_THRESHOLD>(ctx, mq, mx, a, !fold));
    if (stage == 0) {
      // the pilot appended up to 1 024 rows per query: keep the best few by coarse value and re-score only those
      SelectArgs pre = sel;
      pre.keep = pilot_keep;
      pre.max_count = (int32_t)pilot_rows;
      VSK_TRY(launch_select(ctx, pre));
      ivf_save_threshold_kernel<<<qgrid, 256, 0, ctx->stream>>>(cand.thr, pilot_dropped, nq);
      ctx->stats.kernel_launches++;
    }
    // exact values for everything in the lists (the keys kept so far are re-scored too: at most k of them),
    // then the k best exact values stay and the k-th becomes the query's exact threshold
    rerank_kernel<VSK_METRIC_EUCLIDEAN><<<(unsigned)nq, 256, qsm, ctx->stream>>>(q, ix->rows, dim, nullptr, nullptr, cand, rr_total);
    ctx->stats.kernel_launches++;
    sel.max_count = stage == 0 ? pilot_keep : kCandCap;
    sel.by_length = stage == 0 ? 0 : 1;
    VSK_TRY(launch_select(ctx, sel));
    if (stage == 0) {
      // was the coarse pre-selection safe?  (also refreshes the coarse thresholds, which the next launch recomputes)
      ivf_coarse_threshold_kernel<<<qgrid, 256, 0, ctx->stream>>>(cand.thr, qn_tmp, eps, ix->max_xnorm, nq, thr_coarse,
                                                                  pilot_dropped, cand.flags);
      ctx->stats.kernel_launches++;
    }
  }

  // ---- ids back to insertion order, final order ----
  ivf_remap_keys_kernel<<<(unsigned)nq, 128, 0, ctx->stream>>>(cand, nq, ix->list_rows);
  ctx->stats.kernel_launches++;
  VSK_CUDA(ctx, cudaGetLastError());
  SelectArgs fin{};
  fin.cand = cand;
  fin.nq = nq;
  fin.dense_count = -1;
  fin.keep = k;
  fin.out_dist = out_dist;
  fin.out_ids = out_ids;
  fin.k = k;
  fin.metric = VSK_METRIC_EUCLIDEAN;
  fin.id_base = ix->id_base;
  fin.final_sqrt = 1;
  fin.max_count = keep;
  VSK_TRY(launch_select(ctx, fin));

  std::vector<int32_t> flags((size_t)nq);
  int32_t herr = 0;
  unsigned long long hrr = 0;
  VSK_CUDA(ctx, cudaMemcpyAsync(flags.data(), cand.flags, nq * 4, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(&hrr, rr_total, 8, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ctx->stats.reranked_rows += (int64_t)hrr;
  if (herr != 0)
    return fail(ctx, VSK_ERR_TIMEOUT, "tensor-core scan: a bounded pipeline wait ran out (role %d)", herr);
  for (int64_t i = 0; i < nq; ++i)
    if (flags[i]) flagged->push_back((int32_t)i);
  return VSK_OK;
}

constexpr int64_t kLsWindowBytes = 40ll << 20;   // rows a window of list_scan_kernel keeps in L2

template <bool I8>
static int32_t launch_list_scan(Ctx* ctx, const CUtensorMap& mx, const CUtensorMap& mq, const CUtensorMap& mxn, const CUtensorMap& mqn,
                                LsArgs a, int64_t row_bytes) {
  VSK_CUDA(ctx, opt_in_shared(ctx, list_scan_kernel<I8>, kLsSmemBytes));
  const int64_t tiles = ceil_div(a.nq, TN) * ceil_div(a.rows, TM);
  if (tiles <= 0) return VSK_OK;
  a.window = (int32_t)std::max<int64_t>(1, kLsWindowBytes / (row_bytes * TM));
  a.wait_limit = ctx->tuning.wait_limit_log2 > 0 ? (1u << std::min(ctx->tuning.wait_limit_log2, 30)) : 0u;
  if (ctx->tuning.test_stall_scan > 0) {   // testing only, one shot
    a.stall = 1;
    ctx->tuning.test_stall_scan = 0;
  }
  const unsigned grid = (unsigned)std::min<int64_t>(tiles, ctx->prop.multiProcessorCount);
  // room for 256 rows per query (a chunk lists a few times k); what does not fit is appended by the scan itself
  const int64_t total = std::max<int64_t>(1 << 16, std::min<int64_t>(a.nq * 256, 8 << 20));
  void* p;
  VSK_TRY(scratch(ctx, SLOT_LS_LOG, (size_t)total * sizeof(uint2) + (size_t)grid * sizeof(int32_t), &p));
  a.log = (uint2*)p;
  a.log_count = (int32_t*)(a.log + total);
  a.log_cap = total / grid;
  prof_begin(ctx);
  list_scan_kernel<I8><<<grid, AS_THREADS, kLsSmemBytes, ctx->stream>>>(mx, mq, mxn, mqn, a);
  prof_end(ctx);
  tl_mark(ctx, "list_scan");
  ls_scatter_kernel<<<dim3(8, grid), 256, 0, ctx->stream>>>(a.log, a.log_count, a.log_cap, a.cand);
  ctx->stats.kernel_launches += 2;
  ctx->stats.tensor_tiles += tiles;
  VSK_CUDA(ctx, cudaGetLastError());
  return VSK_OK;
}

// Fold columns of the query operand for list_scan_kernel, once per chunk: the row term's constants (8u x4, 4u x4) and the
// pieces of minus the bar.  A row is listed iff  acc = s_q s_x (q.x - |x|^2 / 2)  reaches  bar = -thr s_q s_x / 2, lowered by
// the fp32 accumulation error of its own products.  A bar the columns cannot hold from below flags the query.
// The columns hold |bar| <= kTop = 3.9e9.  With X the bound on the rows' norms, s_q s_x X^2 / 2 is below 2^30 (fold_exp and the
// query scale, choose_scale_kernel), and so is |bar| / (2 |q| / X + 1): only queries of more than 1.3 X can come near kTop.  A bar above
// it is clipped, which lists more rows.
__global__ void ls_fold_queries_kernel(const float* __restrict__ thr, int64_t nq, int64_t nq_pad, const float* scale_q, float scale_x, int fold_exp,
                                       int dim16, int col0, __half* __restrict__ q16, int32_t* __restrict__ flags) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq_pad) return;
  const float s = *scale_q, u = i < nq ? ldexpf(s, -fold_exp) : 0.f;
  float R = i < nq ? -0.5f * *VSK_CHK(thr + i) * s * scale_x : 1e9f;   // the bar
  R = R - fabsf(R) * ((float)dim16 * 2.3841858e-7f + 1e-6f) - 1e-30f;
  constexpr float kTop = 2.0f * kLsBarConst * 60000.f;
  if (!(R >= -kTop)) {                                 // (also what is not a number)
    R = -kTop;
    atomicOr(&flags[i], 2);
  }
  R = fminf(R, kTop);
  const float inv = 1.0f / (2.0f * kLsBarConst);       // minus the bar = 2 c p0 + 2 c p1 + 4 c p2
  const __half p0 = __float2half_rn(-R * inv);
  const float r1 = -R - 2.0f * kLsBarConst * __half2float(p0);
  const __half p1 = __float2half_rn(r1 * inv);
  const __half p2 = __float2half_ru((r1 - 2.0f * kLsBarConst * __half2float(p1)) * (0.5f * inv));   // never below: the bar is not raised
  __align__(16) __half h[16];
#pragma unroll
  for (int j = 0; j < 16; ++j)
    h[j] = j < 8 ? __float2half_rn(j < 4 ? 8.0f * u : 4.0f * u) : j < 10 ? p0 : j < 12 ? p1 : p2;
  uint4* dst = reinterpret_cast<uint4*>(q16 + i * dim16 + col0);
  *VSK_CHK_W(dst) = *reinterpret_cast<const uint4*>(&h[0]);
  *VSK_CHK_W(dst + 1) = *reinterpret_cast<const uint4*>(&h[8]);
}

// The same for int8 operands: 32 bytes b per query with 127 sum(b) >= -bar, the bar rounded down to a step of 127.
// The bytes hold bars from -516 128 to 520 192; accumulators reach 127 x 127 x 384 = 6.2e6.  Codes and queries
// that are not far from centred stay within (N(0,1) data, 384 dimensions: 1e5); where the k-th product lies beyond, the clipped
// bar lists rows that cannot matter, lists may overflow, and the index rests from this path (Index::i8_rest).
__global__ void ls_bar_bytes_kernel(const int32_t* __restrict__ bar, int64_t nq, int64_t nq_pad, int8_t* __restrict__ out,
                                    int32_t* __restrict__ flags) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq_pad) return;
  const int64_t want = i < nq ? -(int64_t)*VSK_CHK(bar + i) : -100000;
  int64_t total = want >= 0 ? (want + kLsBarByte - 1) / kLsBarByte : -((-want) / kLsBarByte);   // rounded up
  if (total > 32 * 127) {   // more rows would have to be listed than the bytes can ask for
    total = 32 * 127;
    atomicOr(&flags[i], 2);
  }
  total = max(total, (int64_t)-32 * 128);
  const int base = (int)(total >= 0 ? total / 32 : -((-total + 31) / 32));
  const int rest = (int)(total - (int64_t)base * 32);   // 0 .. 31 of the bytes are one larger
  __align__(16) int8_t h[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) h[j] = (int8_t)(base + (j < rest ? 1 : 0));
  uint4* dst = reinterpret_cast<uint4*>(out + i * 32);
  *VSK_CHK_W(dst) = *reinterpret_cast<const uint4*>(&h[0]);
  *VSK_CHK_W(dst + 1) = *reinterpret_cast<const uint4*>(&h[16]);
}

// ---- product-quantised rows on the tensor cores -------------------------------------------------------------
// The asymmetric distance of a code row is the squared distance between the query and the row the code decodes to,
// so a batch of queries over m-byte codes is the same contraction as over fp32 rows.  The table scan (pq.cu) does m
// shared-memory gathers per (query, row) and is bound by them (10 000 queries x 10 000 000 rows x 16 segments: 1.6e12
// gathers); the contraction costs 2 (d + 16) flop on the tensor cores instead.  Per chunk of rows:
//   decode     code rows to fp16 operand rows in a bounded work buffer, |x^|^2 / 2 in sixteen folded columns (FoldArgs)
//   contract   tc_scan_kernel with thresholds that allow for the coarse values' error
//   re-score   every listed row from the query's table, summed in segment order: the values the table scan forms,
//              bit for bit; the k best stay and give the next exact threshold
// The thresholds are exact (as in the list scan above), so no certificate is needed: bulk ties of quantised distances
// only lengthen a list, and a query whose list overflows is handed back to the table scan.
constexpr int64_t kPqBlockBytes = 512ll << 20;   // decoded operand rows held at a time
constexpr int PQ_DEC_ROWS = 64;                  // rows per CTA of the decode kernel

// One CTA decodes PQ_DEC_ROWS rows: codes and |x^|^2 (segment sums of the codewords' norms) are staged in shared
// memory, then every thread writes 16-byte pieces of the operand rows.  Bound by the issue of the pieces (a gather from the
// codebook and a store each): 10 000 000 rows of 128 in 12 blocks take 1.22 ms, against 0.45 ms for their 2.9 GB; it was 1.88 ms
// with a division per piece and the 48 columns of padding written as well.
// DS: 2, 4, 8 = the segment length; 16 = any multiple of 8 (a piece lies inside one codeword); 0 = any length.
template <int DS>
__global__ void __launch_bounds__(256) pq_decode16_kernel(const uint8_t* __restrict__ codes, int64_t n, int dim, int dim16, int m,
                                                          int ksub, int ds_rt, const __half* __restrict__ cb16,
                                                          const float* __restrict__ cw2, float scale, int fold, int col0,
                                                          int fold_exp, __half* __restrict__ out, float* __restrict__ aux) {
  extern __shared__ uint8_t sc[];   // [PQ_DEC_ROWS][m]
  __shared__ float n2[PQ_DEC_ROWS];
  const int ds = (DS > 0 && DS <= 8) ? DS : ds_rt;
  const int64_t r0 = (int64_t)blockIdx.x * PQ_DEC_ROWS;
  const int rows = (int)min((int64_t)PQ_DEC_ROWS, n - r0);
  for (int i = threadIdx.x; i < rows * m; i += blockDim.x) sc[i] = __ldg(codes + r0 * m + i);
  __syncthreads();
  {
    // four threads per row
    const int r = threadIdx.x >> 2, part = threadIdx.x & 3;
    float s = 0.f;
    if (r < rows)
      for (int g = part; g < m; g += 4) s += __ldg(cw2 + (int64_t)g * ksub + sc[r * m + g]);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (part == 0 && r < rows) {
      n2[r] = s;
      if (aux) *VSK_CHK_W(aux + r0 + r) = s;
    }
  }
  __syncthreads();
  // Columns past the last K16 step that the contraction takes are not written: no MMA reads them (k16_last_of).
  // The division by the pieces of a row is a multiplication: with inv = (2^20 + e) / pieces, e < pieces, the quotient is exact
  // while t e < 2^20, and t is below 64 pieces: for up to 128 pieces (rows of up to 1 024 columns).
  const int pieces = (fold ? col0 + kFoldCols : (dim + 15) / 16 * 16) >> 3;
  const uint32_t inv = ((1u << 20) + (uint32_t)pieces - 1u) / (uint32_t)pieces;
  for (int t = threadIdx.x; t < rows * pieces; t += blockDim.x) {
    const int r = pieces <= 128 ? (int)(((uint32_t)t * inv) >> 20) : t / pieces, c = (t - r * pieces) * 8;
    __align__(16) __half h[8];
    if (fold && c >= col0 && c < col0 + kFoldCols) {
      // pieces of R = s (|x^|^2 / 2) 2^exp as in prep_rows_kernel
      const float R = ldexpf(0.5f * n2[r] * scale, fold_exp);
      const __half p0 = __float2half_rn(R * 0.0625f);
      const float r1 = R - 16.0f * __half2float(p0);
      const __half p1 = __float2half_rn(r1 * 0.0625f);
      const __half p2 = __float2half_rn((r1 - 16.0f * __half2float(p1)) * 0.0625f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        // fold 2: list_scan_kernel's columns (the row term in eight of them, the constant of the thresholds in the rest)
        if (fold == 2) h[j] = c == col0 ? __hneg(j < 2 ? p0 : j < 4 ? p1 : p2) : __float2half_rn(kLsBarConst);
        else h[j] = __hneg(c == col0 ? (j < 4 ? p0 : p1) : p2);
      }
    } else if (DS > 0 && c + 8 <= dim) {
      constexpr int W = DS > 0 ? (DS < 8 ? DS : 8) : 1;   // halves taken from one codeword
#pragma unroll
      for (int j = 0; j < 8; j += W) {
        const int g = (c + j) / ds;
        const __half* w = cb16 + ((int64_t)g * ksub + sc[r * m + g]) * ds + ((c + j) - g * ds);
        if constexpr (W == 8) *reinterpret_cast<uint4*>(&h[j]) = __ldg(reinterpret_cast<const uint4*>(w));
        else if constexpr (W == 4) *reinterpret_cast<uint2*>(&h[j]) = __ldg(reinterpret_cast<const uint2*>(w));
        else if constexpr (W == 2) *reinterpret_cast<uint32_t*>(&h[j]) = __ldg(reinterpret_cast<const uint32_t*>(w));
        else h[j] = *VSK_CHK(w);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        __half v = __float2half_rn(0.f);
        if (c + j < dim) {
          const int g = (c + j) / ds;
          v = *VSK_CHK(cb16 + ((int64_t)g * ksub + sc[r * m + g]) * ds + ((c + j) - g * ds));
        }
        h[j] = v;
      }
    }
    *VSK_CHK_W(reinterpret_cast<uint4*>(out + (r0 + r) * dim16 + c)) = *reinterpret_cast<const uint4*>(h);
  }
}

// Coarse threshold of a query from its exact one (a rooted table sum v).  v <= T means that the fp32 table sum is at
// most T^2 up to the rounding of the root; the sum's m + ds roundings and those of |q|^2 are covered by the last two
// terms, and eps covers the coarse value against |x^|^2 - 2 q.x^ itself.
__global__ void pq_coarse_threshold_kernel(const float* __restrict__ thr_exact, const float* __restrict__ qnorm,
                                           const float* __restrict__ eps, int64_t nq, float sum_terms, float norm_terms,
                                           float* __restrict__ thr_coarse, int32_t* __restrict__ flags) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  const float t = *VSK_CHK(thr_exact + i);
  float tc = CUDART_INF_F;
  if (!(t < CUDART_INF_F)) atomicOr(&flags[i], kFlagDegenerate);   // (the first rows gave it k values: it is not finite)
  if (!(t == CUDART_INF_F)) {
    const float qn = *VSK_CHK(qnorm + i), t2 = t * t, qn2 = qn * qn;
    tc = (t2 - qn2) + *VSK_CHK(eps + i) + 1.2e-7f * (sum_terms * t2 + norm_terms * qn2);
  }
  *VSK_CHK_W(thr_coarse + i) = tc;
}

// Entries [kept, count) of a query's list are rows of the decoded block (numbered from its first row): their coarse
// values are replaced by the table scan's exact ones, summed in segment order and rooted, and the rows get their
// global numbers.
__global__ void __launch_bounds__(128) pq_rescore_kernel(const float* __restrict__ tables, const uint8_t* __restrict__ codes, int m,
                                                         int ksub, int64_t row0, int kept, CandLists cand,
                                                         unsigned long long* total) {
  const int64_t qi = blockIdx.x;
  const int cnt = min(*VSK_CHK(cand.count + qi), kCandCap);
  uint64_t* keys = cand.keys + qi * kCandCap;
  const float* tab = tables + qi * m * ksub;
  if (threadIdx.x == 0 && cnt > kept) atomicAdd(total, (unsigned long long)(cnt - kept));
  for (int c = kept + threadIdx.x; c < cnt; c += blockDim.x) {
    const int64_t row = row0 + (int64_t)(uint32_t)*VSK_CHK(keys + c);
    const uint8_t* src = codes + row * m;
    float s = 0.f;
#pragma unroll 4
    for (int g = 0; g < m; ++g) s = __fadd_rn(s, __ldg(tab + (int64_t)g * ksub + __ldg(src + g)));
    *VSK_CHK_W(keys + c) = make_key(__fsqrt_rn(s), (uint32_t)row);
  }
}

// Operand constants of a product-quantised index, from its codebooks alone (they never change): fp16 codewords, their
// squared norms, and upper bounds of the decoded rows' norms and residuals.
static int32_t pq_tensor_prepare(Index* ix) {
  Ctx* ctx = ix->ctx;
  if (ix->pq_operands != 0) return VSK_OK;
  const int m = ix->pq_m, ksub = ix->pq_ksub, dim = ix->dim, ds = dim / m;
  const size_t words = (size_t)ksub * dim;
  std::vector<float> cb(words);
  VSK_CUDA(ctx, cudaMemcpyAsync(cb.data(), ix->pq_codebooks, words * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ix->pq_operands = -1;   // not usable, unless all of the following holds
  float absmax = 0.f;
  bool finite = true;
  for (float v : cb) {
    finite = finite && std::isfinite(v);
    absmax = std::max(absmax, std::fabs(v));
  }
  if (!finite || !(absmax < 1e15f) || m > 512) return VSK_OK;   // (the decode kernel stages 64 m bytes of codes)
  float scale = 1.f;
  if (absmax > 0.f) {
    int e;
    std::frexp(absmax, &e);
    if (14 - e > 100) return VSK_OK;   // codewords that are all but zero: the table scan
    scale = std::ldexp(1.f, 14 - e);   // 2^13 <= absmax * scale < 2^14
  }
  std::vector<__half> h(words);
  std::vector<float> cw2((size_t)m * ksub);
  double norm2 = 0.0, norm16 = 0.0, err16 = 0.0;   // sums over the segments of the largest codeword's
  for (int g = 0; g < m; ++g) {
    double a = 0.0, b = 0.0, c = 0.0;
    for (int w = 0; w < ksub; ++w) {
      double x2 = 0.0, h2 = 0.0, e2 = 0.0;
      for (int i = 0; i < ds; ++i) {
        const size_t at = ((size_t)g * ksub + w) * ds + i;
        h[at] = __float2half_rn(cb[at] * scale);
        const double x = cb[at], back = __half2float(h[at]), r = x * scale - back;
        x2 += x * x;
        h2 += back * back;
        e2 += r * r;
      }
      cw2[(size_t)g * ksub + w] = (float)x2;
      a = std::max(a, x2);
      b = std::max(b, h2);
      c = std::max(c, e2);
    }
    norm2 += a;
    norm16 += b;
    err16 += c;
  }
  const float up = 1.0f + 1e-5f;
  ix->dim16 = (int32_t)(ceil_div(dim, TK) * TK);
  ix->fold16 = ctx->tuning.fold_row_term != 0 && (ix->dim16 / TK <= 4 || ix->dim16 - fold_col0(dim) >= kFoldCols);
  if (ix->fold16 && ix->dim16 - fold_col0(dim) < kFoldCols) ix->dim16 += TK;
  const double top = 0.5 * norm2 * scale / 16.0;
  int e = 0;
  if (top > 0.0) e = 14 - (int)std::ceil(std::log2(top));
  ix->fold_exp = std::max(-100, std::min(100, e));
  ix->fold_bmax = (float)(0.5 * norm2) * up;
  ix->scale16 = scale;
  ix->max_xnorm = (float)std::sqrt(norm2) * up;
  ix->max_xnorm16 = (float)std::sqrt(norm16) * up;
  ix->max_xerr16 = (float)std::sqrt(err16) * up;
  ix->min_xnorm_nz = 0.f;
  if (ix->pq_cb16 == nullptr) VSK_TRY(dev_alloc(ctx, (void**)&ix->pq_cb16, words * sizeof(__half)));
  if (ix->pq_cw2 == nullptr) VSK_TRY(dev_alloc(ctx, (void**)&ix->pq_cw2, cw2.size() * sizeof(float)));
  VSK_CUDA(ctx, cudaMemcpyAsync(ix->pq_cb16, h.data(), words * sizeof(__half), cudaMemcpyHostToDevice, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(ix->pq_cw2, cw2.data(), cw2.size() * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ix->pq_operands = 1;
  return VSK_OK;
}

bool pq_tensor_applicable(const Index* ix, int64_t nq, int32_t k) {
  return ix->ctx->search_path == VSK_PATH_TENSOR_RERANK && ix->pq_operands >= 0 && nq >= kPqTensorMinQueries &&
         ix->n >= kPqTensorMinRows && k <= kCandCap / 4;
}

int32_t pq_tensor_search(Index* ix, const float* q, int64_t nq, int32_t k, const float* tables, float* out_dist,
                         int64_t* out_ids, std::vector<int32_t>* flagged, bool* handled) {
  VSK_TRACE("vsk:pq_tensor");
  Ctx* ctx = ix->ctx;
  *handled = false;
  flagged->clear();
  VSK_TRY(pq_tensor_prepare(ix));
  if (ix->pq_operands < 0 || ix->pq_rest.resting()) return VSK_OK;
  const int m = ix->pq_m, ksub = ix->pq_ksub, dim = ix->dim, dim16 = ix->dim16, ds = dim / m;
  const int64_t n = ix->n;
  const bool fold = ix->fold16;
  // a short contraction with the folded row term: queries resident, rows streamed, thresholds folded in too
  const int k16_last = k16_last_of(fold ? fold_col0(dim) + kFoldCols : dim, dim16);
  const bool list = fold && dim16 / TK <= AS_MAX_KB && ls_layout(dim16 / TK, k16_last, false).stages >= 2;
  void* p;
  // the decoded block; without room for it the table scan takes the batch
  const int64_t block = std::min(ceil_div(n, TN) * TN, std::max<int64_t>(TN, kPqBlockBytes / ((int64_t)dim16 * 2) / TN * TN));
  if (scratch(ctx, SLOT_PQ_ROWS, (size_t)block * dim16 * sizeof(__half) + (size_t)block * sizeof(float), &p) != VSK_OK) return VSK_OK;
  __half* rows16 = (__half*)p;
  float* aux = (float*)(rows16 + block * dim16);
  QueryOperands qo;
  VSK_TRY(prepare_query_operands(ix, q, nq, &qo));
  const float* qnorm = qo.eps + nq;   // |q| as the operand preparation measured it
  CUtensorMap mq, mx, mqn, mxn;
  VSK_TRY(make_map(ctx, qo.q16, list ? ceil_div(nq, TN) * TN : nq, dim16, list ? TN : TM, &mq));
  VSK_TRY(make_map_narrow(ctx, qo.q16, ceil_div(nq, TN) * TN, dim16, TN, &mqn));
  CandLists cand;
  VSK_TRY(cand_lists(ctx, nq, &cand));
  VSK_TRY(launch_init_cand(ctx, cand, nq));
  VSK_TRY(scratch(ctx, SLOT_TC_D, (size_t)nq * sizeof(float), &p));
  CandLists cand_coarse = cand;
  cand_coarse.thr = (float*)p;
  TcArgs a{};
  a.nq = nq;
  a.kblocks = dim16 / TK;
  a.k16_last = k16_last;
  a.mode = SCAN_THRESHOLD;
  a.alpha = qo.alpha;
  a.beta = fold ? nullptr : aux;
  a.cand = cand_coarse;
  a.cap = kCandCap;
  a.err = qo.err;
  SelectArgs sel{};
  sel.cand = cand;
  sel.nq = nq;
  sel.keep = k;
  sel.k = k;
  // the first rows by the table scan: exact values, and a threshold to start from
  int64_t seen = std::min<int64_t>(n, schedule_dense_rows(ctx, k));
  VSK_TRY(pq_table_scan(ix, tables, nq, nullptr, cand, SCAN_DENSE, 0, seen));
  sel.dense_count = (int32_t)seen;
  sel.max_count = (int32_t)seen;
  VSK_TRY(launch_select(ctx, sel));
  sel.dense_count = -1;
  sel.max_count = kCandCap;
  sel.by_length = 1;
  const int64_t growth = nq <= 2048 ? std::max(16, ctx->tuning.chunk_growth) : std::max(1, ctx->tuning.chunk_growth);
  PinnedBuf& hb = ctx->host_flags[ctx->lane];
  VSK_TRY(pinned_reserve(ctx, &hb, (size_t)nq * 4 + 16));
  char* hbuf = (char*)hb.p;
  const int32_t* hflags = (const int32_t*)(hbuf + 16);
  auto count_overflowed = [&] {
    int64_t bad = 0;
    for (int64_t i = 0; i < nq; ++i) bad += hflags[i] != 0 && !(hflags[i] & kFlagDegenerate);
    return bad;
  };
  bool looked = false;
  while (seen < n) {
    int64_t chunk = std::min(schedule_chunk(seen, k, 0), std::max<int64_t>(1024, growth * seen));
    chunk = std::max<int64_t>(TN, chunk / TN * TN);
    chunk = std::min(std::min(chunk, block), n - seen);
    if (!looked && 16 * seen >= n) {
      // Most of the work is still ahead: if lists of many queries have overflowed already (rows that tie in bulk), the
      // table scan, which can pass over a tied row, takes the whole batch.
      VSK_CUDA(ctx, cudaMemcpyAsync(hbuf + 16, cand.flags, (size_t)nq * 4, cudaMemcpyDeviceToHost, ctx->stream));
      VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      const int64_t over = count_overflowed();
      if (kPqRestOneIn * over > nq) {
        ix->pq_rest.note(nq, over, kPqRestOneIn);
        return VSK_OK;
      }
      looked = true;
    }
    const unsigned dgrid = (unsigned)ceil_div(chunk, PQ_DEC_ROWS);
    const size_t dsm = (size_t)PQ_DEC_ROWS * m;
#define VSK_PQ_DEC(DS_)                                                                                                          \
    pq_decode16_kernel<DS_><<<dgrid, 256, dsm, ctx->stream>>>(ix->pq_codes + seen * m, chunk, dim, dim16, m, ksub, ds, ix->pq_cb16, \
                                                              ix->pq_cw2, ix->scale16, list ? 2 : fold ? 1 : 0, fold_col0(dim), ix->fold_exp,  \
                                                              rows16, fold ? nullptr : aux)
    if (ds == 8) VSK_PQ_DEC(8);
    else if (ds % 8 == 0) VSK_PQ_DEC(16);
    else if (ds == 4) VSK_PQ_DEC(4);
    else if (ds == 2) VSK_PQ_DEC(2);
    else VSK_PQ_DEC(0);
#undef VSK_PQ_DEC
    tl_mark(ctx, "pq_decode");
    pq_coarse_threshold_kernel<<<(unsigned)ceil_div(nq, 256), 256, 0, ctx->stream>>>(
        cand.thr, qnorm, qo.eps, nq, (float)(m + ds + 8), (float)(ceil_div(dim, 32) + 16), cand_coarse.thr,
        cand.flags);
    ctx->stats.kernel_launches += 2;
    VSK_CUDA(ctx, cudaGetLastError());
    if (list) {
      VSK_TRY(make_map(ctx, rows16, chunk, dim16, TM, &mx));
      VSK_TRY(make_map_narrow(ctx, rows16, chunk, dim16, TM, &mxn));
      const int64_t nq_pad = ceil_div(nq, TN) * TN;
      ls_fold_queries_kernel<<<(unsigned)(nq_pad / 256), 256, 0, ctx->stream>>>(cand_coarse.thr, nq, nq_pad, qo.scale, ix->scale16, ix->fold_exp,
                                                                                   dim16, fold_col0(dim), qo.q16, cand.flags);
      ctx->stats.kernel_launches++;
      LsArgs la{};
      la.rows = chunk;
      la.nq = nq;
      la.kblocks = dim16 / TK;
      la.k16_last = k16_last;
      la.cand = cand;
      la.err = qo.err;
      VSK_TRY(launch_list_scan<false>(ctx, mx, mq, mxn, mqn, la, (int64_t)dim16 * 2));
    } else {
      VSK_TRY(make_map(ctx, rows16, chunk, dim16, TN, &mx));
      a.row_begin = 0;
      a.row_end = chunk;
      VSK_TRY(launch_tc<SCAN_THRESHOLD>(ctx, mq, mx, a, !fold));
    }
    pq_rescore_kernel<<<(unsigned)nq, 128, 0, ctx->stream>>>(tables, ix->pq_codes, m, ksub, seen, (int)std::min<int64_t>(k, seen), cand, qo.rr_total);
    ctx->stats.kernel_launches++;
    VSK_CUDA(ctx, cudaGetLastError());
    tl_mark(ctx, "pq_rescore");
    VSK_TRY(launch_select(ctx, sel));
    seen += chunk;
  }
  SelectArgs fin{};
  fin.cand = cand;
  fin.nq = nq;
  fin.dense_count = -1;
  fin.keep = k;
  fin.out_dist = out_dist;
  fin.out_ids = out_ids;
  fin.k = k;
  fin.id_base = ix->id_base;
  fin.max_count = k;
  VSK_TRY(launch_select(ctx, fin));
  VSK_CUDA(ctx, cudaMemcpyAsync(hbuf, qo.err, 4, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(hbuf + 8, qo.rr_total, 8, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(hbuf + 16, cand.flags, (size_t)nq * 4, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  int32_t herr;
  unsigned long long hrr;
  memcpy(&herr, hbuf, 4);
  memcpy(&hrr, hbuf + 8, 8);
  ctx->stats.reranked_rows += (int64_t)hrr;
  if (herr != 0)
    return fail(ctx, VSK_ERR_TIMEOUT, "tensor-core scan: a bounded pipeline wait ran out (role %d)", herr);
  for (int64_t i = 0; i < nq; ++i)
    if (hflags[i]) flagged->push_back((int32_t)i);
  ix->pq_rest.note(nq, count_overflowed(), kPqRestOneIn);
  *handled = true;
  return VSK_OK;
}

// ---- int8 codes against int8 queries (dotProduct) -----------------------------------------------------------
// sum_i q_i x^_i = sum_i q~_i c_i - K with q~ = q / scale, c the codes and K = sum_i q_i offset_i / scale_i.  With q~ rounded
// to 8 bits (one scale s per query) the contraction runs on the codes as they are stored, at twice the fp16 rate, half
// the operand bytes and no operand copy of the rows, and its accumulators are exact integers.  What is lost is the
// query's rounding, |e| C at most (C = largest norm of a code row): too wide for the certificate of the fp16 path,
// which compares the k-th value with one a few keys further down, so the thresholds are exact instead (every listed row
// is re-scored after each chunk), as in the list scan: a row is listed iff  A = sum_i q8_i c_i  reaches
//   s (K - T - |e| C - rounding),   T the k-th exact value so far.
// 10 000 queries x 6.25 million rows x 384, k = 10: 40.6 ms on the fp16 path, 20.0 here (27.8 on the general kernel, which rows of
// more than three K blocks take).
struct I8Query {
  float inv_step;    // s: q8 = round(s q~)
  float slack;       // |e| C plus the fp32 roundings of the exact values, in true units
  double offset;     // K
};

// One warp per query.  A query that is not finite or all but zero has no 8-bit form (every row would be listed): it is flagged, its
// bar is out of reach, and it is re-run by itself.
__global__ void i8_query_kernel(const float* __restrict__ q, int64_t nq, int dim, int stride, const float* __restrict__ scale,
                                const float* __restrict__ offset, float max_code_norm, float max_xnorm, int8_t* __restrict__ out,
                                I8Query* __restrict__ info, int32_t* __restrict__ flags) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= nq) return;
  const int lane = threadIdx.x & 31;
  const float* p = q + row * dim;
  float amax = 0.f, q2 = 0.f, t2 = 0.f;
  double k = 0.0;
  bool finite = true;
  for (int i = lane; i < dim; i += 32) {
    const float v = __ldg(p + i), sc = __ldg(scale + i), t = __fdiv_rn(v, sc);
    finite = finite && isfinite(t) && isfinite(v);
    amax = fmaxf(amax, fabsf(t));
    q2 = fmaf(v, v, q2);
    t2 = fmaf(t, t, t2);
    k += (double)v * (double)__ldg(offset + i) / (double)sc;
  }
  finite = __all_sync(0xffffffffu, finite);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    q2 += __shfl_xor_sync(0xffffffffu, q2, o);
    t2 += __shfl_xor_sync(0xffffffffu, t2, o);
    k += __shfl_xor_sync(0xffffffffu, k, o);
  }
  const bool usable = finite && amax > 1e-30f && amax < 1e30f;
  const float s = usable ? 127.0f / amax : 1.0f;
  float e2 = 0.f;
  for (int i = lane; i < stride; i += 32) {
    int c = 0;
    if (usable && i < dim) {
      const float t = __fdiv_rn(__ldg(p + i), __ldg(scale + i));
      c = max(-127, min(127, __float2int_rn(t * s)));
      const float e = fmaf((float)c, -amax * (1.0f / 127.0f), t);
      e2 = fmaf(e, e, e2);
    }
    *VSK_CHK_W(out + row * stride + i) = (int8_t)c;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, o);
  if (lane == 0) {
    const float qn = sqrtf(q2), tn = sqrtf(t2);
    I8Query r;
    r.inv_step = s;
    r.offset = k;
    // the step and q~ are rounded to 2^-22 at worst; an exact value is a sum of dim products of q with x^ = (c - offset)
    // / scale, whose roundings are below (dim + 8) 2^-23 |q| |x^|
    r.slack = (sqrtf(e2) * 1.0001f + 1e-6f * tn) * max_code_norm + 1.2e-7f * (float)(dim + 8) * qn * max_xnorm;
    if (!usable) {
      r.slack = -CUDART_INF_F;
      *VSK_CHK_W(flags + row) = kFlagDegenerate;   // (the flags have just been cleared)
    }
    *VSK_CHK_W(info + row) = r;
  }
}

// The accumulator a row must reach, from the query's exact threshold (values are -(q.x^)).
__global__ void i8_bar_kernel(const float* __restrict__ thr_exact, const I8Query* __restrict__ info, int64_t nq,
                              int32_t* __restrict__ bar) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  const I8Query r = *VSK_CHK(info + i);
  const double at = floor((double)r.inv_step * (r.offset - (double)*VSK_CHK(thr_exact + i) - (double)r.slack)) - 1.0;
  // not a number or below every accumulator: every row is listed (and the list overflows)
  *VSK_CHK_W(bar + i) = r.slack == -CUDART_INF_F ? INT_MAX : !(at > -2147483647.0) ? INT_MIN : at > 2147483646.0 ? INT_MAX : (int32_t)at;
}

// Largest norm of a code row and of its decoded row (the stored codes themselves are the operand).
__global__ void i8_row_stats_kernel(const int8_t* __restrict__ codes, int64_t n, int dim, const float* __restrict__ scale,
                                    const float* __restrict__ offset, PrepStats* stats) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  float cmax = 0.f, xmax = 0.f;
  for (int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < n; row += warps) {
    const int8_t* p = codes + row * dim;
    float c2 = 0.f, x2 = 0.f;
    for (int i = lane; i < dim; i += 32) {
      const float c = (float)__ldg(p + i), xh = __fdiv_rn(__fsub_rn(c, __ldg(offset + i)), __ldg(scale + i));
      c2 = fmaf(c, c, c2);
      x2 = fmaf(xh, xh, x2);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      c2 += __shfl_xor_sync(0xffffffffu, c2, o);
      x2 += __shfl_xor_sync(0xffffffffu, x2, o);
    }
    cmax = fmaxf(cmax, c2);
    if (isnan(x2) || x2 > xmax) xmax = x2;   // a decoded value that is not a number stays: nothing compares greater
  }
  if (lane == 0) {
    const float up = 1.0f + 1e-5f;
    atomicMax(&stats->max_norm16, __float_as_uint(sqrtf(cmax) * up));
    atomicMax(&stats->max_norm, __float_as_uint(fabsf(sqrtf(xmax) * up)));
  }
}

__global__ void i8_pad_rows_kernel(const int8_t* __restrict__ codes, int64_t n, int dim, int stride, int8_t* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * stride) return;
  const int64_t r = i / stride;
  const int c = (int)(i - r * stride);
  *VSK_CHK_W(out + i) = c < dim ? __ldg(codes + r * dim + c) : (int8_t)0;
}

// Once per index state: the norms of the error bound, and a copy with rows padded to 16 bytes (TMA strides) where the
// dimension is not a multiple of 16.
static int32_t i8_prepare(Index* ix) {
  Ctx* ctx = ix->ctx;
  if (ix->n8 == ix->n) return VSK_OK;
  dev_free(ix->rows8);
  ix->rows8 = nullptr;
  ix->stride8 = (int32_t)(ceil_div(ix->dim, 16) * 16);
  if (ix->stride8 != ix->dim) {
    VSK_TRY(dev_alloc(ctx, (void**)&ix->rows8, (size_t)ix->n * ix->stride8));
    i8_pad_rows_kernel<<<(unsigned)ceil_div(ix->n * ix->stride8, 256), 256, 0, ctx->stream>>>(ix->codes, ix->n, ix->dim, ix->stride8, ix->rows8);
    ctx->stats.kernel_launches++;
  }
  void* p;
  VSK_TRY(scratch(ctx, SLOT_TC_A, sizeof(PrepStats), &p));
  VSK_CUDA(ctx, cudaMemsetAsync(p, 0, sizeof(PrepStats), ctx->stream));
  i8_row_stats_kernel<<<(unsigned)std::min<int64_t>(ceil_div(ix->n, 8), 148 * 8), 256, 0, ctx->stream>>>(
      ix->codes, ix->n, ix->dim, ix->sq_scale, ix->sq_offset, (PrepStats*)p);
  ctx->stats.kernel_launches++;
  VSK_CUDA(ctx, cudaGetLastError());
  PrepStats h;
  VSK_CUDA(ctx, cudaMemcpyAsync(&h, p, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  memcpy(&ix->max_code_norm, &h.max_norm16, 4);
  memcpy(&ix->max_xnorm8, &h.max_norm, 4);
  ix->n8 = ix->n;
  return VSK_OK;
}

constexpr int kI8RestOneIn = 64;   // more than one query in so many that overflows costs what the integer contraction gains

bool i8_search_applicable(const Index* ix, int32_t k) {
  // 127 * 128 * dim below 2^31: no accumulator can overflow
  return ix->kind == INDEX_FLAT_I8 && ix->metric == VSK_METRIC_DOT_PRODUCT && ix->ctx->search_path == VSK_PATH_TENSOR_RERANK &&
         k <= kCandCap / 4 && ix->dim <= 12 * 1024 && ix->n >= kI8MinRows;
}

int32_t i8_search(Index* ix, const float* q, int64_t nq, int32_t k, float* out_dist, int64_t* out_ids, bool* handled) {
  VSK_TRACE("vsk:i8_scan");
  Ctx* ctx = ix->ctx;
  *handled = false;
  if (ix->i8_rest.resting()) return VSK_OK;
  VSK_TRY(i8_prepare(ix));
  const float limit = 1e30f;
  if (!(ix->max_code_norm < limit) || !(ix->max_xnorm8 < limit)) return VSK_OK;
  const int dim = ix->dim, stride = ix->stride8;
  const int64_t n = ix->n;
  void* p;
  const int64_t nq_pad = ceil_div(nq, TN) * TN;   // (list_scan_kernel's whole blocks)
  VSK_TRY(scratch(ctx, SLOT_Q16, (size_t)nq_pad * stride, &p));
  int8_t* q8 = (int8_t*)p;
  VSK_CUDA(ctx, cudaMemsetAsync(q8 + nq * stride, 0, (size_t)(nq_pad - nq) * stride, ctx->stream));
  VSK_TRY(scratch(ctx, SLOT_QAUX, (size_t)nq * (sizeof(I8Query) + 4), &p));
  I8Query* info = (I8Query*)p;
  int32_t* bar = (int32_t*)(info + nq);
  // up to three K blocks: queries resident, rows streamed, the bars folded in
  const int32_t kblocks = (int32_t)ceil_div(dim, 2 * TK), k_last = (int32_t)(ceil_div(dim, 32) - 4 * (kblocks - 1));
  const bool list = ls_layout(kblocks, k_last, true).stages >= 2;
  VSK_TRY(scratch(ctx, SLOT_TC_C, (size_t)nq_pad * 32, &p));
  int8_t* bar8 = (int8_t*)p;
  VSK_TRY(scratch(ctx, SLOT_TC_B, 64, &p));
  VSK_CUDA(ctx, cudaMemsetAsync(p, 0, 64, ctx->stream));
  const float* alpha = (const float*)p + 2;
  int32_t* err = (int32_t*)p + 3;
  unsigned long long* rr_total = (unsigned long long*)((char*)p + 16);
  CUtensorMap mq, mx, mb;
  const int8_t* rows8 = ix->rows8 ? ix->rows8 : ix->codes;
  VSK_TRY(make_map_i8(ctx, q8, list ? nq_pad : nq, dim, stride, list ? TN : TM, &mq));
  VSK_TRY(make_map_i8(ctx, rows8, n, dim, stride, list ? TM : TN, &mx));
  VSK_TRY(make_map_bytes(ctx, bar8, nq_pad, TN, &mb));
  CandLists cand;
  VSK_TRY(cand_lists(ctx, nq, &cand));
  VSK_TRY(launch_init_cand(ctx, cand, nq));
  i8_query_kernel<<<(unsigned)ceil_div(nq, 8), 256, 0, ctx->stream>>>(q, nq, dim, stride, ix->sq_scale, ix->sq_offset, ix->max_code_norm,
                                                                      ix->max_xnorm8, q8, info, cand.flags);
  ctx->stats.kernel_launches++;
  TcArgs a{};
  a.nq = nq;
  a.kblocks = kblocks;
  a.k16_last = k_last;
  a.mode = SCAN_THRESHOLD;
  a.alpha = alpha;
  a.cand = cand;
  a.cand.thr = (float*)bar;
  a.cap = kCandCap;
  a.err = err;
  // the first rows by the fp32 scan: exact values, and a threshold to start from
  int64_t seen = std::min<int64_t>(n, schedule_dense_rows(ctx, k));
  ExactScanArgs ea{};
  ea.metric = ix->metric;
  ea.mode = SCAN_DENSE;
  ea.q = q;
  ea.x_codes = ix->codes;
  ea.sq_scale = ix->sq_scale;
  ea.sq_offset = ix->sq_offset;
  ea.dim = dim;
  ea.nq = nq;
  ea.row_end = seen;
  ea.bm_hint = nq <= 32 ? 32 : nq <= 64 ? 64 : 0;
  ea.cand = cand;
  VSK_TRY(launch_exact_scan(ctx, ea));
  SelectArgs sel{};
  sel.cand = cand;
  sel.nq = nq;
  sel.keep = k;
  sel.k = k;
  sel.dense_count = (int32_t)seen;
  sel.max_count = (int32_t)seen;
  VSK_TRY(launch_select(ctx, sel));
  sel.dense_count = -1;
  sel.max_count = kCandCap;
  sel.by_length = 1;
  PinnedBuf& hb = ctx->host_flags[ctx->lane];
  VSK_TRY(pinned_reserve(ctx, &hb, (size_t)nq * 4 + 16));
  char* hbuf = (char*)hb.p;
  const int32_t* hflags = (const int32_t*)(hbuf + 16);
  auto count_overflowed = [&] {
    int64_t bad = 0;
    for (int64_t i = 0; i < nq; ++i) bad += hflags[i] != 0 && !(hflags[i] & kFlagDegenerate);
    return bad;
  };
  const size_t qsm = (size_t)dim * sizeof(float);   // (i8_search_applicable: at most 48 KB)
  if (2 * qsm > 48 * 1024)
    VSK_CUDA(ctx, cudaFuncSetAttribute(rerank_i8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * qsm)));
  const int64_t growth = nq <= 2048 ? std::max(16, ctx->tuning.chunk_growth) : std::max(1, ctx->tuning.chunk_growth);
  bool looked = nq < 256;   // a small batch is cheap to scan twice: no look between its chunks
  while (seen < n) {
    // half of the plain schedule's chunk: the bar admits about twice the rows the exact threshold would
    int64_t chunk = std::min(schedule_chunk(seen, k, 0) / 2, std::max<int64_t>(1024, growth * seen));
    chunk = std::max<int64_t>(TN, chunk / TN * TN);
    chunk = std::min(chunk, n - seen);
    if (!looked && 16 * seen >= n) {
      // most of the work is still ahead: where many lists have overflowed already (norms far apart, so that |e| C is wide
      // against the spread of the values), the fp16 path takes the batch
      VSK_CUDA(ctx, cudaMemcpyAsync(hbuf + 16, cand.flags, (size_t)nq * 4, cudaMemcpyDeviceToHost, ctx->stream));
      VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      const int64_t over = count_overflowed();
      if (kI8RestOneIn * over > nq) {
        ix->i8_rest.note(nq, over, kI8RestOneIn);
        return VSK_OK;
      }
      looked = true;
    }
    i8_bar_kernel<<<(unsigned)ceil_div(nq, 256), 256, 0, ctx->stream>>>(cand.thr, info, nq, bar);
    ctx->stats.kernel_launches++;
    a.row_begin = seen;
    a.row_end = seen + chunk;
    if (list) {
      ls_bar_bytes_kernel<<<(unsigned)(nq_pad / 256), 256, 0, ctx->stream>>>(bar, nq, nq_pad, bar8, cand.flags);
      ctx->stats.kernel_launches++;
      VSK_TRY(make_map_i8(ctx, rows8 + seen * stride, chunk, dim, stride, TM, &mx));
      LsArgs la{};
      la.rows = chunk;
      la.nq = nq;
      la.row_id0 = seen;
      la.kblocks = kblocks;
      la.k16_last = k_last;
      la.cand = cand;
      la.err = err;
      VSK_TRY(launch_list_scan<true>(ctx, mx, mq, mx, mb, la, stride));
    } else if (tc_epilogue_warps(a.kblocks, false) == 16) VSK_TRY((launch_tc_ew<SCAN_THRESHOLD, 16, true>(ctx, mq, mx, a, false)));
    else VSK_TRY((launch_tc_ew<SCAN_THRESHOLD, 8, true>(ctx, mq, mx, a, false)));
    rerank_i8_kernel<<<(unsigned)nq, 256, 2 * qsm, ctx->stream>>>(q, ix->codes, dim, ix->sq_scale, ix->sq_offset, cand, rr_total);
    ctx->stats.kernel_launches++;
    VSK_CUDA(ctx, cudaGetLastError());
    tl_mark(ctx, "rerank");
    VSK_TRY(launch_select(ctx, sel));
    seen += chunk;
  }
  SelectArgs fin{};
  fin.cand = cand;
  fin.nq = nq;
  fin.dense_count = -1;
  fin.keep = k;
  fin.out_dist = out_dist;
  fin.out_ids = out_ids;
  fin.k = k;
  fin.metric = ix->metric;
  fin.id_base = ix->id_base;
  fin.max_count = k;
  VSK_TRY(launch_select(ctx, fin));
  VSK_CUDA(ctx, cudaMemcpyAsync(hbuf, err, 4, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(hbuf + 8, rr_total, 8, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(hbuf + 16, cand.flags, (size_t)nq * 4, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  int32_t herr;
  unsigned long long hrr;
  memcpy(&herr, hbuf, 4);
  memcpy(&hrr, hbuf + 8, 8);
  ctx->stats.reranked_rows += (int64_t)hrr;
  if (herr != 0)
    return fail(ctx, VSK_ERR_TIMEOUT, "tensor-core scan: a bounded pipeline wait ran out (role %d)", herr);
  std::vector<int32_t> bad;
  for (int64_t i = 0; i < nq; ++i)
    if (hflags[i]) bad.push_back((int32_t)i);
  // a few queries are re-run by themselves, whatever share of the batch they are; many send the batch to the fp16 path
  const int64_t over = count_overflowed();
  ix->i8_rest.note(nq, over, kI8RestOneIn);
  if (over > 8 && kI8RestOneIn * over > nq) return VSK_OK;
  if (!bad.empty()) VSK_TRY(fp32_search_subset(ix, q, bad, k, nullptr, nullptr, out_dist, out_ids));
  *handled = true;
  return VSK_OK;
}

// ---- public: tensor-core nearest-centroid assignment (used by kmeans.cu) ---------------------------
int32_t tensor_assign_prepare(Ctx* ctx, const float* rows, int64_t n, int32_t dim, TensorAssign* ta, bool one_call) {
  ta->n = n;
  ta->dim = dim;
  // Short contractions keep a block of centroids resident (assign_scan_kernel): the operands then carry 16 more
  // columns for the folded |c|^2 / 2 term.  Longer ones (more than four k-blocks with those columns) take the general kernel.
  ta->stationary = fold_col0(dim) + kFoldCols <= AS_MAX_KB * TK;
  ta->dim16 = (int32_t)(ceil_div(ta->stationary ? fold_col0(dim) + kFoldCols : dim, TK) * TK);
  // stationary kernel: `keys` is the hit log (a hit or two per row as a rule; six entries per row of room)
  const struct { void** p; size_t bytes; } need[] = {
      {(void**)&ta->rows16, (size_t)n * ta->dim16 * sizeof(__half)},
      {(void**)&ta->stats, (size_t)n * 4 * sizeof(float)},
      {(void**)&ta->keys, (size_t)n * (ta->stationary ? kAssignLogPerRow : kAssignCap) * sizeof(uint64_t)},
      {(void**)&ta->best, (size_t)n * sizeof(unsigned long long)},
      {(void**)&ta->count, (size_t)n * sizeof(int32_t)},
      {(void**)&ta->thr, (size_t)n * sizeof(float)},
      {(void**)&ta->bad_rows, (size_t)n * sizeof(int32_t)},
      {&ta->small, 256}};
  size_t total = 0;
  for (const auto& b : need) total += (b.bytes + 255) / 256 * 256;
  char* block = one_call ? (char*)arena_take(ctx, total) : nullptr;
  if (block) {
    ta->arena = ctx;
    for (const auto& b : need) {
      *b.p = block;
      block += (b.bytes + 255) / 256 * 256;
    }
  } else {
    for (const auto& b : need) VSK_TRY(dev_alloc(ctx, b.p, b.bytes));
  }
  VSK_CUDA(ctx, cudaMemsetAsync(ta->small, 0, 256, ctx->stream));
  // small: [0] absmax(rows) [1] scale_x [2] absmax(cent) [3] scale_c [4] alpha [5] err [6] bad_count, then PrepStats at +64
  unsigned* sm = (unsigned*)ta->small;
  absmax_kernel<<<1184, 256, 0, ctx->stream>>>(rows, n * (int64_t)dim, sm + 0);
  choose_scale_kernel<<<1, 1, 0, ctx->stream>>>(sm + 0, 0, (float*)sm + 1);
  float* st = (float*)ta->stats;
  if (dim % 4 == 0 && dim <= 256 && (reinterpret_cast<uintptr_t>(rows) & 15) == 0) {
    prep_rows_wide_kernel<<<(unsigned)ceil_div(n, 8), 256, 0, ctx->stream>>>(rows, n, dim, ta->dim16, (float*)sm + 1, ta->rows16, st, st + n, st + 2 * n);
    ctx->stats.kernel_launches++;
  } else {
    launch_prep<VSK_METRIC_DOT_PRODUCT>(ctx, rows, n, dim, ta->dim16, (float*)sm + 1, ta->rows16, nullptr, st, st + n, st + 2 * n, nullptr);
  }
  ctx->stats.kernel_launches += 2;
  VSK_CUDA(ctx, cudaGetLastError());
  VSK_TRY(make_map(ctx, ta->rows16, n, ta->dim16, TM, (CUtensorMap*)ta->map_rows));
  VSK_TRY(make_map_narrow(ctx, ta->rows16, n, ta->dim16, TM, (CUtensorMap*)ta->map_rows_narrow));
  return VSK_OK;
}

void tensor_assign_release(TensorAssign* ta) {
  if (ta->arena) {
    cudaStreamSynchronize(ta->arena->stream);   // (a call that failed part-way may have left work behind)
    arena_return(ta->arena);
  } else {
    dev_free(ta->rows16); dev_free(ta->stats); dev_free(ta->keys); dev_free(ta->best); dev_free(ta->count);
    dev_free(ta->thr); dev_free(ta->bad_rows); dev_free(ta->small);
  }
  dev_free(ta->prev_cent); dev_free(ta->shift);
  *ta = TensorAssign{};
}

int32_t tensor_assign(Ctx* ctx, TensorAssign* ta, const float* rows, const float* centroids, int32_t k,
                      int32_t* assign, float* dist, bool assign_holds_previous) {
  VSK_TRACE("vsk:assign");
  static_assert(sizeof(CUtensorMap) <= sizeof(ta->map_rows), "tensor map storage too small");
  const int64_t n = ta->n;
  const int dim = ta->dim, dim16 = ta->dim16;
  unsigned* sm = (unsigned*)ta->small;
  float* fsm = (float*)ta->small;
  PrepStats* cs = (PrepStats*)((char*)ta->small + 64);
  float* st = (float*)ta->stats;
  float* eps = st + 3 * n;
  // centroid operand: fp16 rows, |c|^2, stats
  void* p;
  VSK_TRY(scratch(ctx, SLOT_TC_C, (size_t)k * dim16 * sizeof(__half), &p));
  __half* c16 = (__half*)p;
  VSK_TRY(scratch(ctx, SLOT_TC_D, (size_t)k * sizeof(float), &p));
  float* caux = (float*)p;
  PrepStats init{0u, 0u, 0u, 0u, 0x7f800000u};
  VSK_CUDA(ctx, cudaMemcpyAsync(cs, &init, sizeof(init), cudaMemcpyHostToDevice, ctx->stream));
  VSK_CUDA(ctx, cudaMemsetAsync(sm + 2, 0, 4, ctx->stream));
  VSK_CUDA(ctx, cudaMemsetAsync(sm + 5, 0, 8, ctx->stream));
  absmax_kernel<<<64, 256, 0, ctx->stream>>>(centroids, (int64_t)k * dim, sm + 2);
  choose_scale_kernel<<<1, 1, 0, ctx->stream>>>(sm + 2, 0, fsm + 3);
  FoldArgs cfold{0, 0, 0};
  if (ta->stationary) {
    // words 24..27 of `small`: max |c|^2, the fold exponent, (unused), the data side's constant
    VSK_CUDA(ctx, cudaMemsetAsync(sm + 24, 0, 16, ctx->stream));
    max_sq_kernel<<<(unsigned)ceil_div(k, 8), 256, 0, ctx->stream>>>(centroids, k, dim, sm + 24);
    assign_fold_setup_kernel<<<1, 1, 0, ctx->stream>>>(sm + 24, fsm + 3, fsm + 1, (int*)sm + 25, fsm + 27);
    // word 30: the constant the data operand's fold columns hold (0 = none yet; a real constant is a power of two)
    assign_fill_fold_kernel<<<(unsigned)ceil_div(n * (kFoldCols / 8), 256), 256, 0, ctx->stream>>>(ta->rows16, n, dim16, fold_col0(dim), fsm + 27, fsm + 30);
    VSK_CUDA(ctx, cudaMemcpyAsync(fsm + 30, fsm + 27, sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    ctx->stats.kernel_launches += 3;
    cfold = FoldArgs{1, fold_col0(dim), 0, (const int*)sm + 25};
  }
  launch_prep<VSK_METRIC_EUCLIDEAN>(ctx, centroids, k, dim, dim16, fsm + 3, c16, caux, nullptr, nullptr, nullptr, cs, cfold);
  assign_bound_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, ctx->stream>>>(st, st + n, st + 2 * n, n, fsm + 1, fsm + 3, cs, dim16, eps, fsm + 4,
                                                                         ta->stationary ? 1 : 0);
  ctx->stats.kernel_launches += 3;
  VSK_CUDA(ctx, cudaGetLastError());
  CUtensorMap mc;
  VSK_TRY(make_map(ctx, c16, k, dim16, TN, &mc));
  const CUtensorMap& mr = *(const CUtensorMap*)ta->map_rows;
  CUtensorMap mcn;
  VSK_TRY(make_map_narrow(ctx, c16, k, dim16, TN, &mcn));
  const CUtensorMap& mrn = *(const CUtensorMap*)ta->map_rows_narrow;
  if (ta->stationary) {
    AsArgs sa{};
    sa.n = n;
    sa.k = k;
    sa.kblocks = dim16 / TK;
    sa.k16_last = k16_last_of(fold_col0(dim) + kFoldCols, dim16);
    sa.max_stages = ctx->tuning.assign_stages;
    sa.narrow_ok = 1;
    sa.alpha = fsm + 4;
    sa.thr = ta->thr;
    // the hit log lives in the rows' key lists (n x kAssignCap words of 8 bytes), its per-CTA counts in `count`
    sa.log = reinterpret_cast<uint2*>(ta->keys);
    sa.log_total = n * (int64_t)kAssignLogPerRow;
    sa.log_count = ta->count;
    sa.best_value = reinterpret_cast<unsigned*>(ta->best);
    sa.err = (int32_t*)(sm + 5);
    // The centroids of the previous call and how far each has moved since: rows whose centroid has hardly moved take
    // their threshold from the triangle inequality instead of a read of the row (assign_prev_threshold_kernel).
    if (ta->prev_k != k) {
      dev_free(ta->prev_cent);
      dev_free(ta->shift);
      ta->prev_cent = nullptr;
      ta->shift = nullptr;
      ta->prev_k = 0;
      VSK_TRY(dev_alloc(ctx, (void**)&ta->prev_cent, (size_t)k * dim * sizeof(float)));
      VSK_TRY(dev_alloc(ctx, (void**)&ta->shift, (size_t)k * sizeof(float)));
      ta->prev_k = k;
      ta->have_prev = false;
    }
    const bool bound_ok = assign_holds_previous && ta->have_prev && ta->bound_allowed && dist != nullptr;
    if (bound_ok) {
      assign_shift_kernel<<<(unsigned)ceil_div(k, 8), 256, 0, ctx->stream>>>(centroids, ta->prev_cent, k, dim, ta->shift);
      ctx->stats.kernel_launches++;
    }
    unsigned sgrid = 0;
    int64_t log_cap = 0;
    // one pass: thresholds (or the coarse arg-min of a first iteration), threshold scan, exact decisions
    auto pass = [&](bool with_bound) -> int32_t {
      VSK_CUDA(ctx, cudaMemsetAsync(sm + 5, 0, 8, ctx->stream));
      if (assign_holds_previous) {
        launch_prev_threshold(ctx, rows, n, dim, centroids, assign, eps, ta->thr, ta->count, with_bound ? dist : nullptr,
                              ta->shift, st + 2 * n, 0.02f);
      } else {
        VSK_CUDA(ctx, cudaMemsetAsync(sa.best_value, 0xff, (size_t)n * sizeof(unsigned), ctx->stream));
        VSK_TRY(launch_assign_scan<SCAN_ARGMIN>(ctx, mr, mc, mrn, mcn, sa));
        assign_value_threshold_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, ctx->stream>>>(sa.best_value, eps, n, ta->thr, ta->count);
      }
      VSK_CUDA(ctx, cudaMemsetAsync(ta->best, 0xff, (size_t)n * sizeof(unsigned long long), ctx->stream));
      tl_mark(ctx, "assign_thresholds");
      VSK_TRY(launch_assign_scan<SCAN_THRESHOLD>(ctx, mr, mc, mrn, mcn, sa, &sgrid, &log_cap));
      if (dim % 4 == 0 && ((uintptr_t)rows & 15) == 0 && ((uintptr_t)centroids & 15) == 0)
        assign_log_exact_kernel<true><<<dim3(64, sgrid), 256, 0, ctx->stream>>>(rows, dim, centroids, sa.log, sa.log_count, log_cap, ta->best);
      else
        assign_log_exact_kernel<false><<<dim3(64, sgrid), 256, 0, ctx->stream>>>(rows, dim, centroids, sa.log, sa.log_count, log_cap, ta->best);
      tl_mark(ctx, "assign_exact");
      // writes nothing when the scan raised an error: the previous assignment survives for a repeat
      assign_log_decode_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, ctx->stream>>>(ta->best, n, assign, dist, ta->bad_rows, (int32_t*)(sm + 6),
                                                                                (const int32_t*)(sm + 5));
      ctx->stats.kernel_launches += 4;
      VSK_CUDA(ctx, cudaGetLastError());
      return VSK_OK;
    };
    VSK_TRY(pass(bound_ok));
    if (bound_ok) {
      // The looser thresholds list more centroids per row; data without gaps between its clusters can fill the hit
      // log.  Then the pass is repeated once with exact thresholds, and the bound is not tried again on this data.
      int32_t e0 = 0;
      VSK_CUDA(ctx, cudaMemcpyAsync(&e0, sm + 5, 4, cudaMemcpyDeviceToHost, ctx->stream));
      VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      if (e0 == 9) {
        ta->bound_allowed = false;
        VSK_TRY(pass(false));
      }
    }
    // remember these centroids for the next call's shifts
    VSK_CUDA(ctx, cudaMemcpyAsync(ta->prev_cent, centroids, (size_t)k * dim * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    ta->have_prev = true;
  } else {

  TcArgs a{};
  a.nq = n;
  a.row_begin = 0;
  a.row_end = k;
  a.kblocks = dim16 / TK;
  a.k16_last = k16_last_of(dim, dim16);
  a.alpha = fsm + 4;
  a.beta = caux;
  a.row_tile_fastest = 1;
  a.err = (int32_t*)(sm + 5);
  a.best = ta->best;
  a.cap = kAssignCap;
  a.cand.keys = ta->keys;
  a.cand.count = ta->count;
  a.cand.thr = ta->thr;
  a.cand.flags = nullptr;
  a.cand.nq = n;
  if (assign_holds_previous) {
    launch_prev_threshold(ctx, rows, n, dim, centroids, assign, eps, ta->thr, ta->count, nullptr, nullptr, nullptr, 0.f);
  } else {
    VSK_CUDA(ctx, cudaMemsetAsync(ta->best, 0xff, (size_t)n * sizeof(unsigned long long), ctx->stream));
    a.mode = SCAN_ARGMIN;
    VSK_TRY(launch_tc<SCAN_ARGMIN>(ctx, mr, mc, a, true));
    assign_threshold_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, ctx->stream>>>(ta->best, eps, n, ta->thr, ta->count);
  }
  a.mode = SCAN_THRESHOLD;
  VSK_TRY(launch_tc<SCAN_THRESHOLD>(ctx, mr, mc, a, true));
  assign_exact_kernel<<<(unsigned)ceil_div(n, 8), 256, 0, ctx->stream>>>(rows, n, dim, centroids, ta->keys, ta->count, assign, dist,
                                                                         ta->bad_rows, (int32_t*)(sm + 6), tc_epilogue_warps(a.kblocks, true) / 4);
  ctx->stats.kernel_launches += 2;
  VSK_CUDA(ctx, cudaGetLastError());
  }
  int32_t h[2] = {0, 0};
  VSK_CUDA(ctx, cudaMemcpyAsync(h, sm + 5, 8, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (h[0] == 9) {
    // a CTA's hit log ran full (rows with very many near-ties): the fp32 tile decides for every row
    ctx->stats.fallback_queries += n;
    ExactScanArgs e{};
    e.metric = VSK_METRIC_EUCLIDEAN;
    e.mode = SCAN_ARGMIN;
    e.q = rows;
    e.nq = n;
    e.x = centroids;
    e.dim = dim;
    e.row_begin = 0;
    e.row_end = k;
    e.best = ta->best;
    VSK_CUDA(ctx, cudaMemsetAsync(ta->best, 0xff, (size_t)n * sizeof(unsigned long long), ctx->stream));
    VSK_TRY(launch_exact_scan(ctx, e));
    VSK_CUDA(ctx, cudaMemsetAsync(sm + 6, 0, 4, ctx->stream));
    assign_log_decode_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, ctx->stream>>>(ta->best, n, assign, dist, ta->bad_rows, (int32_t*)(sm + 6),
                                                                              nullptr);
    ctx->stats.kernel_launches++;
    VSK_CUDA(ctx, cudaGetLastError());
    VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return VSK_OK;
  }
  if (h[0] != 0) return fail(ctx, VSK_ERR_TIMEOUT, "tensor-core assignment: a bounded pipeline wait ran out (role %d)", h[0]);
  if (h[1] > 0) {
    // rows with too many near-ties (or none listed): the fp32 tile decides
    const int64_t m = h[1];
    ctx->stats.fallback_queries += m;
    VSK_CUDA(ctx, cudaMemsetAsync(ta->best, 0xff, (size_t)m * sizeof(unsigned long long), ctx->stream));
    ExactScanArgs e{};
    e.metric = VSK_METRIC_EUCLIDEAN;
    e.mode = SCAN_ARGMIN;
    e.q = rows;
    e.nq = m;
    e.q_subset = ta->bad_rows;
    e.x = centroids;
    e.dim = dim;
    e.row_begin = 0;
    e.row_end = k;
    e.best = ta->best;
    VSK_TRY(launch_exact_scan(ctx, e));
    scatter_best_kernel<<<(unsigned)ceil_div(m, 256), 256, 0, ctx->stream>>>(ta->best, ta->bad_rows, m, assign, dist);
    ctx->stats.kernel_launches++;
    VSK_CUDA(ctx, cudaGetLastError());
  }
  return VSK_OK;
}

}  // namespace vsk
