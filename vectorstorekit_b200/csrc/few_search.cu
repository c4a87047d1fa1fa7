// Top-k of a few queries in one launch: scan, selection and final order.
//
// A call with one query over a small store is bound by launches, not by bytes: 10 000 rows of 128 floats cross HBM in
// 0.8 us, and the chunked schedule spends a dozen launches on them (109 us for the whole call; 26 us this way, its query in the launch's arguments and its results staged in pinned memory).  Here every
// CTA streams its share of the rows (the inner loop of stream_scan.cu: each row read once, 16-byte loads), keeps its k
// best keys per query in shared memory - appends below a threshold, a block-wide selection when the list fills up - and
// writes them out; the last CTA to finish merges the lists.  The merge needs few of the G k keys written: the k-th
// smallest of the CTAs' best keys bounds the result (k rows lie at or below it), so only CTAs whose best key is within
// it - k of them - are read.  Values are the same direct fp32 formulas, ties go by id, and the row masks are applied
// before a key is listed.
//
// SEG: every query walks the rows of its own probed lists of an IVF index (one grid row per query), found from the probe
// list and the list offsets on the device: no row list is written and the host is not asked in between (one query, 10 of
// 1 024 lists over 1 million rows, 60 000 rows in all: 143 us for the chunked schedule, 56 this way; 75 with two rows per step that
// were waited for, rounds sized by the mean list, an id looked up per listed row and the query copied first).
#include <math_constants.h>

#include <algorithm>
#include <cstring>

#include "block_select.cuh"
#include "common.cuh"
#include "stream_rows.cuh"
#include "tensor_scan.cuh"

namespace vsk {
namespace {

constexpr int FEW_THREADS = 256;
constexpr int FEW_WARPS = FEW_THREADS / 32;
constexpr int kFewShort = 96;      // keys a CTA hands over as they are: shortening a list costs more than the merge's test of its keys
constexpr int kFewRank = 256;      // keys the merge orders by counting the smaller ones (one per thread, no barrier)
constexpr int FEW_LIST = 1024;     // keys per query a CTA holds
constexpr int FEW_ROUND = 512;     // rows per round at most: a round's keys fit behind FEW_LIST - FEW_ROUND listed ones
constexpr int FEW_MAX_CTAS = 1024; // lists per query the merge looks at (the selection holds 8 keys per thread)
static_assert(FEW_LIST - FEW_ROUND >= kFewMaxK && FEW_MAX_CTAS <= FEW_THREADS * SEL_ITEMS, "few-query list sizes");

struct FewKernelArgs {
  FewArgs a;
  int32_t round;        // rows per CTA and round, a multiple of FEW_WARPS * rows per warp step (SEG: the kernel's own)
  int32_t stride;       // room of a CTA's list of one query in `part`
  uint64_t* part;       // [nq][grid][stride] each CTA's best keys (unordered) ...
  uint64_t* part_min;   // [nq][grid] ... the smallest of them (all ones: none)
  int32_t* part_n;      // [nq][grid] ... and how many
  unsigned* ticket;     // [nq] CTAs of the query that have finished; left at zero
};

// A host call's one query, in the launch's arguments: no copy to the device before the launch (1.8 us, and 7.5 more until the
// kernel behind it began).
constexpr int kFewInline = 1024;
template <bool INL> struct FewInline { float q[kFewInline]; };
template <> struct FewInline<false> {};
template <bool INL>
__device__ __forceinline__ float few_query(const FewInline<INL>& iq, const float* q, int64_t i) {
  if constexpr (INL) return iq.q[i];
  else return *VSK_CHK(q + i);
}

struct FewScratch {     // the selection's words
  int hist[256];
  int bin, less, in_bin, out;
};

// Shortens list[0..cnt) to its k smallest keys (cnt > k) and returns the largest of them; every thread takes part.
__device__ __forceinline__ uint64_t few_compact(uint64_t* list, int cnt, int k, FewScratch& s) {
  uint64_t key[SEL_ITEMS];
#pragma unroll
  for (int i = 0; i < SEL_ITEMS; ++i) {
    const int at = threadIdx.x + i * FEW_THREADS;
    key[i] = at < cnt ? list[at] : kEmptyKey;
  }
  if (threadIdx.x == 0) s.out = 0;
  __syncthreads();
  const uint64_t pivot = block_radix_select(key, k, s.hist, &s.bin, &s.less, &s.in_bin);
#pragma unroll
  for (int i = 0; i < SEL_ITEMS; ++i)
    if (key[i] <= pivot && key[i] != kEmptyKey) list[atomicAdd(&s.out, 1)] = key[i];
  __syncthreads();
  return pivot;
}

// After a round of rows: lists that a further round could overfill are shortened to their `keep` smallest keys and tighten their
// query's threshold; after the last round those that do not fit `stride` are.
__device__ __forceinline__ void few_end_round(uint64_t* lists, int nq, int keep, int stride, bool last, int* s_cnt, uint64_t* s_thr, FewScratch& s) {
  __syncthreads();
#pragma unroll 1
  for (int i = 0; i < nq; ++i) {
    const int cnt = s_cnt[i];
    if (cnt > (last ? stride : FEW_LIST - FEW_ROUND)) {
      const uint64_t pivot = few_compact(lists + (size_t)i * FEW_LIST, cnt, keep, s);
      if (threadIdx.x == 0) {
        s_cnt[i] = s.out;
        s_thr[i] = pivot;
      }
    }
  }
  __syncthreads();
}

// Writes this CTA's lists of queries [pos, pos + nq) with their lengths and smallest keys.
__device__ __forceinline__ void few_write_lists(const FewKernelArgs& ka, const uint64_t* lists, int pos, int nq, const int* s_cnt) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 1
  for (int i = 0; i < nq; ++i) {
    const int64_t l = (int64_t)(pos + i) * gridDim.x + blockIdx.x;
    const uint64_t* list = lists + (size_t)i * FEW_LIST;
    const int cnt = s_cnt[i];
    for (int j = threadIdx.x; j < cnt; j += FEW_THREADS) *VSK_CHK_W(ka.part + l * ka.stride + j) = list[j];
    if (warp == 0) {
      uint64_t best = kEmptyKey;
      for (int j = lane; j < cnt; j += 32) best = min(best, list[j]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
      if (lane == 0) {
        *VSK_CHK_W(ka.part_min + l) = best;
        *VSK_CHK_W(ka.part_n + l) = cnt;
      }
    }
  }
}

// The k smallest of list[0..cnt) in order, and their distances and ids out; every thread takes part.
__device__ __forceinline__ void few_order(uint64_t* list, int cnt, int k, bool root, int64_t id_base, float* out_dist, int64_t* out_ids) {
  auto put = [&](int j, uint64_t key, bool has) {
    float d = has ? ordered_to_float((uint32_t)(key >> 32)) : CUDART_INF_F;
    if (has && root) d = sqrtf(d);
    *VSK_CHK_W(out_dist + j) = d;
    *VSK_CHK_W(out_ids + j) = has ? (int64_t)(uint32_t)key + id_base : -1;
  };
  if (cnt <= kFewRank) {   // keys are distinct: a key's place is the number of smaller ones
    const uint64_t mine = (int)threadIdx.x < cnt ? list[threadIdx.x] : kEmptyKey;
    int below = 0;
    for (int j = 0; j < cnt; ++j) below += list[j] < mine;
    if ((int)threadIdx.x < cnt && below < k) put(below, mine, true);
    for (int j = cnt + threadIdx.x; j < k; j += FEW_THREADS) put(j, 0ull, false);
    return;
  }
  const int P = next_pow2(cnt);
  for (int i = cnt + threadIdx.x; i < P; i += FEW_THREADS) list[i] = kEmptyKey;
  __syncthreads();
  bitonic_sort(list, P);
  for (int j = threadIdx.x; j < k; j += FEW_THREADS) put(j, j < cnt ? list[j] : 0ull, j < cnt);
}

// Merges the lists of the launch's query `pos` and writes the result of query `out`.  `list` has room for FEW_LIST keys, `cand` for FEW_MAX_CTAS list numbers.
__device__ __forceinline__ void few_merge(const FewKernelArgs& ka, int64_t pos, int64_t out, int lists, uint64_t* list, unsigned short* cand,
                                          FewScratch& s) {
  __shared__ int n_cand, n_list, n_have;
  const FewArgs& a = ka.a;
  const int k = a.k;
  const uint64_t* mins = ka.part_min + pos * lists;
  uint64_t key[SEL_ITEMS];
  if (threadIdx.x == 0) { n_cand = 0; n_list = 0; n_have = 0; }
  __syncthreads();
  int have = 0;
#pragma unroll
  for (int i = 0; i < SEL_ITEMS; ++i) {
    const int at = threadIdx.x + i * FEW_THREADS;
    key[i] = at < lists ? __ldcg(VSK_CHK(mins + at)) : kEmptyKey;
    have += key[i] != kEmptyKey;
  }
  if (have) atomicAdd(&n_have, have);
  __syncthreads();
  // at least k rows lie at or below the k-th smallest best key
  uint64_t bound = kEmptyKey - 1;
  if (n_have >= k) bound = block_radix_select(key, k, s.hist, &s.bin, &s.less, &s.in_bin);
#pragma unroll
  for (int i = 0; i < SEL_ITEMS; ++i)
    if (key[i] <= bound && key[i] != kEmptyKey) cand[atomicAdd(&n_cand, 1)] = (unsigned short)(threadIdx.x + i * FEW_THREADS);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nc = n_cand;
  int cnt = 0;
  // All of them at once as a rule - few of their keys are within the bound; lists that hold more than there is room for, a
  // batch at a time, shortened in between.
  int batch = max(nc, 1);
  for (int c0 = 0; c0 < nc; c0 += batch) {
    for (int c = c0 + warp; c < min(nc, c0 + batch); c += FEW_WARPS) {
      const int64_t l = pos * lists + cand[c];
      const int n = __ldcg(VSK_CHK(ka.part_n + l));
      for (int i = lane; i < ka.stride; i += 32) {   // (the keys come with their number: what lies behind it is old)
        const uint64_t v = __ldcg(VSK_CHK(ka.part + l * ka.stride + i));
        if (i < n && v <= bound) {
          const int at = atomicAdd(&n_list, 1);
          if (at < FEW_LIST) list[at] = v;
        }
      }
    }
    __syncthreads();
    cnt = n_list;
    __syncthreads();
    if (cnt > FEW_LIST) {   // (the first attempt only)
      batch = (FEW_LIST - k) / ka.stride;
      c0 = -batch;
      if (threadIdx.x == 0) n_list = 0;
    } else if (cnt > max(k, kFewRank) || (cnt > k && batch < nc)) {
      const uint64_t pivot = few_compact(list, cnt, k, s);
      bound = min(bound, pivot);
      cnt = s.out;
      if (threadIdx.x == 0) n_list = cnt;
    }
    __syncthreads();
  }
  few_order(list, cnt, k, a.final_sqrt, a.id_base, a.out_dist + out * k, a.out_ids + out * k);
}

// FEW_ROWS rows per warp step.  CH > 0 (one query, 16-byte loads): rows of at most CH * 128 dimensions, CH loads per row and
// lane, those of the next step issued before this one is reduced.
template <int METRIC, int NQ, bool VEC, bool SEG, int FEW_ROWS, int CH, bool INL>
__global__ void __launch_bounds__(FEW_THREADS, NQ > 4 ? 2 : 3) few_topk_kernel(const __grid_constant__ FewKernelArgs ka,
                                                                              const __grid_constant__ FewInline<INL> iq) {
  static_assert(CH == 0 || (NQ == 1 && VEC), "short rows: one query");
  static_assert(!SEG || NQ == 1, "per-query lists are scanned one query per grid row");
  static_assert(!INL || NQ == 1, "one query travels in the arguments");
  const FewArgs& a = ka.a;
  extern __shared__ __align__(16) uint8_t smem[];
  // [NQ][FEW_LIST] keys, then [NQ][dim] queries, then (SEG) [nprobe + 1] first positions and [nprobe] first rows of the lists
  uint64_t* lists = reinterpret_cast<uint64_t*>(smem);
  float* sq = reinterpret_cast<float*>(smem + (size_t)NQ * FEW_LIST * 8);
  int64_t* seg_pos = reinterpret_cast<int64_t*>(smem + (size_t)NQ * FEW_LIST * 8 + ((size_t)NQ * a.dim * 4 + 7) / 8 * 8);
  int64_t* seg_row = seg_pos + (SEG ? a.nprobe + 1 : 0);
  __shared__ FewScratch fs;
  __shared__ uint64_t s_thr[NQ], s_qm[NQ], s_any;
  __shared__ float s_qn[NQ];
  __shared__ int s_cnt[NQ];
  __shared__ unsigned s_last;
  const int dim = a.dim, k = a.k;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qp = SEG ? (int)blockIdx.y : 0;                         // position in this launch
  const int qb = (SEG && a.q_subset) ? *VSK_CHK(a.q_subset + qp) : qp;         // first query of this CTA
  const int nq_here = SEG ? 1 : (int)a.nq;
  for (int i = threadIdx.x; i < NQ * dim; i += FEW_THREADS) sq[i] = i < nq_here * dim ? few_query<INL>(iq, a.q, (int64_t)qb * dim + i) : 0.f;
  if (threadIdx.x < NQ) {
    s_thr[threadIdx.x] = kEmptyKey - 1;
    s_cnt[threadIdx.x] = 0;
    s_qm[threadIdx.x] = (int)threadIdx.x < nq_here ? (a.q_masks ? *VSK_CHK(a.q_masks + qb + threadIdx.x) : ~0ull) : 0ull;
  }
  if (SEG && warp == 0) {
    // first position of every probed list (an out-of-range probe is an empty list)
    int64_t run = 0;
    for (int p0 = 0; p0 < a.nprobe; p0 += 32) {
      const int p = p0 + lane;
      int64_t beg = 0, len = 0;
      if (p < a.nprobe) {
        const int64_t l = *VSK_CHK(a.probes + (int64_t)qb * a.nprobe + p);
        if (l >= 0 && l < a.nlist) {
          beg = *VSK_CHK(a.list_offsets + l);
          len = *VSK_CHK(a.list_offsets + l + 1) - beg;
        }
      }
      int64_t incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      if (p < a.nprobe) {
        seg_pos[p] = run + incl - len;
        seg_row[p] = beg;
      }
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) seg_pos[a.nprobe] = run;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t any = 0;
    for (int i = 0; i < NQ; ++i) any |= s_qm[i];
    s_any = any;
  }
  if (METRIC == VSK_METRIC_COSINE)
    for (int i = warp; i < NQ; i += FEW_WARPS) {   // |q|, summed as the row norms are
      float ss = 0.f;
      for (int c = lane; c < dim; c += 32) ss = fmaf(sq[i * dim + c], sq[i * dim + c], ss);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane == 0) s_qn[i] = sqrtf(ss);
    }
  __syncthreads();
  const uint64_t any_mask = s_any;
  const int64_t n = SEG ? seg_pos[a.nprobe] : a.n;

  constexpr int V = FEW_ROWS * NQ;
  constexpr int OWNER_SHIFT = 5 - Log2<V>::value;
  int round = ka.round;
  if (SEG) {   // the lists' true length: as few rounds as their size allows, the rows spread evenly over them
    const int64_t share = (n + gridDim.x - 1) / gridDim.x, rounds = (share + FEW_ROUND - 1) / FEW_ROUND;
    constexpr int kStep = FEW_WARPS * FEW_ROWS;
    round = n > 0 ? (int)min((int64_t)FEW_ROUND, ((share + rounds - 1) / rounds + kStep - 1) / kStep * kStep) : kStep;
  }
  const int64_t stride = (int64_t)gridDim.x * round;
  int cur = 0;   // SEG: the list of the current position
  // rows n0 .. of the warp's step; a row that no query of the batch may see is not live, and not read
  auto locate = [&](int64_t n0, int64_t r1, uint32_t (&rid)[FEW_ROWS], uint64_t (&rmask)[FEW_ROWS], bool (&live)[FEW_ROWS]) {
#pragma unroll
    for (int r = 0; r < FEW_ROWS; ++r) {
      const int64_t at = n0 + r;
      const bool has = at < r1;
      rid[r] = has ? (uint32_t)at : 0u;
      if (SEG && has) {   // positions only grow: the warp's current list serves until the next one starts
        while (cur + 1 < a.nprobe && seg_pos[cur + 1] <= at) ++cur;
        rid[r] = (uint32_t)(seg_row[cur] + (at - seg_pos[cur]));
      }
      rmask[r] = (a.row_masks && has) ? __ldg(a.row_masks + rid[r]) : ~0ull;
      live[r] = has && (rmask[r] & any_mask) != 0;
    }
  };
  // the step's partial sums to values, and those at or below the threshold to the lists
  auto list_step = [&](float (&acc)[V], int64_t n0, const uint32_t (&rid)[FEW_ROWS], const uint64_t (&rmask)[FEW_ROWS], const bool (&live)[FEW_ROWS]) {
    warp_reduce_scatter<V>(acc, lane);
    if ((lane & ((1 << OWNER_SHIFT) - 1)) == 0) {
      const int j = lane >> OWNER_SHIFT;
      const int r = j / NQ, i = j - r * NQ;
      bool liver = live[0];
      uint32_t ridr = rid[0];
      uint64_t rmaskr = rmask[0];
#pragma unroll
      for (int t = 1; t < FEW_ROWS; ++t)
        if (r == t) { liver = live[t]; ridr = rid[t]; rmaskr = rmask[t]; }
      if (liver && i < nq_here && (rmaskr & s_qm[i]) != 0) {
        float v = acc[0];
        if (METRIC == VSK_METRIC_COSINE) v = 1.0f - v / (s_qn[i] * __ldg(a.xnorm + ridr) + 1e-8f);
        else if (METRIC == VSK_METRIC_DOT_PRODUCT) v = -v;
        // With ids of their own (id_remap) rows are listed by number and get their ids at the round's end, all at once: by
        // value, that is, and one that only ties the threshold is listed whatever its id.
        const uint64_t key = make_key(v, a.id_remap ? 0u : ridr);
        // a value that is not a number is listed among the first rows only, as the chunked schedule does
        if (key <= s_thr[i] && (!isnan(v) || n0 + r < a.nan_rows))
          lists[i * FEW_LIST + atomicAdd(&s_cnt[i], 1)] = make_key(v, ridr);
      }
    }
  };
  int done = 0;   // keys of the list that carry their ids already (id_remap comes with one query per CTA)
  for (int64_t r0 = (int64_t)blockIdx.x * round; r0 < n; r0 += stride) {
    const int64_t r1 = min(n, r0 + round);
    int64_t n0 = r0 + warp * FEW_ROWS;
    if constexpr (CH > 0) {
      const int nv = dim >> 2;
      const float4* sq4 = reinterpret_cast<const float4*>(sq);
      float4 qv[CH];
#pragma unroll
      for (int c = 0; c < CH; ++c) qv[c] = lane + 32 * c < nv ? sq4[lane + 32 * c] : make_float4(0.f, 0.f, 0.f, 0.f);
      // (one query: a live row is one the query may see, its mask is not needed again)
      uint64_t rmask[FEW_ROWS];
      uint32_t rid[FEW_ROWS];
      float4 x[FEW_ROWS][CH];
      auto fetch = [&](const bool (&live)[FEW_ROWS]) {
#pragma unroll
        for (int r = 0; r < FEW_ROWS; ++r)
#pragma unroll
          for (int c = 0; c < CH; ++c)
            x[r][c] = (live[r] && lane + 32 * c < nv) ? __ldg(reinterpret_cast<const float4*>(a.x + (int64_t)rid[r] * dim) + lane + 32 * c)
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
      };
      bool live[FEW_ROWS];
      if (n0 < r1) {
        locate(n0, r1, rid, rmask, live);
        fetch(live);
      }
      for (; n0 < r1; n0 += FEW_WARPS * FEW_ROWS) {
        float acc[V];
#pragma unroll
        for (int r = 0; r < FEW_ROWS; ++r) {
          acc[r] = 0.f;
#pragma unroll
          for (int c = 0; c < CH; ++c) {
            if (lane + 32 * c >= nv) continue;
            tile::accum<METRIC>(acc[r], qv[c].x, x[r][c].x);
            tile::accum<METRIC>(acc[r], qv[c].y, x[r][c].y);
            tile::accum<METRIC>(acc[r], qv[c].z, x[r][c].z);
            tile::accum<METRIC>(acc[r], qv[c].w, x[r][c].w);
          }
        }
        // the next step's rows are on their way while this one's sums are exchanged and listed
        uint32_t was[FEW_ROWS];
        bool had[FEW_ROWS];
#pragma unroll
        for (int r = 0; r < FEW_ROWS; ++r) {
          was[r] = rid[r];
          had[r] = live[r];
          rmask[r] = ~0ull;
        }
        const int64_t n1 = n0 + FEW_WARPS * FEW_ROWS;
        if (n1 < r1) {
          locate(n1, r1, rid, rmask, live);
          fetch(live);
#pragma unroll
          for (int r = 0; r < FEW_ROWS; ++r) rmask[r] = ~0ull;
        }
        list_step(acc, n0, was, rmask, had);
      }
    } else {
      for (; n0 < r1; n0 += FEW_WARPS * FEW_ROWS) {
        bool live[FEW_ROWS];
        uint32_t rid[FEW_ROWS];
        uint64_t rmask[FEW_ROWS];
        locate(n0, r1, rid, rmask, live);
        float acc[V];
#pragma unroll
        for (int j = 0; j < V; ++j) acc[j] = 0.f;
        stream_accumulate<METRIC, NQ, VEC, FEW_ROWS>(acc, a.x, dim, sq, rid, live, lane);
        list_step(acc, n0, rid, rmask, live);
      }
    }
    if (NQ == 1 && a.id_remap) {
      __syncthreads();
      const int cnt = s_cnt[0];
      for (int j = done + threadIdx.x; j < cnt; j += FEW_THREADS)
        lists[j] = (lists[j] & 0xffffffff00000000ull) | (uint32_t)*VSK_CHK(a.id_remap + (uint32_t)lists[j]);
    }
    few_end_round(lists, nq_here, k, ka.stride, r0 + stride >= n, s_cnt, s_thr, fs);
    if (NQ == 1 && a.id_remap) {
      done = s_cnt[0];
      __syncthreads();   // the next round's first keys are counted in s_cnt: not before every thread has read it
    }
  }
  // ---- this CTA's lists, and the merge by the last one to arrive ----
  few_write_lists(ka, lists, qp, nq_here, s_cnt);
  if (NQ > 1) return;   // several queries: few_merge_kernel merges them side by side
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(ka.ticket + qp, 1u);
  __syncthreads();
  if (s_last != gridDim.x - 1) return;
  __threadfence();
  if (threadIdx.x == 0) *VSK_CHK_W(ka.ticket + qp) = 0u;
  // the query's staging area is free now: list numbers go there (the launch makes it large enough)
  few_merge(ka, qp, qb, (int)gridDim.x, lists, reinterpret_cast<unsigned short*>(smem + (size_t)NQ * FEW_LIST * 8), fs);
}

// ---- the same over the fp16 operand copy ----------------------------------------------------------------------------
// A large store is bound by the bytes of its rows: one query over 1 million x 768 reads 3 GB of fp32 rows, or 1.5 GB of the
// fp16 copy the tensor path keeps (that path padded the query to a tile of 128 and reached 3.4 TB/s: 490 us).  The queries
// stay in fp32, so a coarse value is off by no more than |q| E_x and its own summation (eps).  Every CTA keeps its
// k + kFewMargin best coarse keys; the last step lists every row within 2 eps of the k-th best, re-scores those with the
// direct formulas and orders them.  A query for which that list or one CTA's share of it does not fit is flagged and run
// over the fp32 rows.
constexpr int kFewMargin = 64;
constexpr int FEWH_ROWS = 4;   // rows per warp step: four 16-byte loads in flight per lane

struct FewHalf {
  const __half* x16;      // [n][dim16], s x (cosine: s x / |x|)
  const float* aux;       // |x|^2 (euclidean)
  int32_t dim16;
  float inv_scale;        // 1 / s
  float err, norm;        // largest |s x - x16| / s and |x16| / s of a row
  float max_norm, min_norm_nz;
  int32_t* flags;         // [nq] (pinned host memory), set to 0 or 1
};

// |coarse - exact| for every row, in coarse units (bound_kernel's terms with an unrounded query)
template <int METRIC>
__device__ __forceinline__ float few_eps(const FewHalf& h, int dim, float qn) {
  const float q = METRIC == VSK_METRIC_COSINE ? 1.0f : qn;
  float e = q * h.err + 1.2e-7f * (float)(dim + 16) * q * h.norm;
  if (METRIC == VSK_METRIC_EUCLIDEAN) {
    e = 2.0f * e + 2.4e-7f * (float)(dim + 16) * h.max_norm * h.max_norm +
        1.2e-7f * (h.max_norm * h.max_norm + 2.0f * qn * h.max_norm) + 1.2e-7f * (float)(dim + 16) * qn * h.max_norm + 1.2e-7f * (float)(dim / 32 + 8) * qn * qn;
  } else if (METRIC == VSK_METRIC_COSINE) {
    const float den = qn * h.min_norm_nz;
    e += den > 0.f ? 1e-8f / (den + 1e-8f) + 4.8e-7f : 4.8e-7f;
  }
  return e * 1.0001f + 1e-30f;
}

template <int METRIC>
__device__ __forceinline__ void few_refine(const FewKernelArgs& ka, const FewHalf& h, int lists, int64_t pos, const float* q, uint64_t* list,
                                           unsigned short* cand, FewScratch& fs);

template <int METRIC, int NQ, bool INL>
__global__ void __launch_bounds__(FEW_THREADS, NQ > 4 ? 2 : 3) few_coarse_kernel(const __grid_constant__ FewKernelArgs ka, FewHalf h,
                                                                                const __grid_constant__ FewInline<INL> iq) {
  const FewArgs& a = ka.a;
  extern __shared__ __align__(16) uint8_t smem[];
  uint64_t* lists = reinterpret_cast<uint64_t*>(smem);                       // [NQ][FEW_LIST]
  float4* sq = reinterpret_cast<float4*>(smem + (size_t)NQ * FEW_LIST * 8);  // [NQ][2][dim16 / 8]: halves of 8 dimensions
  __shared__ FewScratch fs;
  __shared__ uint64_t s_thr[NQ];
  __shared__ float s_qn[NQ];
  __shared__ int s_cnt[NQ];
  const int dim = a.dim, keep = a.k + kFewMargin, nv = h.dim16 >> 3;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = (int)a.nq;
  if (threadIdx.x < NQ) {
    s_thr[threadIdx.x] = kEmptyKey - 1;
    s_cnt[threadIdx.x] = 0;
  }
  for (int i = warp; i < NQ; i += FEW_WARPS) {
    float ss = 0.f;
    for (int c = lane; c < dim; c += 32) {
      const float v = i < nq ? few_query<INL>(iq, a.q, (int64_t)i * dim + c) : 0.f;
      ss = fmaf(v, v, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float qn = sqrtf(ss), f = METRIC == VSK_METRIC_COSINE ? (qn > 0.f ? 1.0f / qn : 0.f) : 1.0f;
    if (lane == 0) s_qn[i] = qn;
    for (int c = lane; c < h.dim16; c += 32) {
      const float v = (i < nq && c < dim) ? few_query<INL>(iq, a.q, (int64_t)i * dim + c) * f : 0.f;
      reinterpret_cast<float*>(sq)[((i * 2 + ((c >> 2) & 1)) * nv + (c >> 3)) * 4 + (c & 3)] = v;
    }
  }
  __syncthreads();
  constexpr int V = FEWH_ROWS * NQ;
  constexpr int OWNER_SHIFT = 5 - Log2<V>::value;
  const float alpha = (METRIC == VSK_METRIC_EUCLIDEAN ? -2.0f : -1.0f) * h.inv_scale;
  const int64_t n = a.n, stride = (int64_t)gridDim.x * ka.round;
  for (int64_t r0 = (int64_t)blockIdx.x * ka.round; r0 < n; r0 += stride) {
    const int64_t r1 = min(n, r0 + ka.round);
    for (int64_t n0 = r0 + warp * FEWH_ROWS; n0 < r1; n0 += FEW_WARPS * FEWH_ROWS) {
      float acc[V];
#pragma unroll
      for (int j = 0; j < V; ++j) acc[j] = 0.f;
      const uint4* p[FEWH_ROWS];
#pragma unroll
      for (int r = 0; r < FEWH_ROWS; ++r) p[r] = reinterpret_cast<const uint4*>(h.x16 + min(n0 + r, n - 1) * h.dim16);
      for (int c = lane; c < nv; c += 32) {
        uint4 x[FEWH_ROWS];
#pragma unroll
        for (int r = 0; r < FEWH_ROWS; ++r) x[r] = __ldg(p[r] + c);
        float2 f[FEWH_ROWS][4];
#pragma unroll
        for (int r = 0; r < FEWH_ROWS; ++r) {
          f[r][0] = __half22float2(*reinterpret_cast<const __half2*>(&x[r].x));
          f[r][1] = __half22float2(*reinterpret_cast<const __half2*>(&x[r].y));
          f[r][2] = __half22float2(*reinterpret_cast<const __half2*>(&x[r].z));
          f[r][3] = __half22float2(*reinterpret_cast<const __half2*>(&x[r].w));
        }
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
          const float4 lo = sq[(i * 2) * nv + c], hi = sq[(i * 2 + 1) * nv + c];
#pragma unroll
          for (int r = 0; r < FEWH_ROWS; ++r) {
            float& s = acc[r * NQ + i];
            s = fmaf(lo.x, f[r][0].x, s); s = fmaf(lo.y, f[r][0].y, s); s = fmaf(lo.z, f[r][1].x, s); s = fmaf(lo.w, f[r][1].y, s);
            s = fmaf(hi.x, f[r][2].x, s); s = fmaf(hi.y, f[r][2].y, s); s = fmaf(hi.z, f[r][3].x, s); s = fmaf(hi.w, f[r][3].y, s);
          }
        }
      }
      warp_reduce_scatter<V>(acc, lane);
      if ((lane & ((1 << OWNER_SHIFT) - 1)) == 0) {
        const int j = lane >> OWNER_SHIFT;
        const int r = j / NQ, i = j - r * NQ;
        if (n0 + r < r1 && i < nq) {
          float v = acc[0] * alpha;
          if (METRIC == VSK_METRIC_EUCLIDEAN) v += __ldg(h.aux + n0 + r);
          const uint64_t key = make_key(v, (uint32_t)(n0 + r));
          if (key <= s_thr[i]) lists[i * FEW_LIST + atomicAdd(&s_cnt[i], 1)] = key;
        }
      }
    }
    few_end_round(lists, nq, keep, ka.stride, r0 + stride >= n, s_cnt, s_thr, fs);
  }
  few_write_lists(ka, lists, 0, nq, s_cnt);
  if (NQ > 1) return;   // several queries: few_refine_kernel takes them side by side
  __shared__ unsigned s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(ka.ticket, 1u);
  __syncthreads();
  if (s_last != gridDim.x - 1) return;
  __threadfence();
  if (threadIdx.x == 0) *VSK_CHK_W(ka.ticket) = 0u;
  // the query as it is, where its halves were; behind it the list numbers
  float* qs = reinterpret_cast<float*>(sq);
  for (int c = threadIdx.x; c < dim; c += FEW_THREADS) qs[c] = few_query<INL>(iq, a.q, c);
  __syncthreads();
  few_refine<METRIC>(ka, h, (int)gridDim.x, 0, qs, lists, reinterpret_cast<unsigned short*>(qs + h.dim16), fs);
}

// The rows within 2 eps of the k-th best coarse value, re-scored with the direct formulas and ordered.
template <int METRIC>
__device__ __forceinline__ void few_refine(const FewKernelArgs& ka, const FewHalf& h, int lists, int64_t pos, const float* q, uint64_t* list,
                                           unsigned short* cand, FewScratch& fs) {
  __shared__ int n_cand, n_list, n_have, s_bad;
  __shared__ float s_qn;
  const FewArgs& a = ka.a;
  const int k = a.k, keep = k + kFewMargin, dim = a.dim;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) { n_cand = 0; n_list = 0; n_have = 0; s_bad = 0; }
  if (warp == 0) {
    float ss = 0.f;
    for (int c = lane; c < dim; c += 32) ss = fmaf(*VSK_CHK(q + c), *VSK_CHK(q + c), ss);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) s_qn = sqrtf(ss);
  }
  __syncthreads();
  const float qn = s_qn, band = 2.0f * few_eps<METRIC>(h, dim, qn);
  uint64_t key[SEL_ITEMS];
  int have = 0;
#pragma unroll
  for (int i = 0; i < SEL_ITEMS; ++i) {
    const int at = threadIdx.x + i * FEW_THREADS;
    key[i] = at < lists ? __ldcg(VSK_CHK(ka.part_min + pos * lists + at)) : kEmptyKey;
    have += key[i] != kEmptyKey;
  }
  if (have) atomicAdd(&n_have, have);
  __syncthreads();
  // rows at or below `value` + band; what is not a number leaves every row in
  auto widened = [&](uint64_t kth) {
    const float b = ordered_to_float((uint32_t)(kth >> 32)) + band;
    return b < CUDART_INF_F ? ((uint64_t)float_to_ordered(b) << 32) | 0xffffffffull : kEmptyKey - 1;
  };
  uint64_t bound = kEmptyKey - 1;
  if (n_have >= k) bound = widened(block_radix_select(key, k, fs.hist, &fs.bin, &fs.less, &fs.in_bin));
#pragma unroll
  for (int i = 0; i < SEL_ITEMS; ++i)
    if (key[i] <= bound && key[i] != kEmptyKey) cand[atomicAdd(&n_cand, 1)] = (unsigned short)(threadIdx.x + i * FEW_THREADS);
  __syncthreads();
  const int nc = n_cand;
  for (int c = warp; c < nc; c += FEW_WARPS) {
    const int64_t l = pos * lists + cand[c];
    const int m = __ldcg(VSK_CHK(ka.part_n + l));
    bool all = m >= keep;   // a shortened list whose every key is within the bound may have dropped such a row
    for (int i = lane; i < m; i += 32) {
      const uint64_t v = __ldcg(VSK_CHK(ka.part + l * ka.stride + i));
      if (v <= bound) {
        const int at = atomicAdd(&n_list, 1);
        if (at < FEW_LIST) list[at] = v;
      } else {
        all = false;
      }
    }
    if (__all_sync(0xffffffffu, all) && lane == 0) s_bad = 1;
  }
  __syncthreads();
  int cnt = n_list;
  if (cnt > FEW_LIST || s_bad != 0 || !(band < CUDART_INF_F)) {
    if (threadIdx.x == 0) *VSK_CHK_W(h.flags + pos) = 1;
    return;
  }
  if (cnt > k) {   // the k-th best of all, then only what is within the band of it
#pragma unroll
    for (int i = 0; i < SEL_ITEMS; ++i) {
      const int at = threadIdx.x + i * FEW_THREADS;
      key[i] = at < cnt ? list[at] : kEmptyKey;
    }
    if (threadIdx.x == 0) fs.out = 0;
    __syncthreads();
    bound = widened(block_radix_select(key, k, fs.hist, &fs.bin, &fs.less, &fs.in_bin));
#pragma unroll
    for (int i = 0; i < SEL_ITEMS; ++i)
      if (key[i] <= bound && key[i] != kEmptyKey) list[atomicAdd(&fs.out, 1)] = key[i];
    __syncthreads();
    cnt = fs.out;
  }
  // exact values, summed as the tensor path's re-scoring sums them: four rows per warp step
  constexpr int RR = 4;
  for (int c0 = warp * RR; c0 < cnt; c0 += FEW_WARPS * RR) {
    uint32_t id[RR];
    float s[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      id[r] = (uint32_t)list[min(c0 + r, cnt - 1)];
      s[r] = 0.f;
    }
    for (int i = lane; i < dim; i += 32) {
      const float qv = *VSK_CHK(q + i);
#pragma unroll
      for (int r = 0; r < RR; ++r) {
        const float xv = __ldg(a.x + (int64_t)id[r] * dim + i);
        tile::accum<METRIC>(s[r], qv, xv);
      }
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < RR; ++r) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
      if (lane == 0 && c0 + r < cnt) {
        float v = s[r];
        if (METRIC == VSK_METRIC_COSINE) v = 1.0f - v / (qn * __ldg(a.xnorm + id[r]) + 1e-8f);
        else if (METRIC == VSK_METRIC_DOT_PRODUCT) v = -v;
        list[c0 + r] = make_key(v, id[r]);
      }
    }
  }
  __syncthreads();
  few_order(list, cnt, k, METRIC == VSK_METRIC_EUCLIDEAN, a.id_base, a.out_dist + pos * k, a.out_ids + pos * k);
  if (threadIdx.x == 0) *VSK_CHK_W(h.flags + pos) = 0;
}

template <int METRIC>
__global__ void __launch_bounds__(FEW_THREADS) few_refine_kernel(FewKernelArgs ka, FewHalf h, int lists) {
  __shared__ uint64_t list[FEW_LIST];
  __shared__ unsigned short cand[FEW_MAX_CTAS];
  __shared__ FewScratch fs;
  few_refine<METRIC>(ka, h, lists, blockIdx.x, ka.a.q + (int64_t)blockIdx.x * ka.a.dim, list, cand, fs);
}

__global__ void __launch_bounds__(FEW_THREADS) few_merge_kernel(FewKernelArgs ka, int lists) {
  __shared__ uint64_t list[FEW_LIST];
  __shared__ unsigned short cand[FEW_MAX_CTAS];
  __shared__ FewScratch fs;
  few_merge(ka, blockIdx.x, blockIdx.x, lists, list, cand, fs);
}

template <int NQ>
size_t few_smem(const FewArgs& a) {
  size_t b = ((size_t)NQ * a.dim * 4 + 7) / 8 * 8;
  if (a.probes) b += (size_t)(2 * a.nprobe + 1) * 8;
  b = std::max<size_t>(b, FEW_MAX_CTAS * sizeof(unsigned short));   // the merge's list numbers go here
  return (size_t)NQ * FEW_LIST * 8 + b;
}
constexpr size_t kFewMaxSmem = 110 * 1024;   // two CTAs per SM

// The query of a host call that has not been copied to the device yet (HostQuery), when it fits the arguments.
const float* few_inline_query(const Ctx* ctx, const FewArgs& a) {
  return a.nq == 1 && a.dim <= kFewInline && ctx->host_query.pending && ctx->host_query.dev == a.q ? ctx->host_query.host : nullptr;
}

template <int METRIC, int NQ, bool VEC, bool SEG, int ROWS, int CH, bool INL>
int32_t few_launch_as(Ctx* ctx, FewKernelArgs ka, const float* host_q) {
  const FewArgs& a = ka.a;
  auto kern = few_topk_kernel<METRIC, NQ, VEC, SEG, ROWS, CH, INL>;
  const size_t smem = few_smem<NQ>(a);
  if (smem > 48 * 1024) VSK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int sms = ctx->prop.multiProcessorCount;
  const int per_sm = std::max(1, std::min(NQ > 4 ? 2 : 3, (int)(220 * 1024 / (smem + 3072))));
  // 32 rows per CTA at least; per-query lists share the machine.  SEG: the mean list's length is known, but probed lists are the
  // longer ones, and the kernel takes their true lengths
  const int64_t rows = std::max<int64_t>(SEG ? 2 * a.n : a.n, 1);
  const int64_t nseg = SEG ? a.nq : 1;
  constexpr int kStep = FEW_WARPS * ROWS;
  const int64_t grid = std::min({ceil_div(rows, 32), std::max<int64_t>(1, (int64_t)sms * per_sm / nseg), (int64_t)FEW_MAX_CTAS});
  // rounds of whole warp steps, such that the last one is spread evenly
  const int64_t share = ceil_div(rows, grid);
  ka.round = (int32_t)std::min<int64_t>(FEW_ROUND, ceil_div(ceil_div(share, ceil_div(share, (int64_t)FEW_ROUND)), kStep) * kStep);
  ka.stride = std::max(a.k, kFewShort);
  void* p;
  const size_t lists = (size_t)a.nq * grid;
  VSK_TRY(scratch(ctx, SLOT_FEW, lists * ((size_t)ka.stride * 8 + 8 + 4), &p));
  ka.part = (uint64_t*)p;
  ka.part_min = ka.part + lists * ka.stride;
  ka.part_n = (int32_t*)(ka.part_min + lists);
  FewInline<INL> iq;
  if constexpr (INL) memcpy(iq.q, host_q, (size_t)a.dim * sizeof(float));
  prof_begin(ctx);
  kern<<<dim3((unsigned)grid, (unsigned)nseg), FEW_THREADS, smem, ctx->stream>>>(ka, iq);
  prof_end(ctx);
  ctx->stats.kernel_launches++;
  if (NQ > 1) {
    few_merge_kernel<<<(unsigned)a.nq, FEW_THREADS, 0, ctx->stream>>>(ka, (int)grid);
    ctx->stats.kernel_launches++;
  }
  VSK_CUDA(ctx, cudaGetLastError());
  return VSK_OK;
}

// One query over rows of at most 256 dimensions: four 16-byte loads per lane and step, the next step's already on their way
// (the general form takes two rows per step and waits for them).  Whole call, general form / this, rows of 256 dimensions: 400 000
// rows 104 / 94 us (cosine 115 / 99), 100 000 rows 46.6 / 43.4; of 160: 100 000 rows 42.5 / 41.8; 10 000 rows, stored or probed: the same.
template <int METRIC, int NQ, bool VEC, bool SEG, bool INL>
int32_t few_launch_one(Ctx* ctx, const FewKernelArgs& ka, const float* host_q) {
  if constexpr (VEC) {
    if (ka.a.dim <= 128) return few_launch_as<METRIC, NQ, VEC, SEG, 4, 1, INL>(ctx, ka, host_q);
    if (ka.a.dim <= 256) return few_launch_as<METRIC, NQ, VEC, SEG, 2, 2, INL>(ctx, ka, host_q);
  }
  return few_launch_as<METRIC, NQ, VEC, SEG, 2, 0, INL>(ctx, ka, host_q);
}

template <int METRIC, int NQ, bool VEC, bool SEG>
int32_t few_launch(Ctx* ctx, const FewKernelArgs& ka) {
  if constexpr (NQ == 1)
    if (const float* host_q = few_inline_query(ctx, ka.a)) return few_launch_one<METRIC, NQ, VEC, SEG, true>(ctx, ka, host_q);
  VSK_TRY(host_query_upload(ctx));
  if constexpr (NQ == 1) return few_launch_one<METRIC, NQ, VEC, SEG, false>(ctx, ka, nullptr);
  else return few_launch_as<METRIC, NQ, VEC, SEG, 2, 0, false>(ctx, ka, nullptr);
}

template <int METRIC>
int32_t few_metric(Ctx* ctx, const FewKernelArgs& ka, bool vec) {
  const FewArgs& a = ka.a;
  if (a.nq <= 1) return vec ? few_launch<METRIC, 1, true, false>(ctx, ka) : few_launch<METRIC, 1, false, false>(ctx, ka);
  if (a.nq <= 2) return vec ? few_launch<METRIC, 2, true, false>(ctx, ka) : few_launch<METRIC, 2, false, false>(ctx, ka);
  if (a.nq <= 4) return vec ? few_launch<METRIC, 4, true, false>(ctx, ka) : few_launch<METRIC, 4, false, false>(ctx, ka);
  return vec ? few_launch<METRIC, 8, true, false>(ctx, ka) : few_launch<METRIC, 8, false, false>(ctx, ka);
}

}  // namespace

namespace {

template <int METRIC, int NQ, bool INL>
int32_t few_half_launch(Ctx* ctx, FewKernelArgs ka, const FewHalf& h, const float* host_q) {
  const FewArgs& a = ka.a;
  auto kern = few_coarse_kernel<METRIC, NQ, INL>;
  const size_t smem = (size_t)NQ * (FEW_LIST * 8 + (size_t)h.dim16 * 4) + (NQ == 1 ? FEW_MAX_CTAS * sizeof(unsigned short) : 0);
  if (smem > 48 * 1024) VSK_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int per_sm = std::max(1, std::min(NQ > 4 ? 2 : 3, (int)(220 * 1024 / (smem + 3072))));
  constexpr int kStep = FEW_WARPS * FEWH_ROWS;
  const int64_t grid = std::min<int64_t>(ceil_div(a.n, kStep), (int64_t)ctx->prop.multiProcessorCount * per_sm);
  const int64_t share = ceil_div(a.n, grid);
  ka.round = (int32_t)std::min<int64_t>(FEW_ROUND, ceil_div(ceil_div(share, ceil_div(share, (int64_t)FEW_ROUND)), kStep) * kStep);
  ka.stride = a.k + kFewMargin;
  void* p;
  const size_t lists = (size_t)a.nq * grid;
  VSK_TRY(scratch(ctx, SLOT_FEW, lists * ((size_t)ka.stride * 8 + 8 + 4), &p));
  ka.part = (uint64_t*)p;
  ka.part_min = ka.part + lists * ka.stride;
  ka.part_n = (int32_t*)(ka.part_min + lists);
  FewInline<INL> iq;
  if constexpr (INL) memcpy(iq.q, host_q, (size_t)a.dim * sizeof(float));
  prof_begin(ctx);
  kern<<<(unsigned)grid, FEW_THREADS, smem, ctx->stream>>>(ka, h, iq);
  prof_end(ctx);
  ctx->stats.kernel_launches++;
  if (NQ > 1) {
    few_refine_kernel<METRIC><<<(unsigned)a.nq, FEW_THREADS, 0, ctx->stream>>>(ka, h, (int)grid);
    ctx->stats.kernel_launches++;
  }
  VSK_CUDA(ctx, cudaGetLastError());
  return VSK_OK;
}

template <int METRIC>
int32_t few_half_metric(Ctx* ctx, const FewKernelArgs& ka, const FewHalf& h) {
  if (const float* host_q = few_inline_query(ctx, ka.a)) return few_half_launch<METRIC, 1, true>(ctx, ka, h, host_q);
  VSK_TRY(host_query_upload(ctx));
  if (ka.a.nq <= 1) return few_half_launch<METRIC, 1, false>(ctx, ka, h, nullptr);
  if (ka.a.nq <= 2) return few_half_launch<METRIC, 2, false>(ctx, ka, h, nullptr);
  if (ka.a.nq <= 4) return few_half_launch<METRIC, 4, false>(ctx, ka, h, nullptr);
  return few_half_launch<METRIC, 8, false>(ctx, ka, h, nullptr);
}

}  // namespace

// zeroed once: the last CTA of a query leaves its ticket at zero
static int32_t few_tickets(Ctx* ctx, unsigned** out) {
  unsigned*& tickets = ctx->few_tickets[ctx->lane];
  if (!tickets) {
    VSK_TRY(dev_alloc(ctx, (void**)&tickets, kStreamScanMaxSegQueries * sizeof(unsigned)));
    VSK_CUDA(ctx, cudaMemsetAsync(tickets, 0, kStreamScanMaxSegQueries * sizeof(unsigned), ctx->stream));
  }
  *out = tickets;
  return VSK_OK;
}

int32_t few_search_half(Index* ix, const FewArgs& a, bool* handled) {
  VSK_TRACE("vsk:few_search_half");
  Ctx* ctx = ix->ctx;
  *handled = false;
  const size_t staged = a.nq <= 1 ? 1 : a.nq <= 2 ? 2 : a.nq <= 4 ? 4 : 8;
  if (ctx->search_path != VSK_PATH_TENSOR_RERANK || !ctx->tuning.stream_scan || a.k < 1 || a.k > kFewMaxK || a.nq < 1 ||
      a.nq > kStreamScanMaxQueries || a.row_masks || staged * (FEW_LIST * 8 + (size_t)(a.dim + 80) * 4) > kFewMaxSmem)
    return VSK_OK;
  VSK_TRY(tensor_prepare_index(ix));
  FewHalf h{};
  h.x16 = ix->rows16;
  h.aux = ix->row_aux;
  h.dim16 = ix->dim16;
  h.inv_scale = 1.0f / ix->scale16;
  h.err = ix->max_xerr16 * h.inv_scale;
  h.norm = ix->max_xnorm16 * h.inv_scale;
  h.max_norm = ix->max_xnorm;
  h.min_norm_nz = ix->min_xnorm_nz;
  PinnedBuf& hb = ctx->host_flags[ctx->lane];   // the kernel's flags go straight to the host
  VSK_TRY(pinned_reserve(ctx, &hb, (size_t)a.nq * 4));
  h.flags = (int32_t*)hb.p;
  FewKernelArgs ka{};
  ka.a = a;
  VSK_TRY(few_tickets(ctx, &ka.ticket));
  switch (a.metric) {
    case VSK_METRIC_EUCLIDEAN: VSK_TRY(few_half_metric<VSK_METRIC_EUCLIDEAN>(ctx, ka, h)); break;
    case VSK_METRIC_COSINE: VSK_TRY(few_half_metric<VSK_METRIC_COSINE>(ctx, ka, h)); break;
    default: VSK_TRY(few_half_metric<VSK_METRIC_DOT_PRODUCT>(ctx, ka, h)); break;
  }
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  int64_t bad = 0;
  for (int64_t i = 0; i < a.nq; ++i) bad += ((const int32_t*)hb.p)[i] != 0;
  *handled = true;
  if (bad == 0) return VSK_OK;
  ctx->stats.fallback_queries += bad;
  return few_search(ctx, a);   // the fp32 rows: all of these few queries again
}

bool few_search_applies(const Ctx* ctx, const FewArgs& a) {
  // (the fp32 search path is the chunked schedule by definition)
  if (ctx->search_path != VSK_PATH_TENSOR_RERANK || !ctx->tuning.stream_scan || a.k < 1 || a.k > kFewMaxK || a.nq < 1 || a.dim < 1) return false;
  if (a.probes) return a.metric == VSK_METRIC_EUCLIDEAN && a.nq <= kStreamScanMaxSegQueries && few_smem<1>(a) <= kFewMaxSmem;
  if (a.nq > kStreamScanMaxQueries) return false;
  return (a.nq <= 1 ? few_smem<1>(a) : a.nq <= 2 ? few_smem<2>(a) : a.nq <= 4 ? few_smem<4>(a) : few_smem<8>(a)) <= kFewMaxSmem;
}

int32_t few_search(Ctx* ctx, const FewArgs& a) {
  VSK_TRACE("vsk:few_search");
  FewKernelArgs ka{};
  ka.a = a;
  ka.a.nan_rows = schedule_dense_rows(ctx, a.k);
  VSK_TRY(few_tickets(ctx, &ka.ticket));
  const bool vec = a.dim % 4 == 0 && (reinterpret_cast<uintptr_t>(a.x) & 15) == 0;
  if (a.probes)
    return vec ? few_launch<VSK_METRIC_EUCLIDEAN, 1, true, true>(ctx, ka) : few_launch<VSK_METRIC_EUCLIDEAN, 1, false, true>(ctx, ka);
  switch (a.metric) {
    case VSK_METRIC_EUCLIDEAN: return few_metric<VSK_METRIC_EUCLIDEAN>(ctx, ka, vec);
    case VSK_METRIC_COSINE: return few_metric<VSK_METRIC_COSINE>(ctx, ka, vec);
    case VSK_METRIC_DOT_PRODUCT: return few_metric<VSK_METRIC_DOT_PRODUCT>(ctx, ka, vec);
    case VSK_METRIC_MANHATTAN: return few_metric<VSK_METRIC_MANHATTAN>(ctx, ka, vec);
    default: return fail(ctx, VSK_ERR_UNSUPPORTED_OPERATION, "metric %d is not supported", a.metric);
  }
}

}  // namespace vsk
