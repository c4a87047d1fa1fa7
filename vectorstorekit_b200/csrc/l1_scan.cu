// Manhattan batches: an 8-bit filter in front of the exact formula.
//
// sum |q - x| has no matrix form, so the fp32 tile spends two FP32-pipe instructions per (query, row, dimension) and is bound
// by them (10 000 queries x 2.5 million eligible rows x 256: 573 ms).  The byte form has one instruction for four
// dimensions: vabsdiff4 with accumulate, at half the FP32 rate (measured in registers: 226 dimensions per clock and SM
// against 54 for the fp32 form).  Rows and queries are rounded to bytes on one grid, x ~ lo[d] + step u with the same step in
// every dimension, so the byte sum S bounds the distance D from both sides:
//   |D - step S| <= E_q + E_x,   E = the measured L1 distance between a vector and its rounded form (E_x: largest over rows).
// Per chunk of rows a query lists the rows whose S can still mean D <= T (T: its exact k-th value so far), the listed rows are
// re-scored with the fp32 formula and the k best are kept: thresholds are exact, so rounding only lengthens lists, and a
// query whose list overflows is handed to the fp32 scan.
//
// Tile: 256 threads, 8 x 8 pairs each, BM queries x 16 384 / BM rows (a narrow query tile keeps the padding of a group of
// queries that share a filter small).  Operands lie in shared memory as they do in memory, 64 bytes of a row per stage,
// fetched by cp.async; a 16-byte shared load feeds 32 instructions.  Rows are padded to 80 bytes there and a thread's rows
// are RG apart, so that the eight lanes of a shared-memory phase fall into different banks.
#include <math_constants.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "tensor_scan.cuh"

namespace vsk {
namespace {

constexpr int L1_THREADS = 256;
constexpr int L1_CHUNK = 64;        // bytes of a row per stage
constexpr int L1_PITCH = L1_CHUNK + 16;
constexpr int L1_STAGES = 2;

struct L1Args {
  const uint8_t* q8;          // [nq][stride] by list position
  const uint8_t* x8;          // [n][stride]
  int32_t stride;             // bytes of a row, a multiple of 16
  int64_t nq;
  int64_t row_begin, row_end; // positions (of x_rows when given)
  const int32_t* x_rows;
  const uint64_t* row_masks;  // or null
  const uint64_t* q_masks;
  const int32_t* q_subset;
  const int32_t* bar;         // [nq] largest byte sum that is listed
  CandLists cand;
};

__device__ __forceinline__ void sad4(uint32_t& acc, uint32_t a, uint32_t b) {
  asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %0;" : "+r"(acc) : "r"(a), "r"(b));
}
__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(VSK_CHK(reinterpret_cast<const uint4*>(src))) : "memory");
}

template <int BM> struct L1Tile {
  static constexpr int QG = BM / 8;                 // query groups of 8
  static constexpr int RG = L1_THREADS / QG;        // row groups of 8
  static constexpr int BN = RG * 8;
  static constexpr int STAGE = (BM + BN) * L1_PITCH;
  static constexpr size_t SMEM = (size_t)L1_STAGES * STAGE + BN * sizeof(int32_t);
};

template <int BM>
__global__ void __launch_bounds__(L1_THREADS, 2) l1_scan_kernel(L1Args a) {
  using T = L1Tile<BM>;
  extern __shared__ __align__(16) uint8_t sm[];
  int32_t* s_row = reinterpret_cast<int32_t*>(sm + (size_t)L1_STAGES * T::STAGE);
  // query tile fastest: CTAs that run together share their rows in L2
  const int64_t qtiles = (a.nq + BM - 1) / BM;
  const int64_t m0 = ((int64_t)blockIdx.x % qtiles) * BM;
  const int64_t n0 = a.row_begin + ((int64_t)blockIdx.x / qtiles) * T::BN;
  // a position past the end reads the last row again; its sums are dropped
  for (int i = threadIdx.x; i < T::BN; i += L1_THREADS) {
    const int64_t n = min(n0 + i, a.row_end - 1);
    s_row[i] = a.x_rows ? __ldg(a.x_rows + n) : (int32_t)n;
  }
  __syncthreads();
  const int nsteps = a.stride >> 4, nchunks = (nsteps + 3) >> 2;
  // a thread copies the same 16-byte piece of every 64th row
  const int frow = threadIdx.x >> 2, part = threadIdx.x & 3;
  const uint8_t* fq[(BM + 63) / 64];
#pragma unroll
  for (int i = 0; i < (BM + 63) / 64; ++i) fq[i] = a.q8 + min(m0 + frow + 64 * i, a.nq - 1) * a.stride + part * 16;
  const uint8_t* fx = a.x8 + part * 16;
  auto fetch = [&](int c) {
    uint8_t* st = sm + (c % L1_STAGES) * T::STAGE + frow * L1_PITCH + part * 16;
    if (part < nsteps - 4 * c) {   // (the last chunk may hold fewer than four pieces)
#pragma unroll
      for (int i = 0; i < (BM + 63) / 64; ++i)
        if (BM >= 64 || frow < BM) cp16(st + i * 64 * L1_PITCH, fq[i] + c * L1_CHUNK);
#pragma unroll
      for (int i = 0; i < T::BN / 64; ++i)
        cp16(st + (BM + i * 64) * L1_PITCH, fx + (int64_t)s_row[frow + i * 64] * a.stride + c * L1_CHUNK);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int rg = threadIdx.x % T::RG, qg = threadIdx.x / T::RG;
  uint32_t acc[8][8];   // [query qg * 8 + j][row rg + RG * i]
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[j][i] = 0u;
  fetch(0);
  for (int c = 0; c < nchunks; ++c) {
    if (c + 1 < nchunks) {
      fetch(c + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const uint8_t* st = sm + (c % L1_STAGES) * T::STAGE;
    const uint8_t* sq = st + qg * 8 * L1_PITCH;
    const uint8_t* sx = st + (BM + rg) * L1_PITCH;
    const int parts = min(4, nsteps - 4 * c);
#pragma unroll 1
    for (int s = 0; s < parts; ++s) {
      uint4 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const uint4*>(sx + i * T::RG * L1_PITCH + s * 16);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint4 q = *reinterpret_cast<const uint4*>(sq + j * L1_PITCH + s * 16);
#pragma unroll
        for (int i = 0; i < 8; ++i) sad4(acc[j][i], q.x, x[i].x);
#pragma unroll
        for (int i = 0; i < 8; ++i) sad4(acc[j][i], q.y, x[i].y);
#pragma unroll
        for (int i = 0; i < 8; ++i) sad4(acc[j][i], q.z, x[i].z);
#pragma unroll
        for (int i = 0; i < 8; ++i) sad4(acc[j][i], q.w, x[i].w);
      }
    }
    __syncthreads();   // the stage may be filled again
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int64_t m = m0 + qg * 8 + j;
    if (m >= a.nq) continue;
    const int bar = __ldg(a.bar + m);
    uint32_t low = acc[j][0];
#pragma unroll
    for (int i = 1; i < 8; ++i) low = min(low, acc[j][i]);
    if ((int)low > bar) continue;
    const uint64_t qm = a.q_masks ? __ldg(a.q_masks + (a.q_subset ? (int64_t)__ldg(a.q_subset + m) : m)) : ~0ull;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int at = rg + T::RG * i;
      if ((int)acc[j][i] > bar || n0 + at >= a.row_end) continue;
      const int32_t row = s_row[at];
      if (a.row_masks && (__ldg(a.row_masks + row) & qm) == 0ull) continue;
      const int pos = atomicAdd(&a.cand.count[m], 1);
      if (pos < kCandCap) *VSK_CHK_W(a.cand.keys + m * kCandCap + pos) = make_key(0.f, (uint32_t)row);
    }
  }
}

// Exact values (sum |q - x| in fp32, in dimension order: the fp32 tile's value bit for bit) for the rows listed since the
// last compaction - the keys of value zero, as the scan leaves them; a kept row at distance zero is formed again.  A thread
// per row with four 16-byte loads in flight (VEC) or sixteen scalar ones; a small group of queries takes several CTAs per
// query (blockIdx.y), as the gathers are bound by their latency (156 queries: 64 us a launch with one).
constexpr int L1_RS_THREADS = 128;
template <bool VEC>
__global__ void __launch_bounds__(L1_RS_THREADS) l1_rescore_kernel(const float* __restrict__ q, const float* __restrict__ x, int dim,
                                                                   const int32_t* __restrict__ q_subset, CandLists cand,
                                                                   unsigned long long* total) {
  extern __shared__ __align__(16) float qs[];
  const int64_t pos = blockIdx.x, qi = q_subset ? (int64_t)__ldg(q_subset + pos) : pos;
  const int cnt = min(*VSK_CHK(cand.count + pos), kCandCap);
  uint64_t* keys = cand.keys + pos * kCandCap;
  for (int i = threadIdx.x; i < dim; i += L1_RS_THREADS) qs[i] = __ldg(q + qi * dim + i);
  __syncthreads();
  int formed = 0;
  for (int c = blockIdx.y * L1_RS_THREADS + threadIdx.x; c < cnt; c += gridDim.y * L1_RS_THREADS) {
    const uint64_t key = *VSK_CHK(keys + c);
    if ((uint32_t)(key >> 32) != 0x80000000u) continue;
    const float* p = x + (int64_t)(uint32_t)key * dim;
    float s = 0.f;
    int d = 0;
    for (; d + 16 <= dim; d += 16) {
      float v[16];
      if (VEC) {
#pragma unroll
        for (int u = 0; u < 4; ++u) *reinterpret_cast<float4*>(&v[4 * u]) = __ldg(reinterpret_cast<const float4*>(p + d) + u);
      } else {
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = __ldg(p + d + u);
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) s += fabsf(qs[d + u] - v[u]);
    }
    for (; d < dim; ++d) s += fabsf(qs[d] - __ldg(p + d));
    *VSK_CHK_W(keys + c) = make_key(s, (uint32_t)key);
    ++formed;
  }
  // rows formed by this CTA, one atomic per CTA (the query is done with, its first word takes the sum: with a static word beside
  // it the widest rows would no longer fit into 48 KB)
  int* sum = reinterpret_cast<int*>(qs);
  __syncthreads();
  if (threadIdx.x == 0) *sum = 0;
  __syncthreads();
  if (formed) atomicAdd(sum, formed);
  __syncthreads();
  if (threadIdx.x == 0 && *sum) atomicAdd(total, (unsigned long long)*sum);
}

// Largest byte sum at which a row can still be at or below the query's exact threshold; the fp32 sums compared are off by
// (dim + 8) 2^-23 of their size at most.  A query that is not finite lists nothing and is re-run by itself.
__global__ void l1_bar_kernel(const float* __restrict__ thr, const float* __restrict__ eq, int64_t nq, float ex, float step, int dim,
                              int32_t* __restrict__ bar, int32_t* __restrict__ flags) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  if (!(*VSK_CHK(eq + i) < CUDART_INF_F)) {
    atomicOr(&flags[i], kFlagDegenerate);
    *VSK_CHK_W(bar + i) = -1;
    return;
  }
  const double t = *VSK_CHK(thr + i);
  const double at = (t * (1.0 + 1.2e-7 * (dim + 8)) + (double)eq[i] + (double)ex) / (double)step + 1.0;
  *VSK_CHK_W(bar + i) = at < 2147483000.0 ? (int32_t)at : INT_MAX;   // (also for what is not a number: every row is listed)
}

// lowest and highest value of every dimension
__global__ void l1_range_kernel(const float* __restrict__ x, int64_t n, int dim, int64_t rows_per_block, unsigned* __restrict__ omin,
                                unsigned* __restrict__ omax) {
  const int64_t r0 = (int64_t)blockIdx.y * rows_per_block, r1 = min(n, r0 + rows_per_block);
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= dim) return;
  float mn = CUDART_INF_F, mx = -CUDART_INF_F;
#pragma unroll 8
  for (int64_t r = r0; r < r1; ++r) {
    const float v = __ldg(x + r * dim + d);
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
  atomicMin(omin + d, float_to_ordered(mn));
  atomicMax(omax + d, float_to_ordered(mx));
}

// One warp per row: bytes u = round((x - lo) / step) in [0, 255], zero behind dim, and the row's L1 distance to its rounded
// form (an upper bound; `mag` = largest magnitude of lo + step u, whose fp32 roundings it covers).  Rows of a subset are
// taken through `subset`; err_max (or null) takes the largest of all rows, err (or null) one per row.
__global__ void l1_bytes_kernel(const float* __restrict__ x, int64_t n, int dim, int stride, const int32_t* __restrict__ subset,
                                const float* __restrict__ lo, float step, float mag, uint8_t* __restrict__ out, float* __restrict__ err,
                                unsigned* err_max) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const float inv = 1.0f / step;
  float worst = 0.f;
  for (int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < n; row += warps) {
    const float* p = x + (subset ? (int64_t)__ldg(subset + row) : row) * dim;
    float e = 0.f, big = 0.f;
    for (int w = lane; w < stride >> 2; w += 32) {
      uint32_t word = 0;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int d = 4 * w + b;
        if (d < dim) {
          const float v = __ldg(p + d), l = __ldg(lo + d);
          const int u = max(0, min(255, __float2int_rn((v - l) * inv)));
          e += fabsf(v - fmaf(step, (float)u, l));
          big = fmaxf(big, fabsf(v));
          word |= (uint32_t)u << (8 * b);
        }
      }
      *VSK_CHK_W(reinterpret_cast<uint32_t*>(out + row * stride) + w) = word;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      e += __shfl_xor_sync(0xffffffffu, e, o);
      big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
    }
    e = e * (1.0f + 1e-5f) + 2.4e-7f * (float)dim * (big + mag);
    if (err && lane == 0) *VSK_CHK_W(err + row) = e;
    if (isnan(e) || e > worst) worst = e;   // what is not a number stays: nothing compares greater than it
  }
  if (err_max && lane == 0) atomicMax(err_max, __float_as_uint(fabsf(worst)));
}

// The byte copy of the index rows and the largest rounding of a row (once per index state).
int32_t l1_prepare(Index* ix) {
  Ctx* ctx = ix->ctx;
  if (ix->n_u8 == ix->n) return VSK_OK;
  ix->l1_ok = false;
  dev_free(ix->rows_u8);
  ix->rows_u8 = nullptr;
  const int dim = ix->dim;
  ix->stride_u8 = (int32_t)(ceil_div(dim, 16) * 16);
  if (!ix->l1_lo) VSK_TRY(dev_alloc(ctx, (void**)&ix->l1_lo, (size_t)dim * sizeof(float)));
  void* p;
  VSK_TRY(scratch(ctx, SLOT_TC_A, (size_t)dim * 8 + 16, &p));
  unsigned* omin = (unsigned*)p;
  unsigned* omax = omin + dim;
  unsigned* worst = omax + dim;
  VSK_CUDA(ctx, cudaMemsetAsync(omin, 0xff, (size_t)dim * 4, ctx->stream));
  VSK_CUDA(ctx, cudaMemsetAsync(omax, 0, (size_t)dim * 4 + 4, ctx->stream));
  const int64_t rpb = std::max<int64_t>(64, ceil_div(ix->n, 4096));
  l1_range_kernel<<<dim3((unsigned)ceil_div(dim, 128), (unsigned)ceil_div(ix->n, rpb)), 128, 0, ctx->stream>>>(ix->rows, ix->n, dim, rpb, omin, omax);
  ctx->stats.kernel_launches++;
  std::vector<unsigned> h((size_t)dim * 2);
  VSK_CUDA(ctx, cudaMemcpyAsync(h.data(), omin, (size_t)dim * 8, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  std::vector<float> lo((size_t)dim);
  float range = 0.f, mag = 0.f;
  bool finite = true;
  for (int d = 0; d < dim; ++d) {
    const float a = ordered_to_float(h[(size_t)d]), b = ordered_to_float(h[(size_t)dim + d]);
    finite = finite && std::isfinite(a) && std::isfinite(b) && b >= a;
    lo[(size_t)d] = a;
    range = std::max(range, b - a);
    mag = std::max(mag, std::max(std::fabs(a), std::fabs(b)));
  }
  ix->n_u8 = ix->n;   // looked at, usable or not
  if (!finite || !(mag < 1e30f)) return VSK_OK;
  const float step = range > 1e-30f ? range / 255.0f : 1.0f;
  if (dev_alloc(ctx, (void**)&ix->rows_u8, (size_t)ix->n * ix->stride_u8) != VSK_OK) return VSK_OK;   // no room: the fp32 scan
  VSK_CUDA(ctx, cudaMemcpyAsync(ix->l1_lo, lo.data(), (size_t)dim * 4, cudaMemcpyHostToDevice, ctx->stream));
  l1_bytes_kernel<<<(unsigned)std::min<int64_t>(ceil_div(ix->n, 8), 148 * 16), 256, 0, ctx->stream>>>(
      ix->rows, ix->n, dim, ix->stride_u8, nullptr, ix->l1_lo, step, mag, ix->rows_u8, nullptr, worst);
  ctx->stats.kernel_launches++;
  VSK_CUDA(ctx, cudaGetLastError());
  float ex = 0.f;
  VSK_CUDA(ctx, cudaMemcpyAsync(&ex, worst, 4, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ix->l1_step = step;
  ix->l1_mag = mag;
  ix->l1_ex = ex;
  ix->l1_ok = ex < 1e30f;
  return VSK_OK;
}

template <int BM>
int32_t l1_launch(Ctx* ctx, const L1Args& a) {
  using T = L1Tile<BM>;
  VSK_CUDA(ctx, cudaFuncSetAttribute(l1_scan_kernel<BM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM));
  const int64_t tiles = ceil_div(a.nq, BM) * ceil_div(a.row_end - a.row_begin, T::BN);
  if (tiles > 0x7fffffffLL) return fail(ctx, VSK_ERR_INVALID_BUFFER_SIZE, "too many tiles in one launch");
  prof_begin(ctx);
  l1_scan_kernel<BM><<<(unsigned)tiles, L1_THREADS, T::SMEM, ctx->stream>>>(a);
  prof_end(ctx);
  ctx->stats.kernel_launches++;
  VSK_CUDA(ctx, cudaGetLastError());
  tl_mark(ctx, "l1_scan");
  return VSK_OK;
}

}  // namespace

bool l1_applicable(const Index* ix, int64_t n, int64_t nq, int32_t k) {
  // (a byte sum stays below 2^31)
  return ix->kind == INDEX_FLAT_F32 && ix->metric == VSK_METRIC_MANHATTAN && ix->ctx->search_path == VSK_PATH_TENSOR_RERANK &&
         nq >= kL1MinQueries && n >= kL1MinRows && k <= kCandCap / 4 && ix->dim <= 12 * 1024 &&
         !(ix->n_u8 == ix->n && !ix->l1_ok);
}

// Whether the byte filter takes a batch (or filter group) of nq queries over n rows: with w = nq n dim steps of the fp32 tile,
//   the copy exists     w >= 1e9.  The filter's launches cost 110 us more than the tile's and save 0.064 ns per 1 000 steps:
//                       us, tile / filter: 65 536 rows x 128, 64 queries (0.5e9) 163 / 209, 128 (1.1e9) 241 / 234; 16 384 x
//                       256, 128 (0.5e9) 213 / 241, 512 (2.1e9) 350 / 285; 1 million x 256, 256 (6.6e10) 5 458 / 1 404.
//   no copy of the rows it has to be made, 0.7 ms plus 7 ps per element (1 million x 256: 2.5 ms, 262 144 x 256: 0.9): when the
//   as they are         batches since rows were last added, this one included, would have saved that, 1.1e10 steps and 110 per
//                       element.  Adding and searching in turn thus stays with the tile unless the batch is large (1 million x
//                       256, 64 queries: tile 1.35 ms, copy and filter 3 - 10 ms; 256: 5.5 and 3.9 ms).
//   never made, small   up to 16 million elements the first batch makes it, at 0.8 ms at most: rows that are loaded once are
//                       searched often.
constexpr int64_t kL1SmallElems = 16ll << 20;
static bool l1_pays(Index* ix, int64_t n, int64_t nq, L1Call* call) {
  const double per_query = (double)n * ix->dim, work = per_query * (double)nq;
  const double ahead = per_query * (double)std::max(nq, call->queries);   // groups to come have about as many rows
  call->queries -= nq;
  if (ix->l1_lo == nullptr && ix->n * ix->dim <= kL1SmallElems) return true;
  if (work < 1e9) return false;
  if (ix->n_u8 == ix->n || ix->l1_work + ahead >= 1.1e10 + 110.0 * (double)ix->n * ix->dim) return true;
  ix->l1_work += work;
  return false;
}

int32_t l1_topk(Index* ix, const ExactScanArgs& proto, int64_t n, int64_t nq, const int32_t* sub_dev, int32_t k, float* out_dist,
                int64_t* out_ids, L1Call* call, bool* handled) {
  L1Pending pending;
  VSK_TRY(l1_issue(ix, proto, n, nq, sub_dev, k, out_dist, out_ids, call, handled, &pending));
  return *handled ? l1_collect(ix, &pending, call) : VSK_OK;
}

int32_t l1_issue(Index* ix, const ExactScanArgs& proto, int64_t n, int64_t nq, const int32_t* sub_dev, int32_t k, float* out_dist,
                 int64_t* out_ids, L1Call* call, bool* handled, L1Pending* pending) {
  VSK_TRACE("vsk:l1_scan");
  Ctx* ctx = ix->ctx;
  *handled = false;
  if (!l1_pays(ix, n, nq, call)) return VSK_OK;
  if (!call->asked) {
    call->asked = true;
    call->allowed = !ix->l1_rest.resting();
  }
  if (!call->allowed) return VSK_OK;
  VSK_TRY(l1_prepare(ix));
  if (!ix->l1_ok) return VSK_OK;
  const int dim = ix->dim, stride = ix->stride_u8;
  void* p;
  VSK_TRY(scratch(ctx, SLOT_Q16, (size_t)nq * stride, &p));
  uint8_t* q8 = (uint8_t*)p;
  VSK_TRY(scratch(ctx, SLOT_QAUX, (size_t)nq * 8 + 16, &p));
  unsigned long long* total = (unsigned long long*)p;
  float* eq = (float*)((char*)p + 16);
  int32_t* bar = (int32_t*)(eq + nq);
  VSK_CUDA(ctx, cudaMemsetAsync(total, 0, 8, ctx->stream));
  l1_bytes_kernel<<<(unsigned)ceil_div(nq, 8), 256, 0, ctx->stream>>>(proto.q, nq, dim, stride, sub_dev, ix->l1_lo, ix->l1_step, ix->l1_mag,
                                                                      q8, eq, nullptr);
  ctx->stats.kernel_launches++;
  CandLists cand;
  VSK_TRY(cand_lists(ctx, nq, &cand));
  VSK_TRY(launch_init_cand(ctx, cand, nq));
  // the first rows by the fp32 scan: exact values, and a threshold to start from
  int64_t seen = std::min<int64_t>(n, schedule_dense_rows(ctx, k));
  ExactScanArgs ea = proto;
  ea.mode = SCAN_DENSE;
  ea.nq = nq;
  ea.q_subset = sub_dev;
  ea.cand = cand;
  ea.row_begin = 0;
  ea.row_end = seen;
  VSK_TRY(launch_exact_scan(ctx, ea));
  tl_mark(ctx, "l1_dense");
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
  L1Args a{};
  a.q8 = q8;
  a.x8 = ix->rows_u8;
  a.stride = stride;
  a.nq = nq;
  a.x_rows = proto.x_rows;
  a.row_masks = proto.row_masks;
  a.q_masks = proto.q_masks;
  a.q_subset = sub_dev;
  a.bar = bar;
  a.cand = cand;
  // the widest query tile that pads the batch by no more than a tenth over the narrowest
  const int64_t pad32 = ceil_div(nq, 32) * 32;
  const int bm = 10 * ceil_div(nq, 128) * 128 <= 11 * pad32 ? 128 : 10 * ceil_div(nq, 64) * 64 <= 11 * pad32 ? 64 : 32;
  const size_t qsm = (size_t)dim * sizeof(float);
  const bool vec = dim % 4 == 0 && (reinterpret_cast<uintptr_t>(ix->rows) & 15) == 0;
  while (seen < n) {
    // a quarter of the plain schedule's chunk (the rounding admits a few times the rows the exact threshold would), and at
    // most seven times what has been seen: a listed row costs a gather
    int64_t chunk = std::min(schedule_chunk(seen, k, 0) / 4, 7 * seen);
    chunk = std::min(std::max<int64_t>(chunk, 1024), n - seen);
    l1_bar_kernel<<<(unsigned)ceil_div(nq, 256), 256, 0, ctx->stream>>>(cand.thr, eq, nq, ix->l1_ex, ix->l1_step, dim, bar, cand.flags);
    ctx->stats.kernel_launches++;
    a.row_begin = seen;
    a.row_end = seen + chunk;
    if (bm == 128) VSK_TRY(l1_launch<128>(ctx, a));
    else if (bm == 64) VSK_TRY(l1_launch<64>(ctx, a));
    else VSK_TRY(l1_launch<32>(ctx, a));
    const dim3 rgrid((unsigned)nq, (unsigned)std::max<int64_t>(1, std::min<int64_t>(8, 8 * ctx->prop.multiProcessorCount / nq)));
    if (vec) l1_rescore_kernel<true><<<rgrid, L1_RS_THREADS, qsm, ctx->stream>>>(proto.q, ix->rows, dim, sub_dev, cand, total);
    else l1_rescore_kernel<false><<<rgrid, L1_RS_THREADS, qsm, ctx->stream>>>(proto.q, ix->rows, dim, sub_dev, cand, total);
    ctx->stats.kernel_launches++;
    VSK_CUDA(ctx, cudaGetLastError());
    tl_mark(ctx, "l1_rescore");
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
  fin.q_subset = sub_dev;
  fin.max_count = k;
  VSK_TRY(launch_select(ctx, fin));
  PinnedBuf& hb = ctx->host_flags[ctx->lane];
  VSK_TRY(pinned_reserve(ctx, &hb, (size_t)nq * 8 + 16));
  int32_t* hflags = (int32_t*)((char*)hb.p + 16);
  int32_t* hsub = hflags + nq;
  VSK_CUDA(ctx, cudaMemcpyAsync(hb.p, total, 8, cudaMemcpyDeviceToHost, ctx->stream));
  VSK_CUDA(ctx, cudaMemcpyAsync(hflags, cand.flags, (size_t)nq * 4, cudaMemcpyDeviceToHost, ctx->stream));
  if (sub_dev) VSK_CUDA(ctx, cudaMemcpyAsync(hsub, sub_dev, (size_t)nq * 4, cudaMemcpyDeviceToHost, ctx->stream));
  pending->active = true;
  pending->proto = proto;
  pending->n = n;
  pending->nq = nq;
  pending->sub_dev = sub_dev;
  pending->k = k;
  pending->out_dist = out_dist;
  pending->out_ids = out_ids;
  *handled = true;
  return VSK_OK;
}

// Waits for the lane's stream, and runs the queries whose list overflowed again on the fp32 scan.
int32_t l1_collect(Index* ix, L1Pending* pending, L1Call* call) {
  Ctx* ctx = ix->ctx;
  const L1Pending pd = *pending;
  pending->active = false;
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const PinnedBuf& hb = ctx->host_flags[ctx->lane];
  const int32_t* hflags = (const int32_t*)((const char*)hb.p + 16);
  const int32_t* hsub = hflags + pd.nq;
  unsigned long long hrr;
  memcpy(&hrr, hb.p, 8);
  ctx->stats.reranked_rows += (int64_t)hrr;
  std::vector<int32_t> bad;
  for (int64_t i = 0; i < pd.nq; ++i) {
    if (hflags[i]) bad.push_back(pd.sub_dev ? hsub[i] : (int32_t)i);
    call->bad += hflags[i] != 0 && !(hflags[i] & kFlagDegenerate);
  }
  call->seen += pd.nq;
  if (bad.empty()) return VSK_OK;
  void* p;
  VSK_TRY(scratch(ctx, SLOT_SUBSET, bad.size() * sizeof(int32_t), &p));
  VSK_CUDA(ctx, cudaMemcpyAsync(p, bad.data(), bad.size() * sizeof(int32_t), cudaMemcpyHostToDevice, ctx->stream));
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ctx->stats.fallback_queries += (int64_t)bad.size();
  return fp32_topk(ctx, pd.proto, pd.n, (int64_t)bad.size(), (const int32_t*)p, pd.k, ix->id_base, pd.out_dist, pd.out_ids, 0);
}

}  // namespace vsk
