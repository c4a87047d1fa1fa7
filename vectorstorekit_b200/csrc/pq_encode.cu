// Product-quantised encoding on the tensor cores: the code of a (row, segment) pair is the codeword of largest
// x.c - |c|^2 / 2, one contraction of the segment's rows with its 256 codewords.
//
//   operands   rows and codewords relative to the segment's mean codeword and scaled by a power of two, each fp32 value as
//              the sum of two fp16 ones (h + l; what is left is below 2^-22 of it).  One accumulator holds
//              xh.ch + xl.ch + xh.cl - |c|^2 / 2, the last as three fp16 pieces against ones: one K16 step of
//              tcgen05.mma for segments of 2 and 4 dimensions, two for 8, four for 16.
//   choice     the epilogue keeps the largest accumulator of every four codewords (two instructions per four values) and
//              then looks only at the fours that reach the largest of all less the bound of every rounding involved
//              (one four as a rule); their exact sums, formed as Codebook.encode forms them
//              (ProductQuantizerCodebook.swift:12-30), decide, so codes equal the exact encoder's bit for bit.
//
// 1 million x 128, 16 segments: 2.29 ms for the short-form kernel of pq.cu, 0.52 here (8 segments of 4: 0.82 -> 0.24, 32 of 2:
// 2.57 -> 0.86, 8 of 16: 1.86 -> 0.40).  What bounds it now: the epilogue's instructions - 62 % of the issue slots and of the
// pipe that does maxima, shifts and comparisons, 47 % of the shared-memory pipe (codewords of the fours, at addresses of the lanes'
// choosing), the tensor pipe is at 22 %.  Holding the 64 maxima of a row takes the registers: with 32 columns per load, with the
// columns in two halves, or with four groups of 96 registers some of them spilled, and next to 220 KB of shared memory there
// is no L1 left to spill to (0.61 - 0.87 ms).
//
// A CTA keeps the operand and the fp32 codewords of a group of segments (32 dimensions, 16 of segments of two) in shared
// memory and walks 128-row tiles: warp 0 fetches the fp32 rows by TMA, warps 2 and 3 turn them into operands, warp 1 issues
// the MMAs of one (tile, segment) after the other into two accumulators, and three groups of four warps take them in turn,
// a row per lane, so that one group's choice runs beside the next one's tensor-memory reads.  Planes of eight columns
// (16 bytes per row, no swizzle) make up the operands, so that the steps share them: the descriptor's leading offset is the
// distance between the two planes of a step.
#include <cuda.h>
#include <math_constants.h>

#include <algorithm>

#include "common.cuh"
#include "pq_encode.cuh"
#include "tc_ptx.cuh"
#include "tensor_scan.cuh"

namespace vsk {
namespace {

using namespace tc;

constexpr int PE_EPI0 = 4;           // first epilogue warp
constexpr int PE_GROUPS = 3;
constexpr int PE_THREADS = 32 * (PE_EPI0 + 4 * PE_GROUPS);   // TMA, MMA, two operand warps, three groups of four epilogue warps: 128 registers each
constexpr int PE_RAW = 3;            // fp32 tiles in flight
constexpr int PE_PLANE_A = TM * 16;  // 2 KB: 128 rows x 8 columns
constexpr int PE_PLANE_B = TN * 16;  // 4 KB: 256 codewords x 8 columns
constexpr float kPePad = 60000.f;    // |c|^2 / 2 of a column without a codeword, in operand units

// Planes, steps and sizes by segment length.  Columns of the contraction, x side | c side:
//   2: [h0 h1 l0 l1 h0 h1 1 1][1 0 ..] | [c0 c1 c0 c1 d0 d1 n0 n1][n2 0 ..]      (c, d: high and low part, n: -|c|^2 / 2)
//   4: [h l][h 1 1 1 0] | [c c][d n0 n1 n2 0]
//   8: [l][h][1 1 1 0 ..] | [c][n][c][d]: steps h.c + 1.n and l.c + h.d
//  16: [h h][l l][1 1 1 0 ..][0] | [c c][d d][n][0]: steps h.c, l.c, h.d, 1.n
// SEGS segments to a CTA, NA / NB planes per segment, a_plane / b_plane: first plane of a step.
template <int DS> struct PeShape;
template <> struct PeShape<2> {
  static constexpr int SEGS = 8, NA = 2, NB = 2, STEPS = 1;
  static __host__ __device__ constexpr int a_plane(int) { return 0; }
  static __host__ __device__ constexpr int b_plane(int) { return 0; }
};
template <> struct PeShape<4> {
  static constexpr int SEGS = 8, NA = 2, NB = 2, STEPS = 1;
  static __host__ __device__ constexpr int a_plane(int) { return 0; }
  static __host__ __device__ constexpr int b_plane(int) { return 0; }
};
template <> struct PeShape<8> {
  static constexpr int SEGS = 4, NA = 3, NB = 4, STEPS = 2;
  static __host__ __device__ constexpr int a_plane(int k) { return 1 - k; }
  static __host__ __device__ constexpr int b_plane(int k) { return 2 * k; }
};
template <> struct PeShape<16> {
  static constexpr int SEGS = 2, NA = 6, NB = 6, STEPS = 4;
  static __host__ __device__ constexpr int a_plane(int k) { return k == 1 ? 2 : k == 3 ? 4 : 0; }
  static __host__ __device__ constexpr int b_plane(int k) { return k < 2 ? 0 : 2 * k - 2; }
};

template <int DS>
struct PeSmem {
  using P = PeShape<DS>;
  static constexpr int FLOATS = P::SEGS * DS;               // of a row, per group of segments: 32 (16 for DS = 2)
  static constexpr int CB_FOUR = 4 * DS * 4 + 16;           // bytes of four codewords, padded: an odd number of 16-byte words,
                                                            // so that lanes that look at different fours spread over the banks
  uint8_t b[P::SEGS * P::NB * PE_PLANE_B];
  uint8_t raw[PE_RAW][TM * FLOATS * 4];                     // (each a multiple of 1 024 bytes: the swizzle's atom)
  uint8_t a[2][P::SEGS * P::NA * PE_PLANE_A];
  uint8_t cb[P::SEGS * 64 * CB_FOUR];
  __align__(16) float shift[P::SEGS * DS];                  // - mean of the codewords, in operand units
  float scale[P::SEGS], cmax[P::SEGS];                      // operand scale; largest |c - mean| in operand units
  uint64_t raw_full[PE_RAW], raw_empty[PE_RAW];
  uint64_t a_full[2], a_empty[2];
  uint64_t tmem_full[PE_GROUPS], tmem_empty[2];
  uint64_t drain;
  uint32_t tmem_base;
  volatile int abort_flag;
  int32_t err;
};

struct PeArgs {
  const float* x;
  int64_t n;
  int32_t dim, m, ksub;
  int32_t groups;          // of segments; CTA b takes group b % groups and the row tiles b / groups, + gridDim / groups, ...
  const float* cb;
  uint8_t* codes;
  uint64_t neg_zero;       // two fp32 -0 (f32x2_mul)
  int32_t* err;            // pinned host word, zero before the launch
  uint32_t wait_limit;
};

__device__ __forceinline__ uint32_t half_bits(float v) { return (uint32_t)__half_as_ushort(__float2half_rn(v)); }
__device__ __forceinline__ uint32_t pack2(uint32_t lo, uint32_t hi) { return lo | (hi << 16); }
__device__ __forceinline__ uint32_t half2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
// v = h + l as two halves each, two values at a time
__device__ __forceinline__ void split_half2(float v0, float v1, uint32_t& h, uint32_t& l) {
  const __half2 hh = __floats2half2_rn(v0, v1);
  const float2 back = __half22float2(hh);
  h = half2_bits(hh);
  l = half2_bits(__floats2half2_rn(v0 - back.x, v1 - back.y));
}
constexpr uint32_t kOne16 = 0x3c00u;

// Two fp32 operations per instruction, each rounded by itself.
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f32x2_split(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t f32x2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a b, as a fused operation with -0 (which changes nothing): a product and the sum that takes it are not contracted into one
// operation then, as the assembler does with the two-wide ones whatever their rounding modifiers (-0 comes from memory, so that it
// cannot see it is one)
__device__ __forceinline__ uint64_t f32x2_mul(uint64_t a, uint64_t b, uint64_t neg_zero) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(neg_zero));
  return r;
}

// float number of dimension i of codeword c in a segment's fp32 copy: minus the codewords, two side by side, so that one
// instruction works on both; four make a padded group
template <int DS>
__device__ __forceinline__ int cb_at(int c, int i) { return (c >> 2) * (4 * DS + 4) + ((c >> 1) & 1) * 2 * DS + 2 * i + (c & 1); }

// byte of 16-byte chunk `c` of row `r` of a staged fp32 tile (what TMA's 128-byte, or 64-byte, swizzle wrote)
template <int FLOATS>
__device__ __forceinline__ int raw_at(int r, int c) {
  return FLOATS == 32 ? r * 128 + ((c ^ (r & 7)) << 4) : r * 64 + ((c ^ ((r >> 1) & 3)) << 4);
}

// 16 consecutive columns of this thread's tensor-memory lane, without the wait
__device__ __forceinline__ void tc_ld16_issue(uint32_t taddr, float (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
        "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr)
      : "memory");
}

// the largest of four columns (a volatile operation, so that it stays before the loads that follow: hoisted above it,
// they cost the registers of another set of columns)
__device__ __forceinline__ float max_four(float a, float b, float c, float d) {
  float m;
  asm volatile("{\n\t.reg .f32 t;\n\tmax.f32 t, %1, %2, %3;\n\tmax.f32 %0, t, %4;\n\t}" : "=f"(m) : "f"(a), "f"(b), "f"(c), "f"(d));
  return m;
}

// segment s of staged row r
template <int DS>
__device__ __forceinline__ void pe_row(const uint8_t* raw, int r, int s, float (&x)[DS]) {
  constexpr int FLOATS = PeSmem<DS>::FLOATS;
  if constexpr (DS == 2) {
    *reinterpret_cast<float2*>(x) = *reinterpret_cast<const float2*>(raw + raw_at<FLOATS>(r, s >> 1) + (s & 1) * 8);
  } else {
#pragma unroll
    for (int j = 0; j < DS / 4; ++j) *reinterpret_cast<float4*>(&x[4 * j]) = *reinterpret_cast<const float4*>(raw + raw_at<FLOATS>(r, s * (DS / 4) + j));
  }
}

template <int DS>
__global__ void __launch_bounds__(PE_THREADS, 1) pq_encode_tensor_kernel(const __grid_constant__ CUtensorMap map_x, PeArgs a) {
  extern __shared__ uint8_t smem_raw[];
  using P = PeShape<DS>;
  using Smem = PeSmem<DS>;
  constexpr int FLOATS = Smem::FLOATS, CB_FOUR = Smem::CB_FOUR;
  Smem* sm = reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t wait_limit = a.wait_limit ? a.wait_limit : WAIT_LIMIT;
  const int group = (int)(blockIdx.x % a.groups);
  const int seg0 = group * P::SEGS, ns = min(P::SEGS, a.m - seg0);   // this CTA's segments
  const int n = (int)a.n, tiles = (int)((a.n + TM - 1) / TM);        // (n + TM is below 2^31)
  const int t0 = (int)(blockIdx.x / a.groups), t_step = (int)(gridDim.x / a.groups);
  const int count = t0 < tiles ? (tiles - t0 + t_step - 1) / t_step : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < PE_RAW; ++s) {
      mbar_init(&sm->raw_full[s], 1);
      mbar_init(&sm->raw_empty[s], 2 + 4 * ns);   // the operand warps, and every segment's epilogue warps
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm->a_full[b], 2);
      mbar_init(&sm->a_empty[b], 1);
      mbar_init(&sm->tmem_empty[b], 4);
    }
    for (int g = 0; g < PE_GROUPS; ++g) mbar_init(&sm->tmem_full[g], 1);
    mbar_init(&sm->drain, 1);
    sm->abort_flag = 0;
    sm->err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // ---- the group's codewords: fp32 copy; mean and scale; operand planes ----
  constexpr int CB_FLOATS = 64 * CB_FOUR / 4;
  float* cbs0 = reinterpret_cast<float*>(sm->cb);
  for (int e = threadIdx.x; e < ns * TN * DS; e += PE_THREADS) {
    const int s = e / (TN * DS), c = e / DS % TN, i = e % DS;
    cbs0[s * CB_FLOATS + cb_at<DS>(c, i)] =
        c < a.ksub ? -*VSK_CHK(a.cb + ((int64_t)(seg0 + s) * a.ksub + c) * DS + i) : -CUDART_INF_F;
  }
  __syncthreads();
  if (warp < ns) {   // a warp per segment
    const float* cbs = cbs0 + warp * CB_FLOATS;
    float t[DS];
#pragma unroll
    for (int i = 0; i < DS; ++i) t[i] = 0.f;
    for (int c = lane; c < a.ksub; c += 32)
#pragma unroll
      for (int i = 0; i < DS; ++i) t[i] -= cbs[cb_at<DS>(c, i)];
#pragma unroll
    for (int i = 0; i < DS; ++i) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t[i] += __shfl_xor_sync(0xffffffffu, t[i], o);
      t[i] /= (float)a.ksub;
    }
    float top = 0.f;
    for (int c = lane; c < a.ksub; c += 32)
#pragma unroll
      for (int i = 0; i < DS; ++i) top = fmaxf(top, fabsf(cbs[cb_at<DS>(c, i)] + t[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    float s = 1.f;
    if (top > 0.f && top < CUDART_INF_F) {
      int e;
      frexpf(top, &e);                                  // the largest entry becomes 8 .. 16, so that |c|^2 / 2 fits fp16
      s = ldexpf(1.f, min(120, 4 - e));                 // (e is at most 128: 2^-124 at least, a normal number)
    }
#pragma unroll
    for (int i = 0; i < DS; ++i)
      if (lane == i) sm->shift[warp * DS + i] = -t[i] * s;
    if (lane == 0) {
      sm->scale[warp] = s;
      sm->cmax[warp] = 0.f;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < ns * TN; e += PE_THREADS) {   // (whole warps on one segment)
    const int s = e / TN, c = e - s * TN;
    uint8_t* planes = sm->b + s * P::NB * PE_PLANE_B + c * 16;
    uint32_t h[DS / 2], l[DS / 2];   // pairs of halves
    const bool has = c < a.ksub;
    const float scale = sm->scale[s];
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < DS; i += 2) {
      float v[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        v[u] = has ? fmaf(-cbs0[s * CB_FLOATS + cb_at<DS>(c, i + u)], scale, sm->shift[s * DS + i + u]) : 0.f;
        q = fmaf(v[u], v[u], q);
      }
      split_half2(v[0], v[1], h[i / 2], l[i / 2]);
    }
    float most = q;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
    if (lane == 0) atomicMax(reinterpret_cast<int*>(&sm->cmax[s]), __float_as_int(sqrtf(most) * 1.00001f));   // (not negative)
    const float norm = has ? 0.5f * q : kPePad;
    const __half n0 = __float2half_rn(norm);
    const float r1 = norm - __half2float(n0);
    const __half n1 = __float2half_rn(r1);
    const uint32_t m01 = 0x80008000u ^ pack2((uint32_t)__half_as_ushort(n0), (uint32_t)__half_as_ushort(n1)),
                   m2 = 0x8000u ^ half_bits(r1 - __half2float(n1));
    uint4* pl[P::NB];
#pragma unroll
    for (int p = 0; p < P::NB; ++p) pl[p] = reinterpret_cast<uint4*>(planes + p * PE_PLANE_B);
    if constexpr (DS == 2) {
      *pl[0] = make_uint4(h[0], h[0], l[0], m01);
      *pl[1] = make_uint4(m2, 0u, 0u, 0u);
    } else if constexpr (DS == 4) {
      *pl[0] = make_uint4(h[0], h[1], h[0], h[1]);
      *pl[1] = make_uint4(l[0], l[1], m01, m2);
    } else if constexpr (DS == 8) {
      *pl[0] = make_uint4(h[0], h[1], h[2], h[3]);
      *pl[1] = make_uint4(m01, m2, 0u, 0u);
      *pl[2] = make_uint4(h[0], h[1], h[2], h[3]);
      *pl[3] = make_uint4(l[0], l[1], l[2], l[3]);
    } else {
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        *pl[p] = make_uint4(h[4 * p], h[4 * p + 1], h[4 * p + 2], h[4 * p + 3]);
        *pl[2 + p] = make_uint4(l[4 * p], l[4 * p + 1], l[4 * p + 2], l[4 * p + 3]);
      }
      *pl[4] = make_uint4(m01, m2, 0u, 0u);
      *pl[5] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  // the constant columns of the row operand: written once, the operand warps leave them alone
  for (int e = threadIdx.x; e < 2 * ns * TM; e += PE_THREADS) {
    const int b = e / (ns * TM), s = (e / TM) % ns, r = e % TM;
    uint8_t* planes = sm->a[b] + s * P::NA * PE_PLANE_A + r * 16;
    const uint32_t one2 = pack2(kOne16, kOne16);
    if constexpr (DS == 2) {
      *reinterpret_cast<uint4*>(planes + PE_PLANE_A) = make_uint4(kOne16, 0u, 0u, 0u);
    } else if constexpr (DS == 4) {
      *reinterpret_cast<uint2*>(planes + PE_PLANE_A + 8) = make_uint2(one2, kOne16);
    } else if constexpr (DS == 8) {
      *reinterpret_cast<uint4*>(planes + 2 * PE_PLANE_A) = make_uint4(one2, kOne16, 0u, 0u);
    } else {
      *reinterpret_cast<uint4*>(planes + 4 * PE_PLANE_A) = make_uint4(one2, kOne16, 0u, 0u);
      *reinterpret_cast<uint4*>(planes + 5 * PE_PLANE_A) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sm->tmem_base;

  if (warp == 0) {
    // ---------------- TMA producer: the fp32 rows ----------------
    if (lane == 0) {
      uint32_t issued = 0, issued_ph = 0;
      int st = 0;
      uint32_t ph = 0;
      for (int i = 0; i < count; ++i) {
        if (!mbar_wait(&sm->raw_empty[st], ph ^ 1u, &sm->abort_flag, &sm->err, 1, wait_limit)) break;
        mbar_expect_tx(&sm->raw_full[st], (uint32_t)sizeof(sm->raw[0]));
        tma_load_2d(sm->raw[st], &map_x, &sm->raw_full[st], seg0 * DS, (t0 + i * t_step) * TM);
        issued |= 1u << st;
        issued_ph = (issued_ph & ~(1u << st)) | (ph << st);
        if (++st == PE_RAW) { st = 0; ph ^= 1u; }
      }
      // copies still in flight must land before the CTA's shared memory is released
      for (int s = 0; s < PE_RAW; ++s)
        if (issued & (1u << s))
          for (uint32_t it = 0; it < wait_limit; ++it) {
            if (mbar_try_wait(&sm->raw_full[s], (issued_ph >> s) & 1u)) break;
            __nanosleep(64);
          }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      // K-major planes without a swizzle: 8-row groups 128 bytes apart, the second eight columns one plane further on
      constexpr uint32_t hi = (uint32_t)(128 >> 4) | (1u << 14);
      constexpr uint32_t lead_a = (uint32_t)(PE_PLANE_A >> 4) << 16, lead_b = (uint32_t)(PE_PLANE_B >> 4) << 16;
      const uint32_t b0 = (smem_u32(sm->b) >> 4) | lead_b;
      uint32_t buf = 0, ph = 0, acc = 0, aph = 0, g = 0;
      bool ok = true;
      for (int i = 0; ok && i < count; ++i) {
        if (!mbar_wait(&sm->a_full[buf], ph, &sm->abort_flag, &sm->err, 3, wait_limit)) break;
        tc_fence_after();
        const uint32_t a0 = (smem_u32(sm->a[buf]) >> 4) | lead_a;
        for (int s = 0; s < ns; ++s) {
          if (!mbar_wait(&sm->tmem_empty[acc], aph ^ 1u, &sm->abort_flag, &sm->err, 2, wait_limit)) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < P::STEPS; ++k)
            tc_mma(tmem_base + acc * (uint32_t)TN, desc_pack(a0 + (uint32_t)((s * P::NA + P::a_plane(k)) * (PE_PLANE_A >> 4)), hi),
                   desc_pack(b0 + (uint32_t)((s * P::NB + P::b_plane(k)) * (PE_PLANE_B >> 4)), hi), kIdesc, k ? 1u : 0u);
          tc_commit(&sm->tmem_full[g]);
          g = g + 1 == PE_GROUPS ? 0u : g + 1;
          aph = acc ? aph ^ 1u : aph;
          acc ^= 1u;
        }
        if (ok) tc_commit(&sm->a_empty[buf]);
        ph = buf ? ph ^ 1u : ph;
        buf ^= 1u;
      }
      // all issued MMAs must retire before tensor memory is freed
      tc_commit(&sm->drain);
      for (uint32_t it = 0; it < wait_limit; ++it) {
        if (mbar_try_wait(&sm->drain, 0)) break;
        __nanosleep(64);
      }
    }
  } else if (warp < PE_EPI0) {
    // ---------------- operand warps: 64 rows each, 16 rows x two 16-byte chunks per step ----------------
    // (rows 0 2 4 6 | 1 3 5 7 | ... per eight lanes: with the swizzle neither the loads nor the stores meet in a bank)
    const int row16 = ((lane >> 4) << 3) | (((lane >> 1) & 3) << 1) | ((lane >> 3) & 1);
    int st = 0;
    uint32_t rph = 0, buf = 0, ph = 0;
    // a lane's columns are the same in every row: their shifts and scales stay in registers
    float4 shift[FLOATS / 8];
    float2 scale[FLOATS / 8];
#pragma unroll
    for (int j = 0; j < FLOATS / 8; ++j) {
      const int f = (2 * j + (lane & 1)) * 4, s = min(f / DS, ns - 1), s2 = DS == 2 ? min(f / DS + 1, ns - 1) : s;
      shift[j] = make_float4(sm->shift[s * DS + f % DS], sm->shift[s * DS + f % DS + 1], sm->shift[s2 * DS + (f + 2) % DS],
                             sm->shift[s2 * DS + (f + 2) % DS + 1]);
      scale[j] = make_float2(sm->scale[s], sm->scale[s2]);
    }
    for (int i = 0; i < count; ++i) {
      bool got = mbar_wait(&sm->raw_full[st], rph, &sm->abort_flag, &sm->err, 5, wait_limit) &&
                 mbar_wait(&sm->a_empty[buf], ph ^ 1u, &sm->abort_flag, &sm->err, 6, wait_limit);
      if (!__all_sync(0xffffffffu, got)) break;
      const uint8_t* raw = sm->raw[st];
      uint8_t* out = sm->a[buf];
#pragma unroll 1
      for (int rg = 0; rg < 4; ++rg) {
        const int r = (warp - 2) * 64 + rg * 16 + row16;
        float4 v[FLOATS / 8];
#pragma unroll
        for (int j = 0; j < FLOATS / 8; ++j) v[j] = *reinterpret_cast<const float4*>(raw + raw_at<FLOATS>(r, 2 * j + (lane & 1)));
#pragma unroll
        for (int j = 0; j < FLOATS / 8; ++j) {
          const int f = (2 * j + (lane & 1)) * 4;   // first of four floats
          const int s = f / DS, d = f % DS;
          uint8_t* planes = out + s * P::NA * PE_PLANE_A + r * 16;   // (a segment past the last one: planes nobody multiplies)
          uint32_t h01, l01, h23, l23;
          split_half2(fmaf(v[j].x, scale[j].x, shift[j].x), fmaf(v[j].y, scale[j].x, shift[j].y), h01, l01);
          split_half2(fmaf(v[j].z, scale[j].y, shift[j].z), fmaf(v[j].w, scale[j].y, shift[j].w), h23, l23);
          if constexpr (DS == 2) {
            const uint32_t one2 = pack2(kOne16, kOne16);
            *reinterpret_cast<uint4*>(planes) = make_uint4(h01, l01, h01, one2);
            *reinterpret_cast<uint4*>(planes + P::NA * PE_PLANE_A) = make_uint4(h23, l23, h23, one2);
          } else if constexpr (DS == 4) {
            *reinterpret_cast<uint4*>(planes) = make_uint4(h01, h23, l01, l23);
            *reinterpret_cast<uint2*>(planes + PE_PLANE_A) = make_uint2(h01, h23);
          } else if constexpr (DS == 8) {
            *reinterpret_cast<uint2*>(planes + (d >> 2) * 8) = make_uint2(l01, l23);
            *reinterpret_cast<uint2*>(planes + PE_PLANE_A + (d >> 2) * 8) = make_uint2(h01, h23);
          } else {
            uint8_t* p = planes + (d >> 3) * PE_PLANE_A + ((d >> 2) & 1) * 8;
            *reinterpret_cast<uint2*>(p) = make_uint2(h01, h23);
            *reinterpret_cast<uint2*>(p + 2 * PE_PLANE_A) = make_uint2(l01, l23);
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&sm->raw_empty[st]);
        mbar_arrive(&sm->a_full[buf]);
      }
      if (++st == PE_RAW) { st = 0; rph ^= 1u; }
      ph = buf ? ph ^ 1u : ph;
      buf ^= 1u;
    }
  } else {
    // ---------------- epilogue: group g takes (tile, segment) pairs g, g + 3, ...; a row per lane ----------------
    const int g = (warp - PE_EPI0) >> 2, quarter = warp & 3;
    const int et = quarter * 32 + lane;
    uint32_t ph = 0, acc = (uint32_t)g & 1u;
    // In units of (|x| + |c|)^2: 2^-22 per column and product of the contraction, the fp16 pairs, the norm, and the exact
    // sums' own rounding.
    constexpr float kBand = (16.f * P::STEPS + 4.f) * 2.3841858e-7f * 1.02f + (float)(DS + 2) * 5.9604645e-8f * 1.05f;
    // tile, segment and raw stage of this group's next pair, carried along
    int tile = 0, s = g, st = 0;
    uint32_t rph = 0;
    auto settle = [&]() {
      while (s >= ns) {
        s -= ns;
        ++tile;
        if (++st == PE_RAW) { st = 0; rph ^= 1u; }
      }
    };
    settle();
#pragma unroll 1
    for (; tile < count; s += PE_GROUPS, settle(), ph ^= 1u, acc ^= (uint32_t)PE_GROUPS & 1u) {
      if (!__all_sync(0xffffffffu, mbar_wait(&sm->tmem_full[g], ph, &sm->abort_flag, &sm->err, 4, wait_limit))) break;
      tc_fence_after();
      const uint32_t trow = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * (uint32_t)TN;
      float top4[64], v0[16], v1[16];
      tc_ld16_issue(trow, v0);
#pragma unroll
      for (int c = 0; c < 16; c += 2) {   // the next sixteen columns are on their way while these are looked at
        tc_ld_wait();
        tc_ld16_issue(trow + (uint32_t)(c * 16 + 16), v1);
#pragma unroll
        for (int j = 0; j < 4; ++j) top4[4 * c + j] = max_four(v0[4 * j], v0[4 * j + 1], v0[4 * j + 2], v0[4 * j + 3]);
        tc_ld_wait();
        if (c < 14) tc_ld16_issue(trow + (uint32_t)(c * 16 + 32), v0);
#pragma unroll
        for (int j = 0; j < 4; ++j) top4[4 * c + 4 + j] = max_four(v1[4 * j], v1[4 * j + 1], v1[4 * j + 2], v1[4 * j + 3]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm->tmem_empty[acc]);
      // how far below the best a codeword may lie (the row is staged long since: its operand has been multiplied)
      if (!__all_sync(0xffffffffu, mbar_wait(&sm->raw_full[st], rph, &sm->abort_flag, &sm->err, 7, wait_limit))) break;
      __align__(16) float x[DS], shift[DS];
      pe_row<DS>(sm->raw[st], et, s, x);
      if constexpr (DS == 2) {
        *reinterpret_cast<float2*>(shift) = *reinterpret_cast<const float2*>(sm->shift + s * 2);
      } else {
#pragma unroll
        for (int j = 0; j < DS; j += 4) *reinterpret_cast<float4*>(&shift[j]) = *reinterpret_cast<const float4*>(sm->shift + s * DS + j);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm->raw_empty[st]);
      float x2 = 0.f;
      const float scale = sm->scale[s];
#pragma unroll
      for (int d = 0; d < DS; ++d) {
        const float v = fmaf(x[d], scale, shift[d]);
        x2 = fmaf(v, v, x2);
      }
      const int row = (t0 + tile * t_step) * TM + et;
      const float r = sqrtf(x2) * 1.00001f + sm->cmax[s];
      const float band = r * r * kBand + r * 2.4e-7f + scale * scale * 1e-37f;
      float b4[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b4[j] = fmaxf(top4[j], top4[j + 4]);
#pragma unroll
        for (int i = 8; i < 64; i += 8) b4[j] = max3(b4[j], top4[j + i], top4[j + i + 4]);
      }
      const float bar = fmaxf(max3(b4[0], b4[1], b4[2]), b4[3]) - band;
      // bit j: no codeword of four j reaches the bar (the sign of the difference)
      uint32_t below0 = 0u, below1 = 0u;
#pragma unroll
      for (int j = 31; j >= 0; --j) {
        below0 = __funnelshift_l(__float_as_uint(top4[j] - bar), below0, 1);
        below1 = __funnelshift_l(__float_as_uint(top4[32 + j] - bar), below1, 1);
      }
      // a row that fp16 cannot hold (and what is not a number) takes the exact sums over all codewords
      const bool plain = r < 60000.f && band < CUDART_INF_F;
      uint32_t hit0 = plain ? ~below0 : 0u, hit1 = plain ? ~below1 : 0u;
      float low = CUDART_INF_F;
      int code = 0;
      uint64_t xx[DS];
#pragma unroll
      for (int j = 0; j < DS; ++j) xx[j] = f32x2(x[j], x[j]);
      const uint8_t* cbs = sm->cb + s * 64 * CB_FOUR;
      while (__any_sync(0xffffffffu, (hit0 | hit1) != 0u)) {
        if ((hit0 | hit1) != 0u) {
          const int f = hit0 ? __ffs((int)hit0) - 1 : __ffs((int)hit1) + 31;
          hit1 = hit0 ? hit1 : hit1 & (hit1 - 1u);
          hit0 &= hit0 - 1u;   // (zero stays zero)
          const uint8_t* four = cbs + f * CB_FOUR;
#pragma unroll
          for (int p = 0; p < 2; ++p) {   // codewords 4 f + 2 p and the next
            uint64_t d2 = 0ull;
#pragma unroll
            for (int j = 0; j < DS; j += 2) {
              const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(four + p * DS * 8 + j * 8);
              uint64_t e = f32x2_add(xx[j], w.x);
              d2 = f32x2_add(d2, f32x2_mul(e, e, a.neg_zero));
              e = f32x2_add(xx[j + 1], w.y);
              d2 = f32x2_add(d2, f32x2_mul(e, e, a.neg_zero));
            }
            float d0, d1;
            f32x2_split(d2, d0, d1);
            if (d0 < low) { low = d0; code = 4 * f + 2 * p; }
            if (d1 < low) { low = d1; code = 4 * f + 2 * p + 1; }
          }
        }
      }
      for (unsigned todo = __ballot_sync(0xffffffffu, !plain && row < n); todo; todo &= todo - 1u) {
        const int src = __ffs((int)todo) - 1;
        const int c = pq_exact_code_warp<DS>(a.x + (int64_t)(row - lane + src) * a.dim + (int64_t)(seg0 + s) * DS,
                                             a.cb + (int64_t)(seg0 + s) * a.ksub * DS, a.ksub, lane, false);
        if (lane == src) code = c;
      }
      if (row < n) *VSK_CHK_W(a.codes + (int64_t)row * a.m + seg0 + s) = (uint8_t)code;
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && sm->err != 0) *VSK_CHK_W(a.err) = sm->err;
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

template <int DS>
int32_t launch(Ctx* ctx, PeArgs a) {
  using P = PeShape<DS>;
  CUtensorMap map;
  VSK_TRY(make_map_rows_f32(ctx, a.x, a.n, a.dim, PeSmem<DS>::FLOATS, TM, &map));
  a.groups = (int32_t)ceil_div(a.m, P::SEGS);
  const int64_t tiles = ceil_div(a.n, TM);
  const int64_t per = std::max<int64_t>(1, std::min<int64_t>(tiles, ctx->prop.multiProcessorCount / a.groups));
  constexpr size_t smem = sizeof(PeSmem<DS>) + 1024;
  static_assert(smem <= 227 * 1024, "shared memory of a CTA");
  VSK_CUDA(ctx, opt_in_shared(ctx, pq_encode_tensor_kernel<DS>, smem));
  pq_encode_tensor_kernel<DS><<<(unsigned)(a.groups * per), PE_THREADS, smem, ctx->stream>>>(map, a);
  ctx->stats.kernel_launches++;
  VSK_CUDA(ctx, cudaGetLastError());
  return VSK_OK;
}

}  // namespace

bool pq_encode_tensor_applies(const float* x, int64_t n, int32_t dim, int32_t m, int32_t ksub) {
  const int ds = dim / m;
  // At 65 536 pairs (131 072 for two dimensions) the set-up of the codewords is earned back: 16 segments of 8, calls timed from
  // Python, this / the other: 4 096 rows 53 / 54 us, 10 000 58 / 78, 65 536 86 / 199; 8 of 2: 10 000 rows 52 / 51, 65 536 65 / 83.
  return (ds == 2 || ds == 4 || ds == 8 || ds == 16) && ksub > 128 && n * m >= (ds == 2 ? 131072 : 65536) && n <= 0x7fffff00LL &&
         dim % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
}

int32_t pq_encode_tensor(Ctx* ctx, const float* cb, int32_t dim, int32_t m, int32_t ksub, const float* x, int64_t n, uint8_t* codes) {
  // a wait that runs out is said in a pinned word the kernel can address: no copy before or after the launch
  PinnedBuf& hb = ctx->host_flags[ctx->lane];
  VSK_TRY(pinned_reserve(ctx, &hb, 16));
  volatile int32_t* herr = (volatile int32_t*)hb.p;
  *herr = 0;
  PeArgs a{};
  a.x = x;
  a.n = n;
  a.dim = dim;
  a.m = m;
  a.ksub = ksub;
  a.cb = cb;
  a.codes = codes;
  a.neg_zero = 0x8000000080000000ull;
  a.err = (int32_t*)hb.p;
  a.wait_limit = ctx->tuning.wait_limit_log2 > 0 ? (1u << std::min(ctx->tuning.wait_limit_log2, 30)) : 0u;
  switch (dim / m) {
    case 2: VSK_TRY(launch<2>(ctx, a)); break;
    case 4: VSK_TRY(launch<4>(ctx, a)); break;
    case 8: VSK_TRY(launch<8>(ctx, a)); break;
    default: VSK_TRY(launch<16>(ctx, a)); break;
  }
  VSK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (*herr != 0) return fail(ctx, VSK_ERR_TIMEOUT, "product-quantised encoding: a bounded pipeline wait ran out (role %d)", (int)*herr);
  return VSK_OK;
}

}  // namespace vsk
