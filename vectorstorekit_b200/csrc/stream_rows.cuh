// The inner loop of the scans for a few queries: queries staged in shared memory, a warp streams ROWS rows at a time and
// forms the reference's direct formulas (tile::accum) for every (row, query) pair.
#pragma once
#include "common.cuh"
#include "tile_core.cuh"

namespace vsk {

// v[0..V) per lane -> the total over the warp of v[j] on the lanes with (lane >> (5 - log2 V)) == j, in v[0].
// Each stage halves the values a lane still carries: a lane keeps the half its lane bit selects and hands the
// other half to its partner, so V values cost V - 1 + (5 - log2 V) shuffles instead of 5 V.
template <int V>
__device__ __forceinline__ void warp_reduce_scatter(float (&v)[V], int lane) {
  int off = 16;
#pragma unroll
  for (int c = V; c > 1; c >>= 1) {
    const int h = c >> 1;
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int j = 0; j < h; ++j) {
      const float keep = upper ? v[j + h] : v[j];
      const float send = upper ? v[j] : v[j + h];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
    off >>= 1;
  }
  for (; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
}

template <int V> struct Log2 { static constexpr int value = 1 + Log2<V / 2>::value; };
template <> struct Log2<1> { static constexpr int value = 0; };

// acc[r * NQ + i] += this lane's share of the pair (row rid[r], query i).  VEC: dim is a multiple of 4 and the rows start on
// 16-byte boundaries.  A row that is not live is not read.
template <int METRIC, int NQ, bool VEC, int ROWS>
__device__ __forceinline__ void stream_accumulate(float (&acc)[ROWS * NQ], const float* __restrict__ x, int dim, const float* sq,
                                                  const uint32_t (&rid)[ROWS], const bool (&live)[ROWS], int lane) {
  if (VEC) {
    const int nv = dim >> 2;
    const float4* p[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) p[r] = reinterpret_cast<const float4*>(x + (int64_t)rid[r] * dim);
    const float4* sq4 = reinterpret_cast<const float4*>(sq);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c = lane; c < nv; c += 64) {
      // four 16-byte loads in flight per lane before the first is used
      const int c2 = c + 32;
      const bool two = c2 < nv;
      float4 xv[ROWS][2];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        xv[r][0] = live[r] ? __ldg(p[r] + c) : zero;
        xv[r][1] = (live[r] && two) ? __ldg(p[r] + c2) : zero;
      }
#pragma unroll
      for (int i = 0; i < NQ; ++i) {
        const float4 q = sq4[i * nv + c];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          tile::accum<METRIC>(acc[r * NQ + i], q.x, xv[r][0].x);
          tile::accum<METRIC>(acc[r * NQ + i], q.y, xv[r][0].y);
          tile::accum<METRIC>(acc[r * NQ + i], q.z, xv[r][0].z);
          tile::accum<METRIC>(acc[r * NQ + i], q.w, xv[r][0].w);
        }
      }
      if (two) {
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
          const float4 q = sq4[i * nv + c2];
#pragma unroll
          for (int r = 0; r < ROWS; ++r) {
            tile::accum<METRIC>(acc[r * NQ + i], q.x, xv[r][1].x);
            tile::accum<METRIC>(acc[r * NQ + i], q.y, xv[r][1].y);
            tile::accum<METRIC>(acc[r * NQ + i], q.z, xv[r][1].z);
            tile::accum<METRIC>(acc[r * NQ + i], q.w, xv[r][1].w);
          }
        }
      }
    }
  } else {
    // four scalar loads per row in flight
    for (int k = lane; k < dim; k += 128) {
      float xv[ROWS][4];
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int u = 0; u < 4; ++u) xv[r][u] = (live[r] && k + 32 * u < dim) ? __ldg(x + (int64_t)rid[r] * dim + k + 32 * u) : 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (k + 32 * u >= dim) break;
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
          const float q = sq[i * dim + k + 32 * u];
#pragma unroll
          for (int r = 0; r < ROWS; ++r) tile::accum<METRIC>(acc[r * NQ + i], q, xv[r][u]);
        }
      }
    }
  }
}

}  // namespace vsk
