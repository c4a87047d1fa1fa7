// Exact sums of the product-quantised encoders, and the encoder on the tensor cores (pq_encode.cu).
#pragma once
#include <math_constants.h>

#include "common.cuh"

namespace vsk {

// one term of a squared distance, every operation rounded by itself (the order and the roundings of Codebook.encode)
__device__ __forceinline__ float pq_sqdiff_accum(float acc, float a, float b) {
  const float diff = __fsub_rn(a, b);
  return __fadd_rn(acc, __fmul_rn(diff, diff));
}

// The code of one (row, segment) by the exact sums, over codewords first, first + step, ...: smallest value, lowest code.
template <int DS>
__device__ __forceinline__ void pq_exact_code(const float* __restrict__ seg, const float* __restrict__ cb, int ksub, int first, int step,
                                              bool wide, float& low, int& code) {
  __align__(16) float x[DS];
#pragma unroll
  for (int i = 0; i < DS; ++i) x[i] = __ldg(seg + i);
  low = CUDART_INF_F;
  code = 0;
#pragma unroll 1
  for (int c = first; c < ksub; c += step) {
    __align__(16) float w[DS];
    if (wide) {
#pragma unroll
      for (int i = 0; i + 4 <= DS; i += 4) *reinterpret_cast<float4*>(&w[i]) = __ldg(reinterpret_cast<const float4*>(cb + c * DS + i));
    } else {
#pragma unroll
      for (int i = 0; i < DS; ++i) w[i] = __ldg(cb + c * DS + i);
    }
    float d = 0.f;
#pragma unroll
    for (int i = 0; i < DS; ++i) d = pq_sqdiff_accum(d, x[i], w[i]);
    if (d < low) { low = d; code = c; }
  }
}

// ... by a whole warp, a codeword per lane; every lane gets the code
template <int DS>
__device__ __forceinline__ int pq_exact_code_warp(const float* __restrict__ seg, const float* __restrict__ cb, int ksub, int lane, bool wide) {
  float low;
  int code;
  pq_exact_code<DS>(seg, cb, ksub, lane, 32, wide, low, code);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float l2 = __shfl_xor_sync(0xffffffffu, low, o);
    const int c2 = __shfl_xor_sync(0xffffffffu, code, o);
    if (l2 < low || (l2 == low && c2 < code)) { low = l2; code = c2; }
  }
  return code;
}

// Whether the encoder on the tensor cores takes the call, and is the faster one.
bool pq_encode_tensor_applies(const float* x, int64_t n, int32_t dim, int32_t m, int32_t ksub);
// x: [n][dim], codes: [n][m], device pointers; drains the stream.
int32_t pq_encode_tensor(Ctx* ctx, const float* cb, int32_t dim, int32_t m, int32_t ksub, const float* x, int64_t n, uint8_t* codes);

}  // namespace vsk
