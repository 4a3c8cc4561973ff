// Three bf16 planes whose exact sum is an fp32 value (see linear_f32.cu).
#pragma once

#include "dfl_common.cuh"

namespace dfl {

constexpr int kPlanes = 3;

// An infinity is 1 (of its sign), 0 and itself.  A product takes plane 2 of one operand with plane 0 of the other only, so
// that an infinity meets each element it is multiplied with exactly once, by its sign and size; in plane 0 it would also meet
// the other operand's planes 1 and 2, which are zeros or of the other sign, and give NaN.
__device__ __forceinline__ void split3(float x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c) {
  const bool infinite = isinf(x);
  a = __float2bfloat16_rn(infinite ? copysignf(1.0f, x) : x);
  if (isinf(__bfloat162float(a))) a = __ushort_as_bfloat16((unsigned short)(__float_as_uint(x) >> 16));   // rounded up: truncate
  const float r1 = infinite ? 0.0f : x - __bfloat162float(a);   // exact
  b = __float2bfloat16_rn(r1);
  c = __float2bfloat16_rn(infinite ? x : r1 - __bfloat162float(b));
}

// Four elements of one row as packed plane words.  The looks at infinities, and at what rounding would make one, are left out where
// the sum of the magnitudes says that there are none (a NaN fails the comparison).
__device__ __forceinline__ void split3x4(const float (&f)[4], uint2 (&out)[kPlanes]) {
  if ((fabsf(f[0]) + fabsf(f[1])) + (fabsf(f[2]) + fabsf(f[3])) < 3.0e38f) {
    uint32_t w[kPlanes][2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float a = f[2 * j], b = f[2 * j + 1];
      const __nv_bfloat162 h0 = __floats2bfloat162_rn(a, b);
      const float2 f0 = __bfloat1622float2(h0);
      const float ra = a - f0.x, rb = b - f0.y;
      const __nv_bfloat162 h1 = __floats2bfloat162_rn(ra, rb);
      const float2 f1 = __bfloat1622float2(h1);
      const __nv_bfloat162 h2 = __floats2bfloat162_rn(ra - f1.x, rb - f1.y);
      w[0][j] = *reinterpret_cast<const uint32_t*>(&h0);
      w[1][j] = *reinterpret_cast<const uint32_t*>(&h1);
      w[2][j] = *reinterpret_cast<const uint32_t*>(&h2);
    }
#pragma unroll
    for (int q = 0; q < kPlanes; ++q) out[q] = make_uint2(w[q][0], w[q][1]);
    return;
  }
  __nv_bfloat16 p[kPlanes][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) split3(f[j], p[0][j], p[1][j], p[2][j]);
#pragma unroll
  for (int q = 0; q < kPlanes; ++q) {
    const __nv_bfloat162 lo = __halves2bfloat162(p[q][0], p[q][1]), hi = __halves2bfloat162(p[q][2], p[q][3]);
    out[q] = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  }
}

// Eight probabilities into four packed words of each plane.
__device__ __forceinline__ void split_eight(const float* p, uint32_t (&w)[kPlanes][4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float a = p[2 * j], b = p[2 * j + 1];   // probabilities: finite, no special cases
    const __nv_bfloat162 h0 = __floats2bfloat162_rn(a, b);
    const float2 f0 = __bfloat1622float2(h0);
    const float ra = a - f0.x, rb = b - f0.y;
    const __nv_bfloat162 h1 = __floats2bfloat162_rn(ra, rb);
    const float2 f1 = __bfloat1622float2(h1);
    const __nv_bfloat162 h2 = __floats2bfloat162_rn(ra - f1.x, rb - f1.y);
    w[0][j] = *reinterpret_cast<const uint32_t*>(&h0);
    w[1][j] = *reinterpret_cast<const uint32_t*>(&h1);
    w[2][j] = *reinterpret_cast<const uint32_t*>(&h2);
  }
}

}  // namespace dfl
