// Three bf16 planes whose exact sum is an fp32 value (see linear_f32.cu).
#pragma once

#include "dfl_common.cuh"

namespace dfl {

constexpr int kPlanes = 3;

__device__ __forceinline__ void split3(float x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c) {
  a = __float2bfloat16_rn(x);
  float af = __bfloat162float(a);
  if (isinf(af)) {   // rounding a finite value up to infinity: truncate instead
    a = __ushort_as_bfloat16((unsigned short)(__float_as_uint(x) >> 16));
    af = __bfloat162float(a);
  }
  const float r1 = isinf(af) ? 0.0f : x - af;   // exact
  b = __float2bfloat16_rn(r1);
  c = __float2bfloat16_rn(r1 - __bfloat162float(b));
}

// Four elements of one row as packed plane words.
__device__ __forceinline__ void split3x4(const float (&f)[4], uint2 (&out)[kPlanes]) {
  __nv_bfloat16 p[kPlanes][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) split3(f[j], p[0][j], p[1][j], p[2][j]);
#pragma unroll
  for (int q = 0; q < kPlanes; ++q) {
    const __nv_bfloat162 lo = __halves2bfloat162(p[q][0], p[q][1]), hi = __halves2bfloat162(p[q][2], p[q][3]);
    out[q] = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  }
}

}  // namespace dfl
