// Pieces shared by the two files of the 16-bit tcgen05 GEMM (linear_tc.cu: large persistent tiles, linear_tile.cu: one tile
// per CTA).
#pragma once

#include "dfl_common.cuh"
#include "tcgen05_ptx.cuh"

namespace dfl {

// Epilogue of one accumulator chunk of a head-major output whose rows cannot leave as whole boxes: 32 consecutive columns [n, n+32) of
// output row m, as fp32 bit patterns in r.  Adds the bias, rounds to T and stores 32 (or 16) bytes at a time.  (With branches for
// row-major outputs and GELU, which no launch reached, the operator at 16 x 24 heads x 256 x d 32 took 56.0 us; 52.8 without.)
template <typename T>
__device__ __forceinline__ void store_chunk(const GemmDesc& g, const uint32_t (&r)[32], int m, int n, int hd, const T* bias) {
  const int which = n / hd, rem = n - which * hd;
  const int h = rem / g.head_dim, dd = rem - h * g.head_dim;
  const int row = g.row_groups ? __ldg(g.row_groups + (m >> 5)) + (m & 31) : m;
  const int b = row / g.rows_per_seq, l = row - b * g.rows_per_seq;
  T* out = reinterpret_cast<T*>(which == 0 ? g.out[0] : (which == 1 ? g.out[1] : g.out[2]));
  T* dst = out + (((long long)b * g.heads + h) * g.rows_per_seq + l) * g.head_dim + dd;
  // 32-byte stores (one full sector per thread and instruction) where the destination allows them
  const bool wide = (reinterpret_cast<uintptr_t>(dst) & 31u) == 0;
  uint4 held = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[v * 8 + j]);
    if (bias) {
      const uint4 braw = __ldg(reinterpret_cast<const uint4*>(bias + n + v * 8));
      const T* bh = reinterpret_cast<const T*>(&braw);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += Elem<T>::to_f(bh[j]);
    }
    uint4 packed;
    T* ph = reinterpret_cast<T*>(&packed);
#pragma unroll
    for (int j = 0; j < 8; ++j) ph[j] = Elem<T>::from_f(f[j]);
    if (wide && (v & 1) != 0) {
      asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst + (v - 1) * 8), "r"(held.x), "r"(held.y),
                   "r"(held.z), "r"(held.w), "r"(packed.x), "r"(packed.y), "r"(packed.z), "r"(packed.w) : "memory");
    } else if (wide) {
      held = packed;
    } else {
      *reinterpret_cast<uint4*>(dst + v * 8) = packed;
    }
  }
}

// tcgen05 GEMM family members; the dispatcher is launch_gemm_tc (linear_tc.cu).
struct TilePlan {
  int bn;      // output columns per tile, a multiple of 32 up to 256
  int split;   // CTAs (or CTA pairs) of a cluster that share one tile's inner product
  int pair;    // 1: two CTAs per 256-row tile (cta_group::2)
};
int launch_gemm_tile(const GemmDesc& g, const TilePlan& plan, cudaStream_t stream);

}  // namespace dfl
