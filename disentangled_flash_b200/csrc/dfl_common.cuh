// Shared host/device helpers for the B200 disentangled-attention library.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>
#include <mutex>

#include "../../include/dfl_b200.h"

namespace dfl {

// ---------------------------------------------------------------- errors ---
// Last error detail, per host thread.  Written only on failure paths.
inline char* last_error_buffer() {
  static thread_local char buf[512] = {0};
  return buf;
}

inline int fail(int status, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(last_error_buffer(), 512, fmt, ap);
  va_end(ap);
  return status;
}

inline int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
  return DFL_OK;
}

// What a kernel writes to the status word when one of its waits expires: the number of the wait plus its kernel's hundred, so
// that the code says which kernel of a forward it was.  98 (dfl_embed_layernorm: an index) and 99 (the self test) are no waits
// of these.
enum WaitCodes {
  kWaitsAttention = 100, kWaitsGemmPair = 200, kWaitsGemmTile = 300, kWaitsAttentionRel = 400, kWaitsGemmF32 = 500,
  kWaitsAttentionF32 = 600, kWaitsAttentionF32Rel = kWaitsAttentionF32 + 100
};
inline const char* kernel_of_wait(int code) {
  switch (code / 100 * 100) {
    case kWaitsAttention: return "attention_tc_kernel";
    case kWaitsGemmPair: return "gemm_tc_pair_kernel";
    case kWaitsGemmTile: return "gemm_tile_kernel";
    case kWaitsAttentionRel: return "attention_rel_kernel";
    case kWaitsGemmF32: return "gemm_f32_kernel";
    case kWaitsAttentionF32: return "attention_f32_kernel";
    case kWaitsAttentionF32Rel: return "attention_f32_rel_kernel";
  }
  return code == 99 ? "the self test" : "unknown";
}

// Launchers keep their one-time configuration (shared-memory opt-in, SM count, symbol addresses) per device.
constexpr int kMaxDevices = 64;

// One-time launch configuration of one kernel instance, kept per device: the opt-in to large dynamic shared
// memory is a per-device attribute of the kernel, and the grid of a persistent kernel follows the device's SM
// count.  One object per kernel instance (a function-local static of its launcher); first calls from several
// host threads are serialised.
struct KernelDeviceConfig {
  std::mutex mutex;
  int smem_opted_in[kMaxDevices] = {0};
  int sm_count[kMaxDevices] = {0};
};
template <typename Kernel>
inline int configure_kernel(KernelDeviceConfig& cfg, Kernel kernel, int smem_bytes, int* sm_count, const char* what) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return fail(DFL_ERR_LAUNCH, "%s: current device: %s", what, cudaGetErrorString(e));
  std::lock_guard<std::mutex> lock(cfg.mutex);
  if (smem_bytes > cfg.smem_opted_in[dev]) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "%s: shared-memory opt-in: %s", what, cudaGetErrorString(e));
    cfg.smem_opted_in[dev] = smem_bytes;
  }
  if (cfg.sm_count[dev] == 0) {
    int count = 0;
    e = cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess || count < 1) return fail(DFL_ERR_LAUNCH, "%s: SM count: %s", what, cudaGetErrorString(e));
    cfg.sm_count[dev] = count;
  }
  if (sm_count) *sm_count = cfg.sm_count[dev];
  return DFL_OK;
}

// Launch with programmatic stream serialization: the kernel's CTAs may be scheduled, and run up to their
// `griddepcontrol.wait`, while the previous kernel of the stream is still draining; everything that touches global
// memory comes after that wait, which returns when the previous kernel has completed and its writes are visible.
// This takes the launch latency and the kernel's set-up (barrier initialisation, tensor-memory allocation, descriptor
// prefetch) off the path between two dependent kernels.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_clusters_after_predecessor(void (*kernel)(KArgs...), dim3 grid, dim3 block, int cluster,
                                                     size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 0 ? 2 : 1;   // 0: no cluster, or the kernel's own __cluster_dims__
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_after_predecessor(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                            cudaStream_t stream, Args... args) {
  return launch_clusters_after_predecessor(kernel, grid, block, 0, smem, stream, args...);
}
// Device side of the above: wait for the previous kernel of the stream (no-op for a plain launch).
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel of the stream be scheduled as soon as every CTA of this grid has called it (its own
// wait_for_predecessor() still holds it back until this grid has completed).  Called only after this kernel's own
// wait: whatever ran before this kernel is then complete when the next kernel starts its set-up.
__device__ __forceinline__ void release_successor() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

inline size_t dtype_size(int dtype) { return dtype == DFL_F32 ? 4 : 2; }

// ------------------------------------------------------------ conversions ---
template <typename T> struct Elem;
template <> struct Elem<float> {
  static __device__ __forceinline__ float to_f(float v) { return v; }
  static __device__ __forceinline__ float from_f(float v) { return v; }
};
template <> struct Elem<__half> {
  static __device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half from_f(float v) { return __float2half_rn(v); }
};
template <> struct Elem<__nv_bfloat16> {
  static __device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float v) { return __float2bfloat16_rn(v); }
};

// Round an fp32 value through T (identity for float).
template <typename T>
__device__ __forceinline__ float round_through(float v) {
  return Elem<T>::to_f(Elem<T>::from_f(v));
}

// Non-zero test of one mask element of 1, 4 or 8 bytes.
__device__ __forceinline__ bool mask_keep(const void* mask, int elem_size, long long idx) {
  if (elem_size == 1) return reinterpret_cast<const uint8_t*>(mask)[idx] != 0;
  if (elem_size == 4) return reinterpret_cast<const uint32_t*>(mask)[idx] != 0;
  return reinterpret_cast<const unsigned long long*>(mask)[idx] != 0ull;
}

// ------------------------------------------------- kernel launch wrappers ---
// One function per kernel family; defined in the matching .cu file.
int launch_position_lut(int L, int buckets, int max_pos, int span, int uses_bias, int32_t* lut,
                        int64_t* active, int32_t* n_active, cudaStream_t stream);
int launch_gather_slots(const void* src, const int64_t* active, void* dst, int heads, int n_src,
                        int n_active, int d, int dtype, cudaStream_t stream);

// Generic batched "NT" GEMM description used by both GEMM families:
//   C_z[m, n] = sum_k X_z[m, k] * W_{z % w_mod}[n, k] (+ bias[n])
// with either a head-split epilogue (QKV / position projection) or a plain
// row-major epilogue with leading dimension ldc (position scores).
struct GemmDesc {
  const void* x;
  const void* w;
  const void* bias;
  void* out[3];
  int M, N, K;
  int batch;            // grid.z
  long long stride_x;   // elements between X_z
  long long stride_w;   // elements between W_z'
  int w_mod;            // W index = z % w_mod
  long long stride_c;   // elements between C_z (row-major epilogue)
  int ldc;              // row-major epilogue leading dimension; columns [N, ldc) zero-filled
  int head_split;       // 1: head-split epilogue, 0: row-major
  int heads, head_dim, rows_per_seq;
  int dtype;
  int* status;          // device status word of the call, or null (the tcgen05 GEMM then uses the library's word)
  int activation;       // DFL_ACT_*: applied after the bias (row-major epilogue only)
  // 1-D convolution as a GEMM over taps (the 16-bit tensor-core kernels): k-step (tap, kb) multiplies rows
  // m + tap - taps/2 of X_z (rows outside [0, M) read as zero: 'same' padding) with weight matrix W[tap].
  int taps;             // 0 or 1: plain GEMM
  const void* row_mask; // [batch, M] or null: output rows whose element is zero are set to 0 before the activation
  int row_mask_elem;    // element size of row_mask: 1, 4 or 8 bytes
  // Packed input rows (head-split epilogue of the tensor-core kernels only): rows 32g .. 32g+31 of X are written to
  // rows row_groups[g] .. +31 of the [out_seqs * rows_per_seq] output row space.  Null: row m goes to row m.
  const int* row_groups;
  int out_seqs;         // sequences of the output tensors when row_groups is set (else M / rows_per_seq)
  // 1: the kernel before this one in the stream is one of this library's that waited for its own predecessor and
  // does not write W or the bias, so that W may be read before that kernel has finished (see release_successor())
  int weights_early;
  int out_planes;       // linear_f32.cu: write the result (batch 1) as bf16 planes [3][...] instead of fp32
};

// tanh for the GEMM epilogues of 16-bit outputs: 1 - 2 / (1 + e^(2x)) with approximate exp2 and reciprocal
// (absolute error ~1e-7; exact limits +-1).
__device__ __forceinline__ float tanh_fast(float x) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * 2.8853900817779268f));   // 2 log2(e)
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
  return fmaf(-2.0f, r, 1.0f);
}

// GELU, 0.5 x (1 + erf(x / sqrt 2)), for the GEMM epilogues.
// Exact form (strict FP32 kernels): the CUDA library's erff.
__device__ __forceinline__ float gelu_erf_exact(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
// Form for BF16 outputs: erf by the rational approximation 7.1.26 of Abramowitz & Stegun,
// erf(z) = 1 - (a1 t + ... + a5 t^5) exp(-z^2), t = 1 / (1 + p z), z >= 0, absolute error below 1.5e-7, with one approximate
// reciprocal and one approximate exp2 (relative error ~1e-7 each).  Its error stays small beside the result far into the negative
// tail, whose results BF16's exponent range holds: 1.6e-3 of the result at -5, 6.5e-3 at -7, 1.5e-2 at -9 (gelu_erf_pair: 3.3e-3,
// 0.3, 1).
__device__ __forceinline__ float gelu_erf_fast(float x) {
  // gelu(x) = max(x, 0) - |x| * q(t) * exp(-z^2),  z = |x| / sqrt 2,  q(t) = 0.5 (a1 t + ... + a5 t^5).
  // With w = z * sqrt(log2 e): exp(-z^2) = exp2(-w^2) and 1 + p z = 1 + (p / sqrt(log2 e)) w.
  const float ax = fabsf(x);
  const float w = ax * 0.84932180028801904f;            // sqrt(log2(e) / 2)
  float t, e;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(0.27273748088f, w, 1.0f)));   // p / sqrt(log2 e)
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-w * w));
  float q = fmaf(0.5307027145f, t, -0.7265760135f);      // a5 / 2, a4 / 2
  q = fmaf(q, t, 0.7107068705f);                          // a3 / 2
  q = fmaf(q, t, -0.142248368f);                          // a2 / 2
  q = fmaf(q, t, 0.127414796f);                           // a1 / 2
  return fmaf(-(ax * (q * t)), e, fmaxf(x, 0.0f));
}

// Two fp32 values in one register pair; Blackwell adds and multiplies both with one instruction.
__device__ __forceinline__ unsigned long long pack_f32x2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// GELU of two values, for FP16 outputs:
//   gelu(x) = max(x, 0) - |x| Phi(-|x|),   Phi(-t) = 2^p(t),  t >= 0,
// p the degree-8 polynomial that fits log2(erfc(t / sqrt 2) / 2) on [0, 6.5] with the weight t Phi(-t), that is, with the
// error's weight in the result (Lawson's iteration on least squares; its leading coefficient is negative, so p keeps falling
// beyond the fit).  Absolute error below 2.5e-7 (gelu_erf_fast: 3.3e-7), and relative to the result 4e-4 at worst in the
// negative tail down to -4.5 (9e-4).  Below -4.5 the error relative to the result grows (4.9e-2 at -6); in absolute terms it is below
// 7e-9 there, a tenth of the step between FP16's smallest numbers.  One special-function instruction an element where gelu_erf_fast
// has two, which bound the epilogue (16 lanes a cycle and SM): 16384 x 3072 x 768 fp16 77.5 -> 72.9 us (65 without an activation),
// 12288 rows 61.8 -> 55.0, 512 x 6144 x 1536 13.3 -> 12.7.  On single values, without the packed multiply-adds, 2 to 3 % slower.
__device__ __forceinline__ void gelu_erf_pair(float& a, float& b) {
  const float na = -fabsf(a), nb = -fabsf(b);   // the polynomial is in -t: odd coefficients change their sign
  const unsigned long long t = pack_f32x2(na, nb);
  auto k = [](float c) { return pack_f32x2(c, c); };
  unsigned long long p = fma_f32x2(k(-1.69028031e-06f), t, k(-2.5081631e-05f));
  p = fma_f32x2(p, t, k(-0.000114453323f));
  p = fma_f32x2(p, t, k(0.000323369388f));
  p = fma_f32x2(p, t, k(0.00733342881f));
  p = fma_f32x2(p, t, k(0.0527142401f));
  p = fma_f32x2(p, t, k(-0.459115417f));
  p = fma_f32x2(p, t, k(1.15112327f));
  p = fma_f32x2(p, t, k(-0.999998874f));
  float pa, pb, ea, eb;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(pa), "=f"(pb) : "l"(p));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ea) : "f"(pa));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(eb) : "f"(pb));
  const unsigned long long g = fma_f32x2(t, pack_f32x2(ea, eb), pack_f32x2(fmaxf(a, 0.0f), fmaxf(b, 0.0f)));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(g));
}
// GELU of two values that are rounded to T next.
template <typename T>
__device__ __forceinline__ void gelu_pair(float& a, float& b) {
  if constexpr (__is_same(T, __half)) {
    gelu_erf_pair(a, b);
  } else {
    a = gelu_erf_fast(a);
    b = gelu_erf_fast(b);
  }
}
int launch_gemm_simt(const GemmDesc& g, cudaStream_t stream);
int launch_gemm_tc(const GemmDesc& g, cudaStream_t stream);
// FP32 on the tensor cores: g.x is [3][batch][M][K] and g.w [3][w_mod][N][K] bf16 planes (launch_split_planes).
int launch_gemm_f32_planes(const GemmDesc& g, cudaStream_t stream);
int launch_split_planes(const void* x, void* planes, long long n, cudaStream_t stream);   // n a multiple of 4
int launch_refresh_planes(const DflPlaneSource* sources, int n_sources, long long n_pieces, cudaStream_t stream);
// nn.Conv1d weight [out, in, taps] of 2-byte elements -> [taps, out, in] (in a multiple of 8).  Starts before the kernel ahead of it has finished: that
// one must not write w, nor it or the kernel before it read `out`.
int launch_conv_weight(const void* w, void* out, int c_out, int c_in, int taps, cudaStream_t stream);

int launch_attention_simt(const DflAttnParams& p, cudaStream_t stream);
// FP32 over bf16 planes: p.q, p.k, p.v are [3][B,H,L,d], the scores fp32, the output fp32 or planes [3][B,L,H*d].
bool attention_f32_planes_supported(int head_dim, int seq_len);
int launch_attention_f32_planes(const DflAttnParams& p, int out_planes, cudaStream_t stream);
// The same with the position scores computed in the kernel: p.c2p and p.p2c are unused, pos_key / pos_query [3][H][n_active][d] planes.
// The tables, lut and mask were complete before the kernel ahead of this one in the stream started.
bool attention_f32_rel_supported(int head_dim, int seq_len);
int launch_attention_f32_rel(const DflAttnParams& p, const void* pos_key, const void* pos_query, int n_active, int out_planes,
                             cudaStream_t stream);
int launch_attention_tc(const DflAttnParams& p, cudaStream_t stream);
bool attention_rel_supported(const DflAttnRelParams& p);
// tables_early: rel_key / rel_query were complete before the kernel ahead of this one in the stream started
int launch_attention_rel(const DflAttnRelParams& p, cudaStream_t stream, bool tables_early = false);
bool attention_rel_small_covers(const DflAttnRelParams& p);
int launch_attention_rel_small(const DflAttnRelParams& p, bool tables_early, cudaStream_t stream);
int add_layernorm_max_hidden(size_t elem_size);
int launch_add_layernorm(const void* x, const void* residual, const void* gamma, const void* beta, void* out,
                         long long rows, int hidden, float eps, int dtype, const void* row_mask, int mask_elem,
                         void* out2, const int32_t* out2_rows, void* planes, cudaStream_t stream);
int launch_embed_layernorm(const void* ids, const void* table, long long vocab, const void* pos_ids,
                           const void* pos_table, long long positions, int idx_elem, const void* gamma,
                           const void* beta, void* out, long long rows, int hidden, float eps, int dtype,
                           const void* row_mask, int mask_elem, int* status, cudaStream_t stream);
int launch_copy_rows(const void* src, void* dst, const int32_t* rows, long long n_rows, int row_bytes,
                     cudaStream_t stream);
int launch_selftest_bounded_wait(int* status, uint32_t limit_us, cudaStream_t stream);
int launch_expand_rel_tables(const void* pos, const int32_t* lut, void* rel, int heads, int n_active, int seq_len,
                             int head_dim, int dtype, cudaStream_t stream);

}  // namespace dfl
