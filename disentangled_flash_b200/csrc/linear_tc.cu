// tcgen05 GEMM family for FP16/BF16: fused QKV projection with head-split
// epilogue, relative-embedding projection, and the C2P/P2C position-score GEMMs.
//
// Replaces the library GEMMs on the reference's hot path: F.linear for the
// fused QKV projection plus the three permute().contiguous() copies
// (src/disentangled_flash/_torch.py:284-314), the relative-embedding
// projections (_torch.py:143-158) and torch.matmul x2 for the position scores
// (src/disentangled_flash/kernel.py:574-585).
//
//   C_z[m,n] = sum_k X_z[m,k] * W_{z % w_mod}[n,k] (+ bias[n]),  fp32 accumulation in TMEM
//
// This file: the persistent kernel for large problems and the choice between it and the one-tile-per-CTA kernel of
// linear_tile.cu.  gemm_tc_pair_kernel runs one CTA per SM with 320 threads, in clusters of two CTAs that work on one
// 256-row tile of 128 to 256 columns (cta_group::2): a producer warp streams k-blocks of X and W into a shared-memory
// ring with TMA (128-byte swizzle, K-major) and keeps streaming across tile boundaries, the MMA warp issues tcgen05.mma
// into one of two 256-column TMEM accumulators, and eight epilogue warps drain the finished accumulator (tcgen05.ld, one
// row per thread, 64-column chunks), add the bias, apply the activation, round to the output type, stage 32 x 64 blocks
// in shared memory and write them with tiled bulk stores, head-major [B,H,L,d] or row-major - while the MMA warp already
// fills the other accumulator.
#include <cstring>

#include "linear_epilogue.cuh"

namespace dfl {

// ------------------------------------------------------------------ tensor maps
namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn resolve_encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}
}  // namespace

int encode_tensor_map_3d(CUtensorMap* map, const void* base, uint64_t inner, uint64_t rows, uint64_t batch,
                         uint64_t row_stride_bytes, uint64_t batch_stride_bytes, uint32_t box_inner,
                         uint32_t box_rows, int swizzle_bytes) {
  EncodeTiledFn encode = resolve_encode_tiled();
  if (!encode) return fail(DFL_ERR_DRIVER, "cuTensorMapEncodeTiled entry point not available");
  if ((row_stride_bytes & 15) || (batch_stride_bytes & 15))
    return fail(DFL_ERR_ALIGNMENT, "tensor-map strides must be multiples of 16 bytes");
  const cuuint64_t dims[3] = {inner, rows, batch};
  const cuuint64_t strides[2] = {row_stride_bytes, batch_stride_bytes};
  const cuuint32_t box[3] = {box_inner, box_rows, 1};
  const cuuint32_t elem_strides[3] = {1, 1, 1};
  CUtensorMapSwizzle sw = swizzle_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                          : swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                          : swizzle_bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B
                                                : CU_TENSOR_MAP_SWIZZLE_NONE;
  CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(base), dims, strides, box,
                      elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(DFL_ERR_DRIVER, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return DFL_OK;
}

int encode_tensor_map_4d(CUtensorMap* map, const void* base, const uint64_t (&dims)[4], const uint64_t (&strides)[3],
                         const uint32_t (&box)[4]) {
  EncodeTiledFn encode = resolve_encode_tiled();
  if (!encode) return fail(DFL_ERR_DRIVER, "cuTensorMapEncodeTiled entry point not available");
  if ((strides[0] & 15) || (strides[1] & 15) || (strides[2] & 15))
    return fail(DFL_ERR_ALIGNMENT, "tensor-map strides must be multiples of 16 bytes");
  const cuuint64_t d[4] = {dims[0], dims[1], dims[2], dims[3]}, st[3] = {strides[0], strides[1], strides[2]};
  const cuuint32_t bx[4] = {box[0], box[1], box[2], box[3]}, elem_strides[4] = {1, 1, 1, 1};
  CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 4, const_cast<void*>(base), d, st, bx, elem_strides,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(DFL_ERR_DRIVER, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return DFL_OK;
}

int encode_tensor_map_pieces(CUtensorMap* map, const void* base, uint64_t inner, uint64_t rows, uint64_t batch,
                             uint64_t row_stride_bytes, uint64_t batch_stride_bytes, uint32_t box_rows,
                             uint32_t box_batch, uint32_t box_pieces) {
  if (box_pieces > 1 && inner % 64) return fail(DFL_ERR_BAD_ARG, "rows of whole 128-byte pieces expected");
  const uint64_t dims[4] = {box_pieces > 1 ? 64 : inner, rows, batch, box_pieces > 1 ? inner / 64 : 1};
  const uint64_t strides[3] = {row_stride_bytes, batch_stride_bytes, box_pieces > 1 ? 128 : row_stride_bytes};
  const uint32_t box[4] = {64, box_rows, box_batch, box_pieces};
  return encode_tensor_map_4d(map, base, dims, strides, box);
}

// Library-owned status word for kernels whose caller passes none.
__device__ int g_gemm_status = 0;

namespace {

constexpr int TM = 128, TN = 256;  // rows per CTA, columns of an accumulator (the widest tile)
constexpr int kEpilogueWarps = 8;   // warp w drains TMEM lanes 32*(w&3).. of accumulator columns 128*(w>>2)..
constexpr int kTmaWarp = 8, kMmaWarp = 9;
constexpr int kThreads = 320;
constexpr int kTmemCols = 512;      // two 256-column accumulators: epilogue of tile i overlaps main loop of tile i+1
constexpr int kMaxSmem = 232448;
constexpr int kWaits = kWaitsGemmPair;

// Output staging for the tiled-store epilogue: per epilogue warp one buffer of 32 rows x 64 columns (128-byte
// rows in the 128-byte swizzle pattern of the output tensor maps).  Two warps share a scheduler, so one converts
// while the other's store drains its buffer.
constexpr int kStageRows = 32, kStageCols = 64;
constexpr int kStageBufBytes = kStageRows * kStageCols * 2;   // 4 KB
constexpr int kStagingBytes = 8 * kStageBufBytes;              // one buffer per epilogue warp = 32 KB

struct OutMaps {
  CUtensorMap m[3];
};

// Whether the output can be written as 32-row x 64-column boxes: row-major always (the tensor map clips at ldc and
// M); head-major when a box neither straddles two heads (head_dim a multiple of 64) nor two sequences.
__host__ __device__ inline bool tiled_store_ok(const GemmDesc& g) {
  return !g.head_split || (g.head_dim % kStageCols == 0 && g.rows_per_seq % kStageRows == 0);
}

// Drains one warp's 32 lanes x 128 columns of an accumulator.  `taddr` = TMEM address of the warp's lane quarter at
// the accumulator's first column, `m_warp` = output row of lane 0, `n0` = first output column of the tile, `bn` its
// width; the two warps of a lane quarter take alternate chunks, `chunk0` = 0 or 1.
// With `tiled` the rows go through the warp's staging buffers and leave as tiled bulk stores of full 128-byte
// lines (per-thread stores would write every 32-byte sector in two halves from different instructions, and the
// number of store requests, not the math, then bounds GEMMs with a short K).
// CONV: the epilogue of the convolution branch (padding mask of the output row, tanh) is compiled in; plain GEMMs
// take the instantiation without it (the extra code cost them 7 % when it was shared).
// `wait_full` waits for the accumulator, `release` hands it back to the MMA warp: as soon as it is in registers, before the
// arithmetic and the stores of the last chunk, and without waiting for the stores of earlier ones.  With a short K the drain is
// as long as the MMAs of a tile, so both count: 16384 x 3072 x 768 fp16 65.0 -> 63.7 us, with GELU 72.9 -> 68.7, 12288 rows 55.0
// -> 50.4, 2331 x 2304 x 768 13.8 -> 12.9.
template <typename T, bool CONV, typename WaitFull, typename Release>
__device__ __forceinline__ void drain_accumulator(const GemmDesc& g, const CUtensorMap* tmap_out, bool tiled,
                                                  unsigned char* buf, uint32_t taddr, int m_warp, int n0, int bn,
                                                  int chunk0, int z, int lane, WaitFull wait_full, Release release) {
  const int ncols = g.head_split ? g.N : g.ldc;
  const T* bias = reinterpret_cast<const T*>(g.bias);
  const int hd = g.heads * g.head_dim;
  if (!tiled || n0 + chunk0 * kStageCols >= ncols) {
    const bool ready = wait_full();
    const int m = m_warp + lane;
#pragma unroll 1
    for (int c0 = chunk0 * 32; c0 < bn; c0 += 64) {
      const int n = n0 + c0;
      if (n >= ncols || tiled) break;  // warp-uniform
      uint32_t r[32];
      ptx::tmem_ld32(taddr + (uint32_t)c0, r);
      ptx::tmem_wait_ld();
      if (!ready || m >= g.M) continue;
      store_chunk<T>(g, r, m, n, hd, bias);   // head-major: see tiled_store_ok
    }
    release();
    return;
  }
  bool ready = false;
  // padding mask of this thread's output row (convolution epilogue)
  bool keep_row = true;
  if (CONV && g.row_mask && m_warp + lane < g.M) keep_row = mask_keep(g.row_mask, g.row_mask_elem, (long long)z * g.M + m_warp + lane);
#pragma unroll 1
  for (int c0 = chunk0 * kStageCols; c0 < bn; c0 += 2 * kStageCols) {
    const int n = n0 + c0;
    if (n >= ncols) break;  // warp-uniform
    uint4 braw[8];          // requested before anything is waited for: the first touch of a line comes from L2
#pragma unroll
    for (int v = 0; v < 8; ++v)
      braw[v] = bias && n + v * 8 < g.N ? __ldg(reinterpret_cast<const uint4*>(bias + n + v * 8)) : make_uint4(0u, 0u, 0u, 0u);
    if (c0 == chunk0 * kStageCols) ready = wait_full();
    uint32_t r0[32], r1[32];
    ptx::tmem_ld32(taddr + (uint32_t)c0, r0);
    ptx::tmem_ld32(taddr + (uint32_t)c0 + 32u, r1);
    // the previous store of this warp has finished reading the buffer
    if (lane == 0) ptx::bulk_wait_group_read<0>();
    __syncwarp();
    ptx::tmem_wait_ld();
    if (c0 + 2 * kStageCols >= bn || n + 2 * kStageCols >= ncols) release();   // the accumulator has been read
    if (!ready || m_warp >= g.M) continue;  // warp-uniform
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      float f[8];
      const T* bh = reinterpret_cast<const T*>(&braw[v]);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(v < 4 ? r0[v * 8 + j] : r1[(v - 4) * 8 + j]) + Elem<T>::to_f(bh[j]);
      if (CONV && !keep_row) {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = 0.0f;
      }
      if (g.activation == DFL_ACT_GELU) {
#pragma unroll
        for (int j = 0; j < 8; j += 2) gelu_pair<T>(f[j], f[j + 1]);
      } else if (CONV && g.activation == DFL_ACT_TANH) {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = tanh_fast(f[j]);
      }
      uint4 packed;
      T* ph = reinterpret_cast<T*>(&packed);
#pragma unroll
      for (int j = 0; j < 8; ++j) ph[j] = Elem<T>::from_f(f[j]);
      *reinterpret_cast<uint4*>(buf + lane * 128 + ((v ^ (lane & 7)) << 4)) = packed;
    }
    ptx::fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      if (g.head_split) {
        const int which = n / hd, rem = n - which * hd;
        const int h = rem / g.head_dim, dd = rem - h * g.head_dim;
        const int row = g.row_groups ? __ldg(g.row_groups + (m_warp >> 5)) : m_warp;   // a warp's 32 rows: one group
        const int b = row / g.rows_per_seq, l = row - b * g.rows_per_seq;
        ptx::tma_store_3d(&tmap_out[which], buf, dd, l, b * g.heads + h);
      } else {
        ptx::tma_store_3d(&tmap_out[0], buf, n, m_warp, z);
      }
      ptx::bulk_commit_group();
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// CTA-pair form (clusters of two, `cta_group::2`): one 256 x 256 output tile per pair.  Each CTA loads its own 128
// rows of X and 128 of the tile's 256 rows of W per k-step (32 KB for 128 x 256 x 64 of MMA work; a CTA on its own would
// take 48 KB, and the operand stream from L2 is what bounds this GEMM), the leader CTA (cluster rank 0)
// issues M=256, N=256 MMAs that read both CTAs' shared memory and write 128 accumulator lanes in each CTA's TMEM,
// and each CTA's epilogue warps drain their own lanes.  Barriers: the loads of both CTAs report to the leader's
// `full` barriers; the leader's commits arrive on the `empty` / `tmem_full` barriers of both CTAs; the epilogue
// warps of both CTAs arrive on the leader's `tmem_empty` barriers.
constexpr int kPairStages = 6;                       // 6 x 32 KB operand ring per CTA
constexpr int kPairStageBytes = (TM + TN / 2) * 128;  // A 128x64 + half of B 128x64, 2-byte elements
constexpr int kPairStagingOffset = kPairStages * kPairStageBytes;
constexpr int kPairBarrierOffset = kPairStagingOffset + kStagingBytes;
constexpr int kPairSmem = kPairBarrierOffset + 512 + 1024;
static_assert(kPairSmem <= kMaxSmem,
              "operand ring + output staging + barriers must fit the 227 KB a CTA can opt in to");

template <typename T, bool CONV>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                    const __grid_constant__ OutMaps tmap_out, const GemmDesc g, const int num_kb, const int tiles_n,
                    const int tiles_m, const int num_tiles, const int tiled, const int bn) {
  constexpr int BK = 64;
  constexpr int STAGES = kPairStages;
  constexpr int kTileA = TM * BK * 2;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kPairBarrierOffset);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full_bar = empty_bar + STAGES;   // [2]
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;   // [2]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();   // 0 = leader
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&full_bar[s], 1);    // the leader's producer (expect_tx); only the leader's are used
      ptx::mbar_init(&empty_bar[s], 1);   // one commit of the leader's MMA thread, delivered to both CTAs
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&tmem_full_bar[a], 1);
      ptx::mbar_init(&tmem_empty_bar[a], 2 * kEpilogueWarps);  // one lane of each epilogue warp of both CTAs (leader's only)
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == kTmaWarp && lane == 0) {
    ptx::prefetch_tensormap(&tmap_x);
    ptx::prefetch_tensormap(&tmap_w);
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc_pair(tmem_holder, kTmemCols);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();   // the peer's barriers exist before anything is reported to them
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  const uint32_t load_bytes = (uint32_t)kTileA + (uint32_t)(bn / 2) * BK * 2;   // one k-step of one CTA
  wait_for_predecessor();    // the set-up above overlaps the previous kernel's tail; its outputs are read from here on

  auto tile_coords = [&](int tile, int& m0, int& n0, int& z) {
    const int per_z = tiles_n * tiles_m;
    z = tile / per_z;
    const int rem = tile - z * per_z;
    const int tm = rem / tiles_n;
    m0 = tm * (2 * TM);
    n0 = (rem - tm * tiles_n) * bn;
  };

  if (warp == kTmaWarp) {
    // ---------------------------------------------------------- TMA producer (both CTAs; the whole warp, converged)
    const uint32_t ring_addr = ptx::smem_u32(smem), full_addr = ptx::smem_u32(full_bar), leader_full = ptx::map_to_cta(full_addr, 0);
    const int taps = CONV && g.taps > 1 ? g.taps : 1;
    int s = 0;
    uint32_t ph = 1;   // phase of empty_bar[s] to wait for (the first round passes)
    bool ok = true;
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      int m0, n0, z;
      tile_coords(tile, m0, n0, z);
      // k-steps: num_kb = taps x (k-blocks per tap); a plain GEMM has one tap with no row shift
      const int kb_per_tap = CONV ? num_kb / taps : num_kb;
      const int w_batch = z % g.w_mod, x_row = m0 + (int)rank * TM, w_row = n0 + (int)rank * (bn / 2);
      int tap = 0, kb = 0;
      for (int step = 0; step < num_kb; ++step) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&empty_bar[s], ph, abort_flag, g.status, kWaits + 11));
        if (!ok) break;
        if (rank == 0) ptx::mbar_arrive_expect_tx_warp(full_addr + 8u * s, 2u * load_bytes);
        const uint32_t a = ring_addr + (uint32_t)s * kPairStageBytes, bar = leader_full + 8u * s;
        // rows above the first or below the last row of X_z are filled with zeros by the load
        if constexpr (CONV) {
          ptx::tma_load_3d_pair_warp(a, &tmap_x, bar, kb * BK, x_row + tap - (taps >> 1), z);
          ptx::tma_load_3d_pair_warp(a + kTileA, &tmap_w, bar, kb * BK, w_row, taps > 1 ? tap : w_batch);
          if (++kb == kb_per_tap) {
            kb = 0;
            ++tap;
          }
        } else {
          ptx::tma_load_3d_pair_warp(a, &tmap_x, bar, step * BK, x_row, z);
          ptx::tma_load_3d_pair_warp(a + kTileA, &tmap_w, bar, step * BK, w_row, w_batch);
        }
        if (++s == STAGES) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer (leader only)
    if (rank == 0) {   // the whole warp, converged: see umma_ss_f16_warp
      const uint32_t idesc = ptx::make_idesc_f16(__is_same(T, __nv_bfloat16) ? 1 : 0, 2 * TM, bn, 0, 0);
      constexpr uint32_t mode = ptx::swizzle_mode_for_row_bytes(BK * 2);
      const uint64_t adesc0 = ptx::make_smem_desc(ptx::smem_u32(smem), 16, 8 * BK * 2, mode);
      const uint64_t bdesc0 = ptx::make_smem_desc(ptx::smem_u32(smem + kTileA), 16, 8 * BK * 2, mode);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      int lt = 0;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++lt) {
        const int acc = lt & 1;
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&tmem_empty_bar[acc], ((uint32_t)(lt >> 1) & 1u) ^ 1u, abort_flag, g.status, kWaits + 14));
        if (!ok) break;
        ptx::tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * TN;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = __all_sync(0xffffffffu, ptx::mbar_wait(&full_bar[s], ph, abort_flag, g.status, kWaits + 12));
          if (!ok) break;
          ptx::tc_fence_after();
          const uint64_t adesc = adesc0 + (uint64_t)(s * (kPairStageBytes >> 4));
          const uint64_t bdesc = bdesc0 + (uint64_t)(s * (kPairStageBytes >> 4));
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            ptx::umma_ss_f16_pair_warp(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
          ptx::umma_commit_pair_warp(&empty_bar[s]);  // frees the stage in both CTAs
          if (++s == STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
        if (!ok) break;
        ptx::umma_commit_pair_warp(&tmem_full_bar[acc]);  // accumulator complete, both CTAs' epilogues may read
      }
    }
  } else {
    // -------------------------------------------------------------- epilogue (both CTAs, own lanes)
    unsigned char* staging = smem + kPairStagingOffset + warp * kStageBufBytes;
    const int quarter = warp & 3, chunk0 = warp >> 2;
    bool ready = true;
    int lt = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs, ++lt) {
      int m0, n0, z;
      tile_coords(tile, m0, n0, z);
      const int acc = lt & 1;
      auto wait_full = [&] {
        if (ready) ready = ptx::mbar_wait(&tmem_full_bar[acc], (uint32_t)(lt >> 1) & 1u, abort_flag, g.status, kWaits + 13);
        ptx::tc_fence_after();
        return ready;
      };
      auto release = [&] {   // orders tensor-memory reads only: a releasing arrive at cluster scope would wait for the stores
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_peer(ptx::map_to_cta(ptx::smem_u32(&tmem_empty_bar[acc]), 0));
      };
      drain_accumulator<T, CONV>(g, tmap_out.m, tiled != 0, staging,
                           tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * TN),
                           m0 + (int)rank * TM + quarter * 32, n0, bn, chunk0, z, lane, wait_full, release);
    }
    if (lane == 0) ptx::bulk_wait_group<0>();   // the staging buffers are read until the stores complete
  }

  // Nothing of this CTA may still be in use by the peer (its shared memory is read by the leader's MMAs, its
  // barriers receive the leader's commits) when it exits or frees its tensor memory.
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();
  ptx::tc_fence_after();
  if (warp == kMmaWarp) ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
}

// Tensor maps of the outputs for the tiled-store epilogue: boxes of 32 rows x 64 columns, 128-byte swizzle.
// Head-major outputs [B, H, L, d] are described as {d, L, B*H}; the row-major output as {ldc, M, batch}.
template <typename T>
int encode_output_maps(const GemmDesc& g, OutMaps* maps, int* tiled) {
  *tiled = tiled_store_ok(g) ? 1 : 0;
  memset(maps, 0, sizeof(*maps));
  if (!*tiled) return DFL_OK;
  const size_t es = sizeof(T);
  if (g.head_split) {
    const uint64_t seqs = (uint64_t)(g.row_groups ? g.out_seqs : g.M / g.rows_per_seq) * g.heads;
    for (int o = 0; o < 3; ++o) {
      if (!g.out[o]) continue;
      int rc = encode_tensor_map_3d(&maps->m[o], g.out[o], g.head_dim, g.rows_per_seq, seqs, (uint64_t)g.head_dim * es,
                                    (uint64_t)g.rows_per_seq * g.head_dim * es, kStageCols, kStageRows, 128);
      if (rc != DFL_OK) return rc;
    }
    return DFL_OK;
  }
  const uint64_t batch_stride = g.batch > 1 ? (uint64_t)g.stride_c * es : (uint64_t)g.M * g.ldc * es;
  return encode_tensor_map_3d(&maps->m[0], g.out[0], g.ldc, g.M, g.batch, (uint64_t)g.ldc * es, batch_stride,
                              kStageCols, kStageRows, 128);
}

template <typename T, bool CONV>
int launch_pair(const GemmDesc& g, int bn, cudaStream_t stream) {
  constexpr int BK = 64;
  const size_t es = sizeof(T);
  CUtensorMap tmap_x, tmap_w;
  const uint64_t x_batch_stride = g.batch > 1 ? (uint64_t)g.stride_x * es : (uint64_t)g.M * g.K * es;
  const int taps = g.taps > 1 ? g.taps : 1;
  const int w_batches = taps > 1 ? taps : (g.w_mod > 1 ? g.w_mod : 1);
  const uint64_t w_batch_stride = taps > 1 ? (uint64_t)g.N * g.K * es
                                  : (w_batches > 1 ? (uint64_t)g.stride_w * es : (uint64_t)g.N * g.K * es);
  int rc = encode_tensor_map_3d(&tmap_x, g.x, g.K, g.M, g.batch, (uint64_t)g.K * es, x_batch_stride, BK, TM, BK * 2);
  if (rc != DFL_OK) return rc;
  rc = encode_tensor_map_3d(&tmap_w, g.w, g.K, g.N, w_batches, (uint64_t)g.K * es, w_batch_stride, BK, bn / 2, BK * 2);
  if (rc != DFL_OK) return rc;
  OutMaps tmap_out;
  int tiled = 0;
  rc = encode_output_maps<T>(g, &tmap_out, &tiled);
  if (rc != DFL_OK) return rc;

  auto kernel = gemm_tc_pair_kernel<T, CONV>;
  static KernelDeviceConfig config;   // per template instantiation
  int num_sms = 0;
  rc = configure_kernel(config, kernel, kPairSmem, &num_sms, "gemm_tc_pair_kernel");
  if (rc != DFL_OK) return rc;
  GemmDesc gd = g;
  if (!gd.status) {
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&gd.status), g_gemm_status);
    if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "status word: %s", cudaGetErrorString(e));
  }
  const int ncols = g.head_split ? g.N : g.ldc;
  const int tiles_n = (ncols + bn - 1) / bn, tiles_m = (g.M + 2 * TM - 1) / (2 * TM);
  const long long num_tiles = (long long)tiles_n * tiles_m * g.batch;
  if (num_tiles > 0x7fffffff) return fail(DFL_ERR_TOO_LARGE, "gemm_tc: too many tiles");
  const long long max_pairs = num_sms / 2;
  const int pairs = (int)(num_tiles < max_pairs ? num_tiles : max_pairs);
  const int num_kb = taps * ((g.K + BK - 1) / BK);
  cudaError_t le = launch_after_predecessor(kernel, dim3(2 * pairs), dim3(kThreads), kPairSmem, stream, tmap_x, tmap_w,
                                            tmap_out, gd, num_kb, tiles_n, tiles_m, (int)num_tiles, tiled, bn);
  if (le != cudaSuccess) return fail(DFL_ERR_LAUNCH, "gemm_tc_pair_kernel: %s", cudaGetErrorString(le));
  return check_launch("gemm_tc_pair_kernel");
}

// ------------------------------------------------------------------------------------------------ choice of kernel
// Cost of one GEMM in SM cycles, from the quantities that bound it: the MMA rate of the tile width, the rate at which
// an SM takes operands from L2, waves over the SMs, the accumulator drain, and the exchange of a split inner product.
// The constants were fitted to measured launches that loaded 128 rows of X for every tile, weights streaming from HBM, and an X
// load is still charged as 128 rows where a tile has fewer.  Against every plan at 172 sizes (32 to 16384 rows, N and K of hidden
// 768, 1024 and 1536), tiles loading the rows they have, the choice is 1.1 % above the best one on average (1.3 % at row counts
// that do not fill their tiles), within 5 % at 162 of them, and 26 % at worst (1024 x 1536 x 6144: 24.6 against 19.5 us).
// (Measured while an MMA of a narrow tile cost 60 cycles to issue; it costs 36 now, and the drain of a pair's tile is shorter.  The
// plans were not compared again.)
constexpr double kSmIngest = 83.0;      // operand bytes per cycle and SM ...
constexpr double kSharedIngest = 0.46;  // ... and how much slower when every SM pulls
constexpr double kDrain64 = 1460.0;     // draining 64 accumulator columns of a tile that nothing overlaps
constexpr double kTileStart = 1800.0, kPairStart = 8000.0, kNextWave = 1730.0, kPerCta = 15.0;
constexpr double kExchange = 1730.0, kExchangeBytes = 12.7;   // split: fixed cost, bytes per cycle between CTAs

struct GemmChoice {
  bool persistent;
  TilePlan tile;   // persistent: only bn
};

double mma_cycles(int bn, bool pair) {   // per 16-deep step of a 128- (pair: 256-) row tile, issue rate included
  const double wide = 0.508 * bn;
  const double floor_ = pair ? 40.0 : 33.0 + 0.25 * bn;
  return wide > floor_ ? wide : floor_;
}

GemmChoice choose_gemm(int M, int ncols, int K, int batch, int num_sms, bool may_pair) {
  GemmChoice best{};
  double best_cost = 1e30;
  const int kb = (K + 63) / 64;
  auto per_kb = [&](int bn, bool pair, double active) {
    const double mma = 4.0 * mma_cycles(bn, pair);
    const double load = (16384.0 + bn * (pair ? 64.0 : 128.0)) / kSmIngest * (1.0 + kSharedIngest * active / num_sms);
    return mma > load ? mma : load;
  };
  if (may_pair && K >= 64 && M >= 2 * TM) {
    for (int bn = 128; bn <= 256; bn += 64) {
      const long long tiles = (long long)((M + 255) / 256) * ((ncols + bn - 1) / bn) * batch, slots = num_sms / 2;
      const double waves = (double)((tiles + slots - 1) / slots);
      const double cost = kPairStart + waves * kb * per_kb(bn, true, 2.0 * (double)(tiles < slots ? tiles : slots)) + kDrain64 * bn / 64.0;
      if (cost < best_cost) {
        best_cost = cost;
        best = {true, {bn, 1, 1}};
      }
    }
  }
  const int splits[6] = {1, 2, 3, 4, 6, 8};
  for (int pair = 0; pair <= (may_pair && M > 128 ? 1 : 0); ++pair) {
    for (int bn = 32; bn <= 256; bn += 32) {
      const long long tiles = (long long)((M + (pair ? 255 : 127)) / (pair ? 256 : 128)) * ((ncols + bn - 1) / bn) * batch;
      for (int i = 0; i < 6; ++i) {
        const int split = splits[i], cluster = split * (pair ? 2 : 1);
        // a part of a split product takes whole 128-element k-blocks, at least two of them
        if (split > 1 && (bn % (16 * split) || kb < 4 * split || cluster > 8)) continue;
        const long long ctas = tiles * cluster;
        // clusters do not pack every SM of the GPU's processing clusters
        const long long slots = cluster <= 2 ? num_sms : (cluster <= 6 ? num_sms * 132 / 148 : num_sms * 112 / 148);
        const double waves = (double)((ctas + slots - 1) / slots), active = (double)(ctas < slots ? ctas : slots);
        double cost = kTileStart + waves * ((kb + split - 1) / split * per_kb(bn, pair != 0, active) + kDrain64 * bn / 64.0) +
                      (waves - 1.0) * kNextWave + kPerCta * active;
        if (split > 1) cost += kExchange + (split - 1.0) / split * (M < 128 ? M : 128) * bn * 4.0 / kExchangeBytes;
        if (cost < best_cost) {
          best_cost = cost;
          best = {false, {bn, split, pair}};
        }
      }
    }
  }
  return best;
}

// The choice is a function of the sizes alone; a forward asks for the same few over and over, so every host thread
// keeps the last ones.
GemmChoice cached_choice(int M, int ncols, int K, int batch, int num_sms, bool may_pair) {
  struct Entry {
    int key[5];
    GemmChoice choice;
  };
  static thread_local Entry table[64];
  const int key[5] = {M, ncols, K, batch, num_sms * 2 + (may_pair ? 1 : 0)};
  const uint32_t h = ((uint32_t)M * 2654435761u ^ (uint32_t)ncols * 40503u ^ (uint32_t)K * 97u ^ (uint32_t)batch * 7u) >> 3;
  Entry& e = table[h & 63u];
  if (memcmp(e.key, key, sizeof(key)) != 0) {
    e.choice = choose_gemm(M, ncols, K, batch, num_sms, may_pair);
    memcpy(e.key, key, sizeof(key));
  }
  return e.choice;
}

int device_sm_count(int* out) {
  static KernelDeviceConfig config;
  return configure_kernel(config, gemm_tc_pair_kernel<__half, false>, 0, out, "gemm_tc_pair_kernel");
}

template <typename T>
int launch_t(const GemmDesc& g, cudaStream_t stream) {
  if (g.K % 8) return fail(DFL_ERR_ALIGNMENT, "K=%d: rows must be multiples of 16 bytes for TMA", g.K);
  if (g.head_split && (g.head_dim % 32)) return fail(DFL_ERR_UNSUPPORTED, "head_dim must be a multiple of 32");
  if (!g.head_split && (g.ldc % 8)) return fail(DFL_ERR_ALIGNMENT, "ldc must be a multiple of 8");
  if (g.bias && !aligned16(g.bias)) return fail(DFL_ERR_ALIGNMENT, "bias not 16-byte aligned");
  int num_sms = 0;
  if (int rc = device_sm_count(&num_sms)) return rc;
  const int ncols = g.head_split ? g.N : g.ldc;
  const bool conv = g.taps > 1 || g.row_mask || g.activation == DFL_ACT_TANH;
  if (conv) {
    // long sequences: taps as k-steps of the persistent kernel; short ones: several sequences per tile
    if (g.K >= 64 && g.M >= 2 * TM) return launch_pair<T, true>(g, TN, stream);
    const int taps = g.taps > 1 ? g.taps : 1;
    const int rows = g.M <= TM ? (g.M * g.batch + TM - 1) / (TM / g.M * g.M) * TM : (g.M + TM - 1) / TM * TM * g.batch;
    return launch_gemm_tile(g, cached_choice(rows, ncols, g.K * taps, 1, num_sms, false).tile, stream);
  }
  const GemmChoice c = cached_choice(g.M, ncols, g.K, g.batch, num_sms, true);
  return c.persistent ? launch_pair<T, false>(g, c.tile.bn, stream) : launch_gemm_tile(g, c.tile, stream);
}

}  // namespace

int launch_gemm_tc(const GemmDesc& g, cudaStream_t stream) {
  if (g.dtype == DFL_F16) return launch_t<__half>(g, stream);
  if (g.dtype == DFL_BF16) return launch_t<__nv_bfloat16>(g, stream);
  return fail(DFL_ERR_UNSUPPORTED, "tcgen05 GEMM handles FP16/BF16 only");
}

}  // namespace dfl
