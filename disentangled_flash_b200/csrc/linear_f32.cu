// FP32 GEMM on the tensor cores without giving up FP32 accuracy: every operand is the exact sum of three bf16 planes.
//
//   x = x0 + x1 + x2,  |x1| <= 2^-8 |x|,  |x2| <= 2^-16 |x|        (split_planes_kernel; 8 + 8 + 8 significant bits)
//   x . w = x0.w0 + (x0.w1 + x1.w0) + (x0.w2 + x1.w1 + x2.w0) + terms below 2^-23 |x| |w|, which are left out
//
// Each bf16 product is exact in fp32; what the left-out terms (x1.w2, x2.w1: 2^-26 |x||w| rms) add is below the one
// rounding (2^-24 of the running sum) that a fp32 fused multiply-add makes per term.  The tensor core adds a 16-deep
// step into its fp32 accumulator with truncation, so one accumulator never holds more than one 64-deep k-block: within a
// block the five small products come first (their truncation is at 2^-8 of the block's sum) and the four x0.w0 steps
// last, and the epilogue warps add the finished block to sums in registers, rounded to nearest, while the MMA warp fills
// the other accumulator.  Against an fp64 product the result is at least as accurate as the sequential fp32 chain of the
// CUDA-core kernel this replaces on the prepared paths (tests/test_gpu_f32_tensor.py).
// Infinities and NaN come out as a fp32 multiply-add chain gives them (f32_planes.cuh), except beside operands below 2^-134,
// whose leading plane is zero.
//
// What bounds it: six bf16 MMAs per product, a sixth of the bf16 tensor rate; a k-block brings 96 KB for 24 MMAs of a
// 256 x 256 pair tile (3.1 k cycles), far below what an SM can take from L2.
// One tile per CTA (128 rows) or CTA pair (256 rows) x bn columns, inner product optionally split over a cluster, as in
// linear_tile.cu.  Warps 0-7 epilogue, 8 TMA, 9 MMA.
#include "f32_planes.cuh"
#include "linear_epilogue.cuh"

namespace dfl {

__device__ int g_gemm_f32_status = 0;

namespace {

constexpr int kRows = 128, BK = 64;
constexpr int kPlaneA = kRows * BK * 2;
constexpr int kTmaWarp = 8, kMmaWarp = 9, kThreads = 320, kMaxStages = 4, kMaxSmem = 232448;
constexpr int kWaits = kWaitsGemmF32;

struct F32Args {
  int split, stages, num_kb, tiles_m, tiles_n;
  uint32_t ring_bytes;   // operand ring; behind it the receive buffer of a split inner product
};

// planes[q][i] of x[i]; HBM bound (4 bytes in, 6 out).
__global__ void __launch_bounds__(256) split_planes_kernel(const float4* __restrict__ x, uint2* __restrict__ planes, long long n4) {
  wait_for_predecessor();
  release_successor();
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n4; i += gridDim.x * 256ll) {
    const float4 v = x[i];
    const float f[4] = {v.x, v.y, v.z, v.w};
    uint2 out[kPlanes];
    split3x4(f, out);
#pragma unroll
    for (int q = 0; q < kPlanes; ++q) planes[q * n4 + i] = out[q];
  }
}

// Keeps planes equal to the matrices they were made from: compares a digest of every 4 KB piece (1024 elements) with the one
// stored when its planes were written, and splits the piece again where they differ.  A warp per piece; HBM bound, 4 bytes
// per element (a split reads 4 and writes 6): 46 us for 12 layers of hidden 768 (63.7 M elements), 297 us for 24 of 1536
// (510 M, 6.9 TB/s); 138 and 864 us where everything has changed.  Splitting every matrix anew at each layer of each forward
// cost 190 and 630 us.
// The digest is two 64-bit sums over the element's bits x_i and fixed keys k_i: sum (x_2i + k_2i)(x_2i+1 + k_2i+1), the NH
// hash of Black, Halevi, Krawczyk, Krovetz and Rogaway (UMAC, CRYPTO 1999), and sum x_i (k_i | 1).  One changed element always
// shows (an odd factor is invertible mod 2^64); several leave both sums as they were with a chance of about 2^-64.
constexpr int kPieceVecs = DFL_PLANE_PIECE / 4 / 32;   // float4 per lane
__global__ void __launch_bounds__(256, 3) refresh_planes_kernel(const DflPlaneSource* __restrict__ sources, int n_sources, long long n_pieces) {
  wait_for_predecessor();
  release_successor();
  const int lane = threadIdx.x & 31;
  const uint32_t seed = (uint32_t)(lane + 1) * 0x9E3779B1u;
  int at = 0;
  for (long long piece = blockIdx.x * 8ll + (threadIdx.x >> 5); piece < n_pieces; piece += gridDim.x * 8ll) {
    while (at + 1 < n_sources && piece >= sources[at + 1].first_piece) ++at;
    const DflPlaneSource src = sources[at];
    const long long n4 = src.n / 4, local = piece - src.first_piece, first = local * (DFL_PLANE_PIECE / 4) + lane;
    float4 v[kPieceVecs];
    ulonglong2* digest = reinterpret_cast<ulonglong2*>(src.digests) + local;
    const ulonglong2 then = *digest;
#pragma unroll
    for (int j = 0; j < kPieceVecs; ++j)
      v[j] = first + 32 * j < n4 ? __ldcs(reinterpret_cast<const float4*>(src.w) + first + 32 * j) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    unsigned long long nh = 0, linear = 0;
#pragma unroll
    for (int j = 0; j < kPieceVecs; ++j) {
      const uint32_t x[4] = {__float_as_uint(v[j].x), __float_as_uint(v[j].y), __float_as_uint(v[j].z), __float_as_uint(v[j].w)};
      uint32_t k[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        k[c] = seed * (2u * (uint32_t)(4 * j + c) * 0x45D9F3Bu + 0x2C1B3C6Du);
        k[c] ^= k[c] >> 15;
        linear += (unsigned long long)x[c] * (k[c] | 1u);
      }
      nh += (unsigned long long)(x[0] + k[0]) * (x[1] + k[1]) + (unsigned long long)(x[2] + k[2]) * (x[3] + k[3]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      nh += __shfl_xor_sync(0xffffffffu, nh, o);
      linear += __shfl_xor_sync(0xffffffffu, linear, o);
    }
    if (then.x == nh && then.y == linear) continue;   // warp-uniform
    uint2* planes = reinterpret_cast<uint2*>(src.planes);
#pragma unroll
    for (int j = 0; j < kPieceVecs; ++j) {
      if (first + 32 * j >= n4) break;
      const float f[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
      uint2 out[kPlanes];
      split3x4(f, out);
#pragma unroll
      for (int q = 0; q < kPlanes; ++q) planes[q * n4 + first + 32 * j] = out[q];
    }
    __threadfence();   // another stream that sees the digest sees the planes
    __syncwarp();
    if (lane == 0) *digest = make_ulonglong2(nh, linear);
  }
}

// The finished sums of the warp's 32 rows (first output row m0, `rows_live` of them inside the output) and its chunks of 32 columns
// within [begin, end) of the tile, from shared memory, so that eight lanes store one row segment: bias, activation, row-major or
// head-major, in fp32 or as bf16 planes.  `sums`: the warp's first row at the tile's column `begin`, `pitch` bytes from row to row.
// Two rows at a time in one rolled loop: with a row at a time, its place divided out again for every chunk, and infinities looked
// for element by element, a tile of 128 columns took 10.8 k cycles here, after 18.4 k of MMAs (1024 x 2304 x 768).  The kernels of 192 and
// 256 columns hold their sums in registers around it and spill a little more for it: 60 / 136 and 68 / 156 bytes stored / loaded (12 / 4
// and 44 / 72 before).
template <int NCH>
__device__ __forceinline__ void store_sums(const GemmDesc& g, const unsigned char* sums, uint32_t pitch, const float* bias, int m0,
                                           int rows_live, int z, int n0, int ncols, int begin, int end, int side, int lane) {
  const int v = lane & 7, hd = g.heads * g.head_dim;
  const long long plane = g.head_split ? (long long)g.M * hd : (long long)g.M * g.ldc;   // elements of one plane of an output
#pragma unroll 1
  for (int it = 0; it < 8; it += 2) {
    long long place[2];   // element offset of the row
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int m = m0 + (it + u) * 4 + (lane >> 3);
      if (g.head_split) {
        const int b = m / g.rows_per_seq, l = m - b * g.rows_per_seq;
        place[u] = ((long long)b * g.heads * g.rows_per_seq + l) * g.head_dim;
      } else {
        place[u] = (long long)z * g.stride_c + (long long)m * g.ldc;
      }
    }
#pragma unroll 1
    for (int i = 0; i < NCH; ++i) {
      const int c = 64 * i + 32 * side, n = n0 + c;
      if (c < begin || c >= end || n >= ncols) continue;   // warp-uniform
      void* out = g.out[0];
      long long column = n;
      if (g.head_split) {
        const int which = n / hd, rem = n - which * hd, h = rem / g.head_dim;
        out = which == 0 ? g.out[0] : (which == 1 ? g.out[1] : g.out[2]);
        column = (long long)h * g.rows_per_seq * g.head_dim + (rem - h * g.head_dim);
      }
      const float4 b4 = *reinterpret_cast<const float4*>(bias + c + 4 * v);
      float f[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float4 x = *reinterpret_cast<const float4*>(sums + (uint32_t)((it + u) * 4 + (lane >> 3)) * pitch + (uint32_t)(c - begin + 4 * v) * 4u);
        f[u][0] = x.x + b4.x;
        f[u][1] = x.y + b4.y;
        f[u][2] = x.z + b4.z;
        f[u][3] = x.w + b4.w;
      }
      if (g.activation == DFL_ACT_GELU) {
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int j = 0; j < 4; ++j) f[u][j] = gelu_erf_exact(f[u][j]);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        uint2 w[kPlanes];
        if (g.out_planes) split3x4(f[u], w);
        if ((it + u) * 4 + (lane >> 3) >= rows_live || n + 4 * v >= ncols) continue;
        const long long at = place[u] + column + 4 * v;
        if (g.out_planes) {
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(out) + at;
#pragma unroll
          for (int q = 0; q < kPlanes; ++q) *reinterpret_cast<uint2*>(dst + q * plane) = w[q];
        } else {
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + at) = make_float4(f[u][0], f[u][1], f[u][2], f[u][3]);
        }
      }
    }
  }
}

// NCH: 64-column chunks per tile (bn = 64 * NCH).
template <bool PAIR, int NCH>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const GemmDesc g,
                const F32Args a) {
  constexpr int bn = 64 * NCH, w_rows = PAIR ? bn / 2 : bn;
  constexpr uint32_t kTmemCols = 2 * bn <= 128 ? 128 : (2 * bn <= 256 ? 256 : 512);
  constexpr uint32_t plane_w = w_rows * BK * 2, a_bytes = kPlanes * kPlaneA, stage_bytes = a_bytes + kPlanes * plane_w;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* acc_full = empty_bar + kMaxStages;    // [2] a k-block's sums are complete
  uint64_t* acc_empty = acc_full + 2;             // [2] ... and have been added to the registers
  uint64_t* recv_bar = acc_empty + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(recv_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  float* bias_s = reinterpret_cast<float*>(smem + 1024);
  unsigned char* ring = smem + 2048;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const uint32_t leader = PAIR ? (rank & ~1u) : rank, half = PAIR ? (rank & 1u) : 0u;
  const int part = PAIR ? (int)(rank >> 1) : (int)rank;
  const int tile = blockIdx.x / (a.split * (PAIR ? 2 : 1));
  const int per_z = a.tiles_n * a.tiles_m;
  const int z = tile / per_z, rem = tile - z * per_z;
  const int tm = rem / a.tiles_n, n0 = (rem - tm * a.tiles_n) * bn;
  const int row0 = tm * (PAIR ? 2 * kRows : kRows) + (int)half * kRows;
  const int out_rows = g.M - row0 < 0 ? 0 : (g.M - row0 < kRows ? g.M - row0 : kRows);
  const int kb_begin = part * a.num_kb / a.split, kb_end = (part + 1) * a.num_kb / a.split;
  const int n_kb = kb_end - kb_begin;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&acc_full[i], 1);
      ptx::mbar_init(&acc_empty[i], PAIR ? 16 : 8);   // epilogue warps (of both CTAs, the leader's barrier)
    }
    ptx::mbar_init(recv_bar, 1);
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == kTmaWarp && lane == 0) {
    ptx::prefetch_tensormap(&tmap_x);
    ptx::prefetch_tensormap(&tmap_w);
  }
  if (warp == kMmaWarp) {
    if (PAIR) {
      ptx::tmem_alloc_pair(tmem_holder, kTmemCols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(tmem_holder, kTmemCols);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (PAIR || a.split > 1) ptx::cluster_sync_all();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == kTmaWarp) {
    const uint32_t ring_addr = ptx::smem_u32(ring), full_addr = ptx::smem_u32(full_bar);
    const uint32_t full_remote = PAIR ? ptx::map_to_cta(full_addr, leader) : full_addr;
    const int w_z = z % g.w_mod;
    auto load_w = [&](int kb, int s) {
      if (half == 0) ptx::mbar_arrive_expect_tx_warp(full_addr + 8u * s, (PAIR ? 2u : 1u) * stage_bytes);
      ptx::tma_load_4d_warp<PAIR>(ring_addr + s * stage_bytes + a_bytes, &tmap_w, full_remote + 8u * s, kb * BK,
                                  n0 + (int)half * w_rows, 0, w_z);
    };
    auto load_x = [&](int kb, int s) {
      ptx::tma_load_4d_warp<PAIR>(ring_addr + s * stage_bytes, &tmap_x, full_remote + 8u * s, kb * BK, row0, 0, z);
    };
    const int ahead = n_kb < a.stages ? n_kb : a.stages;
    if (!g.weights_early) wait_for_predecessor();
    for (int i = 0; i < ahead; ++i) load_w(kb_begin + i, i);
    if (g.weights_early) wait_for_predecessor();
    for (int i = 0; i < ahead; ++i) load_x(kb_begin + i, i);
    release_successor();
    int s = 0;
    uint32_t ph = 0;
    for (int i = ahead; i < n_kb; ++i) {
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&empty_bar[s], ph, abort_flag, g.status, kWaits + 41))) break;
      load_w(kb_begin + i, s);
      load_x(kb_begin + i, s);
      if (++s == a.stages) {
        s = 0;
        ph ^= 1u;
      }
    }
  } else if (warp == kMmaWarp) {
    if (half == 0 && ptx::elect_one()) {   // one lane, see umma_ss_f16_words
      constexpr uint32_t idesc = ptx::make_idesc_f16(1, PAIR ? 2 * kRows : kRows, bn, 0, 0);
      constexpr uint32_t mode = ptx::swizzle_mode_for_row_bytes(BK * 2);
      const uint64_t desc0 = ptx::make_smem_desc(ptx::smem_u32(ring), 16, 8 * BK * 2, mode);
      const uint32_t first = (uint32_t)desc0, upper = (uint32_t)(desc0 >> 32);
      // The next k-block's two barriers are looked at between the products of this one: answered only after the last of them, they
      // leave the tensor pipe idle for 340 cycles of a k-block of 1.6 k (128 columns) or 3.1 k (256).
      bool landed = false, free = false;
      int s = 0;
      uint32_t ph = 0, desc = first;
      for (int i = 0; i < n_kb; ++i) {
        const int acc = i & 1;
        if (!landed && !ptx::mbar_wait(&full_bar[s], ph, abort_flag, g.status, kWaits + 42)) break;
        if (!free && !ptx::mbar_wait(&acc_empty[acc], ((uint32_t)(i >> 1) & 1u) ^ 1u, abort_flag, g.status, kWaits + 44)) break;
        ptx::tc_fence_after();
        const uint32_t ad = desc, bd = desc + (a_bytes >> 4), d_tmem = tmem_base + (uint32_t)(acc * bn);
        uint64_t* done = &empty_bar[s];
        desc += stage_bytes >> 4;
        if (++s == a.stages) {
          s = 0;
          ph ^= 1u;
          desc = first;
        }
        // (plane of X, plane of W), smallest products first
        constexpr int px[6] = {2, 1, 0, 1, 0, 0}, pw[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          if (q == 4) {
            landed = i + 1 < n_kb && ptx::mbar_test(&full_bar[s], ph);
            free = ptx::mbar_test(&acc_empty[acc ^ 1], ((uint32_t)((i + 1) >> 1) & 1u) ^ 1u);
          }
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            ptx::umma_ss_f16_words<PAIR>(d_tmem, ad + (uint32_t)(px[q] * (kPlaneA >> 4) + 2 * k), bd + (uint32_t)(pw[q] * (plane_w >> 4) + 2 * k),
                                         upper, idesc, q != 0 || k != 0 ? 1u : 0u);
        }
        ptx::umma_commit_one<PAIR>(done, leader);
        ptx::umma_commit_one<PAIR>(&acc_full[acc], leader);
      }
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3, side = warp >> 2;   // this warp's chunks: columns 64 * i + 32 * side
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(side * 32);
    const int ncols = g.head_split ? g.N : g.ldc;
    if (!g.weights_early) wait_for_predecessor();
    for (int c = threadIdx.x; c < bn; c += 256)
      bias_s[c] = g.bias && n0 + c < g.N ? reinterpret_cast<const float*>(g.bias)[n0 + c] : 0.0f;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (g.weights_early) wait_for_predecessor();
    float sum[NCH][32];
#pragma unroll
    for (int i = 0; i < NCH; ++i)
#pragma unroll
      for (int j = 0; j < 32; ++j) sum[i][j] = 0.0f;
    bool ready = true;
    const uint32_t acc_empty_leader = PAIR ? ptx::map_to_cta(ptx::smem_u32(acc_empty), leader) : ptx::smem_u32(acc_empty);
    for (int kb = 0; kb < n_kb; ++kb) {
      const int acc = kb & 1;
      ready = ready && ptx::mbar_wait(&acc_full[acc], (uint32_t)(kb >> 1) & 1u, abort_flag, g.status, kWaits + 43);
      ready = __all_sync(0xffffffffu, ready);
      if (!ready) break;
      ptx::tc_fence_after();
#pragma unroll
      for (int i = 0; i < NCH; ++i) {
        float v[32];
        ptx::tmem_ld32_f(taddr + (uint32_t)(acc * bn + 64 * i), v);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[i][j] += v[j];
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        // (an arrive that also ordered memory at cluster scope, once a k-block, cost an encoder of 8 x 128 tokens 4 %)
        if (PAIR) ptx::mbar_arrive_peer(acc_empty_leader + 8u * acc);
        else ptx::mbar_arrive(&acc_empty[acc]);
      }
    }
    int rows_live = out_rows - quarter * 32;
    if (!ready) rows_live = 0;
    const int r = quarter * 32 + lane, m0 = row0 + quarter * 32;
    if (a.split == 1) {
      // the sums go where the operands were: every warp's last block is complete, so every MMA has read them
      asm volatile("bar.sync 1, 256;" ::: "memory");
      constexpr uint32_t pitch = bn * 4 + 16;
#pragma unroll
      for (int i = 0; i < NCH; ++i) {
        float4* row = reinterpret_cast<float4*>(ring + (uint32_t)r * pitch) + (64 * i + 32 * side) / 4;
#pragma unroll
        for (int j = 0; j < 8; ++j) row[j] = make_float4(sum[i][4 * j], sum[i][4 * j + 1], sum[i][4 * j + 2], sum[i][4 * j + 3]);
      }
      __syncwarp();
      store_sums<NCH>(g, ring + (uint32_t)(quarter * 32) * pitch, pitch, bias_s, m0, rows_live, z, n0, ncols, 0, bn, side, lane);
    } else {
      // Exchange as in gemm_tile_kernel: part p finishes columns [p * unit, (p + 1) * unit), unit a multiple of 32.
      const int unit = bn / a.split;
      const uint32_t pitch = (uint32_t)(unit * 4 + 16), slot_bytes = (uint32_t)kRows * pitch;
      asm volatile("bar.sync 1, 256;" ::: "memory");   // every warp has added its last block: the ring is idle
#pragma unroll
      for (int i = 0; i < NCH; ++i) {
        const int c = 64 * i + 32 * side, dst_part = c / unit;
        if (dst_part == part || r >= out_rows) continue;
        const int q = dst_part > part ? dst_part - part : dst_part - part + a.split;
        float4* row = reinterpret_cast<float4*>(ring + (uint32_t)(q - 1) * slot_bytes + (uint32_t)r * pitch) + (c - dst_part * unit) / 4;
#pragma unroll
        for (int j = 0; j < 8; ++j) row[j] = make_float4(sum[i][4 * j], sum[i][4 * j + 1], sum[i][4 * j + 2], sum[i][4 * j + 3]);
      }
      ptx::fence_proxy_async_smem();
      asm volatile("bar.sync 1, 256;" ::: "memory");
      const uint32_t share = (uint32_t)out_rows * pitch;
      if (threadIdx.x == 0) {
        ptx::mbar_arrive_expect_tx(recv_bar, share * (uint32_t)(a.split - 1));
        for (int q = 1; q < a.split && share != 0; ++q) {
          const int dst_part = part + q < a.split ? part + q : part + q - a.split;
          const uint32_t dst_rank = PAIR ? 2u * (uint32_t)dst_part + half : (uint32_t)dst_part;
          const uint32_t slot = (uint32_t)(part < dst_part ? part : part - 1);
          ptx::bulk_copy_to_cta(ptx::map_to_cta(ptx::smem_u32(ring) + a.ring_bytes + slot * slot_bytes, dst_rank),
                                ptx::smem_u32(ring) + (uint32_t)(q - 1) * slot_bytes, share,
                                ptx::map_to_cta(ptx::smem_u32(recv_bar), dst_rank));
        }
      }
      __syncwarp();
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(recv_bar, 0, abort_flag, g.status, kWaits + 45))) rows_live = 0;
      unsigned char* recv = ring + a.ring_bytes;   // the first sender's slot takes the finished sums
#pragma unroll
      for (int i = 0; i < NCH; ++i) {
        const int c = 64 * i + 32 * side;
        if (c / unit != part || r >= out_rows) continue;
        float4* own = reinterpret_cast<float4*>(recv + (uint32_t)r * pitch) + (c - part * unit) / 4;
        for (int p = 0; p < a.split - 1; ++p) {
          const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const unsigned char*>(own) + (uint32_t)p * slot_bytes);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 s4 = src[j];
            sum[i][4 * j] += s4.x; sum[i][4 * j + 1] += s4.y; sum[i][4 * j + 2] += s4.z; sum[i][4 * j + 3] += s4.w;
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) own[j] = make_float4(sum[i][4 * j], sum[i][4 * j + 1], sum[i][4 * j + 2], sum[i][4 * j + 3]);
      }
      __syncwarp();
      store_sums<NCH>(g, recv + (uint32_t)(quarter * 32) * pitch, pitch, bias_s, m0, rows_live, z, n0, ncols, part * unit,
                      (part + 1) * unit, side, lane);
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (PAIR || a.split > 1) ptx::cluster_sync_all_relaxed();
  ptx::tc_fence_after();
  if (warp == kMmaWarp) {
    if (PAIR) ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
    else ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <bool PAIR, int NCH>
int launch_plan(const GemmDesc& g, int split, cudaStream_t stream) {
  constexpr int bn = 64 * NCH, w_rows = PAIR ? bn / 2 : bn, stage = kPlanes * (kPlaneA + w_rows * BK * 2);
  F32Args a{};
  a.split = split;
  a.num_kb = (g.K + BK - 1) / BK;
  const int ncols = g.head_split ? g.N : g.ldc;
  a.tiles_n = (ncols + bn - 1) / bn;
  a.tiles_m = (g.M + (PAIR ? 2 : 1) * kRows - 1) / ((PAIR ? 2 : 1) * kRows);
  const int w_batches = g.w_mod > 1 ? g.w_mod : 1;
  CUtensorMap tmap_x, tmap_w;
  const uint64_t row = (uint64_t)g.K * 2;
  int rc = encode_tensor_map_4d(&tmap_x, g.x, {(uint64_t)g.K, (uint64_t)g.M, kPlanes, (uint64_t)g.batch},
                                {row, (uint64_t)g.batch * g.M * row, (uint64_t)g.M * row}, {BK, kRows, kPlanes, 1});
  if (rc != DFL_OK) return rc;
  rc = encode_tensor_map_4d(&tmap_w, g.w, {(uint64_t)g.K, (uint64_t)g.N, kPlanes, (uint64_t)w_batches},
                            {row, (uint64_t)w_batches * g.N * row, (uint64_t)g.N * row}, {BK, (uint32_t)w_rows, kPlanes, 1});
  if (rc != DFL_OK) return rc;

  auto kernel = gemm_f32_kernel<PAIR, NCH>;
  static KernelDeviceConfig config;   // per template instantiation
  rc = configure_kernel(config, kernel, kMaxSmem, nullptr, "gemm_f32_kernel");
  if (rc != DFL_OK) return rc;
  const int recv = split > 1 ? (split - 1) * kRows * (bn / split * 4 + 16) : 0;
  const int kb_cta = (a.num_kb + split - 1) / split;
  a.stages = (kMaxSmem - 3072 - recv) / stage;
  if (a.stages > kb_cta) a.stages = kb_cta;
  if (a.stages > kMaxStages) a.stages = kMaxStages;
  if (a.stages < 1) return fail(DFL_ERR_UNSUPPORTED, "gemm_f32: %d columns in %d parts do not fit", bn, split);
  const int need = split > 1 ? recv : kRows * (bn * 4 + 16);   // parked shares, or the finished sums, where the operands were
  a.ring_bytes = (uint32_t)(a.stages * stage > need ? a.stages * stage : need);
  const int smem = 3072 + (int)a.ring_bytes + recv;
  const int cluster = split * (PAIR ? 2 : 1);
  const long long ctas = (long long)a.tiles_n * a.tiles_m * g.batch * cluster;
  if (ctas > 0x7fffffff) return fail(DFL_ERR_TOO_LARGE, "gemm_f32: too many tiles");
  GemmDesc gd = g;
  if (!gd.status) {
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&gd.status), g_gemm_f32_status);
    if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "status word: %s", cudaGetErrorString(e));
  }
  cudaError_t e = launch_clusters_after_predecessor(kernel, dim3((unsigned)ctas), dim3(kThreads), cluster, (size_t)smem, stream,
                                                    tmap_x, tmap_w, gd, a);
  if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "gemm_f32_kernel: %s", cudaGetErrorString(e));
  return check_launch("gemm_f32_kernel");
}

// Tile, pair and split by the same considerations as choose_gemm (linear_tc.cu), with six MMAs per product: nearly every
// size is bound by the MMA rate times the waves over the SMs.  (The cycles of an MMA and of a tile's end were measured while a
// converged warp issued the MMAs and finished tiles left a row at a time; the plans were not compared again.)
struct F32Choice {
  int pair, nch, split;
};
F32Choice choose_f32(int M, int ncols, int K, int batch, int num_sms) {
  const F32Choice shapes[5] = {{0, 1, 1}, {0, 2, 1}, {1, 2, 1}, {1, 3, 1}, {1, 4, 1}};
  F32Choice best = shapes[0];
  double best_cost = 1e30;
  const int kb = (K + BK - 1) / BK;
  for (const F32Choice& c : shapes) {
    if (c.pair && M <= kRows) continue;
    const int bn = 64 * c.nch, rows = c.pair ? 256 : 128;
    const double mma = 24.0 * (c.pair ? 0.508 * bn : (bn == 64 ? 49.0 : 65.0));
    const double load = 3.0 * (16384.0 + bn * (c.pair ? 64.0 : 128.0)) / 60.0;
    const long long tiles = (long long)((M + rows - 1) / rows) * ((ncols + bn - 1) / bn) * batch;
    for (int split = 1; split <= 4; ++split) {
      const int cluster = split * (c.pair ? 2 : 1);
      if (split > 1 && (bn % (32 * split) || kb < 2 * split || cluster > 8)) continue;
      const long long slots = cluster <= 2 ? num_sms : num_sms * 128 / 148, ctas = tiles * cluster;
      const double waves = (double)((ctas + slots - 1) / slots);
      double cost = waves * ((kb + split - 1) / split * (mma > load ? mma : load) + 3500.0 + 300.0 * c.nch);
      if (split > 1) cost += 1700.0 + (split - 1.0) / split * (M < 128 ? M : 128) * bn * 4.0 / 12.7;
      if (cost < best_cost) {
        best_cost = cost;
        best = {c.pair, c.nch, split};
      }
    }
  }
  return best;
}

}  // namespace

int launch_split_planes(const void* x, void* planes, long long n, cudaStream_t stream) {
  const long long n4 = n / 4, wanted = (n4 + 255) / 256;
  const int blocks = (int)(wanted < 148 * 8 ? wanted : 148 * 8);
  cudaError_t e = launch_after_predecessor(split_planes_kernel, dim3(blocks), dim3(256), 0, stream, (const float4*)x, (uint2*)planes, n4);
  if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "split_planes_kernel: %s", cudaGetErrorString(e));
  return check_launch("split_planes_kernel");
}

int launch_refresh_planes(const DflPlaneSource* sources, int n_sources, long long n_pieces, cudaStream_t stream) {
  const long long wanted = (n_pieces + 7) / 8, cap = 148 * 6;
  cudaError_t e = launch_after_predecessor(refresh_planes_kernel, dim3((unsigned)(wanted < cap ? wanted : cap)), dim3(256), 0, stream,
                                           sources, n_sources, n_pieces);
  if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "refresh_planes_kernel: %s", cudaGetErrorString(e));
  return check_launch("refresh_planes_kernel");
}

int launch_gemm_f32_planes(const GemmDesc& g, cudaStream_t stream) {
  if (g.K % 8) return fail(DFL_ERR_ALIGNMENT, "K=%d: plane rows must be multiples of 16 bytes for TMA", g.K);
  if (g.head_split ? g.head_dim % 32 : g.ldc % 8) return fail(DFL_ERR_UNSUPPORTED, "head_dim or ldc not covered");
  static KernelDeviceConfig config;
  int num_sms = 0;
  if (int rc = configure_kernel(config, split_planes_kernel, 0, &num_sms, "gemm_f32_kernel")) return rc;
  const F32Choice c = choose_f32(g.M, g.head_split ? g.N : g.ldc, g.K, g.batch, num_sms);
  if (!c.pair) return c.nch == 1 ? launch_plan<false, 1>(g, c.split, stream) : launch_plan<false, 2>(g, c.split, stream);
  return c.nch == 2 ? launch_plan<true, 2>(g, c.split, stream)
                    : (c.nch == 3 ? launch_plan<true, 3>(g, c.split, stream) : launch_plan<true, 4>(g, c.split, stream));
}

}  // namespace dfl
