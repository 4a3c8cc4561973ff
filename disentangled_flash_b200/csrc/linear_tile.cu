// tcgen05 GEMM for the sizes at which a 256 x 256 tile leaves SMs idle: one output tile of 128 (or, with a CTA pair,
// 256) rows by `bn` columns per CTA, the width and the number of CTAs that share a tile's inner product chosen at
// launch so that one wave covers the GPU.
//
//   C_z[m,n] = act( sum_k X_z[m,k] * W_{z % w_mod}[n,k] + bias[n] )     (GemmDesc; head-split or row-major output)
//
// What bounds it: with a few hundred rows the whole GEMM is 1-3 us of memory time, so what counts is the chain
// launch -> first operand bytes -> k-steps -> store.  Hence
//   * narrow tiles: a tile's k-steps run at the rate of its operand loads; many CTAs with little each load in parallel;
//   * `split` CTAs of a cluster take consecutive k-ranges of one tile and exchange their fp32 accumulators through
//     distributed shared memory (each CTA finishes bn / split columns): K = 3072 at N = 768 has too few tiles otherwise;
//   * the operand ring holds as many k-blocks as shared memory has room for, so all loads of a short inner product are
//     in flight at once;
//   * with `weights_early` the W blocks are requested before the predecessor kernel has finished (they do not depend
//     on it), and the successor is released at once, so that its set-up and its W loads overlap this kernel.
// Warps 0-7 epilogue (32 TMEM lanes x alternate 32-column chunks each), warp 8 TMA, warp 9 MMA issuer and TMEM owner.
#include <type_traits>

#include "linear_epilogue.cuh"

namespace dfl {

__device__ int g_gemm_tile_status = 0;

namespace {

constexpr int kRows = 128;               // rows per CTA (= TMEM lanes)
constexpr int BK = 64;                   // k-block: one 128-byte swizzle row of 2-byte elements
constexpr int kTileA = kRows * BK * 2;   // 16 KB
constexpr int kEpilogueWarps = 8, kTmaWarp = 8, kMmaWarp = 9;
constexpr int kThreads = 320;
constexpr int kMaxStages = 16;
constexpr int kMaxSmem = 232448;
constexpr int kWaits = kWaitsGemmTile;

struct TileArgs {
  int bn, split, stages;
  int num_kb, kb_per_tap;     // k-blocks (of 64 * pieces elements) of the whole inner product, and of one tap
  int pieces;                 // 64-element pieces per k-block: 1 or 2
  int tiles_m, tiles_n;
  int rows;                   // rows per CTA, at most 128
  int seqs_per_tile;          // convolution with short sequences: sequences per tile (else 0)
  int tmem_cols;
  uint32_t ring_bytes;        // operand ring; behind it the receive buffer of a split inner product
  uint32_t recv_bytes;
  uint32_t x_bytes;           // bytes of one X load (a tile of few rows or short sequences holds fewer than 128)
  uint32_t x_piece;           // bytes from one 64-element piece of it to the next
};

// Where an output row starts: row-major, or head-major (the three outputs share the offset of sequence and position).
struct RowPlace {
  long long base;   // elements
};
__device__ __forceinline__ RowPlace place_row(const GemmDesc& g, int m, int z) {
  RowPlace p;
  if (g.head_split) {
    const int row = g.row_groups ? __ldg(g.row_groups + (m >> 5)) + (m & 31) : m;
    const int b = row / g.rows_per_seq, l = row - b * g.rows_per_seq;
    p.base = ((long long)b * g.heads * g.rows_per_seq + l) * g.head_dim;
  } else {
    p.base = (long long)z * g.stride_c + (long long)m * g.ldc;
  }
  return p;
}

// NC (16 or 32) consecutive columns of 32 output rows, one row per lane, n a multiple of NC: bias (fp32, shared memory),
// activation, rounding; the warp's block goes through `stage` (32 x NC elements) so that NC / 8 neighbouring lanes store
// one row segment (a store of 32 separate rows costs the memory pipe 32 passes, and at 128 x 128 per CTA those passes,
// not the math, were the epilogue: 1.7 us against 0.5 us).  `ncols` ends the row (a multiple of 8).
template <typename T, bool CONV, int NC>
__device__ __forceinline__ void emit(const GemmDesc& g, const float (&acc)[NC], const float* bias, unsigned char* stage,
                                     const RowPlace& place, bool live, int n, int ncols, bool keep_row, int lane) {
  constexpr int C = NC / 8;   // 16-byte chunks per row
  // Two warps per scheduler run this: every step is written over all columns at once, so that the latencies overlap.
  float f[NC];
#pragma unroll
  for (int v = 0; v < NC / 4; ++v) {
    const float4 b = *reinterpret_cast<const float4*>(bias + v * 4);
    f[4 * v] = acc[4 * v] + b.x;
    f[4 * v + 1] = acc[4 * v + 1] + b.y;
    f[4 * v + 2] = acc[4 * v + 2] + b.z;
    f[4 * v + 3] = acc[4 * v + 3] + b.w;
  }
  if (CONV && !keep_row) {
#pragma unroll
    for (int j = 0; j < NC; ++j) f[j] = 0.0f;
  }
  if (g.activation == DFL_ACT_GELU) {
#pragma unroll
    for (int j = 0; j < NC; j += 2) gelu_pair<T>(f[j], f[j + 1]);
  } else if (CONV && g.activation == DFL_ACT_TANH) {
#pragma unroll
    for (int j = 0; j < NC; ++j) f[j] = tanh_fast(f[j]);
  }
  uint4 packed[C];
#pragma unroll
  for (int v = 0; v < C; ++v) {
    T* ph = reinterpret_cast<T*>(&packed[v]);
#pragma unroll
    for (int j = 0; j < 8; ++j) ph[j] = Elem<T>::from_f(f[8 * v + j]);
  }
  __syncwarp();               // the warp's previous block has left the staging buffer
#pragma unroll
  for (int v = 0; v < C; ++v)   // eight consecutive lanes write to eight different 16-byte bank groups
    *reinterpret_cast<uint4*>(stage + lane * (NC * 2) + ((v ^ (C == 4 ? (lane >> 1) & 3 : (lane >> 2) & 1)) << 4)) = packed[v];
  __syncwarp();
  T* out = reinterpret_cast<T*>(g.out[0]);
  long long column = n;
  if (g.head_split) {
    const int hd = g.heads * g.head_dim;
    const int which = n / hd, rem = n - which * hd;
    const int h = rem / g.head_dim, dd = rem - h * g.head_dim;
    out = reinterpret_cast<T*>(which == 0 ? g.out[0] : (which == 1 ? g.out[1] : g.out[2]));
    column = (long long)h * g.rows_per_seq * g.head_dim + dd;
  }
  const uint32_t live_rows = __ballot_sync(0xffffffffu, live);
#pragma unroll
  for (int it = 0; it < C; ++it) {
    const int row = it * (32 / C) + lane / C, v = lane % C;
    packed[it] = *reinterpret_cast<const uint4*>(stage + row * (NC * 2) + ((v ^ (C == 4 ? (row >> 1) & 3 : (row >> 2) & 1)) << 4));
  }
#pragma unroll
  for (int it = 0; it < C; ++it) {
    const int row = it * (32 / C) + lane / C, v = lane % C;
    const long long base = __shfl_sync(0xffffffffu, place.base, row);
    if (((live_rows >> row) & 1u) && n + v * 8 < ncols) *reinterpret_cast<uint4*>(out + base + column + v * 8) = packed[it];
  }
}

template <typename T, bool PAIR, bool CONV>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tile_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                 const GemmDesc g, const TileArgs a) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* acc_bar = empty_bar + kMaxStages;
  uint64_t* recv_bar = acc_bar + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(recv_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  float* bias_s = reinterpret_cast<float*>(smem + 1024);   // [bn] bias of the tile's columns
  unsigned char* ring = smem + 2048;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const uint32_t leader = PAIR ? (rank & ~1u) : rank, half = PAIR ? (rank & 1u) : 0u;
  const int part = PAIR ? (int)(rank >> 1) : (int)rank;
  const int w_rows = PAIR ? a.bn / 2 : a.bn;             // rows of W this CTA stages per k-block
  const uint32_t w_bytes = (uint32_t)(w_rows * a.pieces) * BK * 2, a_bytes = (uint32_t)(kTileA * a.pieces);
  const uint32_t stage_bytes = a_bytes + w_bytes;

  // tile coordinates: (z, m, n), n fastest
  const int tile = blockIdx.x / (a.split * (PAIR ? 2 : 1));
  const int per_z = a.tiles_n * a.tiles_m;
  const int z = tile / per_z, rem = tile - z * per_z;
  const int tm = rem / a.tiles_n, n0 = (rem - tm * a.tiles_n) * a.bn;
  int x_row, x_z = z, out_row, out_rows;   // first X row and batch of the load; first output row and row count
  if (CONV && a.seqs_per_tile) {           // whole short sequences: output rows are flat [batch * L]
    x_row = 0;
    x_z = tm * a.seqs_per_tile;
    out_row = x_z * g.M;
    const int left = g.batch - x_z;
    out_rows = (left < a.seqs_per_tile ? left : a.seqs_per_tile) * g.M;
  } else {
    x_row = (tm * (PAIR ? 2 : 1) + (int)half) * a.rows;
    out_row = x_row;
    out_rows = g.M - x_row < a.rows ? g.M - x_row : a.rows;
  }
  if (out_rows < 0) out_rows = 0;          // the second CTA of a pair may lie wholly below the last row
  const int out_z = CONV && a.seqs_per_tile ? 0 : z;

  const int kb_begin = part * a.num_kb / a.split, kb_end = (part + 1) * a.num_kb / a.split;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      ptx::mbar_init(&full_bar[s], 1);
      ptx::mbar_init(&empty_bar[s], 1);
    }
    ptx::mbar_init(acc_bar, 1);
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
      ptx::tmem_alloc_pair(tmem_holder, a.tmem_cols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(tmem_holder, a.tmem_cols);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (PAIR || a.split > 1) ptx::cluster_sync_all();   // the peers' barriers exist before anything is reported to them
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  bool ready = true;
  if (warp == kTmaWarp) {
    // ---------------------------------------------------------- TMA producer (the whole warp, converged)
    const int w_z = z % g.w_mod;
    const uint32_t ring_addr = ptx::smem_u32(ring), full_addr = ptx::smem_u32(full_bar);
    const uint32_t full_remote = PAIR ? ptx::map_to_cta(full_addr, leader) : full_addr;
    auto load_x = [&](int kb, int s) {
      int tap = 0, kk = kb;
      if (CONV) {
        tap = kb / a.kb_per_tap;
        kk = kb - tap * a.kb_per_tap;
      }
      const int row = CONV ? x_row + tap - (g.taps >> 1) : x_row;   // rows outside the sequence read as zeros
      ptx::tma_load_4d_warp<PAIR>(ring_addr + s * stage_bytes, &tmap_x, full_remote + 8u * s, a.pieces == 1 ? kk * BK : 0, row,
                                  x_z, a.pieces == 1 ? 0 : kk * a.pieces);
    };
    auto load_w = [&](int kb, int s) {
      int tap = w_z, kk = kb;
      if (CONV) {
        tap = kb / a.kb_per_tap;
        kk = kb - tap * a.kb_per_tap;
      }
      if (half == 0) ptx::mbar_arrive_expect_tx_warp(full_addr + 8u * s, (PAIR ? 2u : 1u) * (a.x_bytes + w_bytes));
      ptx::tma_load_4d_warp<PAIR>(ring_addr + s * stage_bytes + a_bytes, &tmap_w, full_remote + 8u * s,
                                  a.pieces == 1 ? kk * BK : 0, n0 + (int)half * w_rows, tap, a.pieces == 1 ? 0 : kk * a.pieces);
    };
    const int n_kb = kb_end - kb_begin;
    const int ahead = n_kb < a.stages ? n_kb : a.stages;
    if (!g.weights_early) wait_for_predecessor();
    for (int i = 0; i < ahead; ++i) load_w(kb_begin + i, i);
    if (g.weights_early) wait_for_predecessor();
    for (int i = 0; i < ahead; ++i) load_x(kb_begin + i, i);
    release_successor();
    int s = 0;
    uint32_t ph = 0;   // phase of empty_bar[s] that the next refill waits for
    for (int i = ahead; i < n_kb; ++i) {
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&empty_bar[s], ph, abort_flag, g.status, kWaits + 21))) break;
      load_w(kb_begin + i, s);
      load_x(kb_begin + i, s);
      if (++s == a.stages) {
        s = 0;
        ph ^= 1u;
      }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer (of a pair: the leader's)
    if (half == 0 && ptx::elect_one()) {   // one lane, see umma_ss_f16_words
      const uint32_t idesc = ptx::make_idesc_f16(__is_same(T, __nv_bfloat16) ? 1 : 0, PAIR ? 2 * kRows : kRows, a.bn, 0, 0);
      constexpr uint32_t mode = ptx::swizzle_mode_for_row_bytes(BK * 2);
      const uint64_t desc0 = ptx::make_smem_desc(ptx::smem_u32(ring), 16, 8 * BK * 2, mode);
      const uint32_t first = (uint32_t)desc0, upper = (uint32_t)(desc0 >> 32);
      // in descriptor units: from X to W of a stage, from a stage to the next, and from a piece to the next
      const uint32_t to_w = a_bytes >> 4, stage_next = stage_bytes >> 4, x_next = a.x_piece >> 4, w_next = (uint32_t)(w_rows * BK * 2) >> 4;
      auto issue = [&](uint32_t ad, uint32_t bd, uint32_t accumulate) {   // one piece
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          ptx::umma_ss_f16_words<PAIR>(tmem_base, ad + 2 * k, bd + 2 * k, upper, idesc, k != 0 ? 1u : accumulate);
      };
      const int n_kb = kb_end - kb_begin;
      int s = 0;
      uint32_t ph = 0, desc = first;
      // The next k-block's barrier is looked at between the MMAs of this one: a wait answered only after the last of them leaves the
      // tensor pipe idle.
      bool landed = false, ok = true;
      for (int i = 0; i < n_kb; ++i) {
        ok = landed || ptx::mbar_wait(&full_bar[s], ph, abort_flag, g.status, kWaits + 22);
        if (!ok) break;
        ptx::tc_fence_after();
        uint64_t* done = &empty_bar[s];
        const uint32_t ad = desc, bd = desc + to_w;
        desc += stage_next;
        if (++s == a.stages) {
          s = 0;
          ph ^= 1u;
          desc = first;
        }
        issue(ad, bd, i != 0 ? 1u : 0u);
        landed = i + 1 < n_kb && ptx::mbar_test(&full_bar[s], ph);
        if (a.pieces == 2) issue(ad + x_next, bd + w_next, 1u);
        ptx::umma_commit_one<PAIR>(done, leader);
      }
      if (ok) ptx::umma_commit_one<PAIR>(acc_bar, leader);
    }
    __syncwarp();
  } else {
    // -------------------------------------------------------------- epilogue
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int ncols = g.head_split ? g.N : g.ldc;
    if (!g.weights_early) wait_for_predecessor();
    for (int c = threadIdx.x; c < a.bn; c += kEpilogueWarps * 32)
      bias_s[c] = g.bias && n0 + c < g.N ? Elem<T>::to_f(reinterpret_cast<const T*>(g.bias)[n0 + c]) : 0.0f;
    asm volatile("bar.sync 1, 256;" ::: "memory");   // the eight epilogue warps
    if (g.weights_early) wait_for_predecessor();      // the output may still be read by the kernel before this one
    const RowPlace place = place_row(g, out_row + (r < out_rows ? r : 0), out_z);
    ready = __all_sync(0xffffffffu, ptx::mbar_wait(acc_bar, 0, abort_flag, g.status, kWaits + 23));
    ptx::tc_fence_after();
    const bool live = ready && r < out_rows;
    // staging of the output blocks: in the operand ring once that is idle, behind the receive buffer otherwise
    unsigned char* stage = (a.split == 1 ? ring : ring + a.ring_bytes + a.recv_bytes) + warp * 2048;
    bool keep_row = true;
    if (CONV && live && g.row_mask)
      keep_row = mask_keep(g.row_mask, g.row_mask_elem, (long long)out_z * g.M + out_row + r);
    if (a.split == 1) {
#pragma unroll 1
      for (int c0 = (warp >> 2) * 32; c0 < a.bn; c0 += 64) {
        const int n = n0 + c0;
        if (n >= ncols) break;   // warp-uniform
        float v[32];
        ptx::tmem_ld32_f(taddr + (uint32_t)c0, v);
        ptx::tmem_wait_ld();
        emit<T, CONV, 32>(g, v, bias_s + c0, stage, place, live, n, ncols, keep_row, lane);
      }
    } else {
      // Part p of the cluster finishes columns [p * unit, (p + 1) * unit) of the tile.  Every other part's share is
      // parked in the operand ring (every load and MMA of this CTA is done), one block of out_rows rows (pitch unit + 4
      // floats) per destination, and leaves as one bulk copy per destination; slot = sender, own slot skipped.
      const int unit = a.bn / a.split;
      const uint32_t pitch = (uint32_t)(unit * 4 + 16), slot_bytes = (uint32_t)kRows * pitch;
#pragma unroll 1
      for (int q = 1; q < a.split; ++q) {
        const int dst_part = part + q < a.split ? part + q : part + q - a.split;
        float4* row = reinterpret_cast<float4*>(ring + (uint32_t)(q - 1) * slot_bytes + (uint32_t)r * pitch);
#pragma unroll 1
        for (int c = (warp >> 2) * 16; c < unit; c += 32) {
          uint32_t v[16];
          ptx::tmem_ld16(taddr + (uint32_t)(dst_part * unit + c), v);
          ptx::tmem_wait_ld();
          if (!live) continue;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            row[c / 4 + j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                         __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
        }
      }
      ptx::fence_proxy_async_smem();
      asm volatile("bar.sync 1, 256;" ::: "memory");   // the eight epilogue warps
      const uint32_t share = (uint32_t)out_rows * pitch;
      if (threadIdx.x == 0) {
        ptx::mbar_arrive_expect_tx(recv_bar, share * (uint32_t)(a.split - 1));
        for (int q = 1; q < a.split && share != 0; ++q) {
          const int dst_part = part + q < a.split ? part + q : part + q - a.split;
          const uint32_t dst_rank = PAIR ? 2u * (uint32_t)dst_part + half : (uint32_t)dst_part;
          const uint32_t slot = (uint32_t)(part < dst_part ? part : part - 1);
          ptx::bulk_copy_to_cta(ptx::map_to_cta(ptx::smem_u32(ring + a.ring_bytes) + slot * slot_bytes, dst_rank),
                                ptx::smem_u32(ring) + (uint32_t)(q - 1) * slot_bytes, share,
                                ptx::map_to_cta(ptx::smem_u32(recv_bar), dst_rank));
        }
      }
      ready = __all_sync(0xffffffffu, ptx::mbar_wait(recv_bar, 0, abort_flag, g.status, kWaits + 24)) && ready;
      const unsigned char* recv = ring + a.ring_bytes + (uint32_t)r * pitch;
      auto finish = [&](auto width, int c) {
        constexpr int NC = decltype(width)::value;
        const int n = n0 + part * unit + c;
        if (n >= ncols) return;   // warp-uniform
        float v[NC];
        if constexpr (NC == 32) ptx::tmem_ld32_f(taddr + (uint32_t)(part * unit + c), v);
        else ptx::tmem_ld16_f(taddr + (uint32_t)(part * unit + c), v);
        ptx::tmem_wait_ld();
        if (live && ready) {
          for (int p = 0; p < a.split - 1; ++p) {
            const float4* src = reinterpret_cast<const float4*>(recv + (uint32_t)p * slot_bytes + (uint32_t)c * 4u);
#pragma unroll
            for (int j = 0; j < NC / 4; ++j) {
              const float4 s4 = src[j];
              v[4 * j] += s4.x; v[4 * j + 1] += s4.y; v[4 * j + 2] += s4.z; v[4 * j + 3] += s4.w;
            }
          }
        }
        emit<T, CONV, NC>(g, v, bias_s + part * unit + c, stage, place, live && ready, n, ncols, keep_row, lane);
      };
      if (unit % 32 == 0) {
#pragma unroll 1
        for (int c = (warp >> 2) * 32; c < unit; c += 64) finish(std::integral_constant<int, 32>{}, c);
      } else {
#pragma unroll 1
        for (int c = (warp >> 2) * 16; c < unit; c += 32) finish(std::integral_constant<int, 16>{}, c);
      }
    }
  }

  // Peers may still read this CTA's shared memory (partial tiles, operands of a pair) or report to its barriers.
  ptx::tc_fence_before();
  __syncthreads();
  if (PAIR || a.split > 1) ptx::cluster_sync_all_relaxed();
  ptx::tc_fence_after();
  if (warp == kMmaWarp) {
    if (PAIR) ptx::tmem_dealloc_pair(tmem_base, a.tmem_cols);
    else ptx::tmem_dealloc(tmem_base, a.tmem_cols);
  }
}

template <typename T, bool PAIR, bool CONV>
int launch_typed(const GemmDesc& g, const TilePlan& plan, cudaStream_t stream) {
  const uint64_t es = sizeof(T);
  const int taps = CONV && g.taps > 1 ? g.taps : 1;
  TileArgs a{};
  a.bn = plan.bn;
  a.tmem_cols = a.bn <= 32 ? 32 : (a.bn <= 64 ? 64 : (a.bn <= 128 ? 128 : 256));
  const int ncols = g.head_split ? g.N : g.ldc;
  a.tiles_n = (ncols + a.bn - 1) / a.bn;
  int box_rows = kRows, box_seqs = 1, z_tiles = g.batch;
  if (CONV && g.M <= kRows) {
    a.seqs_per_tile = box_seqs = kRows / g.M < g.batch ? kRows / g.M : g.batch;
    box_rows = g.M;
    a.tiles_m = (g.batch + box_seqs - 1) / box_seqs;
    z_tiles = 1;
  } else {
    a.tiles_m = (g.M + (PAIR ? 2 : 1) * kRows - 1) / ((PAIR ? 2 : 1) * kRows);
    // The rows are dealt out evenly, in groups of eight (a swizzle atom), instead of 128 to each tile but the last: rows beyond the
    // tensor are zeros that a load takes longer for than for data.  us per launch with 128 rows and with the rows there are
    // (W from HBM, fp16): 32 x 2304 x 768 4.8 / 4.1, 32 x 3072 x 768 with GELU 7.3 / 5.0, 8 x 4608 x 1536 9.8 / 6.5, 64 x 6144 x
    // 1536 8.3 / 8.2; 130 x 1536 x 6144 11.9 / 11.1, 333 x 768 x 3072 8.4 / 8.0.  The MMA reads 128 rows; what lies in the others'
    // place, within the stage, ends in accumulator rows that nobody reads.
    const int ctas_m = a.tiles_m * (PAIR ? 2 : 1);
    if (!CONV) box_rows = ((g.M + ctas_m - 1) / ctas_m + 7) / 8 * 8;
  }
  a.rows = CONV ? kRows : box_rows;
  // two 64-element pieces per k-block where the layout allows it: half the barrier round trips per inner product
  a.pieces = g.K % (2 * BK) == 0 && (!CONV || box_rows * box_seqs == kRows) ? 2 : 1;
  a.kb_per_tap = (g.K + BK * a.pieces - 1) / (BK * a.pieces);
  a.num_kb = taps * a.kb_per_tap;
  a.split = plan.split < a.num_kb ? plan.split : a.num_kb;
  if (a.split > 1 && a.bn % (16 * a.split)) return fail(DFL_ERR_UNSUPPORTED, "gemm_tile: %d columns in %d parts", a.bn, a.split);
  a.x_piece = (uint32_t)(box_rows * box_seqs * BK * 2);
  a.x_bytes = (uint32_t)a.pieces * a.x_piece;

  CUtensorMap tmap_x, tmap_w;
  const uint64_t x_stride = g.batch > 1 ? (uint64_t)g.stride_x * es : (uint64_t)g.M * g.K * es;
  const int w_batches = taps > 1 ? taps : (g.w_mod > 1 ? g.w_mod : 1);
  const uint64_t w_stride = taps == 1 && w_batches > 1 ? (uint64_t)g.stride_w * es : (uint64_t)g.N * g.K * es;
  int rc = encode_tensor_map_pieces(&tmap_x, g.x, g.K, g.M, g.batch, (uint64_t)g.K * es, x_stride, box_rows, box_seqs, a.pieces);
  if (rc != DFL_OK) return rc;
  rc = encode_tensor_map_pieces(&tmap_w, g.w, g.K, g.N, w_batches, (uint64_t)g.K * es, w_stride, PAIR ? a.bn / 2 : a.bn, 1, a.pieces);
  if (rc != DFL_OK) return rc;

  // Operand ring: as many k-blocks as the inner product of one CTA has, within all the shared memory there is (the
  // registers of 320 threads leave room for one CTA per SM anyway).
  auto kernel = gemm_tile_kernel<T, PAIR, CONV>;
  static KernelDeviceConfig config;   // per template instantiation
  rc = configure_kernel(config, kernel, kMaxSmem, nullptr, "gemm_tile_kernel");
  if (rc != DFL_OK) return rc;
  const long long tiles = (long long)a.tiles_n * a.tiles_m * z_tiles;
  const int cluster = a.split * (PAIR ? 2 : 1);
  const long long ctas = tiles * cluster;
  if (ctas > 0x7fffffff) return fail(DFL_ERR_TOO_LARGE, "gemm_tile: too many tiles");
  const int stage = a.pieces * (kTileA + (PAIR ? a.bn / 2 : a.bn) * BK * 2);
  const int staging = kEpilogueWarps * 2048;
  const int recv = a.split > 1 ? (a.split - 1) * kRows * (a.bn / a.split * 4 + 16) : 0;
  const int budget = kMaxSmem - 4096 - (a.split > 1 ? recv + staging : 0);
  const int kb_cta = (a.num_kb + a.split - 1) / a.split;
  a.stages = budget / stage;
  if (a.stages > kb_cta) a.stages = kb_cta;
  if (a.stages > kMaxStages) a.stages = kMaxStages;
  if (a.stages < 1) return fail(DFL_ERR_UNSUPPORTED, "gemm_tile: %d columns, split %d do not fit", a.bn, a.split);
  a.ring_bytes = (uint32_t)(a.stages * stage > recv ? a.stages * stage : recv);   // parked shares reuse the ring
  if (a.ring_bytes < (uint32_t)staging) a.ring_bytes = (uint32_t)staging;
  a.recv_bytes = (uint32_t)recv;
  // alignment slack, barriers, bias, ring, receive buffer, output staging
  const int smem = 3072 + (int)a.ring_bytes + (a.split > 1 ? recv + staging : 0);

  GemmDesc gd = g;
  if (!gd.status) {
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&gd.status), g_gemm_tile_status);
    if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "status word: %s", cudaGetErrorString(e));
  }
  cudaError_t e = launch_clusters_after_predecessor(kernel, dim3((unsigned)ctas), dim3(kThreads), cluster, (size_t)smem,
                                                    stream, tmap_x, tmap_w, gd, a);
  if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "gemm_tile_kernel: %s", cudaGetErrorString(e));
  return check_launch("gemm_tile_kernel");
}

template <typename T>
int launch_t(const GemmDesc& g, const TilePlan& plan, cudaStream_t stream) {
  const bool conv = g.taps > 1 || g.row_mask || g.activation == DFL_ACT_TANH;
  if (conv) return launch_typed<T, false, true>(g, plan, stream);
  return plan.pair ? launch_typed<T, true, false>(g, plan, stream) : launch_typed<T, false, false>(g, plan, stream);
}

}  // namespace

int launch_gemm_tile(const GemmDesc& g, const TilePlan& plan, cudaStream_t stream) {
  return g.dtype == DFL_F16 ? launch_t<__half>(g, plan, stream) : launch_t<__nv_bfloat16>(g, plan, stream);
}

}  // namespace dfl
