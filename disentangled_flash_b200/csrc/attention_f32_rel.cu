// FP32 fused disentangled attention with the position scores computed in the kernel (head dims 32 and 64).
//
//   S[i,j] = q_i.k_j + q_i.pos_key[s] + k_j.pos_query[s],  s = lut[i-j+L-1];  scale, mask, softmax, P V as in attention_f32.cu
// (the score products of kernel.py:574-585 and the kernel of kernel.py:137-345, both in the reference's strict FP32)
// Every product is the six plane products of linear_f32.cu, smallest first, and no tensor-core accumulator holds more than one
// 64-deep block, so the scores are what the score GEMMs and attention_f32_kernel give, but for the order of their two sums.
//
// Why one launch: the scores of 8 x 24 heads x 256 positions are 2 x 100 MB; writing them took 2 x 67 us and gathering them, slot
// by slot, most of the attention kernel's 120 us.  Here they exist as tiles in shared memory only.
//
// A (128 query x 128 key) tile needs one window of 255 relative distances; window row w belongs to the pairs with
// n - r + 127 = w (query row r, key n of the tile).  It is walked in pieces of 64 rows, gathered from the pruned tables through
// the slot table by two warps with cp.async (the slots of neighbouring distances are equal or neighbours, not evenly spaced), for each term:
//   C2P piece: D[r, w] = q_r . key table row;   P2C piece: D[n, w] = k_n . query table row     (128 x 64, two accumulators)
// Eight warps read a finished piece from tensor memory and put element (r, w) or (n, w) to row r, key n of the tile in shared
// memory (pitch 132: neither the diagonal writes nor the row reads meet in a bank), C2P first, P2C added to it.  The same warps
// then run the softmax, two threads per query row.
//
// What bounds a tile at d = 64, 21 k cycles: its eight pieces, 1.3 (C2P) and 1.6 k (P2C) each: 24 MMAs of 128 x 64, 33 cycles each
// with Q as the operand (it lives in tensor memory: shared memory has no room for it, and a tensor-memory operand is read
// faster), 49 with K, and the issuer's waits; the conversion of a P2C piece, 1.2 k, and its gathering, 1.1 k, lie beside it.
// The softmax, 4.5 k, and PV, 2.6 k, follow.  An item starts and ends with 2 k and 3 k.  A second issuer with every other piece
// hides the waits, but then the conversions set the same pace.
// us with the projection, three launches / this one: 8 x 12 heads x 128 x d 64 65 / 40, 8 x 24 x 256 352 / 213, 4 x 12 x 512 217 / 146,
// 2 x 12 x 1024 308 / 239, 1 x 12 x 64 34 / 26, 1 x 12 x 3400 1221 / 1037; d 32 8 x 24 x 256 257 / 110, 1 x 24 x 8192 9633 / 7079.  At no
// length from 16 to 8192, with one term or two, 1 to 170 sequences, were the three launches faster.
// One CTA per (batch, head, 128-query tile).  Warps 0-7 convert and softmax, 8-9 gather table pieces and V, 10 loads Q and K,
// issues the MMAs and owns tensor memory: S (128 columns; P's three planes, 192, take its place), O 64, Q 96,
// two accumulators of 64.
#include "f32_planes.cuh"
#include "tcgen05_ptx.cuh"

namespace dfl {

__device__ int g_attn_f32_rel_status = 0;

namespace {

constexpr int BM = 128, BN = 128, kPiece = 64, kStages = 4;
constexpr int kComputeWarps = 8, kLoadWarp = 8, kLoadWarps = 2, kMmaWarp = 10, kThreads = 352;
constexpr int kMaxSmem = 232448;
constexpr int kCode = kWaitsAttentionF32Rel;
constexpr int COL_SP = 0, COL_O = 192, COL_Q = 256, COL_ACC = 384, kTmemCols = 512;
constexpr int kPitch = 132;   // floats per row of the score tile

template <int D>
struct Shape {
  static constexpr int kRowBytes = D * 2, kChunks = kRowBytes / 16;   // one swizzle row per plane
  static constexpr int kKPlane = BN * kRowBytes, kK = kPlanes * kKPlane;
  static constexpr int kPiecePlane = kPiece * kRowBytes, kStage = kPlanes * kPiecePlane;
  static constexpr int offK = 0, offRing = kK, offRel = offRing + kStages * kStage, offBar = offRel + BM * kPitch * 4;
  static constexpr int offMax = offBar + 256;                          // [2 halves][BM] row maxima, then row sums
  static constexpr int offKeep = offMax + 4 * BM * 4;
};

struct Barriers {
  uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2];
  uint64_t q_load, q_full, k_full, s_full, p_full, o_full, pair[4], compute;
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(Barriers) <= 256, "barrier block too large");

template <int D>
__global__ void __launch_bounds__(kThreads, 1)
attention_f32_rel_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const DflAttnParams p, const __nv_bfloat16* __restrict__ pos_key,
                         const __nv_bfloat16* __restrict__ pos_query, const int n_active, const int out_planes, int* status_word) {
  using T = Shape<D>;
  constexpr int HK = BN / 2, OW = D / 2;   // keys and output columns per softmax thread
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + T::offBar);
  volatile int* abort_flag = &bars->abort_flag;
  const int L = p.seq_len, H = p.heads, BH = p.batch * H;
  const int n_qt = (L + BM - 1) / BM, n_kt = (L + BN - 1) / BN;
  uint32_t* keep_s = reinterpret_cast<uint32_t*>(smem + T::offKeep);                    // kept-key bits
  uint16_t* lut_s = reinterpret_cast<uint16_t*>(smem + T::offKeep + (n_kt * BN / 32) * 4);   // [2L-1]
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int bh = blockIdx.x / n_qt, b = bh / H, h = bh - b * H, i0 = (blockIdx.x - bh * n_qt) * BM;
  const bool has_c2p = pos_key != nullptr, has_p2c = pos_query != nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(&bars->full[s], kLoadWarps);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&bars->acc_full[a], 1);
      ptx::mbar_init(&bars->acc_empty[a], kComputeWarps);
    }
    ptx::mbar_init(&bars->q_load, 1);
    ptx::mbar_init(&bars->q_full, kComputeWarps);
    ptx::mbar_init(&bars->k_full, 1);
    ptx::mbar_init(&bars->s_full, 1);
    ptx::mbar_init(&bars->p_full, kComputeWarps);
    ptx::mbar_init(&bars->o_full, 1);
    for (int s = 0; s < 4; ++s) ptx::mbar_init(&bars->pair[s], 2);
    ptx::mbar_init(&bars->compute, kComputeWarps);
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc(&bars->tmem_base, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
    return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag, status_word, code)) != 0;
  };
  // pieces of the window that some pair of the tile inside the sequence needs
  auto first_piece = [&] { return (BM - (L - i0 < BM ? L - i0 : BM)) / kPiece; };
  auto last_piece = [&](int t) { return (BM - 2 + (L - t * BN < BN ? L - t * BN : BN)) / kPiece; };
  auto value_pieces = [&](int t) { return L - t * BN > kPiece ? 2 : 1; };
  // C2P pieces of tile t whose MMAs run before the PV of the tile ahead of it, while the compute warps are in its softmax: as many
  // as there are accumulators (K, which P2C needs, is loaded later)
  auto early_pieces = [&](int t) { return !has_c2p || t == 0 || t == n_kt ? 0 : (last_piece(t) > first_piece() ? 2 : 1); };

  if (warp >= kLoadWarp && warp < kLoadWarp + kLoadWarps) {
    const int tid = (warp - kLoadWarp) * 32 + lane;
#pragma unroll 8
    for (int e = tid; e < 2 * L - 1; e += kLoadWarps * 32) {   // like the tables, there before the projection ahead of this launch
      int slot = p.lut[e];   // entries outside the table (not a table of the builder) are clamped
      slot = slot < 0 ? 0 : (slot >= n_active ? n_active - 1 : slot);
      lut_s[e] = (uint16_t)slot;
    }
    asm volatile("bar.sync 1, 64;" ::: "memory");   // the two gathering warps
    const uint32_t ring = ptx::smem_u32(smem + T::offRing);
    uint32_t issued = 0, signalled = 0;
    bool ok = true;
    auto signal_to = [&](uint32_t upto) {   // the pieces before `upto` have landed: the tensor core may read them
      if (signalled == upto) return;
      ptx::fence_proxy_async_smem();
      __syncwarp();
      for (; signalled != upto; ++signalled)
        if (lane == 0) ptx::mbar_arrive(&bars->full[signalled % kStages]);
    };
    auto drain = [&] {
      ptx::cp_async_wait_group<0>();
      signal_to(issued);
    };
    // 64 rows of each plane into the next stage; row_of(row, valid) gives the row's index in the plane
    auto piece = [&](const __nv_bfloat16* plane0, long long plane_stride, auto row_of) {
      const uint32_t s = issued % kStages, parity = ((issued / kStages) & 1u) ^ 1u;
      if (!__all_sync(0xffffffffu, ptx::mbar_try_wait(&bars->empty[s], parity))) {
        drain();
        ok = wait(&bars->empty[s], parity, kCode + 71);
      }
      if (!ok) return;
#pragma unroll
      for (int it = 0; it < T::kChunks; ++it) {
        const int idx = it * 64 + tid, row = idx / T::kChunks, c = idx % T::kChunks;
        bool valid = true;
        const __nv_bfloat16* src = plane0 + (long long)row_of(row, valid) * D + c * 8;
        const uint32_t swizzled = (uint32_t)(c ^ (T::kRowBytes == 128 ? row & 7 : (row >> 1) & 3)) << 4;
        const uint32_t dst = ring + s * T::kStage + (uint32_t)(row * T::kRowBytes) + swizzled;
#pragma unroll
        for (int q = 0; q < kPlanes; ++q) ptx::cp_async_16_or_zero(dst + q * T::kPiecePlane, src + q * plane_stride, valid);
      }
      ptx::cp_async_commit();
      ++issued;
      ptx::cp_async_wait_group<2>();
      if (issued > 2 && issued - 2 > signalled) signal_to(issued - 2);
    };
    auto table_piece = [&](int t, int term, int pi) {
      const __nv_bfloat16* table = term == 0 ? pos_key : pos_query;
      const int e0 = i0 - t * BN + L - 1 + BM - 1 - pi * kPiece;   // lut index of the piece's first row; rows count down
      piece(table + (long long)h * n_active * D, (long long)H * n_active * D, [&](int row, bool&) {
        int e = e0 - row;   // distances that no pair inside the sequence has: any row will do
        e = e < 0 ? 0 : (e > 2 * L - 2 ? 2 * L - 2 : e);
        return (int)lut_s[e];
      });
    };
    for (int t = 0; t < n_kt && ok; ++t) {
      const int p0 = first_piece(), p1 = last_piece(t);
      for (int term = 0; term < 2; ++term) {
        if (!(term == 0 ? has_c2p : has_p2c)) continue;
        for (int pi = p0 + (term == 0 ? early_pieces(t) : 0); pi <= p1 && ok; ++pi) table_piece(t, term, pi);
      }
      for (int pi = p0; pi < p0 + early_pieces(t + 1) && ok; ++pi) table_piece(t + 1, 0, pi);
      if (t == 0) wait_for_predecessor();   // V is the predecessor's
      for (int v = 0; v < value_pieces(t) && ok; ++v) {
        const int j0 = t * BN + v * kPiece;
        piece(reinterpret_cast<const __nv_bfloat16*>(p.v) + (long long)bh * L * D, (long long)BH * L * D, [&](int row, bool& valid) {
          valid = j0 + row < L;
          return valid ? j0 + row : 0;
        });
      }
    }
    drain();
  } else if (warp == kMmaWarp) {
    constexpr uint32_t mode = ptx::swizzle_mode_for_row_bytes(T::kRowBytes), sbo = 8 * T::kRowBytes;
    constexpr uint32_t idesc_rel = ptx::make_idesc_f16(1, BM, kPiece, 0, 0), idesc_qk = ptx::make_idesc_f16(1, BM, BN, 0, 0);
    constexpr uint32_t idesc_pv = ptx::make_idesc_f16(1, BM, D, 0, 1);
    constexpr int kSteps = D / 16, kVSteps = kPiece / 16;
    constexpr int pa[6] = {2, 1, 0, 1, 0, 0}, pb[6] = {0, 1, 2, 0, 1, 0};   // plane products, smallest first
    const uint64_t kd = ptx::make_smem_desc(ptx::smem_u32(smem + T::offK), 16, sbo, mode);
    const uint64_t rd = ptx::make_smem_desc(ptx::smem_u32(smem + T::offRing), 16, sbo, mode);
    const uint64_t vd = ptx::make_smem_desc(ptx::smem_u32(smem + T::offRing), T::kPiecePlane, sbo, mode);
    uint32_t pc = 0, ac = 0;   // pieces taken from the ring, accumulators filled
    auto load = [&](int off, const CUtensorMap* map, uint64_t* bar, int row) {   // 128 rows of each plane
      if (lane == 0) {
        ptx::mbar_arrive_expect_tx(bar, (uint32_t)T::kK);
        for (int q = 0; q < kPlanes; ++q) ptx::tma_load_3d(smem + off + q * T::kKPlane, map, bar, 0, row, q * BH + bh);
      }
      __syncwarp();
    };
    wait_for_predecessor();
    load(T::offRel, &tmap_q, &bars->q_load, i0);   // Q passes through the score tile's place on its way to tensor memory
    load(T::offK, &tmap_k, &bars->k_full, 0);
    auto mma_piece = [&](int term) -> bool {
      const uint32_t s = pc % kStages, a = ac & 1u;
      if (!wait(&bars->full[s], (pc / kStages) & 1u, kCode + 75) || !wait(&bars->acc_empty[a], ((ac >> 1) & 1u) ^ 1u, kCode + 76)) return false;
      ptx::tc_fence_after();
      const uint32_t d_tmem = tmem_base + COL_ACC + a * kPiece;
      const uint64_t bd = rd + (uint64_t)((s * T::kStage) >> 4);
      if (term == 0) {
#pragma unroll
        for (int q = 0; q < 6; ++q)
#pragma unroll
          for (int k = 0; k < kSteps; ++k)
            ptx::umma_ts_f16_warp(d_tmem, tmem_base + COL_Q + (uint32_t)(pa[q] * (D / 2) + k * 8),
                                  bd + (uint64_t)((pb[q] * T::kPiecePlane + k * 32) >> 4), idesc_rel, q != 0 || k != 0 ? 1u : 0u);
      } else {
#pragma unroll
        for (int q = 0; q < 6; ++q)
#pragma unroll
          for (int k = 0; k < kSteps; ++k)
            ptx::umma_ss_f16_warp(d_tmem, kd + (uint64_t)((pa[q] * T::kKPlane + k * 32) >> 4),
                                  bd + (uint64_t)((pb[q] * T::kPiecePlane + k * 32) >> 4), idesc_rel, q != 0 || k != 0 ? 1u : 0u);
      }
      ptx::umma_commit_warp(&bars->empty[s]);
      ptx::umma_commit_warp(&bars->acc_full[a]);
      ++pc;
      ++ac;
      return true;
    };
    bool ok = wait(&bars->q_full, 0, kCode + 73);
    for (int t = 0; t < n_kt && ok; ++t) {
      const int n_pieces = last_piece(t) - first_piece() + 1, early = early_pieces(t), next_early = early_pieces(t + 1);
      // C2P, P2C, S, then the next tile's first C2P pieces
      const int c2p_end = has_c2p ? n_pieces - early : 0, p2c_end = c2p_end + (has_p2c ? n_pieces : 0);
#pragma unroll 1
      for (int n = 0; n < p2c_end && ok; ++n) {
        if (n == c2p_end) ok = wait(&bars->k_full, (uint32_t)t & 1u, kCode + 74);
        ok = ok && mma_piece(n < c2p_end ? 0 : 1);
      }
      // S takes the place of the previous tile's P, which PV has read by then
      ok = ok && wait(&bars->k_full, (uint32_t)t & 1u, kCode + 78) &&
           (t == 0 || wait(&bars->o_full, (uint32_t)(t - 1) & 1u, kCode + 79));
      if (!ok) break;
      ptx::tc_fence_after();
#pragma unroll
      for (int q = 0; q < 6; ++q)
#pragma unroll
        for (int k = 0; k < kSteps; ++k)
          ptx::umma_ts_f16_warp(tmem_base + COL_SP, tmem_base + COL_Q + (uint32_t)(pa[q] * (D / 2) + k * 8),
                                kd + (uint64_t)((pb[q] * T::kKPlane + k * 32) >> 4), idesc_qk, q != 0 || k != 0 ? 1u : 0u);
      ptx::umma_commit_warp(&bars->s_full);
#pragma unroll 1
      for (int n = 0; n < next_early && ok; ++n) ok = mma_piece(0);
      const int n_v = value_pieces(t);
      ok = ok && wait(&bars->p_full, (uint32_t)t & 1u, kCode + 80);   // ... and S is complete: K's place is free
      if (ok && t + 1 < n_kt) load(T::offK, &tmap_k, &bars->k_full, (t + 1) * BN);
      for (int v = 0; v < n_v && ok; ++v) ok = wait(&bars->full[(pc + v) % kStages], ((pc + v) / kStages) & 1u, kCode + 81);
      if (!ok) break;
      ptx::tc_fence_after();
      uint64_t v_stage[2];
#pragma unroll
      for (int v = 0; v < 2; ++v) v_stage[v] = vd + (uint64_t)((((pc + v) % kStages) * T::kStage) >> 4);
#pragma unroll
      for (int q = 0; q < 6; ++q)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          if (v >= n_v) continue;
#pragma unroll
          for (int k = 0; k < kVSteps; ++k)
            ptx::umma_ts_f16_warp(tmem_base + COL_O, tmem_base + COL_SP + (uint32_t)(pa[q] * (BN / 2) + v * (kPiece / 2) + k * 8),
                                  v_stage[v] + (uint64_t)((pb[q] * T::kPiecePlane + k * 16 * T::kRowBytes) >> 4), idesc_pv,
                                  q != 0 || v != 0 || k != 0 ? 1u : 0u);
        }
      for (int v = 0; v < n_v; ++v, ++pc) ptx::umma_commit_warp(&bars->empty[pc % kStages]);
      ptx::umma_commit_warp(&bars->o_full);
    }
  } else {
    const int hf = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane, i = i0 + r;
    const bool row_ok = i < L;
    const bool q_keep = row_ok && mask_keep(p.mask, p.mask_elem_size, (long long)b * L + i);
    const float scale_log2 = p.scale * 1.4426950408889634f;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    const uint32_t t_s = tmem_base + lanes + COL_SP + hf * HK, t_p = tmem_base + lanes + COL_SP + hf * (HK / 2);
    const uint32_t t_o = tmem_base + lanes + COL_O + hf * OW, t_acc = tmem_base + lanes + COL_ACC + hf * 32;
    float* xmax = reinterpret_cast<float*>(smem + T::offMax);
    float* rel = reinterpret_cast<float*>(smem + T::offRel);
    for (int w = warp; w < n_kt * BN / 32; w += kComputeWarps) {   // (a tile's scores are never ready before all warps are here)
      const int j = w * 32 + lane;
      const uint32_t bits = __ballot_sync(0xffffffffu, j < L && mask_keep(p.mask, p.mask_elem_size, (long long)b * L + j));
      if (lane == 0) keep_s[w] = bits;
    }
    wait_for_predecessor();
    release_successor();
    bool ok = wait(&bars->q_load, 0, kCode + 90);
    {   // this thread's half of its query row, all planes, into tensor memory (a row read by its own thread from global memory:
        // 3.9 k cycles before the first MMA instead of 2 k)
      const unsigned char* q_row = smem + T::offRel + r * T::kRowBytes;
      const int swizzle = T::kRowBytes == 128 ? r & 7 : (r >> 1) & 3;
#pragma unroll
      for (int q = 0; q < kPlanes; ++q) {
        uint32_t words[OW / 2];
#pragma unroll
        for (int c = 0; c < OW / 8; ++c) {
          const uint4 v = *reinterpret_cast<const uint4*>(q_row + q * T::kKPlane + (((hf * (OW / 8) + c) ^ swizzle) << 4));
          words[4 * c] = v.x;
          words[4 * c + 1] = v.y;
          words[4 * c + 2] = v.z;
          words[4 * c + 3] = v.w;
        }
        const uint32_t at = tmem_base + lanes + COL_Q + (uint32_t)(q * (D / 2) + hf * (OW / 2));
        if constexpr (D == 64) ptx::tmem_st16(at, words);
        else ptx::tmem_st8(at, words);
      }
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->q_full);
    }
    float o[OW];
#pragma unroll
    for (int c = 0; c < OW; ++c) o[c] = 0.0f;
    float m_run = -INFINITY, l_run = 0.0f;
    uint32_t ac = 0, syncs = 0;
    auto sync_compute = [&](int code) {   // the eight warps; bounded, unlike a named barrier
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->compute);
      return wait(&bars->compute, syncs++ & 1u, code);
    };
    auto add_output = [&](float corr) {   // o = (o + tile's PV) * corr
#pragma unroll
      for (int c0 = 0; c0 < OW; c0 += 16) {
        float v[16];
        ptx::tmem_ld16_f(t_o + c0, v);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 16; ++c) o[c0 + c] = (o[c0 + c] + v[c]) * corr;
      }
    };
    // 32 columns of the next finished piece
    auto take = [&](float (&v)[32]) -> bool {
      const uint32_t a = ac & 1u;
      if (!wait(&bars->acc_full[a], (ac >> 1) & 1u, kCode + 82)) return false;
      ptx::tc_fence_after();
      ptx::tmem_ld32_f(t_acc + a * kPiece, v);
      ptx::tmem_wait_ld();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->acc_empty[a]);
      ++ac;
      return true;
    };
    for (int t = 0; t < n_kt && ok; ++t) {
      const int p0 = first_piece(), p1 = last_piece(t);
      if (t > 0) ok = sync_compute(kCode + 83);   // every warp has read the previous tile's scores
      if (has_c2p) {
#pragma unroll 1
        for (int pi = p0; pi <= p1 && ok; ++pi) {
          float v[32];
          ok = take(v);
          const int w0 = pi * kPiece + hf * 32, n0 = w0 + r - (BM - 1);   // key of the first column
          const int least = w0 + quarter * 32 - (BM - 1);                  // ... in the warp's first row
          if (!ok || least + 62 < 0 || least >= BN) continue;              // warp-uniform
          float* dst = rel + r * kPitch + n0;
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if ((unsigned)(n0 + c) < (unsigned)BN) dst[c] = v[c];
        }
        if (has_p2c && ok) ok = sync_compute(kCode + 84);
      }
      if (has_p2c) {
#pragma unroll 1
        for (int pi = p0; pi <= p1 && ok; ++pi) {
          float v[32];
          ok = take(v);
          const int w0 = pi * kPiece + hf * 32, r0 = r + BM - 1 - w0;   // query row of the first column (this lane's key is r)
          const int most = quarter * 32 + 31 + BM - 1 - w0;
          if (!ok || most < 0 || most - 62 >= BM) continue;
          float* dst = rel + r0 * kPitch + r;
#pragma unroll
          for (int c0 = 0; c0 < 32; c0 += 16) {
            if (has_c2p) {
              float old[16];
#pragma unroll
              for (int c = 0; c < 16; ++c) old[c] = (unsigned)(r0 - c0 - c) < (unsigned)BM ? dst[-(c0 + c) * kPitch] : 0.0f;
#pragma unroll
              for (int c = 0; c < 16; ++c) v[c0 + c] += old[c];
            }
#pragma unroll
            for (int c = 0; c < 16; ++c)
              if ((unsigned)(r0 - c0 - c) < (unsigned)BM) dst[-(c0 + c) * kPitch] = v[c0 + c];
          }
        }
      }
      if (ok) ok = sync_compute(kCode + 85);
      ok = ok && wait(&bars->s_full, (uint32_t)t & 1u, kCode + 86);
      if (!ok) break;
      ptx::tc_fence_after();
      // Two passes over the row, 16 keys at a time in rolled loops: scores, scaled and masked, back to the row in shared memory
      // and their maximum; then probabilities.  (All 64 in registers and everything unrolled: a CTA's first tile spent 23 k cycles
      // here, mostly on fetching instructions, later ones 9.4 k.)
      const int j0 = t * BN + hf * HK;
      float4* row = reinterpret_cast<float4*>(rel + r * kPitch + hf * HK);
      float mx = -INFINITY;
#pragma unroll 1
      for (int c0 = 0; c0 < HK; c0 += 16) {
        float v[16];
        ptx::tmem_ld16_f(t_s + c0, v);
        const int left = L - (j0 + c0);
        uint32_t bits = keep_s[(j0 + c0) >> 5] >> (c0 & 16);
        if (!q_keep) bits = left >= 16 ? 0xffffu : (left > 0 ? (1u << left) - 1u : 0u);   // attends to all L keys alike
        ptx::tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float4 x = row[c0 / 4 + c];
          const float add[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float scaled = q_keep ? (v[4 * c + k] + add[k]) * scale_log2 : 0.0f;
            v[4 * c + k] = (bits >> (4 * c + k)) & 1u ? scaled : -INFINITY;
            mx = fmaxf(mx, v[4 * c + k]);
          }
          row[c0 / 4 + c] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
        }
      }
      // row maximum over both halves of the tile; both have read S, so that P may take its place
      xmax[(t & 1) * 2 * BM + hf * BM + r] = mx;
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->pair[quarter]);
      ok = wait(&bars->pair[quarter], (uint32_t)t & 1u, kCode + 87);
      if (!ok) break;
      ptx::tc_fence_after();
      const float m_new = fmaxf(m_run, fmaxf(mx, xmax[(t & 1) * 2 * BM + (1 - hf) * BM + r]));
      const float m_use = m_new == -INFINITY ? 0.0f : m_new;
      const float corr = exp2f(m_run - m_use);   // 0 while nothing has been attended to
      m_run = m_new;
      if (t > 0) add_output(corr);   // the previous tile's PV (complete before S was issued), before its scale is left behind
      // (exp2f: ex2.approx.ftz makes zeros of probabilities below 2^-126, and takes 2 % less at d 32, 0.5 % at d 64)
      float sum = 0.0f;
#pragma unroll 1
      for (int c0 = 0; c0 < HK; c0 += 16) {
        float e[16];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float4 x = row[c0 / 4 + c];
          e[4 * c] = exp2f(x.x - m_use);
          e[4 * c + 1] = exp2f(x.y - m_use);
          e[4 * c + 2] = exp2f(x.z - m_use);
          e[4 * c + 3] = exp2f(x.w - m_use);
          sum += (e[4 * c] + e[4 * c + 1]) + (e[4 * c + 2] + e[4 * c + 3]);
        }
        uint32_t lo[kPlanes][4], hi[kPlanes][4];
        split_eight(e, lo);
        split_eight(e + 8, hi);
#pragma unroll
        for (int q = 0; q < kPlanes; ++q) {
          const uint32_t w[8] = {lo[q][0], lo[q][1], lo[q][2], lo[q][3], hi[q][0], hi[q][1], hi[q][2], hi[q][3]};
          ptx::tmem_st8(t_p + (uint32_t)(q * (BN / 2) + c0 / 2), w);
        }
      }
      l_run = l_run * corr + sum;
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->p_full);
    }
    if (ok) {
      float* xsum = xmax + (n_kt & 1) * 2 * BM;   // the parity the last tile did not use
      xsum[hf * BM + r] = l_run;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->pair[quarter]);
      ok = wait(&bars->pair[quarter], (uint32_t)n_kt & 1u, kCode + 89);
      const float inv = 1.0f / (l_run + xsum[(1 - hf) * BM + r]);
      ok = ok && wait(&bars->o_full, (uint32_t)(n_kt - 1) & 1u, kCode + 88);
      ptx::tc_fence_after();
      add_output(inv);
      // through the rows in shared memory, so that D / 4 lanes store a row
#pragma unroll
      for (int c = 0; c < OW; c += 4)
        *reinterpret_cast<float4*>(rel + r * kPitch + hf * OW + c) = make_float4(o[c], o[c + 1], o[c + 2], o[c + 3]);
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->pair[quarter]);
      ok = wait(&bars->pair[quarter], (uint32_t)(n_kt + 1) & 1u, kCode + 91) && ok;
      constexpr int kLanes = D / 4, kRowsAtOnce = 32 / kLanes;
      const int c = lane % kLanes * 4;
#pragma unroll 4
      for (int it = 0; it < 16 / kRowsAtOnce; ++it) {
        const int row = quarter * 32 + hf * 16 + it * kRowsAtOnce + lane / kLanes;
        if (!ok || i0 + row >= L) continue;
        const float4 x = *reinterpret_cast<const float4*>(rel + row * kPitch + c);
        const float f[4] = {x.x, x.y, x.z, x.w};
        const long long at = ((long long)b * L + i0 + row) * ((long long)H * D) + (long long)h * D + c;
        if (out_planes) {
          uint2 w[kPlanes];
          split3x4(f, w);
          const long long plane = (long long)p.batch * L * H * D;
#pragma unroll
          for (int q = 0; q < kPlanes; ++q) *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + q * plane + at) = w[q];
        } else {
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + at) = x;
        }
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) ptx::tmem_dealloc(tmem_base, kTmemCols);
}

template <int D>
int smem_bytes(int L) {
  return Shape<D>::offKeep + (L + BN - 1) / BN * BN / 8 + (2 * L - 1) * 2 + 1024 + 16;
}

template <int D>
int launch_d(const DflAttnParams& p, const void* pos_key, const void* pos_query, int n_active, int out_planes, cudaStream_t stream) {
  using T = Shape<D>;
  const int L = p.seq_len, BH = p.batch * p.heads;
  const uint64_t row = (uint64_t)D * 2, seq = (uint64_t)L * row;
  CUtensorMap tq, tk;
  int rc = encode_tensor_map_3d(&tq, p.q, D, L, (uint64_t)kPlanes * BH, row, seq, D, BM, T::kRowBytes);
  if (rc == DFL_OK) rc = encode_tensor_map_3d(&tk, p.k, D, L, (uint64_t)kPlanes * BH, row, seq, D, BN, T::kRowBytes);
  if (rc != DFL_OK) return rc;
  auto kernel = attention_f32_rel_kernel<D>;
  static KernelDeviceConfig config;   // per instantiation
  rc = configure_kernel(config, kernel, kMaxSmem, nullptr, "attention_f32_rel_kernel");
  if (rc != DFL_OK) return rc;
  int* status_word = p.status;
  if (!status_word) {
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&status_word), g_attn_f32_rel_status);
    if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "status word: %s", cudaGetErrorString(e));
  }
  // never so little shared memory that a second CTA could become resident: each takes all of tensor memory
  const int smem = smem_bytes<D>(L), floor_smem = kMaxSmem / 2 + 1024;
  const long long items = (long long)((L + BM - 1) / BM) * BH;
  if (items > 0x7fffffff) return fail(DFL_ERR_TOO_LARGE, "too many query tiles");
  cudaError_t e = launch_after_predecessor(kernel, dim3((unsigned)items), dim3(kThreads), (size_t)(smem < floor_smem ? floor_smem : smem),
                                           stream, tq, tk, p, reinterpret_cast<const __nv_bfloat16*>(pos_key),
                                           reinterpret_cast<const __nv_bfloat16*>(pos_query), n_active, out_planes, status_word);
  if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "attention_f32_rel_kernel: %s", cudaGetErrorString(e));
  return check_launch("attention_f32_rel_kernel");
}

}  // namespace

bool attention_f32_rel_supported(int head_dim, int seq_len) {
  if (seq_len < 1) return false;
  return head_dim == 64 ? smem_bytes<64>(seq_len) <= kMaxSmem : (head_dim == 32 && smem_bytes<32>(seq_len) <= kMaxSmem);
}

int launch_attention_f32_rel(const DflAttnParams& p, const void* pos_key, const void* pos_query, int n_active, int out_planes,
                             cudaStream_t stream) {
  return p.head_dim == 64 ? launch_d<64>(p, pos_key, pos_query, n_active, out_planes, stream)
                          : launch_d<32>(p, pos_key, pos_query, n_active, out_planes, stream);
}

}  // namespace dfl
