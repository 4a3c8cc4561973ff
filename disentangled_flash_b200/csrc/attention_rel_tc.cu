// tcgen05 fused disentangled attention over position tables laid out by relative distance.
//
// Same result as dfl_pos_scores + dfl_attention_fwd (reference: the two torch.matmul calls at
// src/disentangled_flash/kernel.py:574-585 followed by the Triton kernel kernel.py:137-345).  The tables
// rel_key / rel_query [H, 2L-1, d] hold, in row e, the position projection every (query i, key j) pair with
// x = j - i = e - (L-1) uses, so the two relative terms of a (128 query x 128 key) tile are
//   C2P[i, j] = q_i . rel_key[x]      P2C[i, j] = k_j . rel_query[x]
// with x running over one contiguous window of 255 table rows.  Both are produced by tcgen05.mma from 128-row
// table blocks (L2 resident) and rounded to the input type exactly like the separate score GEMMs round their output;
// converter warps undo the diagonal on the way through shared memory:
//   C2P depends on the query rows only: D[r, m] = q_r . rel_key[x_lo + m] with TMEM lanes = query rows.  The window of a
//       key tile is two 128-column blocks; the next key tile needs one new block.  Converter warps round a block's rows and
//       store each shifted by its row, so that key x of the tile ends up in column x: a softmax thread adds its 64 scores
//       from eight 16-byte loads.
//   P2C is new for every key tile: D[n, m] = k_n . rel_query[x_lo + m] with TMEM lanes = keys n, computed in four
//       parts of 64 table rows through two 64-column accumulators.  Here the diagonal runs across the lanes' columns and
//       the softmax threads need it transposed: converter warps round each key's row and store it, shifted by its key, as
//       row n of a K-major B operand, and S gets it by one more MMA, S += I . tile^T with an identity matrix as A.  The
//       tensor pipe is idle three quarters of the time otherwise; it transposes and adds exactly (one product by 1.0 and
//       zeros, fp32 accumulation).
//
// Persistent: one CTA per SM walks (batch, head, 128-query tile) items in 128-key tiles; every role keeps running
// counters so that the barrier phases carry over from item to item and the loader / MMA issuers run ahead.
//   warps 0-7   softmax: two threads per query row (warps w and w+4 own the same TMEM lanes; each takes 64 of the
//               128 keys of a tile, 32 of the 64 packed P columns and half of the output columns).  One pass: the 64
//               scores stay in registers from the S load to the P store.
//   warps 8-15  converters of the P2C parts (TMEM -> 16-bit -> shared memory), warps 16-23 of the C2P blocks; two warps
//               per TMEM lane quarter and role, one for each accumulator of the role's pair
//   warp 24     issuer of S with the P2C tile added, and TMEM owner
//   warp 25     per-item mask analysis (kept-key bits, skipped key tiles), one item ahead, and TMA producer of Q, K, rel_query
//   warp 26     issuer of the PV and C2P block MMAs and of the loads of V and rel_key, warp 27 of the P2C parts
// What bounds it: a 128 x 128 tile takes 5.4 k cycles, of which a softmax thread works 3.5 k and waits 1.2 k for S; S waits
// for the P2C operand, which the converters fill in 2.5 k once the identity MMA has released it.  No unit is busy: each role is
// a chain of dependent instructions that its warps cannot overlap with themselves, so what helps is more warps a role and
// loads far enough ahead.  us, launch after launch, both terms, no padding, before (one converter warp per quarter and role,
// one loader in MMA order, C2P behind S in one issuer) and now:
//   32 x 12 heads x 512 x d 64 fp16 155 -> 135     64 x 16 x 256 x 64 bf16 109 -> 95     7 x 12 x 333 x 64 bf16 29.1 -> 26.2
//   16 x 24 x 256 x d 32 fp16 46.9 -> 38.6         16 x 8 x 512 x d 128 bf16 104 -> 78
// The same sizes in that order with lengths uniform in [L/2, L], and without padding C2P alone and P2C alone (kernel times):
//   140 -> 121, 114 -> 99, 28.6 -> 25.6, 46.8 -> 41.0, 103 -> 77;   114 -> 94, 84 -> 79, 22.4 -> 20.8, 34.6 -> 32.0, 76 -> 56.6;
//   134 -> 113, 93 -> 79, 25.7 -> 22.5, 40.0 -> 32.3, 85 -> 71
// The converters' register budget matters more than their number: at 48 registers with the next columns in flight while the
// last are stored they spill, and the kernel took 238 us.  The waits, the loader and the MMA loops are rolled: with everything
// unrolled (156 KB of code) a third of the issue slots were lost to instruction fetch.
#include <type_traits>

#include "attention_tc_common.cuh"

namespace dfl {

__device__ int g_attn_rel_status = 0;

namespace {

using attn::Pack2;

constexpr int BM = 128;              // query rows per item (= TMEM lanes)
constexpr int BK = 128;              // keys per tile
constexpr int kSoftmaxWarps = 8;
constexpr int kC2pWarp = 16;         // warps 8-15 convert the P2C parts, 16-23 the C2P blocks
constexpr int kMmaWarp = 24;
constexpr int kTmaWarp = 25;
constexpr int kPvWarp = 26;
constexpr int kPartWarp = 27;
constexpr int kThreads = 896;
constexpr int kSoftmaxRegs = 128;    // 256 x 128 + 512 x 48 + 128 x 56 = 64512 registers
constexpr int kConvRegs = 48;
constexpr int kMiscRegs = 56;
// The kernel is launched with 65536 / kThreads registers per thread, rounded down to the allocation unit of 8: 72.
// `setmaxnreg.inc` waits until the pool holds what it asks for, so the three budgets must not ask for more than the SM has (a wait that nothing could
// bound); `setmaxnreg.dec` with a value above the launch allocation is an illegal instruction.
constexpr int kLaunchRegs = 65536 / kThreads / 8 * 8;
static_assert(8 * 32 * kSoftmaxRegs + 16 * 32 * kConvRegs + 4 * 32 * kMiscRegs <= kThreads * kLaunchRegs,
              "register budgets of the three warpgroup kinds exceed what the launch allocates");
static_assert(kSoftmaxRegs >= kLaunchRegs && kConvRegs <= kLaunchRegs && kMiscRegs <= kLaunchRegs &&
                  kSoftmaxRegs % 8 == 0 && kConvRegs % 8 == 0 && kMiscRegs % 8 == 0,
              "setmaxnreg.inc raises and setmaxnreg.dec lowers the launch allocation, in multiples of 8");
constexpr int kConsumerWarps = 27;   // softmax, converters, MMA issuers: every warp that reads an item slot

constexpr int kItemSlots = 3;        // the loader analyses one item ahead of the one whose tiles it loads
constexpr int kMaxSeqLen = 2048;
constexpr int kMaskWords = kMaxSeqLen / 32;   // kept-key bits per item

// C2P rows: per query row two tiles of 128 16-bit scores, tile T of the CTA's running count in half T & 1, key x of the tile
// at column x: the softmax thread of the row reads its 64 keys as eight 16-byte words.  33 16-byte units per row: eight
// consecutive rows hit different bank groups with those reads, and the converters' 4-byte stores conflict 2-way.
constexpr int ROW_PITCH = 528;
// P2C tile: the B operand of the MMA that adds it to S, K-major without swizzle: 8-row core matrices of 128 bytes, rows =
// keys, K = query rows.  Chunks of eight query rows are STG_CHUNK bytes apart (32 bytes more than 16 core matrices, so
// that the 4-byte stores of 32 neighbouring keys, each shifted by its key, fall into 32 different banks).
constexpr int STG_CHUNK = 16 * 128 + 32;
constexpr int STG_BYTES = 16 * STG_CHUNK;
// Identity operand of that MMA, a strip of 16-byte rows: row 120 + c holds a one in column c.  The two chunks of eight columns
// of a K = 16 step are windows of 128 rows of this strip, EYE_LBO apart: k-step kk of the 128 x 128 identity takes the window
// from row 112 - 16 kk for the upper eight of its columns and the one eight rows further down for the lower eight (the
// P2C operand gives its chunks in that order too: they lie in descending order of the query rows).
constexpr int EYE_ROWS = 248;
constexpr int EYE_LBO = 128;
constexpr int EYE_BYTES = EYE_ROWS * 16;

// TMEM columns (all 512; one CTA per SM)
constexpr int COL_S = 0;      // 128  S = Q K^T of the current tile (fp32)
constexpr int COL_P = 128;    // 64   P of the current tile (16-bit pairs), A operand of the PV MMA
constexpr int COL_O = 192;    // D    O accumulator
                              // XC: 2 x 64   halves of a new C2P block for the 128 query rows, from 256 on; with d = 128
                              // both in turn in the 64 columns from 320 on
constexpr int COL_XP = 384;   // 2 x 64  two of the four parts (64 table rows each) of the P2C accumulator of a key tile
constexpr int kTmemCols = 512;

template <int D>
struct RLayout {
  static_assert(D == 32 || D == 64 || D == 128, "head dims 32, 64 and 128");
  // An operand tile is kSub sub-tiles of at most 64 columns, one swizzled 64- or 128-byte row per tile row.  The tables come
  // in pieces of 64 rows, V at d = 128 too.
  static constexpr int kSub = D > 64 ? 2 : 1;
  static constexpr int kRowBytes = D * 2 / kSub;
  static constexpr int kTile = 128 * D * 2;            // Q tile, K tile
  static constexpr int kTab = 64 * D * 2;              // piece of a table
  static constexpr int kVPieces = D > 64 ? 2 : 1;
  static constexpr int kVRows = 128 / kVPieces;
  static constexpr int kVPiece = kVRows * D * 2;
  static constexpr int kKStages = D > 64 ? 1 : 2;
  static constexpr int kVStages = D == 32 ? 2 : 1;
  // d = 64 and 128 fill shared memory.
  static constexpr int kRkStages = D == 32 ? 4 : (D == 64 ? 3 : 1);
  static constexpr int kRqStages = D == 32 ? 4 : (D == 64 ? 4 : 1);
  // P2C operand tiles.  d 64 has room for a second one only if rel_key has one stage and rel_query two: 132 us against 135 at
  // 32 x 12 heads x 512, but 104 against 95 at 64 x 16 x 256, where items are short and begin with four loads of rel_key.
  static constexpr int kStgs = D == 32 ? 2 : 1;
  static constexpr int kXcCols = 64, kXcs = D > 64 ? 1 : 2;   // C2P accumulators
  static constexpr int kColXc = D > 64 ? 320 : 256;
  static constexpr int offQ = 0;
  static constexpr int offK = offQ + kTile;
  static constexpr int offV = offK + kKStages * kTile;
  static constexpr int offRK = offV + kVStages * kVPiece;
  static constexpr int offRQ = offRK + kRkStages * kTab;
  static constexpr int offRows = offRQ + kRqStages * kTab;
  static constexpr int offStg = offRows + BM * ROW_PITCH;
  static constexpr int offEye = offStg + kStgs * STG_BYTES;
  static constexpr int offBar = offEye + EYE_BYTES;
  static constexpr int kBarBytes = 512;
  // exchange area: [2 parities][2 halves][BM] row maxima (row sums at the end of an item, partial column sums of V)
  static constexpr int offXmax = offBar + kBarBytes;
  static constexpr int offItem = offXmax + (D > 64 ? 8 * D * 4 : 2 * 2 * BM * 4);
  static constexpr int kItemBytes = 304;
  static constexpr int total = offItem + kItemSlots * kItemBytes;
  static_assert(offStg % 16 == 0 && offBar % 16 == 0 && offItem % 16 == 0, "alignment");
  static_assert(total <= 232448, "shared memory budget");
};

// What the loader warp publishes per item.
struct ItemSlot {
  int t_begin, t_end;   // key tiles [t_begin, t_end) are processed
  int any_kept;         // 0: every query row of the tile is padding -> mean-of-V path, no pipeline work; 2: padded rows beside
                        // kept ones, and key tiles that are not walked
  int bh, h, i0;        // batch*heads + head, head, first query row
  int out_rows;         // rows of the sequence the output holds, from out_row0 on: [B,L,H*d], or packed rows (see
  long long out_row0;   // DflAttnRelParams.out_row_base)
  uint32_t kbits[kMaskWords];   // kept-key bits of the batch row, word w = keys [32w, 32w+32)
};
static_assert(sizeof(ItemSlot) <= 304, "item slot too large");

struct RBarriers {
  uint64_t q_full, q_empty;
  uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2];
  uint64_t rk_full[4], rk_empty[4], rq_full[4], rq_empty[4];
  uint64_t s_full, s_free;          // S accumulator: MMA -> softmax, softmax (8 warps) -> MMA
  uint64_t xc_full[2], xc_free[2];  // halves of a C2P block: MMA -> converters (4 warps each) -> MMA
  uint64_t xp_full[2], xp_free[2];  // P2C part accumulators: MMA -> converters (4 warps) -> MMA
  uint64_t pt_ready[2], pt_release[2];   // P2C tiles in shared memory: converters -> MMA (its reads complete) -> converters
  uint64_t p_full, o_ready, o_free; // P stored (8 warps); PV complete; output accumulator read out (8 warps)
  uint64_t c2p_ready, ring_release; // C2P rows of a tile: converters -> softmax -> converters
  uint64_t pair2[4];                // the two warps of a lane quarter: row maximum (row sum) posted
  uint64_t item_full[kItemSlots], item_empty[kItemSlots];
  uint64_t xbar;                    // the eight softmax warps (column sums of V, for padded query rows)
  uint32_t tmem_base;
};
static_assert(sizeof(RBarriers) <= 512, "barrier block too large");

template <int N>
__device__ __forceinline__ void setmaxnreg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

__device__ __forceinline__ uint4 lds_v4(uint32_t saddr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(saddr) : "memory");
  return v;
}
// {hi, lo} >> amount, low 32 bits; amount 0 or 16 (wrap), 16 or 32 (clamp)
__device__ __forceinline__ uint32_t funnel_wrap(uint32_t lo, uint32_t hi, uint32_t amount) {
  uint32_t v;
  asm("shf.r.wrap.b32 %0, %1, %2, %3;" : "=r"(v) : "r"(lo), "r"(hi), "r"(amount));
  return v;
}
__device__ __forceinline__ uint32_t funnel_clamp(uint32_t lo, uint32_t hi, uint32_t amount) {
  uint32_t v;
  asm("shf.r.clamp.b32 %0, %1, %2, %3;" : "=r"(v) : "r"(lo), "r"(hi), "r"(amount));
  return v;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float m;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}
__device__ __forceinline__ void sts_u32(uint32_t saddr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(saddr), "r"(v) : "memory");
}
__device__ __forceinline__ void sts_u32_if(uint32_t saddr, uint32_t v, bool on) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.u32 [%0], %1;\n\t}" ::"r"(saddr), "r"(v), "r"((int)on) : "memory");
}
// ... if bit `bit` of `mask` is set
__device__ __forceinline__ void sts_u32_bit(uint32_t saddr, uint32_t v, uint32_t mask, int bit) {
  asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %2, %3;\n\tsetp.ne.b32 p, t, 0;\n\t@p st.shared.u32 [%0], %1;\n\t}"
               ::"r"(saddr), "r"(v), "r"(mask), "r"(1u << bit) : "memory");
}
__device__ __forceinline__ void sts_u16_if(uint32_t saddr, uint32_t v, bool on) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.u16 [%0], %1;\n\t}" ::"r"(saddr), "h"((unsigned short)v), "r"((int)on) : "memory");
}
// Two scores rounded to T and packed.  FP16 saturates: a score beyond 65504 would be an infinity, and the MMA that adds
// the P2C tile to S multiplies the other rows' entries of that key by zero.
template <typename T>
__device__ __forceinline__ uint32_t pack_scores(float lo, float hi) {
  uint32_t v;
  if constexpr (__is_same(T, __half)) asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
  else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
  return v;
}

// 32 consecutive fp32 TMEM columns of this thread's lane into arr[off .. off+31] (a register array indexed by
// compile-time constants; no address of the array is taken, so it stays in registers across loop iterations).
#define DFL_TMEM_LD32_F(taddr, arr, off)                                                                            \
  asm volatile(                                                                                                     \
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "                                                                     \
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "                                     \
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"                     \
      : "=f"(arr[off + 0]), "=f"(arr[off + 1]), "=f"(arr[off + 2]), "=f"(arr[off + 3]), "=f"(arr[off + 4]),          \
        "=f"(arr[off + 5]), "=f"(arr[off + 6]), "=f"(arr[off + 7]), "=f"(arr[off + 8]), "=f"(arr[off + 9]),          \
        "=f"(arr[off + 10]), "=f"(arr[off + 11]), "=f"(arr[off + 12]), "=f"(arr[off + 13]), "=f"(arr[off + 14]),     \
        "=f"(arr[off + 15]), "=f"(arr[off + 16]), "=f"(arr[off + 17]), "=f"(arr[off + 18]), "=f"(arr[off + 19]),     \
        "=f"(arr[off + 20]), "=f"(arr[off + 21]), "=f"(arr[off + 22]), "=f"(arr[off + 23]), "=f"(arr[off + 24]),     \
        "=f"(arr[off + 25]), "=f"(arr[off + 26]), "=f"(arr[off + 27]), "=f"(arr[off + 28]), "=f"(arr[off + 29]),     \
        "=f"(arr[off + 30]), "=f"(arr[off + 31])                                                                     \
      : "r"(taddr)                                                                                                  \
      : "memory")

// s0 += lo half of w, s1 += hi half of w (w = two packed values of type T), in fp32.
template <typename T>
__device__ __forceinline__ void add_pair(float& s0, float& s1, uint32_t w);
template <>
__device__ __forceinline__ void add_pair<__half>(float& s0, float& s1, uint32_t w) {
  asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tadd.rn.f32.f16 %0, lo, %0;\n\tadd.rn.f32.f16 %1, hi, %1;\n\t}"
      : "+f"(s0), "+f"(s1)
      : "r"(w));
}
template <>
__device__ __forceinline__ void add_pair<__nv_bfloat16>(float& s0, float& s1, uint32_t w) {
  asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tadd.rn.f32.bf16 %0, lo, %0;\n\tadd.rn.f32.bf16 %1, hi, %1;\n\t}"
      : "+f"(s0), "+f"(s1)
      : "r"(w));
}

// Kept-key bits of batch row b, one word of 32 keys per lane: lane l gets words l (lo) and l + 32 (hi).  Warp-collective:
// the mask is read 32 elements at a time, sixteen words in flight.
__device__ __forceinline__ void kept_bits(const DflAttnRelParams& p, int b, int lane, uint32_t& lo, uint32_t& hi) {
  const int L = p.seq_len, n_words = (L + 31) / 32;
  const long long base = (long long)b * L;
  lo = hi = 0;
#pragma unroll 1
  for (int w0 = 0; w0 < n_words; w0 += 16) {
    bool keep[16];
#pragma unroll
    for (int x = 0; x < 16; ++x) {
      const int j = 32 * (w0 + x) + lane;
      keep[x] = j < L && mask_keep(p.mask, p.mask_elem_size, base + j);
    }
#pragma unroll
    for (int x = 0; x < 16; ++x) {
      const uint32_t bits = __ballot_sync(0xffffffffu, keep[x]);
      if (lane == ((w0 + x) & 31)) {
        if (w0 + x < 32) lo = bits;
        else hi = bits;
      }
    }
  }
}

// Key tiles before the first and after the last kept key contribute nothing to a kept query row (their
// probabilities are exactly zero) and are skipped.  A padded query row attends uniformly to all L keys: where a tile has both
// kinds of rows (fold), the softmax threads add the column sums of V over the skipped keys to its padded rows.  A tile of padded
// rows only is the column mean of V (any_kept false).
// Warp-collective: lane l holds the kept-key words l (kb_lo) and l + 32 (kb_hi) of the batch row.
struct TileRange {
  int t_begin, t_end;
  bool any_kept, fold;
};
__device__ __forceinline__ TileRange tile_range(uint32_t kb_lo, uint32_t kb_hi, int i0, int L, int lane) {
  const int n_kt = (L + BK - 1) / BK;
  const uint32_t nz_lo = __ballot_sync(0xffffffffu, kb_lo != 0u);
  const uint32_t nz_hi = __ballot_sync(0xffffffffu, kb_hi != 0u);
  const int qw = i0 >> 5;                       // first mask word of the query tile (a multiple of 4)
  const bool q_hi = qw >= 32;
  const uint32_t kb = q_hi ? kb_hi : kb_lo;
  const int wl = qw & 31;
  const bool in_q = lane >= wl && lane < wl + BM / 32;
  const int rows_here = L - 32 * (lane + (q_hi ? 32 : 0));   // in-range rows of this lane's word
  const uint32_t full = rows_here >= 32 ? 0xffffffffu : (rows_here <= 0 ? 0u : ((1u << rows_here) - 1u));
  const bool any_kept = __ballot_sync(0xffffffffu, in_q && kb != 0u) != 0u;
  const bool any_padded = __ballot_sync(0xffffffffu, in_q && (kb & full) != full) != 0u;
  TileRange r{0, n_kt, any_kept, false};
  if ((nz_lo | nz_hi) != 0u) {
    const int first = nz_lo ? __ffs(nz_lo) - 1 : 32 + __ffs(nz_hi) - 1;
    const int last = nz_hi ? 32 + 31 - __clz(nz_hi) : 31 - __clz(nz_lo);
    r.t_begin = first >> 2;
    r.t_end = (last >> 2) + 1;
    r.fold = any_kept && any_padded && (r.t_begin > 0 || r.t_end < n_kt);
  }
  return r;
}

// D[128 x N] = A[128 x d] * B[N x d]^T, both operands K-major tiles in shared memory; a_sub, b_sub: descriptor units from
// one 64-column sub-tile to the next.  One converged warp.
template <int D>
__device__ __forceinline__ void mma_over_d(uint32_t d_tmem, uint64_t a_desc, uint32_t a_sub, uint64_t b_desc, uint32_t b_sub,
                                           uint32_t idesc) {
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    ptx::umma_ss_f16_warp(d_tmem, a_desc, b_desc, idesc, kk != 0 ? 1u : 0u);
    a_desc += D > 64 && kk == 3 ? a_sub - 6u : 2u;
    b_desc += D > 64 && kk == 3 ? b_sub - 6u : 2u;
  }
}

template <typename T, int D>
__global__ void __launch_bounds__(kThreads, 1)
attention_rel_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                     const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_fk,
                     const __grid_constant__ CUtensorMap tmap_fq, const DflAttnRelParams p, int* status_word,
                     int n_items) {
  using LO = RLayout<D>;
  extern __shared__ __align__(1024) unsigned char smem[];   // the swizzled tiles need the alignment
  RBarriers* bars = reinterpret_cast<RBarriers*>(smem + LO::offBar);
  ItemSlot* slots = reinterpret_cast<ItemSlot*>(smem + LO::offItem);

  const int L = p.seq_len, H = p.heads;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const bool has_c2p = p.rel_key != nullptr, has_p2c = p.rel_query != nullptr;
  int fail_code = 0;   // code of the bounded wait of this thread that expired first, if any

  // ------------------------------------------------------------------ setup (once per CTA)
  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_full, 1);
    ptx::mbar_init(&bars->q_empty, has_c2p ? 2 : 1);          // its issuers: Q K^T, and C2P blocks
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(&bars->k_full[s], 1);
      ptx::mbar_init(&bars->k_empty[s], has_p2c ? 2 : 1);   // its issuers: Q K^T, and P2C parts
      ptx::mbar_init(&bars->v_full[s], 1);
      ptx::mbar_init(&bars->v_empty[s], 1);
    }
    for (int s = 0; s < 4; ++s) {
      ptx::mbar_init(&bars->rk_full[s], 1);
      ptx::mbar_init(&bars->rk_empty[s], 1);
      ptx::mbar_init(&bars->rq_full[s], 1);
      ptx::mbar_init(&bars->rq_empty[s], 1);
    }
    for (int s = 0; s < kItemSlots; ++s) {
      ptx::mbar_init(&bars->item_full[s], 1);
      ptx::mbar_init(&bars->item_empty[s], kConsumerWarps);
    }
    ptx::mbar_init(&bars->s_full, 1);
    ptx::mbar_init(&bars->s_free, kSoftmaxWarps);   // one elected lane per softmax warp
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(&bars->xc_full[s], 1);
      ptx::mbar_init(&bars->xc_free[s], 4);         // converter warps
      ptx::mbar_init(&bars->xp_full[s], 1);
      ptx::mbar_init(&bars->xp_free[s], 4);         // converter warps
      ptx::mbar_init(&bars->pt_ready[s], 8);
      ptx::mbar_init(&bars->pt_release[s], 1);
    }
    ptx::mbar_init(&bars->p_full, kSoftmaxWarps);
    ptx::mbar_init(&bars->o_ready, 1);
    ptx::mbar_init(&bars->o_free, kSoftmaxWarps);
    ptx::mbar_init(&bars->c2p_ready, 8);
    ptx::mbar_init(&bars->ring_release, kSoftmaxWarps);
    for (int s = 0; s < 4; ++s) ptx::mbar_init(&bars->pair2[s], 2);
    ptx::mbar_init(&bars->xbar, kSoftmaxWarps);
    ptx::fence_mbar_init();
  }
  // identity operand: zeros with ones on rows 120 .. 127
  for (int e = threadIdx.x; e < EYE_ROWS; e += kThreads) {
    const int col = e - 120;   // column of the one, if in [0, 8)
    const uint32_t one = __is_same(T, __half) ? 0x3C00u : 0x3F80u;
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = col == 2 * j ? one : (col == 2 * j + 1 ? one << 16 : 0u);
    *reinterpret_cast<uint4*>(smem + LO::offEye + e * 16) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  ptx::fence_proxy_async_smem();
  if (warp == kTmaWarp && lane == 0) {
    ptx::prefetch_tensormap(&tmap_q);
    ptx::prefetch_tensormap(&tmap_k);
    ptx::prefetch_tensormap(&tmap_v);
    ptx::prefetch_tensormap(&tmap_fk);
    ptx::prefetch_tensormap(&tmap_fq);
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc(&bars->tmem_base, kTmemCols);
    ptx::tmem_relinquish();
  }
  // Item order: item = query tile * (batch*heads) + batch*head, so the items of one CTA (stride gridDim) differ in
  // query tile and batch row, which evens out the padding-dependent cost without any bookkeeping.
  const int n_bh = p.batch * H;
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  // A bounded wait whose verdict is the same in every lane of the warp (the tcgen05.ld/st/wait instructions that
  // follow are warp-collective and must not be reached by part of a warp).
  auto wwait = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
    return ptx::mbar_wait_warp(bar, parity, fail_code, code);
  };

  // The set-up above overlaps the tail of the previous kernel of the stream; Q, K, V, the mask and the status word
  // are touched from here on.
  wait_for_predecessor();

  // Every role walks the same item sequence (item number k of this CTA is item blockIdx.x + k * gridDim.x; it uses
  // item slot k % 3 in phase (k / 3) & 1) and keeps its own running counters.  Register budgets are set per
  // warpgroup (warps 0-7: softmax; 8-23: converters; 24-27: the rest), at the head of the branch the whole warpgroup
  // takes.
  if (warp < kSoftmaxWarps) {
    setmaxnreg_inc<kSoftmaxRegs>();
    // ----------------------------------------------------------------- softmax
    const int hf = warp >> 2, q4 = warp & 3;    // key half of the tile, lane quarter
    const int r = q4 * 32 + lane;               // query row of the tile = TMEM lane
    const float cscale = p.scale * 1.4426950408889634f;
    const float slack = attn::kLazyMaxSlack / cscale;
    constexpr int OW = D / 2;                   // output columns per thread
    const uint32_t lane_base = (uint32_t)(q4 * 32) << 16;
    const uint32_t t_s = tmem_base + lane_base + COL_S + hf * 64;
    const uint32_t t_p = tmem_base + lane_base + COL_P + hf * 32;
    const uint32_t t_o = tmem_base + lane_base + COL_O + hf * OW;
    const uint32_t c2p_row = ptx::smem_u32(smem + LO::offRows) + (uint32_t)(r * ROW_PITCH + hf * 128);   // this thread's 64 keys
    float* xchg = reinterpret_cast<float*>(smem + LO::offXmax);
    uint64_t* pair2 = &bars->pair2[q4];
    // Two running counts give every barrier phase of this role: c_t = key tiles started (all items), c_i = items with
    // kept rows finished.  Per tile one phase each of s_full, c2p_ready and o_ready, per tile and per item one of pair2;
    // an item that takes column sums of V (padded rows only, or beside kept ones) uses xbar exactly four times.
    uint32_t c_t = 0, c_i = 0;
    bool ok = true;

    int k = 0;
    for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x, ++k) {
      const int slot = k % kItemSlots;
      ok = wwait(&bars->item_full[slot], (uint32_t)(k / kItemSlots) & 1u, 33);
      if (!ok) break;
      const ItemSlot* sl = &slots[slot];
      const int t_begin = sl->t_begin, n = sl->t_end - sl->t_begin;
      const int kind = sl->any_kept;
      const bool any_kept = kind != 0;
      const int bh = sl->bh, h = sl->h;
      const int i0 = sl->i0;
      const long long out_row0 = sl->out_row0;
      const int out_rows = sl->out_rows;
      if (!any_kept && out_rows <= i0) {
        // a tile of padded positions that the packed output does not hold: nothing to compute, nothing to store
      } else {
        const int i = i0 + r;
        const bool row_ok = i < L;
        const bool q_keep = row_ok && ((sl->kbits[i >> 5] >> (i & 31)) & 1u) != 0u;
        float m_run = -INFINITY, l_run = 0.0f;

        for (int u = 0; u < n && any_kept && ok; ++u) {
          const int t = t_begin + u;
          const uint32_t kb0 = sl->kbits[4 * t + 2 * hf], kb1 = sl->kbits[4 * t + 2 * hf + 1];
          const int n_in = L - t * BK - hf * 64;   // in-range keys among this thread's 64 (may be <= 0 or >= 64)
          const uint32_t tile_phase = c_t & 1u;
          ++c_t;
          ok = wwait(&bars->s_full, tile_phase, 41);
          if (!ok) break;
          ptx::tc_fence_after();

          // Scores of the thread's 64 keys: Q.K plus the P2C term from tensor memory (the MMA issuer has added the
          // term), the C2P term from the thread's row in shared memory.  They stay in registers until P is stored.
          float s[64];
          DFL_TMEM_LD32_F(t_s, s, 0);
          DFL_TMEM_LD32_F(t_s + 32, s, 32);
          if (has_c2p) {
            ok = wwait(&bars->c2p_ready, tile_phase, 42);
            if (!ok) break;
            const uint32_t caddr = c2p_row + (tile_phase ? 256u : 0u);
            uint4 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = lds_v4(caddr + 16u * j);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int half = 0; half < 2; ++half) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int x = 32 * half + 8 * j;
                add_pair<T>(s[x], s[x + 1], w[j].x);
                add_pair<T>(s[x + 2], s[x + 3], w[j].y);
                add_pair<T>(s[x + 4], s[x + 5], w[j].z);
                add_pair<T>(s[x + 6], s[x + 7], w[j].w);
              }
              if (half == 0) {
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = lds_v4(caddr + 64u + 16u * j);
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) {   // S and the C2P row are in registers: both may be overwritten for the next tiles
                  ptx::mbar_arrive(&bars->s_free);
                  ptx::mbar_arrive(&bars->ring_release);
                }
              }
            }
          } else {
            ptx::tmem_wait_ld();
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&bars->s_free);
          }
          // mask: keys >= L and padded keys -> -inf; a padded query row -> 0 on every in-range key
          if (!q_keep) {
#pragma unroll
            for (int x = 0; x < 64; ++x) s[x] = x < n_in ? 0.0f : -INFINITY;
          } else if ((kb0 & kb1) != 0xffffffffu) {
#pragma unroll
            for (int x = 0; x < 32; ++x) {
              if (!((kb0 >> x) & 1u)) s[x] = -INFINITY;
              if (!((kb1 >> x) & 1u)) s[32 + x] = -INFINITY;
            }
          }
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int x = 0; x < 64; x += 2) mx[(x >> 1) & 3] = max3(mx[(x >> 1) & 3], s[x], s[x + 1]);
          const float my_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
          // the row maximum of the tile needs the other half of the keys: exchange through shared memory
          const uint32_t pair_phase = (c_t + c_i + 1u) & 1u;   // c_t - 1 tiles and c_i items before this exchange
          float* xm = xchg + pair_phase * (2 * BM);
          xm[hf * BM + r] = my_max;
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(pair2);
          ok = wwait(pair2, pair_phase, 45);
          if (!ok) break;
          const float tile_max = fmaxf(my_max, xm[(1 - hf) * BM + r]);

          // Lazy reference maximum: m_run moves only when the tile maximum exceeds it by more than 2^8 after scaling,
          // so exp2 arguments stay <= 8 (P <= 256, exact range of both 16-bit types) and O needs rescaling rarely.
          // Both threads of a row see the same m_run and tile_max and take the same decision.
          bool pv_seen = false;   // PV(u-1) known complete
          const bool move = tile_max > m_run + slack;   // also true for the first finite maximum
          if (__any_sync(0xffffffffu, move)) {
            const float m_new = move ? tile_max : m_run;
            const float m_use = m_new == -INFINITY ? 0.0f : m_new;
            const float corr = move ? ptx::ex2_approx((m_run - m_use) * cscale) : 1.0f;   // 0 when m_run = -inf
            m_run = m_new;
            l_run *= corr;
            if (u >= 1) {   // O holds the item's earlier tiles: rescale this thread's half of the columns
              ok = wwait(&bars->o_ready, c_t & 1u, 46);   // PV(u-1): c_t - 2 completed before it
              pv_seen = true;
              if (!ok) break;
              ptx::tc_fence_after();
#pragma unroll
              for (int c0 = 0; c0 < OW; c0 += 16) {
                uint32_t o[16];
                ptx::tmem_ld16(t_o + c0, o);
                ptx::tmem_wait_ld();
#pragma unroll
                for (int x = 0; x < 16; ++x) o[x] = __float_as_uint(__uint_as_float(o[x]) * corr);
                ptx::tmem_st16(t_o + c0, o);
              }
            }
          }
          const float neg_m = -(m_run == -INFINITY ? 0.0f : m_run) * cscale;

          // P = exp2(score * scale - reference), rounded, to the P columns; row sum.
          // The row sum is taken over P as rounded for the tensor core, so that the weights P/l the output is
          // built from sum to one exactly.  (The reference sums the unrounded values, kernel.py:316-333; with the
          // lazy reference maximum the largest P of a row is not the exactly representable 1.0, and an unrounded
          // sum would leave the rounding error of the dominant key uncompensated.)
          float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint32_t packed[16];
#pragma unroll
            for (int x = 0; x < 32; ++x) s[32 * q + x] = fmaf(s[32 * q + x], cscale, neg_m);
#pragma unroll
            for (int x = 0; x < 32; ++x) s[32 * q + x] = ptx::ex2_approx(s[32 * q + x]);
#pragma unroll
            for (int x = 0; x < 32; x += 2) packed[x / 2] = Pack2<T>::pack(s[32 * q + x], s[32 * q + x + 1]);
#pragma unroll
            for (int x = 0; x < 16; ++x) add_pair<T>(sum[(2 * x) & 3], sum[(2 * x + 1) & 3], packed[x]);
            // the P buffer is the A operand of the previous tile's PV until that MMA completes
            if (q == 0 && u >= 1 && !pv_seen) {
              ok = wwait(&bars->o_ready, c_t & 1u, 47);
              if (!ok) break;
              ptx::tc_fence_after();
            }
            ptx::tmem_st16(t_p + 16 * q, packed);
          }
          if (!ok) break;
          l_run += (sum[0] + sum[1]) + (sum[2] + sum[3]);
          ptx::tmem_wait_st();
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&bars->p_full);
        }
        if (!ok) break;

        // ---- row sums, the item's last PV, then normalise and store this thread's half of the output columns
        float total = 0.0f;
        if (any_kept) {
          const uint32_t sum_phase = (c_t + c_i) & 1u;
          float* xs = xchg + sum_phase * (2 * BM);
          xs[hf * BM + r] = l_run;
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(pair2);
          ok = wwait(pair2, sum_phase, 49);
          ++c_i;
          if (!ok) break;
          total = l_run + xs[(1 - hf) * BM + r];
        }
        if (kind != 1) {
          // Padded query rows attend uniformly to all L keys.  Where every row of the tile is one, the outputs are the column mean
          // of V: no score, no softmax.  Beside kept rows their weight is one on every key (their scores are zero, so is their
          // maximum), and the keys of the tiles that were not walked are a column sum of V added to the accumulator: 1.5 k cycles
          // where a tile takes 5.4 k.  Lengths uniform in [256, 512], us: 32 x 12 heads x 512 x d 64 122 -> 118, 16 x 8 x 512 x d 128
          // 78 -> 74.5.  16-byte loads, every thread sums 8 columns over a stride of rows; the row groups of a warp are folded with
          // shuffles and the eight warps through shared memory (the row-exchange words, idle from here to the next item).
          constexpr int kChunks = D / 8;             // 16-byte chunks per row of V
          constexpr int kRowStep = 256 / kChunks;    // rows covered by the 256 threads at once
          const int tid = threadIdx.x, chunk = tid % kChunks;
          const int before = any_kept ? t_begin * BK : L, after = min(L, (t_begin + n) * BK), skipped = any_kept ? before + L - after : L;
          const uint4* V4 = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.v) + (long long)bh * L * D);
          float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
          for (int x = tid / kChunks; x < skipped; x += kRowStep) {
            const int row = x < before ? x : x - before + after;
            const uint4 raw = __ldg(V4 + (long long)row * kChunks + chunk);
            const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] += Elem<T>::to_f(e[j]);
          }
#pragma unroll
          for (int o = kChunks; o < 32; o <<= 1) {
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
          }
          // every warp has read its partner's row sums of the item before
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&bars->xbar);
          ok = wwait(&bars->xbar, 0u, 34);
          if (!ok) break;
          if (lane < kChunks) {
#pragma unroll
            for (int j = 0; j < 8; ++j) xchg[warp * D + lane * 8 + j] = acc[j];
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&bars->xbar);
          ok = wwait(&bars->xbar, 1u, 36);
          if (!ok) break;
          if (tid < D) {
            float column = 0.0f;
#pragma unroll
            for (int w = 0; w < kSoftmaxWarps; ++w) column += xchg[w * D + tid];
            xchg[tid] = column;   // no other thread reads this word of the partial sums
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&bars->xbar);
          ok = wwait(&bars->xbar, 0u, 35);
          if (!ok) break;
          if (!any_kept) {
            const int rows = out_rows - i0 < BM ? out_rows - i0 : BM;
            float mean[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) mean[j] = xchg[chunk * 8 + j] / (float)L;
            const uint4 mine = make_uint4(Pack2<T>::pack(mean[0], mean[1]), Pack2<T>::pack(mean[2], mean[3]),
                                          Pack2<T>::pack(mean[4], mean[5]), Pack2<T>::pack(mean[6], mean[7]));
            T* out = reinterpret_cast<T*>(p.out) + (out_row0 + i0) * ((long long)H * D) + (long long)h * D;
            for (int e = tid; e < rows * kChunks; e += 256)
              *reinterpret_cast<uint4*>(out + (long long)(e / kChunks) * H * D + chunk * 8) = mine;
          } else {
            ok = wwait(&bars->o_ready, (c_t & 1u) ^ 1u, 50);   // the item's last PV
            if (!ok) break;
            ptx::tc_fence_after();
            if (!q_keep) total += (float)skipped;
#pragma unroll 1
            for (int c0 = 0; c0 < OW; c0 += 16) {
              uint32_t o[16];
              ptx::tmem_ld16(t_o + c0, o);
              ptx::tmem_wait_ld();
#pragma unroll
              for (int x = 0; x < 16; ++x) o[x] = __float_as_uint(__uint_as_float(o[x]) + (q_keep ? 0.0f : xchg[hf * OW + c0 + x]));
              ptx::tmem_st16(t_o + c0, o);
            }
            ptx::tmem_wait_st();
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&bars->xbar);   // the exchange words are free again
          ok = wwait(&bars->xbar, 1u, 37);
          if (!ok) break;
        }
        if (any_kept) {
          const float inv = 1.0f / total;
          ok = wwait(&bars->o_ready, (c_t & 1u) ^ 1u, 48);   // the item's last PV: c_t - 1 completed before it
          if (!ok) break;
          ptx::tc_fence_after();
          // Lanes of one row each would touch 32 cache lines per store (1900 cycles an item).  The kGroup lanes of a group
          // transpose their 16-byte chunks instead: lane c of the group ends up with chunk c of every row of the group, and a
          // store covers whole segments.
          constexpr int OC = OW < 32 ? OW : 32;   // columns at a time
          constexpr int kGroup = OC / 8;
          const int row0 = i0 + (r & ~(kGroup - 1)), rows = min(L, out_rows) - row0;
          T* out = reinterpret_cast<T*>(p.out) + (out_row0 + row0) * ((long long)H * D) + (long long)h * D + hf * OW + (lane & (kGroup - 1)) * 8;
#pragma unroll
          for (int c0 = 0; c0 < OW; c0 += OC) {
            uint32_t o[OC];
            attn::tmem_ld_n(t_o + c0, o);
            ptx::tmem_wait_ld();
            if (c0 + OC == OW) {   // the accumulator is in registers: the next item's first PV may overwrite it
              ptx::tc_fence_before();
              __syncwarp();
              if (lane == 0) ptx::mbar_arrive(&bars->o_free);
            }
            uint32_t w[kGroup][4];
#pragma unroll
            for (int x = 0; x < OC / 2; ++x)
              w[x / 4][x % 4] = Pack2<T>::pack(__uint_as_float(o[2 * x]) * inv, __uint_as_float(o[2 * x + 1]) * inv);
#pragma unroll
            for (int bit = 1; bit < kGroup; bit <<= 1) {
              const bool upper = (lane & bit) != 0;
#pragma unroll
              for (int c = 0; c < kGroup; ++c) {
                if (c & bit) continue;
#pragma unroll
                for (int x = 0; x < 4; ++x) {   // the lower lane keeps chunk c and takes the partner's, the upper one chunk c + bit
                  const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? w[c][x] : w[c | bit][x], bit);
                  if (upper) w[c][x] = got;
                  else w[c | bit][x] = got;
                }
              }
            }
#pragma unroll
            for (int c = 0; c < kGroup; ++c)
              if (c < rows) *reinterpret_cast<uint4*>(out + (long long)c * H * D + c0) = make_uint4(w[c][0], w[c][1], w[c][2], w[c][3]);
          }
        }
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->item_empty[slot]);
    }
  } else if (warp < kMmaWarp) {
    setmaxnreg_dec<kConvRegs>();
    // -------------------------------------------------------------- converters
    // Thread (quarter q4, lane) owns TMEM lane 32*q4 + lane of both transit accumulators and moves its row, rounded to T,
    // to where the consumer reads it without a shift of its own:
    //   C2P block c (lane = query row r): column m is the score of key x = m + r of tile c - 1 where that is below 128,
    //     of key x - 128 of tile c otherwise (the block is the upper half of one tile's window and the lower half of the
    //     next one's).  Consecutive m land at consecutive columns of the row buffer, modulo its two tiles.
    //   P2C parts (lane = key n): table column w of the tile's 256 is the score of query row 128 + n - w; the row goes to
    //     row n of the K-major B operand of the MMA that adds the tile to S.
    // Both destinations are shifted by the lane, and a 4-byte store takes two neighbouring columns: for odd (C2P) or even
    // (P2C) rows a funnel shift pairs them from the packed words at hand, and the first and the last of 32 columns are
    // stored by themselves.  No column needs its neighbours in another warp's hands, so each role has two warps per
    // quarter, one for the first and one for the second accumulator of its pair: 32 columns are a chain of some 60
    // instructions, 600 to 1100 cycles, that a warp cannot overlap with itself.
    const int q4 = warp & 3, group = (warp >> 2) & 1;
    const int row = q4 * 32 + lane;
    const bool odd = (row & 1) != 0;
    const uint32_t lane_base = (uint32_t)(q4 * 32) << 16;
    const int row_even = row & ~1;
    uint32_t rel_seen = 0;      // phases of ring_release (one per key tile) waited for so far
    uint32_t tiles_before = 0;  // key tiles of all earlier items
    uint32_t c_x = 0, c_pt = 0; // accumulators of this group converted, P2C tiles completed
    bool ok = true;

    // Half `group` of a C2P block: upper part of running tile `upper`, lower part of tile upper + 1; the first block of an item
    // has no upper part.  The two row buffers must be free: `need` key tiles in total must have been read.
    auto convert_block = [&](bool first, uint32_t upper, uint32_t need) -> bool {
      // word k of a block (columns 2k, 2k+1; for odd rows 2k-1, 2k) goes to column 128 * tile + 2k + row_even
      const uint32_t row_addr = ptx::smem_u32(smem + LO::offRows) + (uint32_t)(row * ROW_PITCH + 2 * row_even);
      const uint32_t shift = odd ? 16u : 32u;
      const uint32_t t_xc = tmem_base + lane_base + LO::kColXc + (LO::kXcs > 1 ? 64 * group : 0);
      if (!wwait(&bars->xc_full[group], c_x & 1u, 18)) return false;
      ++c_x;
      ptx::tc_fence_after();
      while (rel_seen < need) {
        if (!wwait(&bars->ring_release, rel_seen & 1u, 17)) return false;
        ++rel_seen;
      }
#pragma unroll 1
      for (int j = 2 * group; j < 2 * group + 2; ++j) {   // 32 columns at a time
        uint32_t v[32];
        ptx::tmem_ld32(t_xc + 32 * (j & 1), v);
        ptx::tmem_wait_ld();
        uint32_t w[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) w[k] = pack_scores<T>(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
        if (j & 1) {   // in registers: the accumulator is free for the next MMA
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&bars->xc_free[group]);
        }
        const uint32_t head = w[0], tail = w[15];
#pragma unroll
        for (int k = 15; k > 0; --k) w[k] = funnel_clamp(w[k - 1], w[k], shift);
        // column 2k + row_even below 128: tile `upper`; from 128 on: the next tile, whose buffer is the other half
        const uint32_t up = row_addr + (upper & 1u) * 256u + 64u * j, down = row_addr + ((upper & 1u) ? 0u : 256u) - 256u + 64u * j;
        const int turn = j + q4;   // columns of this warp and chunk: 32 * turn .. 32 * turn + 62
        if (turn >= 4 || !first) {
          const uint32_t to = turn >= 4 ? down : up;
          sts_u32_if(to, head, !odd);
          sts_u16_if(to + 2, head, odd);
        }
        if (turn >= 3 || !first) sts_u16_if((turn >= 3 ? down : up) + 64, tail >> 16, odd);
        if (turn == 3) {
          // words below 16 - lane / 2 belong to tile `upper`
          const uint32_t below = (1u << (16 - (lane >> 1))) - 1u, stored = first ? ~below : ~0u;
#pragma unroll
          for (int k = 1; k < 16; ++k) sts_u32_bit(((below >> k) & 1u ? up : down) + 4 * k, w[k], stored, k);
        } else if (turn >= 4 || !first) {
          const uint32_t to = turn >= 4 ? down : up;
#pragma unroll
          for (int k = 1; k < 16; ++k) sts_u32(to + 4 * k, w[k]);
        }
      }
      return true;
    };
    // Parts `group` and `group` + 2 (64 table columns each) of a tile's P2C accumulator.  A quarter's 32 keys take words
    // 16 * q4 + 1 .. 16 * q4 + 79 of the tile's 128: 32-column chunks q4 .. q4 + 4 of the eight, two chunks per part.
    auto convert_parts = [&]() -> bool {
      const uint32_t t_xp = tmem_base + lane_base + COL_XP + 64 * group;
      const uint32_t stg = c_pt % LO::kStgs;
      const uint32_t shift = odd ? 0u : 16u;
      bool waited = false;
#pragma unroll 1
      for (int part = group; part < 4; part += 2) {
        if (!wwait(&bars->xp_full[group], c_x & 1u, 19)) return false;
        ++c_x;
        ptx::tc_fence_after();
        const int begin = max(q4, 2 * part), end = min(q4 + 5, 2 * part + 2);
        if (begin >= end) {   // nothing for this warp's keys: its share of xp_free
          if (lane == 0) ptx::mbar_arrive(&bars->xp_free[group]);
          continue;
        }
        if (!waited && !wwait(&bars->pt_release[stg], (c_pt / LO::kStgs & 1u) ^ 1u, 20)) return false;   // that tile has been read
        waited = true;
#pragma unroll 1
        for (int j = begin; j < end; ++j) {
          uint32_t v[32];
          ptx::tmem_ld32(t_xp + 32 * (j & 1), v);
          ptx::tmem_wait_ld();
          uint32_t w[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) w[k] = pack_scores<T>(__uint_as_float(v[2 * k + 1]), __uint_as_float(v[2 * k]));
          if (j == end - 1) {   // what this warp needs of the part is in registers
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&bars->xp_free[group]);
          }
          const uint32_t head = w[0], tail = w[15];
#pragma unroll
          for (int k = 15; k > 0; --k) w[k] = funnel_wrap(w[k], w[k - 1], shift);
          // word k holds query rows 128 + row_even - 2 (16 j + k) and + 1; 16 query rows down are two chunks of eight
          const int qr = 128 + row_even - 32 * j;
          const uint32_t base = ptx::smem_u32(smem + LO::offStg) + stg * (uint32_t)STG_BYTES + (uint32_t)((row >> 3) * 128 + (row & 7) * 16);
          uint32_t at[4];   // where words 0, 1, 2, 3 (mod 4) go
#pragma unroll
          for (int x = 0; x < 4; ++x) at[x] = base + (uint32_t)((15 - ((qr - 2 * x) >> 3)) * STG_CHUNK + ((qr - 2 * x) & 7) * 2);
          const int turn = j - q4;
          if (turn > 0) {
            sts_u32_if(at[0], head, odd);
            sts_u16_if(at[0], head >> 16, !odd);
          }
          if (turn < 4) sts_u16_if(at[0] + 4 * STG_CHUNK + 2, tail, !odd);
          if (turn >= 1 && turn <= 3) {
#pragma unroll
            for (int k = 1; k < 16; ++k) sts_u32(at[k & 3] + (uint32_t)((k >> 2) * STG_CHUNK), w[k]);
          } else {
            // of the tile's words 1 + row_even / 2 .. 64 + row_even / 2 are query rows of the tile: the first of the quarter's
            // chunks begins below them, the last ends above, at 1 + and at lane / 2
            const uint32_t rows = turn == 0 ? 0xfffffffeu << (lane >> 1) : (2u << (lane >> 1)) - 1u;
#pragma unroll
            for (int k = 1; k < 16; ++k) sts_u32_bit(at[k & 3] + (uint32_t)((k >> 2) * STG_CHUNK), w[k], rows, k);
          }
        }
      }
      return true;
    };

    int k = 0;
    for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x, ++k) {
      const int slot = k % kItemSlots;
      ok = wwait(&bars->item_full[slot], (uint32_t)(k / kItemSlots) & 1u, 32);
      if (!ok) break;
      const ItemSlot* sl = &slots[slot];
      const int n = sl->t_end - sl->t_begin;
      if (sl->any_kept != 0) {
        if (warp >= kC2pWarp) {
          // block 0, then per key tile u block u + 1
          for (int u = -1; u < n && ok && has_c2p; ++u) {
            const uint32_t upper = tiles_before + (uint32_t)u;
            ok = convert_block(u < 0, upper, upper == 0xffffffffu ? 0u : upper);
            if (ok && u >= 0) {
              __syncwarp();
              if (lane == 0) ptx::mbar_arrive(&bars->c2p_ready);
            }
          }
        } else {
          for (int u = 0; u < n && ok && has_p2c; ++u) {
            ok = convert_parts();
            if (!ok) break;
            ptx::fence_proxy_async_smem();   // the tile is read by the tensor core
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&bars->pt_ready[c_pt % LO::kStgs]);
            ++c_pt;
          }
        }
        if (!ok) break;
        tiles_before += (uint32_t)n;
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->item_empty[slot]);
    }
  } else {
    setmaxnreg_dec<kMiscRegs>();
    // Q, K, rel_query and the mask analysis have a warp of their own, rel_key and V are loaded by the issuer of their MMAs.  (One
    // warp for all of them was what the tensor core waited for: 157 us with a lane per stream at 32 x 12 heads x 512 x 64, where
    // this takes 135.)  `count` loads so far: stage = count % stages, phase = (count / stages) & 1.
    auto issue_load = [&](const CUtensorMap* map, int offset, int bytes, uint64_t* full, uint32_t stage, int row, int z) {
      const uint32_t bar = ptx::smem_u32(&full[stage]), to = ptx::smem_u32(smem) + offset + stage * bytes;
      ptx::mbar_arrive_expect_tx_warp(bar, (uint32_t)bytes);
#pragma unroll
      for (int c = 0; c < LO::kSub; ++c) ptx::tma_load_3d_warp(to + c * (bytes / LO::kSub), map, bar, 64 * c, row, z);
    };
    auto load = [&](const CUtensorMap* map, int offset, int bytes, uint64_t* full, uint64_t* empty, uint32_t& count, uint32_t stages,
                    int row, int z, int code) -> bool {
      const uint32_t st = count % stages, ph = (count / stages) & 1u;
      ++count;
      if (!wwait(&empty[st], ph ^ 1u, code)) return false;
      issue_load(map, offset, bytes, full, st, row, z);
      return true;
    };
    if (warp == kTmaWarp) {
      // ------------------------------------------------- mask analysis, Q and K
      uint32_t c_q = 0, c_k = 0, c_rq = 0;
      bool ok = true;
      struct Item {
        int t_begin, n, i0, bh, h;
      };
      // Mask analysis of item number k2 (item it2), published through its slot.  Warp-collective.
      auto analyze = [&](int k2, int it2, Item& f) -> bool {
        const int slot = k2 % kItemSlots;
        const int qt = it2 / n_bh, bh = it2 - qt * n_bh, b = bh / H;
        const int i0 = qt * BM;
        ItemSlot* sl = &slots[slot];
        if (!wwait(&bars->item_empty[slot], ((uint32_t)(k2 / kItemSlots) & 1u) ^ 1u, 30)) return false;
        uint32_t kb_lo, kb_hi;
        kept_bits(p, b, lane, kb_lo, kb_hi);
        const TileRange range = tile_range(kb_lo, kb_hi, i0, L, lane);
        sl->kbits[lane] = kb_lo;
        sl->kbits[lane + 32] = kb_hi;
        if (lane == 0) {
          sl->t_begin = range.t_begin;
          sl->t_end = range.t_end;
          sl->any_kept = range.fold ? 2 : (range.any_kept ? 1 : 0);
          sl->bh = bh;
          sl->h = bh - b * H;
          sl->out_row0 = p.out_row_base ? (long long)p.out_row_base[b] : (long long)b * L;
          sl->out_rows = p.out_row_base ? p.out_row_count[b] : L;
          sl->i0 = i0;
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->item_full[slot]);
        f = {range.t_begin, range.any_kept ? range.t_end - range.t_begin : 0, i0, bh, bh - b * H};
        return true;
      };
      Item cur{}, nxt{};
      int k = 0;
      if ((int)blockIdx.x < n_items) ok = analyze(0, blockIdx.x, cur);
#pragma unroll 1
      for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x, ++k) {
        // K and the rel_query pieces of a tile first: its P2C parts are computed ahead of S, those of the first tile while Q waits
        // for the item before.  The next item is analysed once Q is on its way; the slot it takes is that of the item before
        // the one that is being computed.
        const int row0 = cur.t_begin * BK - cur.i0 - BM + (L - 1);
#pragma unroll 1
        for (int u = 0; u < cur.n && ok; ++u) {
          ok = load(&tmap_k, LO::offK, LO::kTile, bars->k_full, bars->k_empty, c_k, LO::kKStages, (cur.t_begin + u) * BK, cur.bh, 1);
#pragma unroll 1
          for (int part = 0; part < 4 && has_p2c && ok; ++part)
            ok = load(&tmap_fq, LO::offRQ, LO::kTab, bars->rq_full, bars->rq_empty, c_rq, LO::kRqStages, row0 + u * BK + part * 64, cur.h, 12);
          if (u == 0) {
            ok = ok && load(&tmap_q, LO::offQ, LO::kTile, &bars->q_full, &bars->q_empty, c_q, 1, cur.i0, cur.bh, 3);
            if (ok && n_items - it > (int)gridDim.x) ok = analyze(k + 1, it + (int)gridDim.x, nxt);
          }
        }
        if (ok && cur.n == 0 && n_items - it > (int)gridDim.x) ok = analyze(k + 1, it + (int)gridDim.x, nxt);
        cur = nxt;
      }
    } else if (warp == kMmaWarp) {
      // -------------------------------------------------------------- MMA issuer
      // S = Q K^T as soon as the softmax threads have read the previous tile's S, and the P2C tile on top of it as soon as the
      // converters have finished it.  In each issuing role the whole warp walks the items and one elected lane issues
      // (umma_ss_f16_warp); descriptors are precomputed and only their start-address field moves.  The other MMAs have
      // issuers of their own: an issue costs its warp about as long as the MMA runs.
      constexpr int is_bf16 = __is_same(T, __nv_bfloat16) ? 1 : 0;
      constexpr uint32_t idesc_nn = ptx::make_idesc_f16(is_bf16, BM, 128, 0, 0);   // 128 x 128, both K-major
      constexpr uint32_t mode = ptx::swizzle_mode_for_row_bytes(LO::kRowBytes);
      constexpr uint32_t kTileUnits = (uint32_t)LO::kTile >> 4;
      const uint64_t q_desc = ptx::make_smem_desc(ptx::smem_u32(smem + LO::offQ), 16, 8 * LO::kRowBytes, mode);
      const uint64_t k_desc = ptx::make_smem_desc(ptx::smem_u32(smem + LO::offK), 16, 8 * LO::kRowBytes, mode);
      const uint64_t eye_desc = ptx::make_smem_desc(ptx::smem_u32(smem + LO::offEye) + 112 * 16, EYE_LBO, 128, 0);
      const uint64_t stg_desc = ptx::make_smem_desc(ptx::smem_u32(smem + LO::offStg), STG_CHUNK, 128, 0);
      uint32_t c_q = 0, c_k = 0;   // loads consumed; c_k is also the count of S tiles
      bool ok = true;
      int k = 0;
      for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x, ++k) {
        const int slot = k % kItemSlots;
        ok = wwait(&bars->item_full[slot], (uint32_t)(k / kItemSlots) & 1u, 31);
        if (!ok) break;
        const bool any_kept = slots[slot].any_kept != 0;
        const int n = slots[slot].t_end - slots[slot].t_begin;
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->item_empty[slot]);
        if (!any_kept) continue;
        ok = wwait(&bars->q_full, c_q & 1u, 4);
        ++c_q;
#pragma unroll 1
        for (int u = 0; u < n && ok; ++u) {
          const uint32_t kst = c_k % LO::kKStages, stg = c_k % LO::kStgs;
          ok = wwait(&bars->k_full[kst], (c_k / LO::kKStages) & 1u, 5) && wwait(&bars->s_free, (c_k & 1u) ^ 1u, 6);
          if (!ok) break;
          ptx::tc_fence_after();
          mma_over_d<D>(tmem_base + COL_S, q_desc, kTileUnits / LO::kSub, k_desc + kst * kTileUnits, kTileUnits / LO::kSub, idesc_nn);
          ptx::umma_commit_warp(&bars->k_empty[kst]);
          if (u + 1 == n) ptx::umma_commit_warp(&bars->q_empty);
          if (has_p2c) {
            ok = wwait(&bars->pt_ready[stg], (c_k / LO::kStgs) & 1u, 9);
            if (!ok) break;
            ptx::tc_fence_after();
            const uint64_t b_desc = stg_desc + stg * (uint32_t)(STG_BYTES >> 4);
#pragma unroll
            for (int kk = 0; kk < BM / 16; ++kk)
              ptx::umma_ss_f16_warp(tmem_base + COL_S, eye_desc - (uint64_t)(16 * kk), b_desc + (uint64_t)((14 - 2 * kk) * (STG_CHUNK >> 4)),
                                    idesc_nn, 1u);
            ptx::umma_commit_warp(&bars->pt_release[stg]);
          }
          ptx::umma_commit_warp(&bars->s_full);
          ++c_k;
        }
      }
    } else if (warp == kPartWarp) {
      // ------------------------------- P2C parts, as far ahead as their two accumulators allow
      // XP[n, w] = K . rel_query^T over the 64 table rows of one piece
      constexpr uint32_t idesc_part = ptx::make_idesc_f16(__is_same(T, __nv_bfloat16) ? 1 : 0, BM, 64, 0, 0);
      constexpr uint32_t mode = ptx::swizzle_mode_for_row_bytes(LO::kRowBytes);
      constexpr uint32_t kTileUnits = (uint32_t)LO::kTile >> 4, kTabUnits = (uint32_t)LO::kTab >> 4;
      const uint64_t k_desc = ptx::make_smem_desc(ptx::smem_u32(smem + LO::offK), 16, 8 * LO::kRowBytes, mode);
      const uint64_t rq_desc = ptx::make_smem_desc(ptx::smem_u32(smem + LO::offRQ), 16, 8 * LO::kRowBytes, mode);
      uint32_t c_k = 0, c_xp = 0;   // key tiles consumed, parts issued
      bool ok = true;
      int k = 0;
      for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x, ++k) {
        const int slot = k % kItemSlots;
        ok = wwait(&bars->item_full[slot], (uint32_t)(k / kItemSlots) & 1u, 40);
        if (!ok) break;
        const int n = slots[slot].any_kept != 0 && has_p2c ? slots[slot].t_end - slots[slot].t_begin : 0;
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->item_empty[slot]);
#pragma unroll 1
        for (uint32_t x = 0; x < 4u * (uint32_t)n && ok; ++x) {   // part x & 3 of key tile x >> 2
          const uint32_t part = x & 3u, kst = c_k % LO::kKStages, buf = c_xp & 1u, rst = c_xp % LO::kRqStages;
          if (part == 0) ok = wwait(&bars->k_full[kst], (c_k / LO::kKStages) & 1u, 43);
          ok = ok && wwait(&bars->rq_full[rst], (c_xp / LO::kRqStages) & 1u, 15) && wwait(&bars->xp_free[buf], ((c_xp >> 1) & 1u) ^ 1u, 16);
          if (!ok) break;
          ptx::tc_fence_after();
          mma_over_d<D>(tmem_base + COL_XP + 64 * buf, k_desc + kst * kTileUnits, kTileUnits / LO::kSub, rq_desc + rst * kTabUnits,
                        kTabUnits / LO::kSub, idesc_part);
          ptx::umma_commit_warp(&bars->rq_empty[rst]);
          ptx::umma_commit_warp(&bars->xp_full[buf]);
          ++c_xp;
          if (part == 3) {
            ptx::umma_commit_warp(&bars->k_empty[kst]);
            ++c_k;
          }
        }
      }
    } else if (warp == kPvWarp) {
      // ------------------------- C2P half blocks, and O (+)= P . V of every key tile, with the loads of both
      // Whichever can go next goes: the C2P blocks run an item and a half ahead of the PV MMAs, on a cursor of their own.
      constexpr int is_bf16 = __is_same(T, __nv_bfloat16) ? 1 : 0;
      constexpr uint32_t idesc_c = ptx::make_idesc_f16(is_bf16, BM, LO::kXcCols, 0, 0);
      constexpr uint32_t idesc_pv = ptx::make_idesc_f16(is_bf16, BM, D, 0, 1);   // V is MN-major
      constexpr uint32_t mode = ptx::swizzle_mode_for_row_bytes(LO::kRowBytes);
      constexpr uint32_t kTileUnits = (uint32_t)LO::kTile >> 4, kTabUnits = (uint32_t)LO::kTab >> 4;
      constexpr uint32_t kPvStepUnits = (16u * LO::kRowBytes) >> 4;   // 16 keys further down the V tile
      const uint64_t q_desc = ptx::make_smem_desc(ptx::smem_u32(smem + LO::offQ), 16, 8 * LO::kRowBytes, mode);
      const uint64_t rk_desc = ptx::make_smem_desc(ptx::smem_u32(smem + LO::offRK), 16, 8 * LO::kRowBytes, mode);
      const uint64_t v_desc = ptx::make_smem_desc(ptx::smem_u32(smem + LO::offV), LO::kVPiece / LO::kSub, 8 * LO::kRowBytes, mode);
      const int n_mine = (int)blockIdx.x < n_items ? (n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
      // Bounded by a count of passes in which nothing could go (each up to seven polls, 25 to 250 ns).  One more pass then notes
      // the barrier of the last step that could not be taken: an instantiation of its own, since what the loop carries for a
      // report costs it up to 5 % of the kernel (d 64, two key tiles an item).
      constexpr uint32_t kPasses = ptx::kWaitPolls * 4u;
      uint32_t left = kPasses;
      int missing = 0;
      // C2P: items taken, half blocks of the last one still to be loaded and to be issued, coordinates of the next load; counts
      int kc = 0, halves = 0, rk_loads = 0, rk_row = 0, rk_h = 0;
      bool have_q = false;
      uint32_t c_q = 0, c_rk = 0, c_rk_load = 0;
      // PV: items taken, pieces of V of the last one still to be loaded and to be multiplied, coordinates; counts
      int kp = 0, pieces = 0, v_loads = 0, v_row = 0, v_bh = 0;
      bool first = false;               // no piece of the item has been multiplied
      uint32_t c_v = 0, c_v_load = 0, c_t = 0, c_items = 0;
      auto pass = [&](auto report) __attribute__((always_inline)) {
        auto complete = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
          const bool yes = __all_sync(0xffffffffu, ptx::mbar_test(bar, parity));
          if (decltype(report)::value && !yes) missing = code;
          return yes;
        };
        --left;
        if (halves == 0 && kc < n_mine && complete(&bars->item_full[kc % kItemSlots], (uint32_t)(kc / kItemSlots) & 1u, 39)) {
          const ItemSlot* sl = &slots[kc % kItemSlots];   // ours until the PV cursor has taken it too
          ++kc;
          if (sl->any_kept != 0 && has_c2p) {
            halves = rk_loads = 2 * (sl->t_end - sl->t_begin) + 2;
            // table row of column 0 of block 0: pair (row r, key x) of tile u uses column 128 - r + x of blocks u, u + 1
            rk_row = sl->t_begin * BK - sl->i0 - BM + (L - 1);
            rk_h = sl->h;
            have_q = false;
          }
          left = kPasses;
        }
        if (rk_loads > 0 && complete(&bars->rk_empty[c_rk_load % LO::kRkStages], ((c_rk_load / LO::kRkStages) & 1u) ^ 1u, 2)) {
          issue_load(&tmap_fk, LO::offRK, LO::kTab, bars->rk_full, c_rk_load % LO::kRkStages, rk_row, rk_h);
          ++c_rk_load;
          --rk_loads;
          rk_row += 64;
          left = kPasses;
        }
        if (halves > 0) {
          if (!have_q) {
            have_q = complete(&bars->q_full, c_q & 1u, 10);
            if (have_q) ++c_q;
          }
          // its accumulator has been read: by the group's half before, or, with one accumulator, by the other group's
          const uint32_t st = c_rk % LO::kRkStages;
          if (have_q && complete(&bars->rk_full[st], (c_rk / LO::kRkStages) & 1u, 13) &&
              (LO::kXcs > 1 ? complete(&bars->xc_free[c_rk & 1u], ((c_rk >> 1) & 1u) ^ 1u, 14)
                            : c_rk == 0u || complete(&bars->xc_free[(c_rk - 1u) & 1u], ((c_rk - 1u) >> 1) & 1u, 14))) {
            ptx::tc_fence_after();
            mma_over_d<D>(tmem_base + LO::kColXc + (LO::kXcs > 1 ? 64 * (c_rk & 1u) : 0u), q_desc, kTileUnits / LO::kSub,
                          rk_desc + st * kTabUnits, kTabUnits / LO::kSub, idesc_c);
            ptx::umma_commit_warp(&bars->rk_empty[st]);
            ptx::umma_commit_warp(&bars->xc_full[c_rk & 1u]);
            ++c_rk;
            if (--halves == 0) ptx::umma_commit_warp(&bars->q_empty);
            left = kPasses;
          }
        }
        if (pieces == 0 && kp < kc) {
          const int slot = kp % kItemSlots;
          ++kp;
          if (slots[slot].any_kept != 0) {
            pieces = v_loads = (slots[slot].t_end - slots[slot].t_begin) * LO::kVPieces;
            v_row = slots[slot].t_begin * BK;
            v_bh = slots[slot].bh;
            first = true;
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&bars->item_empty[slot]);
          left = kPasses;
        }
        if (v_loads > 0 && complete(&bars->v_empty[c_v_load % LO::kVStages], ((c_v_load / LO::kVStages) & 1u) ^ 1u, 11)) {
          issue_load(&tmap_v, LO::offV, LO::kVPiece, bars->v_full, c_v_load % LO::kVStages, v_row, v_bh);
          ++c_v_load;
          --v_loads;
          v_row += LO::kVRows;
          left = kPasses;
        }
        // A tile's P has been stored; before an item's first, the output accumulator of the previous item with kept rows has been
        // read out (o_free completes one phase per such item, and this warp is never more than one phase behind).
        const uint32_t part_of_tile = c_v % LO::kVPieces, vst = c_v % LO::kVStages;
        if (pieces > 0 && (part_of_tile != 0 || complete(&bars->p_full, c_t & 1u, 7)) && complete(&bars->v_full[vst], (c_v / LO::kVStages) & 1u, 8) &&
            (!first || c_items == 0 || complete(&bars->o_free, (c_items - 1u) & 1u, 38))) {
          ptx::tc_fence_after();
          const uint64_t vt_desc = v_desc + vst * (uint32_t)(LO::kVPiece >> 4);
          const uint32_t p_cols = tmem_base + COL_P + part_of_tile * (LO::kVRows / 2);
#pragma unroll
          for (int kk = 0; kk < LO::kVRows / 16; ++kk)
            ptx::umma_ts_f16_warp(tmem_base + COL_O, p_cols + kk * 8, vt_desc + kk * kPvStepUnits, idesc_pv, !first || kk > 0 ? 1u : 0u);
          ptx::umma_commit_warp(&bars->v_empty[vst]);
          first = false;
          ++c_v;
          --pieces;
          if (part_of_tile == LO::kVPieces - 1) {
            ptx::umma_commit_warp(&bars->o_ready);
            ++c_t;
          }
          if (pieces == 0) ++c_items;
          left = kPasses;
        }
      };
#pragma unroll 1
      while ((kp < n_mine || halves + pieces > 0) && left != 0u) pass(std::false_type{});
      if (left == 0u) {
        pass(std::true_type{});
        fail_code = missing != 0 ? missing : 44;   // 44: it has completed since
      }
    }
  }

  if (fail_code != 0 && status_word != nullptr) atomicCAS(status_word, 0, kWaitsAttentionRel + fail_code);
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) ptx::tmem_dealloc(tmem_base, kTmemCols);
}

// rel[h, e, :] = pos[h, lut[2L-2-e], :]; one thread per 16-byte chunk.
__global__ void expand_rel_tables_kernel(const uint4* __restrict__ pos, const int32_t* __restrict__ lut,
                                         uint4* __restrict__ rel, int heads, int n_active, int n_rows, int chunks) {
  const long long total = (long long)heads * n_rows * chunks;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(idx % chunks);
    const long long he = idx / chunks;
    const int e = (int)(he % n_rows), h = (int)(he / n_rows);
    int slot = lut[n_rows - 1 - e];
    slot = slot < 0 ? 0 : (slot >= n_active ? n_active - 1 : slot);
    rel[idx] = pos[((long long)h * n_active + slot) * chunks + c];
  }
}

template <typename T, int D>
int launch_rel_typed(const DflAttnRelParams& p, cudaStream_t stream) {
  using LO = RLayout<D>;
  const int L = p.seq_len, BH = p.batch * p.heads, R = 2 * L - 1;
  const uint64_t row = (uint64_t)D * sizeof(T), seq = (uint64_t)L * row, table = (uint64_t)R * row;
  CUtensorMap tq, tk, tv, tfk, tfq;
  constexpr int kCols = D / LO::kSub;
  int rc = encode_tensor_map_3d(&tq, p.q, D, L, BH, row, seq, kCols, BM, LO::kRowBytes);
  if (rc == DFL_OK) rc = encode_tensor_map_3d(&tk, p.k, D, L, BH, row, seq, kCols, BK, LO::kRowBytes);
  if (rc == DFL_OK) rc = encode_tensor_map_3d(&tv, p.v, D, L, BH, row, seq, kCols, LO::kVRows, LO::kRowBytes);
  // a disabled term reuses the other table's map; it is never dereferenced
  const void* fk = p.rel_key ? p.rel_key : p.rel_query;
  const void* fq = p.rel_query ? p.rel_query : p.rel_key;
  if (rc == DFL_OK) rc = encode_tensor_map_3d(&tfk, fk, D, R, p.heads, row, table, kCols, 64, LO::kRowBytes);
  if (rc == DFL_OK) rc = encode_tensor_map_3d(&tfq, fq, D, R, p.heads, row, table, kCols, 64, LO::kRowBytes);
  if (rc != DFL_OK) return rc;

  auto kernel = attention_rel_kernel<T, D>;
  static KernelDeviceConfig config;   // per instantiation
  int sm_count = 0;
  rc = configure_kernel(config, kernel, LO::total, &sm_count, "attention_rel_kernel");
  if (rc != DFL_OK) return rc;
  cudaError_t e;
  int* status_word = p.status;
  if (!status_word) {
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&status_word), g_attn_rel_status);
    if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "status word: %s", cudaGetErrorString(e));
  }
  const long long n_items = (long long)BH * ((L + BM - 1) / BM);
  if (n_items > 0x7fffffffLL) return fail(DFL_ERR_TOO_LARGE, "too many (batch, head, query tile) items");
  const int grid = n_items < sm_count ? (int)n_items : sm_count;
  e = launch_after_predecessor(kernel, dim3(grid), dim3(kThreads), LO::total, stream, tq, tk, tv, tfk, tfq, p, status_word,
                               (int)n_items);
  if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "attention_rel_kernel: %s", cudaGetErrorString(e));
  return check_launch("attention_rel_kernel");
}

}  // namespace

bool attention_rel_supported(const DflAttnRelParams& p) {
  // d = 128 beyond 96 positions: plans of shorter buckets have no relative tables at this head dim, which callers rely on.
  // The line is that of the interface, not a crossover: one launch beats three from 16 positions on (us, three / one: 16
  // positions 13.3 / 13.1 for 1 x 8 heads, 51 / 36 for 64 x 8; 96 positions 18.5 / 13.1 and 87 / 36; 512 positions 212 / 97 for
  // 16 x 8 heads).
  return p.dtype != DFL_F32 && (p.head_dim == 32 || p.head_dim == 64 || (p.head_dim == 128 && p.seq_len > 96)) &&
         (p.rel_key || p.rel_query) && p.seq_len >= 1 && p.seq_len <= kMaxSeqLen;
}

template <typename T>
int launch_rel(const DflAttnRelParams& p, cudaStream_t stream) {
  return p.head_dim == 128  ? launch_rel_typed<T, 128>(p, stream)
         : p.head_dim == 64 ? launch_rel_typed<T, 64>(p, stream)
                            : launch_rel_typed<T, 32>(p, stream);
}

int launch_attention_rel(const DflAttnRelParams& p, cudaStream_t stream, bool tables_early) {
  if (!attention_rel_supported(p)) return fail(DFL_ERR_UNSUPPORTED, "configuration not covered by the relative-table kernel");
  if (attention_rel_small_covers(p)) return launch_attention_rel_small(p, tables_early, stream);
  return p.dtype == DFL_F16 ? launch_rel<__half>(p, stream) : launch_rel<__nv_bfloat16>(p, stream);
}

int launch_expand_rel_tables(const void* pos, const int32_t* lut, void* rel, int heads, int n_active, int seq_len,
                             int head_dim, int dtype, cudaStream_t stream) {
  const int chunks = head_dim * (int)dtype_size(dtype) / 16;
  const int n_rows = 2 * seq_len - 1;
  const long long total = (long long)heads * n_rows * chunks;
  const int threads = 256;
  long long blocks = (total + threads - 1) / threads;
  if (blocks > 4096) blocks = 4096;
  expand_rel_tables_kernel<<<(int)blocks, threads, 0, stream>>>(reinterpret_cast<const uint4*>(pos), lut,
                                                                reinterpret_cast<uint4*>(rel), heads, n_active, n_rows,
                                                                chunks);
  return check_launch("expand_rel_tables_kernel");
}

}  // namespace dfl
