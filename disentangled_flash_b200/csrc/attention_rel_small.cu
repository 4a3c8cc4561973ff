// Disentangled attention over position tables laid out by relative distance, for short sequences.
//
// The operation of attention_rel_tc.cu (dfl_attention_rel_fwd) for sequences of at most 128 positions, where that kernel
// has one key tile per item and is a chain of hand-overs between its roles (load, table MMAs, converters, score MMA,
// softmax, PV): 9 us for a batch that needs well under one.  Here a (batch, head) is one CTA, or two with half of the query
// rows each, the whole sequence is in shared memory, and a warp keeps 16 rows of a step in its registers:
//   P2C[j, m] = k_j . rel_query[m]   16 keys a warp against the table rows that the CTA's queries can reach
//   C2P[i, m] = q_i . rel_key[m]     16 queries a warp; both rounded to T and written to shared memory
//   S = Q K^T on the fragments, plus the two scores of its diagonal; mask, softmax, O = P V, normalise.
// With two CTAs a head, two warps share 16 query rows, half of the keys each, and exchange maxima, sums and partial outputs.
// The matrix instruction is the warp-level mma.sync: its result is in the registers of the warp that needs it, where tensor
// memory would bring back the round trips that bound the other kernel; the operands of an item are a few hundred
// instructions of it.  What bounds it is the load latency, then the diagonal gathers, which two CTAs halve.  us per launch, fp16,
// d 64, both terms, attention_rel_tc.cu / one CTA a head / two: 1 x 12 heads x 32 9.2 / 4.0 / 3.3, 4 x 12 x 64 9.4 / 5.6 / 4.4,
// 4 x 12 x 96 9.4 / 8.1 / 5.9, 4 x 12 x 128 9.3 / 10.8 / 7.1, 8 x 12 x 128 9.6 / 11.5 / 9.4.  A forward (hidden 768, 12 layers)
// with one and with two: 4 x 128 tokens as a graph 519 -> 495 us, 8 x 128 623 -> 605.
// Rounding is that of attention_rel_tc.cu: relative terms to T (FP16 saturating), P to T (BF16 up to 64 keys: to two of them), the row sum
// over the rounded P.
#include <type_traits>

#include "attention_tc_common.cuh"

namespace dfl {
namespace {

// NW warps cover LM positions.  PARTS CTAs share a head, each with its part of the query rows and all keys; the PARTS warps
// of 16 query rows then share the keys.
template <int D, int NW, int PARTS>
struct SLayout {
  static constexpr int kThreads = 32 * NW;
  static constexpr int LM = 16 * NW;             // positions covered
  static constexpr int kGroups = NW / PARTS;     // 16-row query groups of a CTA
  static constexpr int kRows = 16 * kGroups;     // its query rows
  static constexpr int kTableRows = LM + kRows;  // table rows its queries can reach (and one more)
  static constexpr int kRowBytes = D * 2;
  static constexpr int kChunks = kRowBytes / 16;
  // 16-bit columns per score row: LM (C2P) or kRows (P2C) + 16, and 10 more so that the gathers of a warp (rows g, columns 2t,
  // shifted by the row) spread over the banks
  static constexpr int kPitchC = LM + 26, kPitchP = kRows + 26;
  static constexpr int offQ = 0;
  static constexpr int offK = offQ + kRows * kRowBytes;
  static constexpr int offV = offK + LM * kRowBytes;
  static constexpr int offRK = offV + LM * kRowBytes;   // later the exchange between the warps of a query group
  static constexpr int offRQ = offRK + kTableRows * kRowBytes;
  // Beyond 64 positions the C2P scores take the place of rel_query, so that two CTAs fit an SM.
  static constexpr bool kReuse = NW > 4;
  static constexpr int kSizeRQ = kTableRows * kRowBytes, kSizeC = kRows * kPitchC * 2;
  static constexpr int offC = kReuse ? offRQ : offRQ + kSizeRQ;
  static constexpr int offP = !kReuse ? offC + kSizeC : offRQ + (kSizeRQ > kSizeC ? kSizeRQ : kSizeC);
  static constexpr int offKeep = offP + LM * kPitchP * 2;
  static constexpr int total = offKeep + LM;
  static_assert(PARTS == 1 || kGroups * (PARTS * 32 + PARTS * (D / 4) * 32) * 4 <= kTableRows * kRowBytes, "exchange area");
};

// byte offset of 16-byte chunk c of a row; eight consecutive rows of one chunk index hit different banks
template <int D>
__device__ __forceinline__ uint32_t chunk_at(int row, int c) {
  return (uint32_t)(row * D * 2 + ((c ^ (D == 64 ? row & 7 : (row >> 1) & 3)) << 4));
}
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <typename T>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (__is_same(T, __half))
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two scores rounded to T and packed; FP16 saturates (see attention_rel_tc.cu)
template <typename T>
__device__ __forceinline__ uint32_t round_scores(float lo, float hi) {
  uint32_t v;
  if constexpr (__is_same(T, __half)) asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
  else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
  return v;
}

template <typename T, int D, int NW, int PARTS>
__global__ void __launch_bounds__(SLayout<D, NW, PARTS>::kThreads)
attention_rel_small_kernel(const DflAttnRelParams p, int tables_early) {
  using LO = SLayout<D, NW, PARTS>;
  constexpr int LM = LO::LM, CH = LO::kChunks, NT = LO::kThreads, QR = LO::kRows, QG = LO::kGroups;
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t base = ptx::smem_u32(smem);
  const int L = p.seq_len, bh = blockIdx.x / PARTS, b = bh / p.heads, h = bh - b * p.heads;
  const int q0 = ((int)blockIdx.x - bh * PARTS) * QR;   // first query row
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const bool has_c2p = p.rel_key != nullptr, has_p2c = p.rel_query != nullptr;
  if (q0 >= L) return;

  // Table row e (x = j - i = e - (L - 1)) goes to row e + LM - L - (LM - QR - q0), which makes every window below independent of
  // L and of the part.  Rows the tables do not have are left as they are: they only reach scores of positions beyond L,
  // which are replaced.
  auto load_tables = [&]() {
    const long long first = (long long)h * (2 * L - 1) * D;
    const int shift = q0 + QR - L;
    const int e0 = shift < 0 ? -shift : 0, e1 = min(2 * L - 1, LO::kTableRows - shift);
    for (int x = e0 * CH + tid; x < e1 * CH; x += NT) {
      const int e = x / CH, c = x - e * CH;
      const uint32_t at = chunk_at<D>(e + shift, c);
      const long long from = first + (long long)e * D + c * 8;
      if (has_c2p) ptx::cp_async_16(smem + LO::offRK + at, reinterpret_cast<const T*>(p.rel_key) + from);
      if (has_p2c) ptx::cp_async_16(smem + LO::offRQ + at, reinterpret_cast<const T*>(p.rel_query) + from);
    }
  };
  if (tables_early) load_tables();
  wait_for_predecessor();
  release_successor();
  {
    const long long first = (long long)bh * L * D;
    for (int x = tid; x < LM * CH; x += NT) {
      const int r = x / CH, c = x - r * CH;
      const uint32_t at = chunk_at<D>(r, c);
      if (r < L) {
        const long long from = first + (long long)r * D + c * 8;
        ptx::cp_async_16(smem + LO::offK + at, reinterpret_cast<const T*>(p.k) + from);
        if (PARTS == 1 || (r >= q0 && r < q0 + QR))
          ptx::cp_async_16(smem + LO::offQ + chunk_at<D>(r - q0, c), reinterpret_cast<const T*>(p.q) + from);
        ptx::cp_async_16(smem + LO::offV + at, reinterpret_cast<const T*>(p.v) + from);
      } else {   // a probability of zero times what was left there must be zero
        *reinterpret_cast<uint4*>(smem + LO::offV + at) = make_uint4(0, 0, 0, 0);
      }
    }
  }
  if (!tables_early) load_tables();
  if (tid < LM) smem[LO::offKeep + tid] = tid < L && mask_keep(p.mask, p.mask_elem_size, (long long)b * L + tid) ? 1 : 0;
  ptx::cp_async_wait_all();
  __syncthreads();

  const int group = warp % QG, share = warp / QG;   // query group; share of its keys
  const int r0 = 16 * group, i0 = q0 + r0;          // first row of the group, in the CTA and in the sequence
  const bool active = i0 < L;
  // 16 rows of `a` against 8 table rows at a time, n in [begin, end), from `row0` on, rounded, to rows dst_row.. of a buffer
  auto relative = [&](const uint32_t (&a)[D / 16][4], int table, int row0, int dst, int dst_row, auto pitch, int begin, int end) {
    constexpr int P = decltype(pitch)::value;
#pragma unroll 2
    for (int n = begin; n < end; ++n) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k2 = 0; k2 < D / 32; ++k2) {
        uint32_t bf[4];
        ldsm(bf, base + table + chunk_at<D>(row0 + 8 * n + (lane & 7), 4 * k2 + (lane >> 3)));
        mma16816<T>(c, a[2 * k2], bf[0], bf[1]);
        mma16816<T>(c, a[2 * k2 + 1], bf[2], bf[3]);
      }
      uint32_t* to = reinterpret_cast<uint32_t*>(smem + dst + ((dst_row + g) * P + 8 * n + 2 * t) * 2);
      to[0] = round_scores<T>(c[0], c[1]);
      to[4 * P] = round_scores<T>(c[2], c[3]);   // eight rows further down
    }
  };
  if (has_p2c && 16 * warp < L) {   // the keys of all parts: one group of 16 a warp
    uint32_t kf[D / 16][4];
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) ldsm(kf[kk], base + LO::offK + chunk_at<D>(16 * warp + (lane & 15), 2 * kk + (lane >> 4)));
    relative(kf, LO::offRQ, 16 * warp, LO::offP, 16 * warp, std::integral_constant<int, LO::kPitchP>{}, 0, (QR + 16) / 8);
  }
  if (LO::kReuse) __syncthreads();   // rel_query has been read
  uint32_t qf[D / 16][4];
  if (active) {
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) ldsm(qf[kk], base + LO::offQ + chunk_at<D>(r0 + (lane & 15), 2 * kk + (lane >> 4)));
    constexpr int kTiles = (LM + 16) / 8 / PARTS;   // of eight columns, a warp's share
    if (has_c2p)
      relative(qf, LO::offRK, QR - 16 - r0, LO::offC, r0, std::integral_constant<int, LO::kPitchC>{}, share * kTiles, (share + 1) * kTiles);
  }
  __syncthreads();
  if (!active) return;

  uint32_t bits[(LM + 31) / 32];   // kept keys
#pragma unroll
  for (int w = 0; w < (LM + 31) / 32; ++w) bits[w] = __ballot_sync(0xffffffffu, 32 * w + lane < LM && smem[LO::offKeep + 32 * w + lane] != 0);
  const bool keep_lo = smem[LO::offKeep + i0 + g] != 0, keep_hi = smem[LO::offKeep + i0 + g + 8] != 0;

  constexpr int KT = LM / 8 / PARTS;   // tiles of eight keys of this warp, from j0 on
  const int j0 = share * 8 * KT;
  float s[KT][4];
  float max_lo = -INFINITY, max_hi = -INFINITY;
  const T* c2p = reinterpret_cast<const T*>(smem + LO::offC) + (r0 + g) * LO::kPitchC + j0 + 15 - g + 2 * t;
  const T* p2c = reinterpret_cast<const T*>(smem + LO::offP) + (j0 + 2 * t) * LO::kPitchP + 2 * t + QR - 1 - r0 - g;
#pragma unroll
  for (int n = 0; n < KT; ++n) {
#pragma unroll
    for (int x = 0; x < 4; ++x) s[n][x] = -INFINITY;
    if (j0 + 8 * n < L) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k2 = 0; k2 < D / 32; ++k2) {
        uint32_t bf[4];
        ldsm(bf, base + LO::offK + chunk_at<D>(j0 + 8 * n + (lane & 7), 4 * k2 + (lane >> 3)));
        mma16816<T>(c, qf[2 * k2], bf[0], bf[1]);
        mma16816<T>(c, qf[2 * k2 + 1], bf[2], bf[3]);
      }
      uint32_t word = bits[n / 4];   // of the tile's keys; j0 is a multiple of 16
      if (PARTS > 1) {
        const int w = (j0 + 8 * n) >> 5;
        word = bits[0];
#pragma unroll
        for (int q = 1; q < (LM + 31) / 32; ++q) word = w == q ? bits[q] : word;
      }
      const uint32_t tile_bits = word >> ((j0 + 8 * n) & 31);
#pragma unroll
      for (int x = 0; x < 4; ++x) {   // row i0 + g + 8 (x >> 1), key j = j0 + 8 n + 2 t + (x & 1); j0 is a multiple of 16
        const int j = j0 + 8 * n + 2 * t + (x & 1), down = 8 * (x >> 1);
        if (has_c2p) c[x] += Elem<T>::to_f(c2p[down * (LO::kPitchC - 1) + 8 * n + (x & 1)]);
        if (has_p2c) c[x] += Elem<T>::to_f(p2c[(8 * n + (x & 1)) * LO::kPitchP + 8 * (n & 1) + (x & 1) - down]);
        const bool kept = (tile_bits >> (2 * t + (x & 1))) & 1u;
        // a padded query attends to all L keys alike
        s[n][x] = (x < 2 ? keep_lo : keep_hi) ? (kept ? c[x] : -INFINITY) : (j < L ? 0.0f : -INFINITY);
      }
      max_lo = fmaxf(max_lo, fmaxf(s[n][0], s[n][1]));
      max_hi = fmaxf(max_hi, fmaxf(s[n][2], s[n][3]));
    }
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    max_lo = fmaxf(max_lo, __shfl_xor_sync(0xffffffffu, max_lo, o));
    max_hi = fmaxf(max_hi, __shfl_xor_sync(0xffffffffu, max_hi, o));
  }
  // Exchange of the two warps of a group, where rel_key was: row maxima and sums [group][share][16], then partial outputs.
  float* const rows_x = reinterpret_cast<float*>(smem + LO::offRK) + group * PARTS * 32;
  float* const out_x = reinterpret_cast<float*>(smem + LO::offRK) + QG * PARTS * 32 + group * PARTS * (D / 4) * 32;
  if (PARTS > 1) {
    if (t == 0) {
      rows_x[share * 32 + g] = max_lo;
      rows_x[share * 32 + g + 8] = max_hi;
    }
    asm volatile("bar.sync %0, 64;" ::"r"(1 + group) : "memory");
    max_lo = fmaxf(max_lo, rows_x[(share ^ 1) * 32 + g]);
    max_hi = fmaxf(max_hi, rows_x[(share ^ 1) * 32 + g + 8]);
  }
  const float cscale = p.scale * 1.4426950408889634f;
  // a row beyond L may hold anything; it is not stored
  const float neg_lo = -max_lo * cscale, neg_hi = -max_hi * cscale;
  // With few keys the 8 bits of a bf16 probability show in the output; what its rounding drops is multiplied as well.
  constexpr bool kSplitP = !__is_same(T, __half) && LM <= 64;
  float sum_lo = 0.f, sum_hi = 0.f;
  float o[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n) {
#pragma unroll
    for (int x = 0; x < 4; ++x) o[n][x] = 0.f;
  }
#pragma unroll
  for (int ks = 0; ks < KT / 2; ++ks) {
    if (j0 + 16 * ks >= L) continue;
    uint32_t pf[4], rest[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {   // fragment register x: keys 16 ks + 8 (x >> 1), row half x & 1
      const float* e = s[2 * ks + (x >> 1)] + 2 * (x & 1);
      const float neg = (x & 1) ? neg_hi : neg_lo;
      const float p0 = ptx::ex2_approx(fmaf(e[0], cscale, neg)), p1 = ptx::ex2_approx(fmaf(e[1], cscale, neg));
      pf[x] = attn::Pack2<T>::pack(p0, p1);
      (x & 1 ? sum_hi : sum_lo) += attn::Pack2<T>::sum2(pf[x]);
      if (kSplitP) {
        rest[x] = attn::Pack2<T>::pack(p0 - __uint_as_float(pf[x] << 16), p1 - __uint_as_float(pf[x] & 0xffff0000u));
        (x & 1 ? sum_hi : sum_lo) += attn::Pack2<T>::sum2(rest[x]);
      }
    }
#pragma unroll
    for (int n2 = 0; n2 < D / 16; ++n2) {
      uint32_t bf[4];
      ldsm_trans(bf, base + LO::offV + chunk_at<D>(j0 + 16 * ks + (lane & 15), 2 * n2 + (lane >> 4)));
      mma16816<T>(o[2 * n2], pf, bf[0], bf[1]);
      mma16816<T>(o[2 * n2 + 1], pf, bf[2], bf[3]);
      if (kSplitP) {
        mma16816<T>(o[2 * n2], rest, bf[0], bf[1]);
        mma16816<T>(o[2 * n2 + 1], rest, bf[2], bf[3]);
      }
    }
  }
#pragma unroll
  for (int x = 1; x < 4; x <<= 1) {
    sum_lo += __shfl_xor_sync(0xffffffffu, sum_lo, x);
    sum_hi += __shfl_xor_sync(0xffffffffu, sum_hi, x);
  }
  // each warp of a group finishes its share of the columns: it hands over its sums of the others
  constexpr int OT = D / 8 / PARTS;   // tiles of eight columns it finishes
  float own[OT][4];
#pragma unroll
  for (int n = 0; n < OT; ++n) {
#pragma unroll
    for (int x = 0; x < 4; ++x) own[n][x] = o[n][x];
  }
  if constexpr (PARTS > 1) {
    if (t == 0) {
      rows_x[share * 32 + 16 + g] = sum_lo;
      rows_x[share * 32 + 24 + g] = sum_hi;
    }
    float* mine = out_x + share * (D / 4) * 32 + lane;
#pragma unroll
    for (int n = 0; n < OT; ++n) {
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        own[n][x] = share == 0 ? o[n][x] : o[OT + n][x];
        mine[(4 * n + x) * 32] = share == 0 ? o[OT + n][x] : o[n][x];
      }
    }
    asm volatile("bar.sync %0, 64;" ::"r"(1 + group) : "memory");
    const float* theirs = out_x + (share ^ 1) * (D / 4) * 32 + lane;
#pragma unroll
    for (int n = 0; n < OT; ++n) {
#pragma unroll
      for (int x = 0; x < 4; ++x) own[n][x] += theirs[(4 * n + x) * 32];
    }
    sum_lo += rows_x[(share ^ 1) * 32 + 16 + g];
    sum_hi += rows_x[(share ^ 1) * 32 + 24 + g];
  }
  const float inv_lo = 1.0f / sum_lo, inv_hi = 1.0f / sum_hi;
  // through the group's rows of Q, so that the stores are 16 bytes wide
  const int first_chunk = share * OT;
#pragma unroll
  for (int n = 0; n < OT; ++n) {
    *reinterpret_cast<uint32_t*>(smem + LO::offQ + chunk_at<D>(r0 + g, first_chunk + n) + 4 * t) = attn::Pack2<T>::pack(own[n][0] * inv_lo, own[n][1] * inv_lo);
    *reinterpret_cast<uint32_t*>(smem + LO::offQ + chunk_at<D>(r0 + g + 8, first_chunk + n) + 4 * t) = attn::Pack2<T>::pack(own[n][2] * inv_hi, own[n][3] * inv_hi);
  }
  __syncwarp();
  const long long out_row0 = p.out_row_base ? (long long)p.out_row_base[b] : (long long)b * L;
  const int rows = p.out_row_base ? min(L, p.out_row_count[b]) : L;
  T* out = reinterpret_cast<T*>(p.out) + out_row0 * ((long long)p.heads * D) + (long long)h * D;
#pragma unroll
  for (int x = lane; x < 16 * OT; x += 32) {
    const int r = x / OT, c = first_chunk + x % OT;
    if (i0 + r < rows)
      *reinterpret_cast<uint4*>(out + (long long)(i0 + r) * p.heads * D + c * 8) = *reinterpret_cast<const uint4*>(smem + LO::offQ + chunk_at<D>(r0 + r, c));
  }
}

template <typename T, int D, int NW, int PARTS>
int launch_small(const DflAttnRelParams& p, bool tables_early, cudaStream_t stream) {
  using LO = SLayout<D, NW, PARTS>;
  auto kernel = attention_rel_small_kernel<T, D, NW, PARTS>;
  static KernelDeviceConfig config;   // per instantiation
  int sm_count = 0;
  if (int rc = configure_kernel(config, kernel, LO::total, &sm_count, "attention_rel_small_kernel")) return rc;
  const cudaError_t e = launch_after_predecessor(kernel, dim3(p.batch * p.heads * PARTS), dim3(LO::kThreads), LO::total, stream, p,
                                                 tables_early ? 1 : 0);
  if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "attention_rel_small_kernel: %s", cudaGetErrorString(e));
  return check_launch("attention_rel_small_kernel");
}

// Sizes of 2, 4, 6 and 8 warps: a row's windows are as wide as the size.  80 positions in six warps instead of eight
// 8.1 -> 7.4 us (4 x 12 heads), a forward of 8 x 96 tokens 553 -> 537 us.
template <typename T, int D, int PARTS>
int launch_rows(const DflAttnRelParams& p, bool tables_early, cudaStream_t stream) {
  return p.seq_len <= 32   ? launch_small<T, D, 2, PARTS>(p, tables_early, stream)
         : p.seq_len <= 64 ? launch_small<T, D, 4, PARTS>(p, tables_early, stream)
                           : launch_small<T, D, 6, PARTS>(p, tables_early, stream);
}

int device_sm_count() {
  static KernelDeviceConfig config;
  int sm_count = 0;
  return configure_kernel(config, attention_rel_small_kernel<__half, 64, 8, 2>, SLayout<64, 8, 2>::total, &sm_count,
                          "attention_rel_small_kernel") == DFL_OK ? sm_count : 0;
}

// Two CTAs a head while that does not take more CTAs than the SMs hold two of; with more heads the second CTA would only repeat
// the loads and the P2C windows.  us per launch, two / one, d 64: 48 items of 64 positions 4.4 / 5.6, 192 6.8 / 6.5, 384
// 10.5 / 7.6; 144 items of 96 positions 7.1 / 8.6, 192 12.4 / 9.9; 48 items of 128 positions 7.1 / 10.8, 144 9.5 / 11.3.
// The line is drawn for d 64.  At d 32 and 65 to 96 positions two CTAs are behind at 192 heads (96 positions: 8.4 / 8.1) and 4 to 17 %
// ahead again from 384 on (12.4 / 14.3, 768 20.8 / 21.6), where one is chosen all the same.
// Beyond 96 positions one CTA a head is never the choice (see attention_rel_small_covers).
template <typename T, int D>
int launch_parts(const DflAttnRelParams& p, bool tables_early, cudaStream_t stream) {
  if (p.seq_len > 96) return launch_small<T, D, 8, 2>(p, tables_early, stream);
  return p.batch * p.heads <= device_sm_count() ? launch_rows<T, D, 2>(p, tables_early, stream)
                                                : launch_rows<T, D, 1>(p, tables_early, stream);
}

}  // namespace

// Up to 96 positions two or more CTAs share an SM and this kernel is ahead at any batch (us, this / attention_rel_tc.cu: d 32, 64
// positions, 768 items 11.2 / 28.5; d 64, 96 positions, 192 items 9.9 / 13.7, 384 17.9 / 18.0, 768 26.9 / 29.6).  Beyond that it is
// ahead while its CTAs, two a head, make one round: two an SM at d 64 (128 positions: 144 items 9.5 / 10.1, 192 15.5 / 13.7), three
// at d 32 (192 items 9.9 / 12.7, 288 13.8 / 13.3).
bool attention_rel_small_covers(const DflAttnRelParams& p) {
  if (p.seq_len > 128 || (p.head_dim != 32 && p.head_dim != 64)) return false;
  if (p.seq_len <= 96) return true;
  return 2ll * p.batch * p.heads <= (p.head_dim == 32 ? 3ll : 2ll) * device_sm_count();
}

int launch_attention_rel_small(const DflAttnRelParams& p, bool tables_early, cudaStream_t stream) {
  if (p.dtype == DFL_F16)
    return p.head_dim == 64 ? launch_parts<__half, 64>(p, tables_early, stream) : launch_parts<__half, 32>(p, tables_early, stream);
  return p.head_dim == 64 ? launch_parts<__nv_bfloat16, 64>(p, tables_early, stream)
                          : launch_parts<__nv_bfloat16, 32>(p, tables_early, stream);
}

}  // namespace dfl
