// Disentangled attention over position tables laid out by relative distance, for short sequences.
//
// The operation of attention_rel_tc.cu (dfl_attention_rel_fwd) for sequences of at most 128 positions, where that kernel
// has one key tile per item and is a chain of hand-overs between its roles (load, table MMAs, converters, score MMA,
// softmax, PV): 11 us for a batch that needs well under one.  Here a (batch, head) is one CTA with one warp per 16 query
// rows, the whole sequence is in shared memory, and every step of a row stays in the registers of its warp:
//   P2C[j, m] = k_j . rel_query[j0 + m]      the warp's 16 keys against the table rows 16 + LM columns wide that any query
//   C2P[i, m] = q_i . rel_key[LM-16-i0 + m]  can reach; both rounded to T and written to shared memory
//   S = Q K^T on the fragments, plus C2P[i, j - i + 15] and P2C[j, j - i + LM - 1]; mask, softmax, O = P V, normalise.
// The matrix instruction is the warp-level mma.sync: its result is in the registers of the warp that needs it, where tensor
// memory would bring back the round trips that bound the other kernel; the operands of an item are a few hundred
// instructions of it.  What bounds it is the load latency, then the diagonal gathers.  us per launch, fp16, d 64, both terms,
// attention_rel_tc.cu -> here: 1 x 12 heads x 32 9.2 -> 4.0, 8 x 24 x 64 13.9 -> 6.5, 64 x 16 x 32 40 -> 8.9, 64 x 16 x 64
// 40 -> 23; 8 x 12 x 128 10.0 -> 10.2 back to back, but 1.2 us a layer less in a forward, where its set-up and its
// table loads overlap the projection.  A forward of 1 x 32 tokens (hidden 768, 12 layers) 463 -> 381 us, of 8 x 64 at hidden 1536
// (24 layers) 1638 -> 1416 us.
// Rounding is that of attention_rel_tc.cu: relative terms to T (FP16 saturating), P to T (BF16 up to 64 keys: to two of them), the row sum
// over the rounded P.
#include "attention_tc_common.cuh"

namespace dfl {
namespace {

template <int D, int NW>
struct SLayout {
  static constexpr int kThreads = 32 * NW;
  static constexpr int LM = 16 * NW;             // positions covered
  static constexpr int kRowBytes = D * 2;
  static constexpr int kChunks = kRowBytes / 16;
  // 16-bit columns per score row: LM + 16, and 10 more so that the gathers of a warp (rows g, columns 2t, shifted by the row)
  // spread over the banks
  static constexpr int kPitch = LM + 26;
  static constexpr int offQ = 0;
  static constexpr int offK = offQ + LM * kRowBytes;
  static constexpr int offV = offK + LM * kRowBytes;
  static constexpr int offRK = offV + LM * kRowBytes;
  static constexpr int offRQ = offRK + 2 * LM * kRowBytes;
  static constexpr int offC = offRQ + 2 * LM * kRowBytes;
  static constexpr int offP = offC + LM * kPitch * 2;
  static constexpr int offKeep = offP + LM * kPitch * 2;
  static constexpr int total = offKeep + LM;
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

template <typename T, int D, int NW>
__global__ void __launch_bounds__(SLayout<D, NW>::kThreads)
attention_rel_small_kernel(const DflAttnRelParams p, int tables_early) {
  using LO = SLayout<D, NW>;
  constexpr int LM = LO::LM, CH = LO::kChunks, NT = LO::kThreads, P = LO::kPitch;
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t base = ptx::smem_u32(smem);
  const int L = p.seq_len, bh = blockIdx.x, b = bh / p.heads, h = bh - b * p.heads;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const bool has_c2p = p.rel_key != nullptr, has_p2c = p.rel_query != nullptr;

  // Table row e (x = j - i = e - (L - 1)) goes to row e + LM - L, which makes every window below independent of L.  Rows
  // the tables do not have are left as they are: they only reach scores of positions beyond L, which are replaced.
  auto load_tables = [&]() {
    const long long first = (long long)h * (2 * L - 1) * D;
    for (int x = tid; x < (2 * L - 1) * CH; x += NT) {
      const int e = x / CH, c = x - e * CH;
      const uint32_t at = chunk_at<D>(e + LM - L, c);
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
        ptx::cp_async_16(smem + LO::offQ + at, reinterpret_cast<const T*>(p.q) + from);
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

  const int i0 = 16 * warp;
  const bool active = i0 < L;
  uint32_t qf[D / 16][4];
  if (active) {
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) ldsm(qf[kk], base + LO::offQ + chunk_at<D>(i0 + (lane & 15), 2 * kk + (lane >> 4)));
    // 16 rows of `a` against LM + 16 table rows from `row0` on, rounded, to rows i0.. of the score buffer
    auto relative = [&](const uint32_t (&a)[D / 16][4], int table, int row0, int dst) {
#pragma unroll 2
      for (int n = 0; n < (LM + 16) / 8; ++n) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k2 = 0; k2 < D / 32; ++k2) {
          uint32_t bf[4];
          ldsm(bf, base + table + chunk_at<D>(row0 + 8 * n + (lane & 7), 4 * k2 + (lane >> 3)));
          mma16816<T>(c, a[2 * k2], bf[0], bf[1]);
          mma16816<T>(c, a[2 * k2 + 1], bf[2], bf[3]);
        }
        uint32_t* to = reinterpret_cast<uint32_t*>(smem + dst + ((i0 + g) * P + 8 * n + 2 * t) * 2);
        to[0] = round_scores<T>(c[0], c[1]);
        to[4 * P] = round_scores<T>(c[2], c[3]);   // eight rows further down
      }
    };
    if (has_p2c) {
      uint32_t kf[D / 16][4];
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) ldsm(kf[kk], base + LO::offK + chunk_at<D>(i0 + (lane & 15), 2 * kk + (lane >> 4)));
      relative(kf, LO::offRQ, i0, LO::offP);
    }
    if (has_c2p) relative(qf, LO::offRK, LM - 16 - i0, LO::offC);
  }
  __syncthreads();
  if (!active) return;

  uint32_t bits[(LM + 31) / 32];   // kept keys
#pragma unroll
  for (int w = 0; w < (LM + 31) / 32; ++w) bits[w] = __ballot_sync(0xffffffffu, smem[LO::offKeep + 32 * w + lane] != 0);
  const bool keep_lo = smem[LO::offKeep + i0 + g] != 0, keep_hi = smem[LO::offKeep + i0 + g + 8] != 0;

  float s[LM / 8][4];
  float max_lo = -INFINITY, max_hi = -INFINITY;
  const T* c2p = reinterpret_cast<const T*>(smem + LO::offC) + (i0 + g) * P + 15 - g + 2 * t;
  const T* p2c = reinterpret_cast<const T*>(smem + LO::offP) + 2 * t * P + 2 * t + LM - 1 - i0 - g;
#pragma unroll
  for (int n = 0; n < LM / 8; ++n) {
#pragma unroll
    for (int x = 0; x < 4; ++x) s[n][x] = -INFINITY;
    if (8 * n < L) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k2 = 0; k2 < D / 32; ++k2) {
        uint32_t bf[4];
        ldsm(bf, base + LO::offK + chunk_at<D>(8 * n + (lane & 7), 4 * k2 + (lane >> 3)));
        mma16816<T>(c, qf[2 * k2], bf[0], bf[1]);
        mma16816<T>(c, qf[2 * k2 + 1], bf[2], bf[3]);
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) {   // row i0 + g + 8 (x >> 1), key j = 8 n + 2 t + (x & 1)
        const int j = 8 * n + 2 * t + (x & 1), down = 8 * (x >> 1);
        if (has_c2p) c[x] += Elem<T>::to_f(c2p[down * (P - 1) + 8 * n + (x & 1)]);
        if (has_p2c) c[x] += Elem<T>::to_f(p2c[(8 * n + (x & 1)) * P + 8 * (n & 1) + (x & 1) - down]);
        const bool kept = (bits[n / 4] >> (8 * (n & 3) + 2 * t + (x & 1))) & 1u;
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
  for (int ks = 0; ks < LM / 16; ++ks) {
    if (16 * ks >= L) continue;
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
      ldsm_trans(bf, base + LO::offV + chunk_at<D>(16 * ks + (lane & 15), 2 * n2 + (lane >> 4)));
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
  const float inv_lo = 1.0f / sum_lo, inv_hi = 1.0f / sum_hi;
  // through the warp's own rows of Q, so that the stores are 16 bytes wide
#pragma unroll
  for (int n = 0; n < D / 8; ++n) {
    *reinterpret_cast<uint32_t*>(smem + LO::offQ + chunk_at<D>(i0 + g, n) + 4 * t) = attn::Pack2<T>::pack(o[n][0] * inv_lo, o[n][1] * inv_lo);
    *reinterpret_cast<uint32_t*>(smem + LO::offQ + chunk_at<D>(i0 + g + 8, n) + 4 * t) = attn::Pack2<T>::pack(o[n][2] * inv_hi, o[n][3] * inv_hi);
  }
  __syncwarp();
  const long long out_row0 = p.out_row_base ? (long long)p.out_row_base[b] : (long long)b * L;
  const int rows = p.out_row_base ? min(L, p.out_row_count[b]) : L;
  T* out = reinterpret_cast<T*>(p.out) + out_row0 * ((long long)p.heads * D) + (long long)h * D;
#pragma unroll
  for (int x = lane; x < 16 * CH; x += 32) {
    const int i = i0 + x / CH, c = x % CH;
    if (i < rows) *reinterpret_cast<uint4*>(out + (long long)i * p.heads * D + c * 8) = *reinterpret_cast<const uint4*>(smem + LO::offQ + chunk_at<D>(i, c));
  }
}

template <typename T, int D, int NW>
int launch_small(const DflAttnRelParams& p, bool tables_early, cudaStream_t stream) {
  using LO = SLayout<D, NW>;
  auto kernel = attention_rel_small_kernel<T, D, NW>;
  static KernelDeviceConfig config;   // per instantiation
  int sm_count = 0;
  if (int rc = configure_kernel(config, kernel, LO::total, &sm_count, "attention_rel_small_kernel")) return rc;
  const cudaError_t e = launch_after_predecessor(kernel, dim3(p.batch * p.heads), dim3(LO::kThreads), LO::total, stream, p,
                                                 tables_early ? 1 : 0);
  if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "attention_rel_small_kernel: %s", cudaGetErrorString(e));
  return check_launch("attention_rel_small_kernel");
}

// Sizes of 2, 4, 6 and 8 warps: a row's windows are as wide as the size.  80 positions in six warps instead of eight
// 8.1 -> 7.4 us (4 x 12 heads), a forward of 8 x 96 tokens 553 -> 537 us.
template <typename T, int D>
int launch_rows(const DflAttnRelParams& p, bool tables_early, cudaStream_t stream) {
  return p.seq_len <= 32   ? launch_small<T, D, 2>(p, tables_early, stream)
         : p.seq_len <= 64 ? launch_small<T, D, 4>(p, tables_early, stream)
         : p.seq_len <= 96 ? launch_small<T, D, 6>(p, tables_early, stream)
                           : launch_small<T, D, 8>(p, tables_early, stream);
}

}  // namespace

// Up to 64 positions several CTAs share an SM and this kernel is ahead at any batch (d 32, 64 positions, 768 items: 10.7
// against 30.5 us).  Beyond that, at d 64 and from 97 positions on at d 32, a CTA takes an SM's shared memory, and a second
// round of them costs more than the other kernel's pipeline over items: as long as there is one round (d 64, 96 positions: 144
// items 8.2 against 10.7 us, 192 items 15.1 against 14.0).  At d 32 and 65 to 96 positions two CTAs fit (90 KB), and one round is
// less than this kernel could be used for: 288 items of 96 positions take 13.9 us in the other one, 7.2 in this.
bool attention_rel_small_covers(const DflAttnRelParams& p) {
  if (p.seq_len > 128 || (p.head_dim != 32 && p.head_dim != 64)) return false;
  if (p.seq_len <= 64) return true;
  static KernelDeviceConfig config;
  int sm_count = 0;
  return configure_kernel(config, attention_rel_small_kernel<__half, 64, 8>, SLayout<64, 8>::total, &sm_count,
                          "attention_rel_small_kernel") == DFL_OK && p.batch * p.heads <= sm_count;
}

int launch_attention_rel_small(const DflAttnRelParams& p, bool tables_early, cudaStream_t stream) {
  if (p.dtype == DFL_F16)
    return p.head_dim == 64 ? launch_rows<__half, 64>(p, tables_early, stream) : launch_rows<__half, 32>(p, tables_early, stream);
  return p.head_dim == 64 ? launch_rows<__nv_bfloat16, 64>(p, tables_early, stream)
                          : launch_rows<__nv_bfloat16, 32>(p, tables_early, stream);
}

}  // namespace dfl
