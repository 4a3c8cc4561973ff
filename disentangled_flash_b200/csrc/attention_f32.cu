// FP32 fused disentangled attention on the tensor cores, position scores from memory: head dim 128, modules without position
// terms, and at head dim 64 sequences whose slot table does not fit beside attention_f32_rel.cu's tiles (3409 positions on; at
// head dim 32 every length fits).
//
// Q, K and V come as three bf16 planes each whose sum is the fp32 value (linear_f32.cu: the QKV projection writes them), the
// position scores C2P / P2C as fp32 [B,H,L,ld].  Semantics of kernel.py:137-345 in fp32 (the reference's strict mode):
//   S[i,j] = q_i.k_j + c2p[i, lut[i-j+L-1]] + p2c[j, lut[i-j+L-1]], scaled; padded keys -> -inf, a padded query row
//   attends uniformly to all L keys; online softmax in base 2; O = P V.
// S takes the six plane products of a fp32-accurate product, smallest first; P is split into planes as it is computed and
// PV takes six products as well.  Every key tile's PV starts from zero in tensor memory and is added to the output in
// registers, so no tensor-core accumulator is carried from tile to tile.
//
// One CTA per (batch, head, 128-query tile), keys in tiles of 128 (64 at head dim 128, where the planes of Q, K and V fill
// shared memory).  What bounds a tile is the softmax side: per (query, key) element two position scores gathered from
// global memory (C2P: one row per lane, L1 hits; P2C: consecutive slots over the lanes of a warp), one exponential and the
// split of P, about 25 instructions, against 24 + 48 MMAs (3.5 k cycles at d = 64).
// Warps 0-7 softmax (two threads per query row, each half of a tile's keys and half of the output columns), warp 8 TMA,
// warp 9 MMA issuer and TMEM owner.
#include "f32_planes.cuh"
#include "tcgen05_ptx.cuh"

namespace dfl {

__device__ int g_attn_f32_status = 0;

namespace {

constexpr int BM = 128, kSoftmaxWarps = 8, kTmaWarp = 8, kMmaWarp = 9, kThreads = 320;
constexpr int kMaxSmem = 232448;
constexpr int kWaits = kWaitsAttentionF32;
constexpr int COL_S = 0, COL_P = 128, COL_O = 320;   // S: BN fp32; P: three planes of BN / 2; O: D fp32
constexpr int kTmemCols = 512;

template <int D>
struct Tiles {
  static constexpr int BN = D == 128 ? 64 : 128;
  static constexpr int kRowBytes = D >= 64 ? 128 : D * 2;      // swizzle span
  static constexpr int kSub = D * 2 / kRowBytes;               // 64-column sub-tiles of a row
  static constexpr int kQSub = BM * kRowBytes, kKSub = BN * kRowBytes;
  static constexpr int kQ = kPlanes * kSub * kQSub, kKV = kPlanes * kSub * kKSub;
  static constexpr int offQ = 0, offK = kQ, offV = offK + kKV, offBar = offV + kKV;
  static constexpr int offMax = offBar + 256;                  // [2 halves][BM] row maxima, then row sums
  static constexpr int offKeep = offMax + 4 * BM * 4;
};

struct Barriers {
  uint64_t q_full, k_full, k_empty, v_full, v_empty, s_full, p_full, o_full, pair[4];
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(Barriers) <= 256, "barrier block too large");

template <int D>
__global__ void __launch_bounds__(kThreads, 1)
attention_f32_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                     const __grid_constant__ CUtensorMap tmap_v, const DflAttnParams p, int out_planes, int* status_word) {
  using T = Tiles<D>;
  constexpr int BN = T::BN, HK = BN / 2, OW = D / 2;   // keys and output columns per softmax thread
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + T::offBar);
  volatile int* abort_flag = &bars->abort_flag;
  const int L = p.seq_len, H = p.heads, BH = p.batch * H;
  const int n_kt = (L + BN - 1) / BN;
  uint32_t* keep_s = reinterpret_cast<uint32_t*>(smem + T::offKeep);                       // kept-key bits
  uint16_t* lut_s = reinterpret_cast<uint16_t*>(smem + T::offKeep + (n_kt * BN / 32) * 4);   // [2L-1]
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int bh = blockIdx.y, b = bh / H, h = bh - b * H, i0 = blockIdx.x * BM;
  const bool has_c2p = p.c2p != nullptr, has_p2c = p.p2c != nullptr;

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_full, 1);
    ptx::mbar_init(&bars->k_full, 1);
    ptx::mbar_init(&bars->k_empty, 1);
    ptx::mbar_init(&bars->v_full, 1);
    ptx::mbar_init(&bars->v_empty, 1);
    ptx::mbar_init(&bars->s_full, 1);
    ptx::mbar_init(&bars->p_full, kSoftmaxWarps);
    ptx::mbar_init(&bars->o_full, 1);
    for (int s = 0; s < 4; ++s) ptx::mbar_init(&bars->pair[s], 2);
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc(&bars->tmem_base, kTmemCols);
    ptx::tmem_relinquish();
  }
  wait_for_predecessor();
  if (has_c2p || has_p2c)
    for (int e = threadIdx.x; e < 2 * L - 1; e += kThreads) {
      int slot = p.lut[e];   // entries outside the score rows (not a table of the builder) are clamped
      slot = slot < 0 ? 0 : (slot >= p.ld_slots ? p.ld_slots - 1 : slot);
      lut_s[e] = (uint16_t)slot;
    }
  for (int w = warp; w < n_kt * BN / 32; w += kThreads / 32) {
    const int j = w * 32 + lane;
    const uint32_t bits = __ballot_sync(0xffffffffu, j < L && mask_keep(p.mask, p.mask_elem_size, (long long)b * L + j));
    if (lane == 0) keep_s[w] = bits;
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  release_successor();
  const uint32_t tmem_base = bars->tmem_base;

  if (warp == kTmaWarp) {
    if (lane == 0) {
      auto load = [&](int off, int sub_bytes, const CUtensorMap* map, uint64_t* bar, int row) {
        for (int q = 0; q < kPlanes; ++q)
          for (int c = 0; c < T::kSub; ++c)
            ptx::tma_load_3d(smem + off + (q * T::kSub + c) * sub_bytes, map, bar, c * 64, row, q * BH + bh);
      };
      ptx::mbar_arrive_expect_tx(&bars->q_full, (uint32_t)T::kQ);
      load(T::offQ, T::kQSub, &tmap_q, &bars->q_full, i0);
      for (int t = 0; t < n_kt; ++t) {
        if (!ptx::mbar_wait(&bars->k_empty, ((uint32_t)t & 1u) ^ 1u, abort_flag, status_word, kWaits + 51)) break;
        ptx::mbar_arrive_expect_tx(&bars->k_full, (uint32_t)T::kKV);
        load(T::offK, T::kKSub, &tmap_k, &bars->k_full, t * BN);
        if (!ptx::mbar_wait(&bars->v_empty, ((uint32_t)t & 1u) ^ 1u, abort_flag, status_word, kWaits + 52)) break;
        ptx::mbar_arrive_expect_tx(&bars->v_full, (uint32_t)T::kKV);
        load(T::offV, T::kKSub, &tmap_v, &bars->v_full, t * BN);
      }
    }
  } else if (warp == kMmaWarp) {
    constexpr uint32_t mode = ptx::swizzle_mode_for_row_bytes(T::kRowBytes), sbo = 8 * T::kRowBytes;
    constexpr uint32_t idesc_qk = ptx::make_idesc_f16(1, BM, BN, 0, 0), idesc_pv = ptx::make_idesc_f16(1, BM, D, 0, 1);
    constexpr int kSteps = T::kRowBytes / 32;
    constexpr int pa[6] = {2, 1, 0, 1, 0, 0}, pb[6] = {0, 1, 2, 0, 1, 0};   // plane products, smallest first
    const uint64_t qd = ptx::make_smem_desc(ptx::smem_u32(smem + T::offQ), 16, sbo, mode);
    const uint64_t kd = ptx::make_smem_desc(ptx::smem_u32(smem + T::offK), 16, sbo, mode);
    const uint64_t vd = ptx::make_smem_desc(ptx::smem_u32(smem + T::offV), T::kKSub, sbo, mode);
    auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
      return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag, status_word, code)) != 0;
    };
    auto issue_s = [&](int t) -> bool {
      if (!wait(&bars->k_full, (uint32_t)t & 1u, kWaits + 53)) return false;
      ptx::tc_fence_after();
#pragma unroll
      for (int q = 0; q < 6; ++q)
#pragma unroll
        for (int c = 0; c < T::kSub; ++c)
#pragma unroll
          for (int k = 0; k < kSteps; ++k)
            ptx::umma_ss_f16_warp(tmem_base + COL_S, qd + (uint64_t)(((pa[q] * T::kSub + c) * T::kQSub + k * 32) >> 4),
                                  kd + (uint64_t)(((pb[q] * T::kSub + c) * T::kKSub + k * 32) >> 4), idesc_qk,
                                  q != 0 || c != 0 || k != 0 ? 1u : 0u);
      ptx::umma_commit_warp(&bars->k_empty);
      ptx::umma_commit_warp(&bars->s_full);
      return true;
    };
    bool ok = wait(&bars->q_full, 0, kWaits + 54) && issue_s(0);
    for (int t = 0; t < n_kt && ok; ++t) {
      ok = wait(&bars->p_full, (uint32_t)t & 1u, kWaits + 55) && wait(&bars->v_full, (uint32_t)t & 1u, kWaits + 56);
      if (!ok) break;
      ptx::tc_fence_after();
#pragma unroll 1
      for (int q = 0; q < 6; ++q) {
        const uint32_t a = tmem_base + COL_P + (uint32_t)(pa[q] * (BN / 2));
        const uint64_t bq = vd + (uint64_t)((pb[q] * T::kSub * T::kKSub) >> 4);
#pragma unroll
        for (int k = 0; k < BN / 16; ++k)
          ptx::umma_ts_f16_warp(tmem_base + COL_O, a + (uint32_t)(k * 8), bq + (uint64_t)((k * 16 * T::kRowBytes) >> 4), idesc_pv,
                                q != 0 || k != 0 ? 1u : 0u);
      }
      ptx::umma_commit_warp(&bars->v_empty);
      ptx::umma_commit_warp(&bars->o_full);
      if (t + 1 < n_kt) ok = issue_s(t + 1);   // S(t) has been read by every softmax thread before P(t) was stored
    }
  } else {
    const int hf = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane, i = i0 + r;
    const bool row_ok = i < L;
    const bool q_keep = row_ok && mask_keep(p.mask, p.mask_elem_size, (long long)b * L + i);
    const float scale_log2 = p.scale * 1.4426950408889634f;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    const uint32_t t_s = tmem_base + lanes + COL_S + hf * HK, t_p = tmem_base + lanes + COL_P + hf * (HK / 2);
    const uint32_t t_o = tmem_base + lanes + COL_O + hf * OW;
    float* xmax = reinterpret_cast<float*>(smem + T::offMax);
    const float* c2p = has_c2p ? reinterpret_cast<const float*>(p.c2p) + ((long long)bh * L + (row_ok ? i : 0)) * p.ld_slots : nullptr;
    const float* p2c = has_p2c ? reinterpret_cast<const float*>(p.p2c) + (long long)bh * L * p.ld_slots : nullptr;
    const uint16_t* lut_i = lut_s + (row_ok ? i : 0) + L - 1;   // slot of key j: lut_i[-j]
    float o[OW];
#pragma unroll
    for (int c = 0; c < OW; ++c) o[c] = 0.0f;
    float m_run = -INFINITY, l_run = 0.0f;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
      return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, abort_flag, status_word, code)) != 0;
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
    // position scores of keys j0 .. j0 + 15
    auto gather = [&](int j0, float (&a)[16], float (&d)[16]) {
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const int j = j0 + c;
        const bool in = row_ok && j < L;
        const int slot = in ? lut_i[-j] : 0;
        a[c] = has_c2p && in ? __ldg(c2p + slot) : 0.0f;
        d[c] = has_p2c && in ? __ldg(p2c + (long long)j * p.ld_slots + slot) : 0.0f;
      }
    };
    for (int t = 0; t < n_kt && ok; ++t) {
      const int j0 = t * BN + hf * HK;
      // The position scores do not depend on S: the first of the tile's are on their way while it is waited for.  us per launch
      // without / with: d 32 8 x 24 heads x 128 35.6 / 35.5, 16 x 24 x 256 178 / 173, 8 x 24 x 512 305 / 295 (its 112 bytes of
      // spills cost less than it gives); d 64 8 x 12 x 128 23.7 / 22.9, 8 x 24 x 256 113 / 108, 8 x 12 x 512 184 / 172 (96
      // bytes, 40 without); d 128 8 x 8 x 128 43.5 / 37.8, 16 x 8 x 256 171 / 143, 8 x 8 x 512 254 / 211; one term alone 2 to 17 %
      // faster.  All of a tile's at once do not fit the registers; rows of C2P copied to shared memory first, 25 -> 29 us.
      float a[16], d[16];
      gather(j0, a, d);
      ok = wait(&bars->s_full, (uint32_t)t & 1u, kWaits + 57);
      if (!ok) break;
      ptx::tc_fence_after();
      float s[HK];
#pragma unroll
      for (int c0 = 0; c0 < HK; c0 += 32) {
        float v[32];
        ptx::tmem_ld32_f(t_s + c0, v);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) s[c0 + c] = v[c];
      }
      if (has_c2p || has_p2c) {
#pragma unroll
        for (int c0 = 0; c0 < HK; c0 += 16) {
          if (c0 > 0) gather(j0 + c0, a, d);
#pragma unroll
          for (int c = 0; c < 16; ++c) s[c0 + c] = (s[c0 + c] + a[c]) + d[c];
        }
      }
      float mx = -INFINITY;
#pragma unroll
      for (int w = 0; w < HK / 32; ++w) {
        const uint32_t bits = keep_s[(j0 >> 5) + w];
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const int j = j0 + 32 * w + c;
          float v = s[32 * w + c] * scale_log2;
          if (!q_keep) v = j < L ? 0.0f : -INFINITY;
          else if (!((bits >> c) & 1u)) v = -INFINITY;
          s[32 * w + c] = v;
          mx = fmaxf(mx, v);
        }
      }
      // row maximum over both halves of the tile
      xmax[(t & 1) * 2 * BM + hf * BM + r] = mx;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->pair[quarter]);
      ok = wait(&bars->pair[quarter], (uint32_t)t & 1u, kWaits + 58);
      if (!ok) break;
      const float m_new = fmaxf(m_run, fmaxf(mx, xmax[(t & 1) * 2 * BM + (1 - hf) * BM + r]));
      const float m_use = m_new == -INFINITY ? 0.0f : m_new;
      const float corr = exp2f(m_run - m_use);   // 0 while nothing has been attended to
      m_run = m_new;
      float sum = 0.0f;
#pragma unroll
      for (int c = 0; c < HK; ++c) {
        s[c] = exp2f(s[c] - m_use);
        sum += s[c];
      }
      l_run = l_run * corr + sum;
      if (t > 0) {   // the previous tile's PV: added before its scale is left behind, and P may be overwritten
        ok = wait(&bars->o_full, (uint32_t)(t - 1) & 1u, kWaits + 59);
        if (!ok) break;
        ptx::tc_fence_after();
        add_output(corr);
      }
#pragma unroll
      for (int c0 = 0; c0 < HK; c0 += 16) {
        uint32_t lo[kPlanes][4], hi[kPlanes][4];
        split_eight(&s[c0], lo);
        split_eight(&s[c0 + 8], hi);
#pragma unroll
        for (int q = 0; q < kPlanes; ++q) {
          const uint32_t w[8] = {lo[q][0], lo[q][1], lo[q][2], lo[q][3], hi[q][0], hi[q][1], hi[q][2], hi[q][3]};
          ptx::tmem_st8(t_p + (uint32_t)(q * (BN / 2) + c0 / 2), w);
        }
      }
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->p_full);
    }
    if (ok) ok = wait(&bars->o_full, (uint32_t)(n_kt - 1) & 1u, kWaits + 60);
    if (ok) {
      ptx::tc_fence_after();
      add_output(1.0f);
      float* xsum = xmax + (n_kt & 1) * 2 * BM;   // the parity the last tile did not use
      xsum[hf * BM + r] = l_run;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->pair[quarter]);
      ok = wait(&bars->pair[quarter], (uint32_t)n_kt & 1u, kWaits + 61);
      if (ok && row_ok) {
        const float inv = 1.0f / (l_run + xsum[(1 - hf) * BM + r]);
        const long long at = ((long long)b * L + i) * ((long long)H * D) + (long long)h * D + hf * OW;
#pragma unroll
        for (int c = 0; c < OW; c += 4) {
          const float f[4] = {o[c] * inv, o[c + 1] * inv, o[c + 2] * inv, o[c + 3] * inv};
          if (out_planes) {
            uint2 w[kPlanes];
            split3x4(f, w);
            const long long plane = (long long)p.batch * L * H * D;
#pragma unroll
            for (int q = 0; q < kPlanes; ++q)
              *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + q * plane + at + c) = w[q];
          } else {
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + at + c) = make_float4(f[0], f[1], f[2], f[3]);
          }
        }
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) ptx::tmem_dealloc(tmem_base, kTmemCols);
}

template <int D>
int launch_d(const DflAttnParams& p, int out_planes, cudaStream_t stream) {
  using T = Tiles<D>;
  const int L = p.seq_len, BH = p.batch * p.heads;
  const uint64_t row = (uint64_t)D * 2, seq = (uint64_t)L * row;
  const uint32_t box_inner = D < 64 ? D : 64;
  CUtensorMap tq, tk, tv;
  int rc = encode_tensor_map_3d(&tq, p.q, D, L, (uint64_t)kPlanes * BH, row, seq, box_inner, BM, T::kRowBytes);
  if (rc == DFL_OK) rc = encode_tensor_map_3d(&tk, p.k, D, L, (uint64_t)kPlanes * BH, row, seq, box_inner, T::BN, T::kRowBytes);
  if (rc == DFL_OK) rc = encode_tensor_map_3d(&tv, p.v, D, L, (uint64_t)kPlanes * BH, row, seq, box_inner, T::BN, T::kRowBytes);
  if (rc != DFL_OK) return rc;
  const int n_kt = (L + T::BN - 1) / T::BN;
  const int smem = T::offKeep + n_kt * T::BN / 8 + (2 * L - 1) * 2 + 1024 + 16;
  if (smem > kMaxSmem) return fail(DFL_ERR_TOO_LARGE, "seq_len %d needs %d bytes of shared memory", L, smem);
  auto kernel = attention_f32_kernel<D>;
  static KernelDeviceConfig config;   // per instantiation
  rc = configure_kernel(config, kernel, kMaxSmem, nullptr, "attention_f32_kernel");
  if (rc != DFL_OK) return rc;
  int* status_word = p.status;
  if (!status_word) {
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&status_word), g_attn_f32_status);
    if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "status word: %s", cudaGetErrorString(e));
  }
  // never so little shared memory that a second CTA could become resident: each takes all of tensor memory
  const int floor_smem = kMaxSmem / 2 + 1024;
  const dim3 grid((L + BM - 1) / BM, BH);
  cudaError_t e = launch_after_predecessor(kernel, grid, dim3(kThreads), (size_t)(smem < floor_smem ? floor_smem : smem), stream, tq,
                                           tk, tv, p, out_planes, status_word);
  if (e != cudaSuccess) return fail(DFL_ERR_LAUNCH, "attention_f32_kernel: %s", cudaGetErrorString(e));
  return check_launch("attention_f32_kernel");
}

}  // namespace

bool attention_f32_planes_supported(int head_dim, int seq_len) {
  return (head_dim == 32 || head_dim == 64 || head_dim == 128) && seq_len >= 1 && seq_len <= (head_dim == 128 ? 4096 : 8192);
}

int launch_attention_f32_planes(const DflAttnParams& p, int out_planes, cudaStream_t stream) {
  if ((long long)p.batch * p.heads > 65535) return fail(DFL_ERR_TOO_LARGE, "batch*heads > 65535");
  switch (p.head_dim) {
    case 32: return launch_d<32>(p, out_planes, stream);
    case 64: return launch_d<64>(p, out_planes, stream);
    case 128: return launch_d<128>(p, out_planes, stream);
  }
  return fail(DFL_ERR_UNSUPPORTED, "head_dim %d not in {32,64,128}", p.head_dim);
}

}  // namespace dfl
