// The layer loop of a prepared encoder (DebertaV2InferenceEncoder.forward_prepared, src/disentangled_flash/
// deberta.py:247-285) as one host function: it carves the activations out of one workspace and issues the library's
// kernels back to back.  From Python a layer costs some 130 us of host time for seven launches, more than its kernels run
// for a batch below about 1500 tokens; here it is about 20 us.  Each kernel after the first knows that its predecessor
// is one of this library's (GemmDesc::weights_early).
#include "dfl_common.cuh"

namespace dfl {
namespace {

constexpr size_t kAlign = 256;
size_t padded(size_t bytes) { return (bytes + kAlign - 1) / kAlign * kAlign; }

// Offsets of the activations inside the workspace.
struct Workspace {
  size_t qkv, context, dense, mixed, inner, state[2], scores[2], total;
  // F32: bf16 planes of the layer's input, of its first output block, and of the FFN's inside (Q, K, V and the context
  // are planes there too)
  size_t state_planes, mixed_planes, inner_planes;
  size_t conv_w;   // conv_w_module: the convolution's weight by taps
};

constexpr size_t kPlaneBytes = 6;   // three bf16 planes per element

// F32 whose attention kernel computes the position scores itself: nothing of them in the workspace
bool scores_in_kernel(const DflEncoderParams& p) { return p.dtype == DFL_F32 && attention_f32_rel_supported(p.head_dim, p.seq_len); }

bool two_call(const DflEncoderParams& p) { return !p.layers[0].rel_key && !p.layers[0].rel_query; }

Workspace plan_workspace(const DflEncoderParams& p) {
  const size_t es = dtype_size(p.dtype), positions = (size_t)p.batch * p.seq_len;
  const size_t rows = p.packed_rows > 0 ? (size_t)p.packed_rows : positions;
  const size_t width = (size_t)p.heads * p.head_dim;
  Workspace w{};
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += padded(bytes);
    return here;
  };
  const bool f32 = p.dtype == DFL_F32, layers = !p.attention_only;
  w.qkv = take(p.packed_rows > 0 && p.row_groups ? 0 : 3 * padded(positions * width * (f32 ? kPlaneBytes : es)));
  if (layers) {
    w.context = take(rows * width * (f32 ? kPlaneBytes : es));
    w.dense = take(rows * p.hidden * es);
    w.mixed = take(rows * p.hidden * es);
    const size_t inner = f32 ? 0 : rows * (size_t)p.ffn, conv = p.conv_w ? positions * (size_t)p.hidden : 0;
    w.inner = take((inner > conv ? inner : conv) * es);   // also the convolution's output
    for (int i = 0; i < 2; ++i) w.state[i] = take(rows * p.hidden * es);
  }
  if (f32) {
    w.state_planes = take(rows * p.hidden * kPlaneBytes);
    if (layers) {
      w.mixed_planes = take(rows * p.hidden * kPlaneBytes);
      w.inner_planes = take(rows * (size_t)p.ffn * kPlaneBytes);
    }
  }
  if (p.conv_w && p.conv_w_module) w.conv_w = take((size_t)p.conv_taps * p.hidden * p.hidden * es);
  if (two_call(p) && !scores_in_kernel(p)) {
    const size_t ld = ((size_t)p.n_active + 7) / 8 * 8;
    for (int i = 0; i < 2; ++i) w.scores[i] = take(positions * p.heads * ld * es);
  }
  w.total = at;
  return w;
}

int validate(const DflEncoderParams& p) {
  if (p.dtype != DFL_F16 && p.dtype != DFL_BF16 && p.dtype != DFL_F32) return fail(DFL_ERR_BAD_ARG, "unknown dtype %d", p.dtype);
  if (p.n_layers < 1 || p.batch < 1 || p.seq_len < 1 || p.hidden < 1 || p.heads < 1 || (p.ffn < 1 && !p.attention_only))
    return fail(DFL_ERR_BAD_ARG, "non-positive size");
  if (p.head_dim != 32 && p.head_dim != 64 && p.head_dim != 128)
    return fail(DFL_ERR_UNSUPPORTED, "head_dim %d not in {32,64,128}", p.head_dim);
  if (p.hidden % 8 || (!p.attention_only && (p.ffn % 8 || !dfl_add_layernorm_supported(p.dtype, p.hidden))))
    return fail(DFL_ERR_UNSUPPORTED, "hidden %d / ffn %d not covered", p.hidden, p.ffn);
  if (!p.layers || !p.outs || !p.outs[p.n_layers - 1] || !p.x || !p.mask || !p.workspace)
    return fail(DFL_ERR_BAD_ARG, "null pointer");
  if (p.mask_elem_size != 1 && p.mask_elem_size != 4 && p.mask_elem_size != 8)
    return fail(DFL_ERR_BAD_ARG, "mask_elem_size must be 1, 4 or 8");
  if (!(p.scale > 0.0f)) return fail(DFL_ERR_BAD_ARG, "scale must be positive");
  if (!aligned16(p.x) || !aligned16(p.workspace)) return fail(DFL_ERR_ALIGNMENT, "tensors must be 16-byte aligned");
  for (int l = 0; l < p.n_layers; ++l) {
    const DflEncoderLayer& y = p.layers[l];
    if (!y.qkv_w || (!p.attention_only && (!y.attn_out_w || !y.attn_norm_w || !y.ffn_in_w || !y.ffn_out_w || !y.ffn_norm_w)))
      return fail(DFL_ERR_BAD_ARG, "layer %d: null weight", l);
    const void* all[16] = {y.qkv_w, y.qkv_b, y.attn_out_w, y.attn_out_b, y.attn_norm_w, y.attn_norm_b, y.ffn_in_w, y.ffn_in_b,
                           y.ffn_out_w, y.ffn_out_b, y.ffn_norm_w, y.ffn_norm_b, y.rel_key, y.rel_query, y.pos_key, y.pos_query};
    for (const void* q : all)
      if (!aligned16(q)) return fail(DFL_ERR_ALIGNMENT, "layer %d: weights must be 16-byte aligned", l);
    if (!aligned16(p.outs[l])) return fail(DFL_ERR_ALIGNMENT, "outs[%d] not 16-byte aligned", l);
    if (!(y.attn_norm_eps >= 0.0f) || !(y.ffn_norm_eps >= 0.0f)) return fail(DFL_ERR_BAD_ARG, "eps must be non-negative");
    if ((!y.rel_key && !y.rel_query) != two_call(p)) return fail(DFL_ERR_BAD_ARG, "layers with and without rel tables");
    // the F32 kernel gathers rows of these tables by the slots of lut, clamped to [0, n_active)
    if (two_call(p) && (y.pos_key || y.pos_query) && (!p.lut || p.n_active < 1))
      return fail(DFL_ERR_BAD_ARG, "layer %d: position tables without a LUT or with n_active %d", l, p.n_active);
  }
  if (p.attention_only && (p.n_layers != 1 || p.packed_rows > 0 || p.conv_w))
    return fail(DFL_ERR_BAD_ARG, "attention_only takes one layer of padded rows");
  if (p.dtype == DFL_F32 && (p.conv_w || p.packed_rows > 0 || !two_call(p)))
    return fail(DFL_ERR_UNSUPPORTED, "F32 has no convolution branch, no packed rows and no rel_key / rel_query form");
  if (p.plane_sources && (p.dtype != DFL_F32 || p.n_plane_sources < 1 || p.n_plane_pieces < 1))
    return fail(DFL_ERR_BAD_ARG, "plane sources are an F32 form, with their counts");
  if (p.dtype == DFL_F32 && !attention_f32_planes_supported(p.head_dim, p.seq_len))
    return fail(DFL_ERR_UNSUPPORTED, "head_dim %d at seq_len %d in F32", p.head_dim, p.seq_len);
  if (p.conv_w && p.conv_w_module && p.conv_taps < 1) return fail(DFL_ERR_BAD_ARG, "conv_taps %d", p.conv_taps);
  // the two-call attention kernels have batch*heads as a grid's second dimension; the rel form has no such limit
  if (two_call(p) && (long long)p.batch * p.heads > 65535) return fail(DFL_ERR_TOO_LARGE, "batch*heads > 65535");
  if (p.packed_rows > 0) {
    if (two_call(p)) return fail(DFL_ERR_UNSUPPORTED, "packed rows need the rel_key / rel_query form");
    if (!p.pack_rows || !p.row_base || !p.row_count) return fail(DFL_ERR_BAD_ARG, "null packed-row table");
    if (p.row_groups) {
      if (p.packed_rows % 32 || p.seq_len % 32) return fail(DFL_ERR_BAD_ARG, "row groups are 32 rows of one sequence");
      if (!p.qkv[0] || !p.qkv[1] || !p.qkv[2]) return fail(DFL_ERR_BAD_ARG, "null qkv buffer");
    }
  }
  return DFL_OK;
}

struct Loop {
  DflEncoderParams& p;
  cudaStream_t stream;
  Workspace w;
  unsigned char* base;

  void* at(size_t offset) const { return base + offset; }

  // out[rows, n] = act(x[rows, k] w^T + b), or the three head-major tensors of the QKV projection
  int gemm(const void* x, const void* weight, const void* bias, void* out, int rows, int n, int k, int activation,
           void* const* heads_out = nullptr, bool out_planes = false) {
    GemmDesc g{};
    g.x = x; g.w = weight; g.bias = bias;
    g.M = rows; g.N = n; g.K = k;
    g.batch = 1; g.w_mod = 1; g.ldc = n;
    g.heads = 1; g.head_dim = n; g.rows_per_seq = rows;
    g.dtype = p.dtype; g.status = p.status; g.activation = activation;
    g.weights_early = p.launches > 0 ? 1 : 0;
    if (heads_out) {
      for (int i = 0; i < 3; ++i) g.out[i] = heads_out[i];
      g.head_split = 1; g.heads = p.heads; g.head_dim = p.head_dim; g.rows_per_seq = p.seq_len;
      if (p.packed_rows > 0 && p.row_groups) {
        g.row_groups = p.row_groups;
        g.out_seqs = p.batch;
      }
    } else {
      g.out[0] = out;
    }
    ++p.launches;
    if (p.dtype == DFL_F32) {
      g.out_planes = out_planes ? 1 : 0;
      return launch_gemm_f32_planes(g, stream);
    }
    return launch_gemm_tc(g, stream);
  }

  int split(const void* x, void* planes, size_t elements) {
    ++p.launches;
    return launch_split_planes(x, planes, (long long)elements, stream);
  }

  // scores[b, h, row, slot] = head[b, h, row, :] . table[h, slot, :] in F32 over the planes of both
  int scores_f32(const void* head, const void* table, void* out, int ld) {
    GemmDesc g{};
    g.x = head; g.w = table; g.out[0] = out;
    g.M = p.seq_len; g.N = p.n_active; g.K = p.head_dim;
    g.batch = p.batch * p.heads; g.w_mod = p.heads;
    g.stride_c = (long long)p.seq_len * ld; g.ldc = ld;
    g.heads = p.heads; g.head_dim = p.head_dim; g.rows_per_seq = p.seq_len;
    g.dtype = p.dtype; g.status = p.status; g.weights_early = 1;
    ++p.launches;
    return launch_gemm_f32_planes(g, stream);
  }

  int norm(const void* x, const void* residual, const void* gamma, const void* beta, void* out, int rows, float eps,
           const void* row_mask = nullptr, void* out2 = nullptr, void* planes = nullptr) {
    ++p.launches;
    return launch_add_layernorm(x, residual, gamma, beta, out, rows, p.hidden, eps, p.dtype, row_mask, p.mask_elem_size, out2,
                                out2 ? p.pack_rows : nullptr, planes, stream);
  }

  int attention(const DflEncoderLayer& y, void* const* qkv, void* out, int layer) {
    if (p.attention_events && cudaEventRecord((cudaEvent_t)p.attention_events[2 * layer], stream) != cudaSuccess)
      return fail(DFL_ERR_LAUNCH, "recording a timing event");
    int rc = DFL_OK;
    if (!two_call(p)) {
      DflAttnRelParams a{};
      a.q = qkv[0]; a.k = qkv[1]; a.v = qkv[2];
      a.rel_key = y.rel_key; a.rel_query = y.rel_query; a.mask = p.mask; a.out = out; a.status = p.status;
      a.batch = p.batch; a.heads = p.heads; a.seq_len = p.seq_len; a.head_dim = p.head_dim;
      a.mask_elem_size = p.mask_elem_size; a.scale = p.scale; a.dtype = p.dtype; a.algo = DFL_ALGO_AUTO;
      if (p.packed_rows > 0) {
        a.out_row_base = p.row_base;
        a.out_row_count = p.row_count;
      }
      ++p.launches;
      rc = launch_attention_rel(a, stream, true);   // the projection ran between the tables and this launch
    } else {
      DflAttnParams a{};
      const int ld = (p.n_active + 7) / 8 * 8;
      const bool in_kernel = (y.pos_key || y.pos_query) && scores_in_kernel(p);
      if (in_kernel) {
      } else if ((y.pos_key || y.pos_query) && p.dtype == DFL_F32) {
        if (y.pos_key) {
          a.c2p = at(w.scores[0]);
          if (int rc2 = scores_f32(qkv[0], y.pos_key, at(w.scores[0]), ld)) return rc2;
        }
        if (y.pos_query) {
          a.p2c = at(w.scores[1]);
          if (int rc2 = scores_f32(qkv[1], y.pos_query, at(w.scores[1]), ld)) return rc2;
        }
        a.ld_slots = ld;
      } else if (y.pos_key || y.pos_query) {
        DflPosScoreParams s{};
        s.q = y.pos_key ? qkv[0] : nullptr; s.k = y.pos_query ? qkv[1] : nullptr;
        s.pos_key = y.pos_key; s.pos_query = y.pos_query;
        s.c2p = y.pos_key ? at(w.scores[0]) : nullptr; s.p2c = y.pos_query ? at(w.scores[1]) : nullptr;
        s.batch = p.batch; s.heads = p.heads; s.seq_len = p.seq_len; s.head_dim = p.head_dim;
        s.n_active = p.n_active; s.ld_slots = ld; s.dtype = p.dtype; s.algo = DFL_ALGO_AUTO; s.status = p.status;
        p.launches += (s.c2p ? 1 : 0) + (s.p2c ? 1 : 0);
        rc = dfl_pos_scores(&s, stream);
        if (rc != DFL_OK) return rc;
        a.c2p = s.c2p; a.p2c = s.p2c; a.ld_slots = ld;
      }
      a.q = qkv[0]; a.k = qkv[1]; a.v = qkv[2]; a.lut = p.lut; a.mask = p.mask; a.out = out; a.status = p.status;
      a.batch = p.batch; a.heads = p.heads; a.seq_len = p.seq_len; a.head_dim = p.head_dim;
      a.mask_elem_size = p.mask_elem_size; a.scale = p.scale; a.dtype = p.dtype; a.algo = DFL_ALGO_AUTO;
      ++p.launches;
      const int out_planes = p.attention_only ? 0 : 1;
      rc = in_kernel ? launch_attention_f32_rel(a, y.pos_key, y.pos_query, p.n_active, out_planes, stream)
                     : (p.dtype == DFL_F32 ? launch_attention_f32_planes(a, out_planes, stream) : dfl_attention_fwd(&a, stream));
    }
    if (rc == DFL_OK && p.attention_events && cudaEventRecord((cudaEvent_t)p.attention_events[2 * layer + 1], stream) != cudaSuccess)
      return fail(DFL_ERR_LAUNCH, "recording a timing event");
    return rc;
  }

  // keep * LayerNorm(state + act(keep * conv1d(x))) -> out
  int convolution(const void* state, void* out) {
    GemmDesc g{};
    g.x = p.x; g.w = p.conv_w_module ? at(w.conv_w) : p.conv_w; g.bias = p.conv_b; g.out[0] = at(w.inner);
    g.M = p.seq_len; g.N = p.hidden; g.K = p.hidden;
    g.batch = p.batch; g.stride_x = g.stride_c = (long long)p.seq_len * p.hidden; g.w_mod = 1; g.ldc = p.hidden;
    g.heads = 1; g.head_dim = p.hidden; g.rows_per_seq = p.seq_len;
    g.dtype = p.dtype; g.status = p.status; g.activation = p.conv_activation;
    g.taps = p.conv_taps; g.row_mask = p.mask; g.row_mask_elem = p.mask_elem_size;
    g.weights_early = 1;
    ++p.launches;
    if (int rc = launch_gemm_tc(g, stream)) return rc;
    return norm(at(w.inner), state, p.conv_norm_w, p.conv_norm_b, out, p.batch * p.seq_len, p.conv_norm_eps, p.mask);
  }

  int run() {
    const bool packed = p.packed_rows > 0;
    const int rows = packed ? p.packed_rows : p.batch * p.seq_len, width = p.heads * p.head_dim;
    // Q, K, V of packed rows: projected from the packed rows where groups of 32 of them have a place in the head-major
    // buffers, from the unpacked state (which every layer then writes as well) otherwise
    const bool grouped = packed && p.row_groups;
    const int qkv_rows = grouped ? rows : p.batch * p.seq_len;
    void* qkv[3];
    for (int i = 0; i < 3; ++i)
      qkv[i] = grouped ? p.qkv[i] : at(w.qkv + (size_t)i * padded((size_t)qkv_rows * width * (p.dtype == DFL_F32 ? kPlaneBytes : dtype_size(p.dtype))));
    if (p.plane_sources) {
      ++p.launches;
      if (int rc = launch_refresh_planes(p.plane_sources, p.n_plane_sources, p.n_plane_pieces, stream)) return rc;
    }
    const void* state = p.x;
    const bool f32 = p.dtype == DFL_F32;
    void* unpacked = p.outs[p.n_layers - 1];
    if (packed) {
      ++p.launches;
      if (int rc = launch_copy_rows(p.x, at(w.state[1]), p.pack_rows, rows, p.hidden * (int)dtype_size(p.dtype), stream)) return rc;
      state = at(w.state[1]);
    }
    if (f32)
      if (int rc = split(state, at(w.state_planes), (size_t)rows * p.hidden)) return rc;
    if (p.attention_only) {
      const DflEncoderLayer& y = p.layers[0];
      if (int rc = gemm(f32 ? at(w.state_planes) : state, y.qkv_w, y.qkv_b, nullptr, rows, 3 * width, p.hidden, DFL_ACT_NONE, qkv, true)) return rc;
      return attention(y, qkv, p.outs[0], 0);
    }
    for (int l = 0; l < p.n_layers; ++l) {
      const DflEncoderLayer& y = p.layers[l];
      const bool last = l == p.n_layers - 1, convolve = l == 0 && p.conv_w;
      void* next = !packed && p.outs[l] ? p.outs[l] : at(w.state[l & 1]);
      const void* input = f32 ? at(w.state_planes) : (packed && !grouped ? (l == 0 ? p.x : unpacked) : state);
      if (int rc = gemm(input, y.qkv_w, y.qkv_b, nullptr, qkv_rows, 3 * width, p.hidden, DFL_ACT_NONE, qkv, true)) return rc;
      if (convolve && p.conv_w_module) {   // after the projection: the previous forward has finished by then
        ++p.launches;
        if (int rc = launch_conv_weight(p.conv_w, at(w.conv_w), p.hidden, p.hidden, p.conv_taps, stream)) return rc;
      }
      if (int rc = attention(y, qkv, at(w.context), l)) return rc;
      if (int rc = gemm(at(w.context), y.attn_out_w, y.attn_out_b, at(w.dense), rows, p.hidden, width, DFL_ACT_NONE)) return rc;
      if (int rc = norm(at(w.dense), state, y.attn_norm_w, y.attn_norm_b, at(w.mixed), rows, y.attn_norm_eps, nullptr, nullptr,
                        f32 ? at(w.mixed_planes) : nullptr)) return rc;
      void* inner = f32 ? at(w.inner_planes) : at(w.inner);
      if (int rc = gemm(f32 ? at(w.mixed_planes) : at(w.mixed), y.ffn_in_w, y.ffn_in_b, inner, rows, p.ffn, p.hidden, DFL_ACT_GELU, nullptr, true)) return rc;
      if (int rc = gemm(inner, y.ffn_out_w, y.ffn_out_b, at(w.dense), rows, p.hidden, p.ffn, DFL_ACT_NONE)) return rc;
      // a packed state is also written out at its unpacked rows where the convolution, the next projection or the caller
      // reads it
      if (int rc = norm(at(w.dense), at(w.mixed), y.ffn_norm_w, y.ffn_norm_b, next, rows, y.ffn_norm_eps, nullptr,
                        packed && (last || convolve || !grouped) ? unpacked : nullptr, f32 && !last ? at(w.state_planes) : nullptr)) return rc;
      if (convolve) {
        if (int rc = convolution(packed ? unpacked : next, packed ? unpacked : next)) return rc;
        if (packed && !last) {
          ++p.launches;
          if (int rc = launch_copy_rows(unpacked, next, p.pack_rows, rows, p.hidden * (int)dtype_size(p.dtype), stream)) return rc;
        }
      }
      state = next;
    }
    return DFL_OK;
  }
};

}  // namespace
}  // namespace dfl

using namespace dfl;

extern "C" {

size_t dfl_encoder_workspace_bytes(const DflEncoderParams* p) {
  if (!p || !p->layers || p->n_layers < 1 || p->batch < 1 || p->seq_len < 1) return 0;
  return plan_workspace(*p).total;
}

int dfl_encoder_fwd(DflEncoderParams* p, void* stream) {
  if (!p) return fail(DFL_ERR_BAD_ARG, "null params");
  p->launches = 0;
  if (int rc = validate(*p)) return rc;
  Loop loop{*p, (cudaStream_t)stream, plan_workspace(*p), static_cast<unsigned char*>(p->workspace)};
  if (p->workspace_bytes < loop.w.total)
    return fail(DFL_ERR_BAD_ARG, "workspace of %zu bytes, %zu needed", p->workspace_bytes, loop.w.total);
  return loop.run();
}

}  // extern "C"
