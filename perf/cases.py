"""The work that users of this framework have it do, as measurable cases.

A case is one call of a public entry point on one batch:

* ``encoder``: ``optimize_deberta(model, sequence_lengths=...)`` once, then ``model.encoder(hidden, mask)`` per batch.
* ``graph``: the same encoder through ``capture_deberta_buckets`` (one CUDA graph per bucket), the small-batch server.
* ``packed``: ``encoder.forward_packed(hidden, mask, lengths)``, the large padded batch without its padding.
* ``embed``: token ids through ``fuse_deberta_embeddings`` and the encoder, the whole backbone.
* ``attention``: ``DisentangledFlashAttention.forward_prepared``, the operator inside a caller's own layer.

Geometries, dtypes, buckets and padding are the ones of the repository's benchmark and tests: 12 layers of hidden 768
(base), 24 of 1024 (large), 24 of 1536 (xlarge); FP16, BF16 and strict FP32; log-bucket positions with 256 buckets;
valid lengths uniform in [L/2, L]; weights N(0, 0.02).
"""

from __future__ import annotations

import torch
from torch import nn
from torch.nn import functional as F

import disentangled_flash_b200 as dfl

GEOMETRY = {
    "base": dict(layers=12, hidden=768, heads=12, ffn=3072, conv=3),
    "large": dict(layers=24, hidden=1024, heads=16, ffn=4096, conv=0),
    "xlarge": dict(layers=24, hidden=1536, heads=24, ffn=6144, conv=3),
}
DTYPE = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
VOCAB = 128100
BUCKETS = 256


# ------------------------------------------------------------------------------------------------------------ cases
def _encoder(path, model, dtype, batch, length):
    return dict(path=path, model=model, dtype=dtype, batch=batch, length=length)


def _attention(dtype, batch, length, heads, head_dim):
    return dict(path="attention", dtype=dtype, batch=batch, length=length, heads=heads, head_dim=head_dim)


def listed():
    return [
        # one short query at a time: latency, launches and host work
        dict(name="base fp16 1x32", **_encoder("encoder", "base", "fp16", 1, 32)),
        # a server that captured its small bucket
        dict(name="base bf16 4x128 graph", **_encoder("graph", "base", "bf16", 4, 128)),
        # reranking a handful of passages
        dict(name="base fp16 8x128", **_encoder("encoder", "base", "fp16", 8, 128)),
        # documents at their own length, no bucket of the tuned sizes, from token ids
        dict(name="base bf16 7x333 ids", **_encoder("embed", "base", "bf16", 7, 333)),
        # the throughput batch of the benchmark, padded and without its padding
        dict(name="base fp16 32x512", **_encoder("encoder", "base", "fp16", 32, 512)),
        dict(name="base fp16 32x512 packed", **_encoder("packed", "base", "fp16", 32, 512)),
        # the largest models: an interactive batch, and a bulk job on one of eight replicas
        dict(name="xlarge bf16 8x64", **_encoder("encoder", "xlarge", "bf16", 8, 64)),
        dict(name="large bf16 64x256", **_encoder("encoder", "large", "bf16", 64, 256)),
        # numerics-critical users: strict FP32
        dict(name="base fp32 8x128", **_encoder("encoder", "base", "fp32", 8, 128)),
        dict(name="xlarge fp32 8x256", **_encoder("encoder", "xlarge", "fp32", 8, 256)),
        # the operator alone, at the head dims the encoders above do not have
        dict(name="attention fp16 16x256 d32", **_attention("fp16", 16, 256, 24, 32)),
        dict(name="attention bf16 16x512 d128", **_attention("bf16", 16, 512, 8, 128)),
    ]


def _log_uniform(rng, low, high):
    return max(low, min(high, round(low * (high / low) ** rng.random())))


def draw(rng):
    if rng.random() < 0.3:
        dtype = rng.choice(("fp16", "bf16", "fp16", "bf16", "fp32"))
        heads, head_dim = rng.choice(((24, 32), (12, 64), (8, 128)))
        length = _log_uniform(rng, 16, 1024)
        most = max(1, (4096 if dtype == "fp32" else 16384) // length)
        return _attention(dtype, _log_uniform(rng, 1, min(64, most)), length, heads, head_dim)
    path = rng.choice(("encoder", "encoder", "encoder", "graph", "packed", "embed"))
    model = rng.choice(("base", "base", "large", "xlarge"))
    dtype = rng.choice(("fp16", "bf16") if path == "packed" else ("fp16", "bf16", "fp16", "bf16", "fp32"))
    length = _log_uniform(rng, 16, 512)
    tokens = {"base": 16384, "large": 8192, "xlarge": 4096}[model] // (8 if dtype == "fp32" else 1)
    if path == "graph":
        tokens = min(tokens, 2048)   # captured buckets are the small ones
    length = min(length, tokens)
    return _encoder(path, model, dtype, _log_uniform(rng, 1, max(1, min(64, tokens // length))), length)


# ------------------------------------------------------------------------- a backbone with Hugging Face's module tree
class _Config:
    def __init__(self, layers, hidden, heads, ffn, conv, head_dim=None):
        self.num_hidden_layers, self.hidden_size, self.num_attention_heads = layers, hidden, heads
        self.attention_head_size = head_dim or hidden // heads
        self.intermediate_size, self.conv_kernel_size = ffn, conv
        self.layer_norm_eps, self.hidden_dropout_prob, self.attention_probs_dropout_prob = 1e-7, 0.1, 0.1
        self.relative_attention, self.max_relative_positions, self.max_position_embeddings = True, -1, 512
        self.position_buckets, self.share_att_key, self.pos_att_type = BUCKETS, True, ("p2c", "c2p")
        self.hidden_act, self.norm_rel_ebd, self.conv_act, self.conv_groups = "gelu", "layer_norm", "tanh", 1


class _Projections(nn.Module):   # the parameters of attention.self; optimize_deberta exchanges the module
    def __init__(self, c):
        super().__init__()
        width = c.num_attention_heads * c.attention_head_size
        self.query_proj, self.key_proj, self.value_proj = (nn.Linear(c.hidden_size, width) for _ in range(3))


class _Output(nn.Module):
    def __init__(self, c, width):
        super().__init__()
        self.dense = nn.Linear(width, c.hidden_size)
        self.LayerNorm = nn.LayerNorm(c.hidden_size, c.layer_norm_eps)
        self.dropout = nn.Dropout(c.hidden_dropout_prob)

    def forward(self, hidden_states, input_tensor):
        return self.LayerNorm(self.dropout(self.dense(hidden_states)) + input_tensor)


class _Attention(nn.Module):
    def __init__(self, c):
        super().__init__()
        self.self = _Projections(c)
        self.output = _Output(c, c.num_attention_heads * c.attention_head_size)


class _Intermediate(nn.Module):
    def __init__(self, c):
        super().__init__()
        self.dense = nn.Linear(c.hidden_size, c.intermediate_size)
        self.intermediate_act_fn = F.gelu

    def forward(self, hidden_states):
        return self.intermediate_act_fn(self.dense(hidden_states))


class _Layer(nn.Module):
    def __init__(self, c):
        super().__init__()
        self.attention, self.intermediate = _Attention(c), _Intermediate(c)
        self.output = _Output(c, c.intermediate_size)


class _Conv(nn.Module):
    def __init__(self, c):
        super().__init__()
        self.conv_act = c.conv_act
        self.conv = nn.Conv1d(c.hidden_size, c.hidden_size, c.conv_kernel_size, padding=(c.conv_kernel_size - 1) // 2)
        self.LayerNorm = nn.LayerNorm(c.hidden_size, c.layer_norm_eps)
        self.dropout = nn.Dropout(c.hidden_dropout_prob)

    def forward(self, hidden_states, residual_states, input_mask):
        out = self.conv(hidden_states.transpose(1, 2)).transpose(1, 2).contiguous()
        keep = input_mask.bool().unsqueeze(-1)
        out = torch.tanh(self.dropout(out.masked_fill(~keep, 0)))
        normed = self.LayerNorm(residual_states + out)
        return normed * keep.to(normed.dtype)


class _Encoder(nn.Module):
    def __init__(self, c):
        super().__init__()
        self.layer = nn.ModuleList(_Layer(c) for _ in range(c.num_hidden_layers))
        self.relative_attention, self.position_buckets = True, c.position_buckets
        self.max_relative_positions = c.max_position_embeddings
        self.rel_embeddings = nn.Embedding(2 * c.position_buckets, c.hidden_size)
        self.norm_rel_ebd = ["layer_norm"]
        self.LayerNorm = nn.LayerNorm(c.hidden_size, c.layer_norm_eps)
        self.conv = _Conv(c) if c.conv_kernel_size else None


class _Embeddings(nn.Module):
    def __init__(self, c, vocab):
        super().__init__()
        self.word_embeddings = nn.Embedding(vocab, c.hidden_size, padding_idx=0)
        self.LayerNorm = nn.LayerNorm(c.hidden_size, c.layer_norm_eps)
        self.dropout = nn.Dropout(c.hidden_dropout_prob)

    def forward(self, input_ids=None, token_type_ids=None, position_ids=None, mask=None, inputs_embeds=None):
        rows = self.LayerNorm(self.word_embeddings(input_ids))
        return self.dropout(rows if mask is None else rows * mask.unsqueeze(-1).to(rows.dtype))


class _Backbone(nn.Module):
    def __init__(self, c, vocab):
        super().__init__()
        self.config, self.embeddings, self.encoder = c, _Embeddings(c, vocab), _Encoder(c)


def _initialise(module, gen):
    with torch.no_grad():
        for child in module.modules():
            if isinstance(child, (nn.Linear, nn.Conv1d, nn.Embedding)):
                child.weight.normal_(0.0, 0.02, generator=gen)
                if getattr(child, "bias", None) is not None:
                    child.bias.normal_(0.0, 0.02, generator=gen)
            elif isinstance(child, nn.LayerNorm):
                child.weight.normal_(1.0, 0.05, generator=gen)
                child.bias.normal_(0.0, 0.02, generator=gen)


# ------------------------------------------------------------------------------------------------------- measurement
def prepare(case, seed):
    device, dtype = torch.device("cuda", torch.cuda.current_device()), DTYPE[case["dtype"]]
    gen = torch.Generator(device).manual_seed(seed)
    batch, length, path = case["batch"], case["length"], case["path"]
    valid = torch.randint(-(-length // 2), length + 1, (batch,), generator=torch.Generator().manual_seed(seed))
    mask = (torch.arange(length)[None, :] < valid[:, None]).to(device)

    if path == "attention":
        c = _Config(1, case["heads"] * case["head_dim"], case["heads"], 0, 0, case["head_dim"])
        with torch.device(device):
            module = dfl.DisentangledFlashAttention(c)
            relative = torch.randn(2 * BUCKETS, c.hidden_size, generator=gen)
        _initialise(module, gen)
        module.to(dtype).eval().prepare_for_inference(relative.to(dtype))
        hidden = torch.randn(batch, length, c.hidden_size, generator=gen, device=device).to(dtype)
        return dict(path=path, module=module, plan=module.prepare_shape(length), hidden=hidden, mask=mask)

    c = _Config(**GEOMETRY[case["model"]])
    with torch.device(device):
        model = _Backbone(c, VOCAB if path == "embed" else 8).eval()
        _initialise(model, gen)
        model.to(dtype)
        dfl.optimize_deberta(model, sequence_lengths=[length])
    state = dict(path=path, model=model, mask=mask)
    if path == "embed":
        dfl.fuse_deberta_embeddings(model)
        ids = torch.randint(1, VOCAB, (batch, length), generator=gen, device=device)
        # a tokenizer's output: int64 ids and int64 mask
        state.update(ids=ids * mask, mask=mask.to(torch.int64))
        return state
    # what the embedding layer hands over: normalised rows, zero at padded positions
    hidden = F.layer_norm(torch.randn(batch, length, c.hidden_size, generator=gen, device=device), (c.hidden_size,))
    state["hidden"] = (hidden * mask.unsqueeze(-1)).to(dtype)
    if path == "packed":
        state["lengths"] = valid.tolist()
    if path == "graph":
        state["bucket"] = dfl.capture_deberta_buckets(model.encoder, batch)[length]
    return state


@torch.inference_mode()
def run(state):
    path, mask = state["path"], state["mask"]
    if path == "attention":
        return state["module"].forward_prepared(state["hidden"], mask, state["plan"])[0]
    if path == "graph":
        return state["bucket"](state["hidden"], mask)
    encoder = state["model"].encoder
    if path == "packed":
        out = encoder.forward_packed(state["hidden"], mask, state["lengths"]).last_hidden_state
        return out * mask.unsqueeze(-1)   # padded positions are unspecified in this form
    hidden = state["hidden"] if path == "encoder" else state["model"].embeddings(input_ids=state["ids"], mask=mask)
    return encoder(hidden, mask, output_hidden_states=False).last_hidden_state


def work(case):
    batch, length = case["batch"], case["length"]
    size = 4 if case["dtype"] == "fp32" else 2
    tokens = batch * length * (0.75 if case["path"] == "packed" else 1.0)
    slots = min(2 * length - 1, 2 * BUCKETS)

    def core(heads, head_dim):   # QK^T and PV, and the two position-score products over the active slots
        return 4.0 * tokens * heads * head_dim * (length + slots)

    if case["path"] == "attention":
        hidden = case["heads"] * case["head_dim"]
        return {"bytes": size * (2.0 * tokens * hidden + 3 * hidden * hidden + 2 * slots * hidden),
                "flops": 6.0 * tokens * hidden * hidden + core(case["heads"], case["head_dim"])}
    g = GEOMETRY[case["model"]]
    hidden, ffn, layers = g["hidden"], g["ffn"], g["layers"]
    weights = layers * (4 * hidden * hidden + 2 * hidden * ffn) + g["conv"] * hidden * hidden
    flops = 2.0 * tokens * weights + layers * core(g["heads"], hidden // g["heads"])
    tables = layers * 2.0 * slots * hidden
    return {"bytes": size * (weights + tables + 2.0 * tokens * hidden), "flops": flops}


def tolerance(case):
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}
    if case["path"] == "attention":
        return {"rel": 2e-3 if case["dtype"] == "fp16" else 1e-2}
    # every layer rounds its state to 11 (FP16) or 8 (BF16) bits; 12 or 24 layers carry the difference on
    return {"rel": 3e-3 if case["dtype"] == "fp16" else 1.5e-2}
