"""The prepared layer loop of one bucket as a single native call (``dfl_encoder_fwd``).

Built by ``DebertaV2InferenceEncoder.prepare_for_inference`` for a bucket whose layers all have the Hugging Face shape;
the encoder's Python loop serves everything else.  In FP32 the weight matrices are held as bf16 planes
(``dfl_split_planes``) for the tensor-core GEMMs, made once per encoder; a weight modified in place after that sends the
calls to the Python loop until the next preparation.  A convolution branch stays the caller's module in FP32.  Holds the pointers of every parameter the loop reads
and compares them with the modules' current ones before each call, so a parameter that was exchanged or moved after the
preparation is never read at its old place.
"""

from __future__ import annotations

import ctypes
from collections.abc import Callable
from typing import Any

import torch
from torch import nn

from . import _cabi
from .attention import fill_attention_fields

_ATTENTION_FIELDS = (("qkv_w", "attention.self", "_cached_qkv_weight"), ("qkv_b", "attention.self", "_cached_qkv_bias"))
_LAYER_FIELDS = (
    ("attn_out_w", "attention.output.dense", "weight"), ("attn_out_b", "attention.output.dense", "bias"),
    ("attn_norm_w", "attention.output.LayerNorm", "weight"), ("attn_norm_b", "attention.output.LayerNorm", "bias"),
    ("ffn_in_w", "intermediate.dense", "weight"), ("ffn_in_b", "intermediate.dense", "bias"),
    ("ffn_out_w", "output.dense", "weight"), ("ffn_out_b", "output.dense", "bias"),
    ("ffn_norm_w", "output.LayerNorm", "weight"), ("ffn_norm_b", "output.LayerNorm", "bias"),
)
_PLANE_FIELDS = ("attn_out_w", "ffn_in_w", "ffn_out_w")   # weight matrices given as planes in FP32
_data_ptr = torch.Tensor.data_ptr


def version_of(tensor: torch.Tensor) -> int:
    """How often ``tensor`` has been modified in place (inference tensors do not count)."""

    return -1 if tensor.is_inference() else tensor._version


def _module_at(root: nn.Module, path: str) -> nn.Module:
    for name in path.split("."):
        root = getattr(root, name)
    return root


class LayerLoop:
    """One bucket of one encoder.  ``build`` returns None where the loop does not cover the encoder."""

    def __init__(self) -> None:
        self.plans: Any = None
        self.length = 0

    @staticmethod
    def build(encoder: nn.Module, length: int, plans: Any, conv_covered: bool) -> "LayerLoop | None":
        first = encoder.layer[0].attention.self
        weight = first.query_proj.weight
        dtype, device = weight.dtype, weight.device
        f32 = dtype == torch.float32
        if device.type != "cuda" or dtype not in (torch.float16, torch.bfloat16, torch.float32):
            return None
        if not (all(a and b for a, b in encoder._fused_output_blocks) and (f32 or all(encoder._fused_intermediates))):
            return None
        if encoder.conv is not None and not (conv_covered or f32):
            return None
        self = LayerLoop()
        self.plans, self.length, self.device, self.dtype, self.f32 = plans, length, device, dtype, f32
        self.attention = [layer.attention.self for layer in encoder.layer]
        hidden, ffn = weight.shape[1], encoder.layer[0].intermediate.dense.weight.shape[0]
        width = first.all_head_size
        if hidden % 8 or ffn % 8 or first.attention_head_size not in (32, 64, 128):
            return None
        if f32 and not _cabi.f32_planes_supported(first.attention_head_size, length):
            return None
        n = len(encoder.layer)
        self.layers = (_cabi.DflEncoderLayer * n)()
        # (owner dict, key) of every tensor the loop reads, and where it was
        self._owners: list[dict] = []
        self._keys: list[str] = []
        self._planes: list[torch.Tensor] = []

        def read(module: nn.Module, key: str) -> torch.Tensor | None:
            for owner in (module._parameters, module._buffers):
                tensor = owner.get(key)
                if tensor is not None:
                    if tensor.dtype != dtype or tensor.device != device or not tensor.is_contiguous():
                        raise _NotCovered
                    self._owners.append(owner)
                    self._keys.append(key)
                    return tensor
            return None

        shapes = {"attn_out_w": (hidden, width), "ffn_in_w": (ffn, hidden),
                  "ffn_out_w": (hidden, ffn), "attn_norm_w": (hidden,), "ffn_norm_w": (hidden,)}
        try:
            for index, layer in enumerate(encoder.layer):
                entry, plan = self.layers[index], plans[index]
                for _, path, key in _ATTENTION_FIELDS:
                    read(_module_at(layer, path), key)
                module = layer.attention.self
                if module._cached_qkv_weight.shape != (3 * width, hidden) or (f32 and module._cached_qkv_planes is None):
                    return None
                fill_attention_fields(entry, module, plan)
                for field, path, key in _LAYER_FIELDS:
                    owner = _module_at(layer, path)
                    tensor = read(owner, key)
                    if field in shapes and (tensor is None or tuple(tensor.shape) != shapes[field]):
                        return None
                    if f32 and field in _PLANE_FIELDS:
                        tensor = encoder._weight_planes_of(tensor)
                        self._planes.append(tensor)
                    setattr(entry, field, None if tensor is None else tensor.data_ptr())
                entry.attn_norm_eps = float(layer.attention.output.LayerNorm.eps)
                entry.ffn_norm_eps = float(layer.output.LayerNorm.eps)
                if (module.has_c2p, module.has_p2c, module.pos_att_type) != (first.has_c2p, first.has_p2c, first.pos_att_type):
                    return None
            p = _cabi.DflEncoderParams()
            if encoder.conv is not None and not f32:
                norm = encoder.conv.LayerNorm
                bias = read(encoder.conv.conv, "bias")
                gamma, beta = read(norm, "weight"), read(norm, "bias")
                read(encoder.conv.conv, "weight")
                self._conv_weight = encoder._conv_weight   # [taps, out, in], permuted at prepare time
                p.conv_w, p.conv_b = self._conv_weight.data_ptr(), None if bias is None else bias.data_ptr()
                p.conv_norm_w, p.conv_norm_b = gamma.data_ptr(), None if beta is None else beta.data_ptr()
                p.conv_taps, p.conv_activation = self._conv_weight.shape[0], encoder._conv_activation_code
                p.conv_norm_eps = float(norm.eps)
        except _NotCovered:
            return None
        self._pointers = self._current_state()
        lut = plans[0].delta_to_local
        p.layers, p.n_layers = self.layers, n
        p.seq_len, p.hidden, p.heads, p.head_dim, p.ffn = length, hidden, first.num_attention_heads, first.attention_head_size, ffn
        p.lut, p.n_active = lut.data_ptr(), plans[0].active_slots.numel()
        p.scale, p.dtype = first._score_scale(), _cabi.dtype_code(dtype)
        self.params, self.n_layers, self.hidden = p, n, hidden
        return self

    def _current_state(self) -> list[int]:
        """Address of every tensor the loop reads; in FP32, where copies of the weights are read, their versions too."""

        tensors = list(map(dict.__getitem__, self._owners, self._keys))
        state = list(map(_data_ptr, tensors))
        return state + list(map(version_of, tensors)) if self.f32 else state

    def covers(self, encoder: nn.Module, plans: Any, hidden: torch.Tensor, mask: torch.Tensor) -> bool:
        """Whether this call can take the native loop (the state it was built from still holds)."""

        if plans is not self.plans or hidden.dtype != self.dtype or hidden.device != self.device or hidden.dim() != 3:
            return False
        if hidden.shape[1] != self.length or hidden.shape[2] != self.hidden or hidden.shape[0] < 1:
            return False
        if mask.shape != hidden.shape[:2] or mask.device != self.device or torch.is_grad_enabled():
            return False
        for fused in encoder._fused_output_blocks:
            if not (fused[0] and fused[1]):
                return False
        if not self.f32 and not all(encoder._fused_intermediates):
            return False
        for module in self.attention:
            if module.training or module._algo != _cabi.ALGO_AUTO:
                return False
        try:
            return self._current_state() == self._pointers
        except (KeyError, TypeError, AttributeError):   # a parameter was deleted or set to None
            return False

    def _call(self, hidden: torch.Tensor, mask: torch.Tensor, outs: Any, status: torch.Tensor | None) -> _cabi.DflEncoderParams:
        if mask.dtype.is_floating_point or mask.element_size() not in (1, 4, 8):
            mask = mask.bool()
        hidden, mask = hidden.contiguous(), mask.contiguous()
        p = _cabi.DflEncoderParams()
        ctypes.pointer(p)[0] = self.params   # a copy: several threads may run one bucket
        p.x, p.mask, p.mask_elem_size, p.batch = hidden.data_ptr(), mask.data_ptr(), mask.element_size(), hidden.shape[0]
        p.status = None if status is None else status.data_ptr()
        p.outs = outs
        p._keep = (hidden, mask)
        return p

    def run(self, hidden: torch.Tensor, mask: torch.Tensor, status: torch.Tensor | None,
            trace: list[torch.Tensor] | None, conv: Callable[[torch.Tensor], torch.Tensor] | None = None) -> torch.Tensor:
        """``conv``: a convolution branch that is not part of the native loop, called with the state after layer 0."""

        if conv is not None:
            first: list[torch.Tensor] = []
            state = conv(self._run(hidden, mask, status, first, 0, 1))
            if state.shape != hidden.shape or state.dtype != self.dtype or state.device != self.device:
                raise ValueError(f"the convolution branch returned {tuple(state.shape)} of {state.dtype} on {state.device}, "
                                 f"the layers take {tuple(hidden.shape)} of {self.dtype} on {self.device}")
            if trace is not None:
                trace.append(state)
            return self._run(state, mask, status, trace, 1, self.n_layers) if self.n_layers > 1 else state
        return self._run(hidden, mask, status, trace, 0, self.n_layers)

    def _run(self, hidden: torch.Tensor, mask: torch.Tensor, status: torch.Tensor | None,
             trace: list[torch.Tensor] | None, begin: int, end: int) -> torch.Tensor:
        n = end - begin
        outs = (ctypes.c_void_p * n)()
        out = torch.empty(hidden.shape, dtype=self.dtype, device=self.device)
        outs[n - 1] = out.data_ptr()
        if trace is not None:
            for layer in range(n - 1):
                state = torch.empty(hidden.shape, dtype=self.dtype, device=self.device)
                outs[layer] = state.data_ptr()
                trace.append(state)
            trace.append(out)
        p = self._call(hidden, mask, outs, status)
        if n != self.n_layers:
            p.n_layers = n
            p.layers = ctypes.cast(ctypes.addressof(self.layers) + begin * ctypes.sizeof(_cabi.DflEncoderLayer),
                                   ctypes.POINTER(_cabi.DflEncoderLayer))
        _cabi.encoder_fwd(p, self.device)
        return out

    def run_packed(self, hidden: torch.Tensor, mask: torch.Tensor, status: torch.Tensor | None, out: torch.Tensor,
                   tables: tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor],
                   qkv: tuple[torch.Tensor, ...] | None) -> None:
        """``tables`` = (pack_rows, row_groups, row_base, row_count); the result goes to the covered rows of ``out``.
        ``qkv``: the head-major buffers of the grouped projection, None where the bucket has no row groups."""

        outs = (ctypes.c_void_p * self.n_layers)()
        outs[self.n_layers - 1] = out.data_ptr()
        p = self._call(hidden, mask, outs, status)
        pack_rows, row_groups, row_base, row_count = tables
        p.packed_rows, p.pack_rows = pack_rows.numel(), pack_rows.data_ptr()
        p.row_base, p.row_count = row_base.data_ptr(), row_count.data_ptr()
        if qkv is not None:
            p.row_groups = row_groups.data_ptr()
            for i in range(3):
                p.qkv[i] = qkv[i].data_ptr()
        _cabi.encoder_fwd(p, self.device)


class _NotCovered(Exception):
    pass


__all__ = ["LayerLoop"]
