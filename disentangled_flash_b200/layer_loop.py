"""The prepared layer loop of one bucket as a single native call (``dfl_encoder_fwd``).

Built by ``DebertaV2InferenceEncoder.prepare_for_inference`` for a bucket whose layers all have the Hugging Face shape;
the encoder's Python loop serves everything else.  A convolution branch stays the caller's module in FP32.

The native call reads the modules' parameters by address.  Before each call the state the addresses were taken from is
compared with the present one: the modules, where and in which form their parameters lie, and the settings that went into
the call.  Whatever was exchanged, moved or changed after the preparation, the call then takes the Python loop, which
reads the modules as they are.
"""

from __future__ import annotations

import ctypes
from collections.abc import Callable
from operator import itemgetter
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
_PLANE_FIELDS = ("attn_out_w", "ffn_in_w", "ffn_out_w")   # weight matrices given as planes in FP32, which follow them
_data_ptr, _dtype = torch.Tensor.data_ptr, torch.Tensor.dtype.__get__
_shape, _stride = torch.Tensor.shape.__get__, torch.Tensor.stride


def _module_at(root: nn.Module, path: str) -> nn.Module:
    for name in path.split("."):
        root = getattr(root, name)
    return root


class LayerLoop:
    """One bucket of one encoder.  ``build`` returns None where the loop does not cover the encoder."""

    def __init__(self) -> None:
        self.plans: Any = None
        self.length = 0
        # The state a call is compared with (see covers()).  A dict of sub-modules or of instance attributes belongs to its
        # module, so an exchanged module shows up in the dict of its parent.
        self._children: list[dict] = []   # module._modules of every module on the way to a parameter
        self._owners: list[dict] = []     # (dict, key) of every tensor the loop reads
        self._keys: list[str] = []
        self._matrices: list[int] = []    # which of them have more than one dimension
        self._settings: list[dict] = []   # (instance attributes, name): eps, training, the activation, ...
        self._names: list[str] = []
        self._hooks: list[dict] = []      # forward hooks of modules the native call stands in for

    @staticmethod
    def build(encoder: nn.Module, length: int, plans: Any, conv_covered: bool) -> "LayerLoop | None":
        first = encoder.layer[0].attention.self
        weight = first.query_proj.weight
        dtype, device = weight.dtype, weight.device
        f32 = dtype == torch.float32
        if dtype not in (torch.float16, torch.bfloat16, torch.float32):
            return None
        if not (all(a and b for a, b in encoder._fused_output_blocks) and (f32 or all(encoder._fused_intermediates))):
            return None
        if encoder.conv is not None and not (conv_covered or f32):
            return None
        self = LayerLoop()
        self.plans, self.length, self.device, self.dtype, self.f32 = plans, length, device, dtype, f32
        self.layer, self.conv = encoder.layer, encoder.conv
        hidden, ffn = weight.shape[1], encoder.layer[0].intermediate.dense.weight.shape[0]
        width = first.all_head_size
        if hidden % 8 or ffn % 8 or first.attention_head_size not in (32, 64, 128):
            return None
        if f32 and not _cabi.f32_planes_supported(first.attention_head_size, length):
            return None
        n = len(encoder.layer)
        self.layers = (_cabi.DflEncoderLayer * n)()

        def read(module: nn.Module, key: str) -> torch.Tensor | None:
            for owner in (module._parameters, module._buffers):
                tensor = owner.get(key)
                if tensor is not None:
                    if tensor.dtype != dtype or tensor.device != device or not tensor.is_contiguous():
                        raise _NotCovered
                    if tensor.data_ptr() % 16:   # a slice of a flat buffer, say: the Python loop's GEMMs take it
                        raise _NotCovered
                    self._owners.append(owner)
                    self._keys.append(key)
                    if tensor.dim() > 1:
                        self._matrices.append(len(self._keys) - 1)
                    return tensor
            self._settings += [module._parameters, module._buffers]   # none, and none may appear
            self._names += [key, key]
            return None

        weights: list[torch.Tensor] = []
        shapes = {"attn_out_w": (hidden, width), "ffn_in_w": (ffn, hidden),
                  "ffn_out_w": (hidden, ffn), "attn_norm_w": (hidden,), "ffn_norm_w": (hidden,)}
        try:
            self._walk(encoder.layer)
            for index, layer in enumerate(encoder.layer):
                entry, plan = self.layers[index], plans[index]
                self._walk(layer, layer.attention, layer.attention.output, layer.intermediate, layer.output)
                for _, path, key in _ATTENTION_FIELDS:
                    read(_module_at(layer, path), key)
                module = layer.attention.self
                if module._cached_qkv_weight.shape != (3 * width, hidden) or (f32 and module._cached_qkv_planes is None):
                    return None
                if module.training or module._algo != _cabi.ALGO_AUTO:
                    return None
                self._watch(module, "training", "_algo", "relative_attention", "pos_att_type")
                fill_attention_fields(entry, module, plan)
                if f32:
                    self._owners.append(module._buffers)
                    self._keys.append("_cached_qkv_planes")
                for field, path, key in _LAYER_FIELDS:
                    tensor = read(_module_at(layer, path), key)
                    if field in shapes and (tensor is None or tuple(tensor.shape) != shapes[field]):
                        return None
                    if f32 and field in _PLANE_FIELDS:
                        weights.append(tensor.detach())
                    else:
                        setattr(entry, field, None if tensor is None else tensor.data_ptr())
                entry.attn_norm_eps = float(layer.attention.output.LayerNorm.eps)
                entry.ffn_norm_eps = float(layer.output.LayerNorm.eps)
                self._watch(layer.attention.output.LayerNorm, "eps")
                self._watch(layer.output.LayerNorm, "eps")
                activation = layer.intermediate.intermediate_act_fn
                self._watch(layer.intermediate, "intermediate_act_fn")
                if isinstance(activation, nn.Module):
                    self._watch(activation, "approximate", "act")
                if f32:   # the Python loop calls this block as the module it is
                    self._stand_in_for(layer.intermediate)
                    self._stand_in_for(layer.intermediate.dense, nn.Linear)
                    if isinstance(activation, nn.Module):
                        self._stand_in_for(activation)
                if (module.has_c2p, module.has_p2c, module.pos_att_type) != (first.has_c2p, first.has_p2c, first.pos_att_type):
                    return None
            p = _cabi.DflEncoderParams()
            if f32:
                self._weights = encoder._planes_following(weights)
                for index, planes in enumerate(self._weights.planes):
                    setattr(self.layers[index // 3], _PLANE_FIELDS[index % 3], planes.data_ptr())
                p.plane_sources, p.n_plane_sources = self._weights.sources.data_ptr(), self._weights.n_sources
                p.n_plane_pieces = self._weights.n_pieces
            if encoder.conv is not None and not f32:
                self._walk(encoder.conv)
                norm = encoder.conv.LayerNorm
                bias = read(encoder.conv.conv, "bias")
                gamma, beta = read(norm, "weight"), read(norm, "bias")
                weight = read(encoder.conv.conv, "weight")
                self._conv_weight = encoder._conv_weight   # [taps, out, in], permuted at prepare time
                # a bucket for which the Python loop calls the module, which reads its weight at the call, does so too
                p.conv_w_module = not encoder._conv_fused[length]
                p.conv_w = (weight if p.conv_w_module else self._conv_weight).data_ptr()
                p.conv_b = None if bias is None else bias.data_ptr()
                p.conv_norm_w, p.conv_norm_b = gamma.data_ptr(), None if beta is None else beta.data_ptr()
                p.conv_taps, p.conv_activation = self._conv_weight.shape[0], encoder._conv_activation_code
                p.conv_norm_eps = float(norm.eps)
                self._watch(norm, "eps")
                if not encoder._conv_fused[length]:   # the Python loop calls this branch as the module it is
                    self._watch(encoder.conv, "conv_act")
                    self._stand_in_for(encoder.conv)
                    self._stand_in_for(encoder.conv.conv, nn.Conv1d)
                    self._stand_in_for(norm, nn.LayerNorm)
                    dropout = encoder.conv._modules.get("dropout")
                    if dropout is not None:
                        if dropout.training:
                            return None
                        self._stand_in_for(dropout)
                        self._watch(dropout, "training")
        except _NotCovered:
            return None
        self._pick = itemgetter(*self._matrices)
        state = self._current_state()
        self._state = (*state[:4], list(map(dict.copy, self._children)), *state[5:])
        lut = plans[0].delta_to_local
        p.layers, p.n_layers = self.layers, n
        p.seq_len, p.hidden, p.heads, p.head_dim, p.ffn = length, hidden, first.num_attention_heads, first.attention_head_size, ffn
        p.lut, p.n_active = lut.data_ptr(), plans[0].active_slots.numel()
        p.scale, p.dtype = first._score_scale(), _cabi.dtype_code(dtype)
        self.params, self.n_layers, self.hidden = p, n, hidden
        return self

    def _walk(self, *modules: nn.Module) -> None:
        self._children += [module._modules for module in modules]

    def _watch(self, module: nn.Module, *names: str) -> None:
        self._settings += [module.__dict__] * len(names)
        self._names += names

    def _stand_in_for(self, module: nn.Module, kind: type[nn.Module] | None = None) -> None:
        """The native call does what ``module`` does: not if it (a ``kind``) has a forward of its own, or hooks."""

        if kind is not None and type(module).forward is not kind.forward:
            raise _NotCovered
        self._watch(module, "forward")
        self._hooks += [module._forward_hooks, module._forward_pre_hooks]

    def _current_state(self) -> tuple:
        """What the addresses in the native call depend on, some 30 us for 12 layers: per tensor the address and the type,
        of a matrix also its form (``.data = other`` changes them under the same name)."""

        tensors = list(map(dict.__getitem__, self._owners, self._keys))
        matrices = self._pick(tensors)
        return (list(map(_data_ptr, tensors)), list(map(_dtype, tensors)), list(map(_shape, matrices)), list(map(_stride, matrices)),
                self._children, list(map(dict.get, self._settings, self._names)))

    def covers(self, encoder: nn.Module, plans: Any, hidden: torch.Tensor, mask: torch.Tensor) -> bool:
        """Whether this call can take the native loop (the state it was built from still holds)."""

        if plans is not self.plans or hidden.dtype != self.dtype or hidden.device != self.device or hidden.dim() != 3:
            return False
        if hidden.shape[1] != self.length or hidden.shape[2] != self.hidden or hidden.shape[0] < 1:
            return False
        if mask.shape != hidden.shape[:2] or mask.device != self.device or torch.is_grad_enabled():
            return False
        if encoder.layer is not self.layer or encoder.conv is not self.conv or any(self._hooks):
            return False
        for fused in encoder._fused_output_blocks:
            if not (fused[0] and fused[1]):
                return False
        if not self.f32 and not all(encoder._fused_intermediates):
            return False
        try:
            return self._current_state() == self._state
        except (KeyError, TypeError, AttributeError, RuntimeError):   # a parameter was deleted, or set to or from None
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
            if begin > 0:
                p.plane_sources = None   # done by the call for the first layers
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
