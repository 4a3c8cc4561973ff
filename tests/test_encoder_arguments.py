"""Arguments of ``dfl_encoder_fwd`` that its kernels could not use are refused on the host, before anything is launched."""

import ctypes

import pytest
import torch

from disentangled_flash_b200 import _cabi


def _params(dtype, head_dim):
    """One attention layer over addresses that nothing reads: the call is refused before its first launch."""
    layers, outs = (_cabi.DflEncoderLayer * 1)(), (ctypes.c_void_p * 1)(1 << 20)
    layers[0].qkv_w = layers[0].pos_key = layers[0].pos_query = 1 << 20
    p = _cabi.DflEncoderParams()
    p.layers, p.outs, p.n_layers, p.attention_only = layers, outs, 1, 1
    p.x = p.mask = p.workspace = p.lut = 1 << 20
    p.batch, p.seq_len, p.heads, p.head_dim, p.hidden = 1, 64, 2, head_dim, 2 * head_dim
    p.mask_elem_size, p.scale, p.dtype, p.n_active = 1, 0.1, dtype, 127
    p.held = layers, outs
    return p


@pytest.mark.skipif(torch.cuda.is_available(), reason="a host check, over addresses that are none of a GPU's")
@pytest.mark.parametrize("dtype", (_cabi.DFL_F32, _cabi.DFL_F16))
@pytest.mark.parametrize("head_dim", (32, 64, 128))
@pytest.mark.parametrize("terms", ("both", "pos_key", "pos_query"))
@pytest.mark.parametrize("field,value", (("n_active", 0), ("n_active", -3), ("lut", None)))
def test_position_tables_need_slots(dtype, head_dim, terms, field, value):
    lib = _cabi.load_library()
    p = _params(dtype, head_dim)
    for name in ("pos_key", "pos_query"):
        if terms not in ("both", name):
            setattr(p.layers[0], name, None)
    p.workspace_bytes = lib.dfl_encoder_workspace_bytes(ctypes.byref(p)) + (1 << 20)
    setattr(p, field, value)
    assert lib.dfl_encoder_fwd(ctypes.byref(p), None) == _cabi.DFL_ERR_BAD_ARG
    assert b"LUT" in lib.dfl_last_error() and p.launches == 0
