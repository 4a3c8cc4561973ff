"""When the native layer loop may serve a call, and what it checks on the way: everything that needs no GPU.  The loops are
built over CPU modules whose prepared buffers are made by hand, and the native call is replaced by a recorder."""

import pytest
import torch
from torch import nn

import hf_modules
import disentangled_flash_b200 as df
from disentangled_flash_b200 import _cabi
from disentangled_flash_b200.layer_loop import LayerLoop


@pytest.mark.parametrize("wrong", (lambda x: x[:, :-1], lambda x: x.half(), lambda x: x.to("meta"), lambda x: x[..., :8]))
def test_a_convolution_branch_that_changes_the_state_is_refused(monkeypatch, wrong):
    loop = LayerLoop()
    loop.dtype, loop.device, loop.n_layers = torch.float32, torch.device("cpu"), 2
    runs = []
    monkeypatch.setattr(loop, "_run", lambda hidden, *a: runs.append(a[-2:]) or hidden)
    hidden, mask = torch.zeros(2, 4, 16), torch.ones(2, 4, dtype=torch.bool)
    with pytest.raises(ValueError, match="convolution branch"):
        loop.run(hidden, mask, None, None, wrong)
    assert runs == [(0, 1)]
    loop.run(hidden, mask, None, None, lambda state: state)
    assert runs[1:] == [(0, 1), (1, 2)]


def test_the_convolution_module_gets_the_mask_as_the_caller_gave_it(monkeypatch):
    """Hugging Face's ConvLayer computes ``1 - input_mask``, which a boolean mask does not allow."""

    cfg = df.DebertaAttentionConfig(hidden_size=64, num_attention_heads=2, attention_head_size=32, num_hidden_layers=1,
                                    intermediate_size=128, max_position_embeddings=64, position_buckets=32, conv_kernel_size=3)
    encoder = df.DebertaV2InferenceEncoder(hf_modules.Encoder(cfg), cfg).eval()
    loop, seen = LayerLoop(), []
    loop.dtype, loop.device, loop.f32, loop.n_layers = torch.float32, torch.device("cpu"), True, 1
    monkeypatch.setattr(loop, "_run", lambda hidden, mask, *a: seen.append(mask) or hidden)
    monkeypatch.setattr(encoder, "_layer_loop", lambda *a: loop)
    monkeypatch.setattr(encoder.conv, "forward", lambda x, state, mask: seen.append(mask) or state)
    mask = torch.ones(2, 4)
    with torch.no_grad():
        encoder.forward_prepared(torch.zeros(2, 4, 64), mask, ())
    assert seen[0].dtype == torch.bool and seen[1] is mask
