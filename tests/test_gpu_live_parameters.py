"""A prepared encoder reads the blocks around the attention as they are at the call: modules exchanged and parameters changed
after the preparation give what the encoder's Python loop, which calls them live, gives."""

import pytest
import torch
from torch import nn

import hf_modules
import disentangled_flash_b200 as df

pytestmark = pytest.mark.gpu
dev = "cuda"


def prepared(dtype, length, conv=0, batch=2, inference=False):
    cfg = df.DebertaAttentionConfig(hidden_size=256, num_attention_heads=4, attention_head_size=64, num_hidden_layers=2,
                                    intermediate_size=512, max_position_embeddings=512, position_buckets=64,
                                    norm_rel_ebd="layer_norm", conv_kernel_size=conv)
    gen = torch.Generator().manual_seed(3)
    with torch.inference_mode(inference):
        backbone = hf_modules.Backbone(cfg, vocab_size=8).eval()
        hf_modules.initialize_parameters(backbone, 5, std=0.05)
        backbone.to(dev, dtype)
        df.optimize_deberta(backbone, sequence_lengths=[length])
    hidden = torch.randn(batch, length, 256, generator=gen).to(dtype).to(dev)
    mask = (torch.arange(length)[None, :] < torch.tensor([length] * (batch - 1) + [max(1, length // 2)])[:, None]).to(dev)
    assert length in backbone.encoder._layer_loops
    return backbone.encoder, hidden, mask


def both(encoder, hidden, mask):
    """What the encoder gives, and what its Python loop gives."""

    with torch.inference_mode():
        got = encoder(hidden, mask).last_hidden_state.float().cpu()
        loops, encoder._layer_loops = encoder._layer_loops, {}
        want = encoder(hidden, mask).last_hidden_state.float().cpu()
        encoder._layer_loops = loops
    return got, want


def assert_follows(encoder, hidden, mask, before, dtype):
    got, want = both(encoder, hidden, mask)
    scale = want.norm()
    # two layers, a few roundings of the state apart (FP32: of the sums)
    assert (got - want).norm() / scale < {torch.float32: 1e-5, torch.float16: 4e-3, torch.bfloat16: 3e-2}[dtype]
    assert (got - before).norm() / scale > 0.1   # the change matters


@pytest.mark.parametrize("dtype", (torch.float16, torch.float32))
def test_exchanged_modules_are_used(dtype):
    encoder, hidden, mask = prepared(dtype, 64)
    before, _ = both(encoder, hidden, mask)
    torch.manual_seed(1)
    encoder.layer[1].output.dense = nn.Linear(512, 256).to(dev, dtype)
    assert_follows(encoder, hidden, mask, before, dtype)
