"""More (sequence, head) pairs than a grid's second dimension holds: the relative-table form has no such limit, alone and in
the native layer loop (short sequences: one CTA per pair; longer ones: items of a persistent kernel)."""

import pytest
import torch

import hf_modules
import disentangled_flash_b200 as df

pytestmark = pytest.mark.gpu
dev = "cuda"


@pytest.mark.parametrize("length", (8, 130))
def test_more_than_65535_sequences_times_heads(length):
    heads, batch = 32, 2050   # 65600 pairs
    cfg = df.DebertaAttentionConfig(hidden_size=32, num_attention_heads=heads, attention_head_size=32, num_hidden_layers=1,
                                    intermediate_size=64, max_position_embeddings=512, position_buckets=64,
                                    norm_rel_ebd="layer_norm", conv_kernel_size=0)
    backbone = hf_modules.Backbone(cfg, vocab_size=8).eval()
    backbone.encoder.layer[0].attention.output.dense = torch.nn.Linear(heads * 32, 32)
    hf_modules.initialize_parameters(backbone, 5, std=0.05)
    df.optimize_deberta(backbone.to(dev, torch.float16), sequence_lengths=[length])
    encoder = backbone.encoder
    hidden = torch.randn(batch, length, 32, generator=torch.Generator().manual_seed(2)).half().to(dev)
    mask = torch.ones(batch, length, dtype=torch.bool, device=dev)
    mask[::3, length // 2:] = False
    module = encoder.layer[0].attention.self
    with torch.inference_mode():
        whole = encoder(hidden, mask).last_hidden_state
        halves = torch.cat([encoder(h, m).last_hidden_state for h, m in zip(hidden.split(batch // 2), mask.split(batch // 2))])
        context = module.forward_prepared(hidden, mask, module.prepare_shape(length))[0]
    encoder.check_device_status()
    assert context.shape == (batch, length, heads * 32) and torch.isfinite(context).all()
    # the same sums, perhaps split otherwise: a rounding step or two of fp16 around values of a few units
    assert (whole.float() - halves.float()).abs().max() < 2e-2
