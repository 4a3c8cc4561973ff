"""The FP32 forward on the tensor cores (bf16 planes, ``linear_f32.cu``) at ragged sizes: as close to an fp64 evaluation of
the same encoder as the IEEE-fp32 kernels are, and the split exact over the range of fp32."""

import pytest
import torch

pytestmark = pytest.mark.gpu
dev = "cuda"


def test_planes_sum_to_the_value_exactly():
    from disentangled_flash_b200 import _cabi as c

    gen = torch.Generator().manual_seed(3)
    x = torch.randn(4096, generator=gen) * torch.exp2(torch.randint(-90, 120, (4096,), generator=gen).float())
    x[:8] = torch.tensor([0.0, -0.0, 1.0, torch.finfo(torch.float32).max, -torch.finfo(torch.float32).max, 1 + 2.0 ** -23,
                          3.3895e38, 2.0 ** -100])
    planes = c.split_planes(x.to(dev)).cpu().double()
    assert torch.equal(planes.sum(0), x.double())


@pytest.mark.parametrize("hidden,heads,d,ffn,batch,length,conv", (
    (256, 8, 32, 512, 3, 17, 0), (264, 3, 32, 1000, 1, 1, 0), (768, 12, 64, 3072, 2, 130, 3), (1024, 8, 128, 1032, 1, 257, 0),
    (768, 12, 64, 3072, 9, 100, 0),
))
def test_encoder_is_as_accurate_as_the_fp32_kernels(hidden, heads, d, ffn, batch, length, conv):
    import hf_modules
    import disentangled_flash_b200 as df
    from oracle.encoder import oracle_encoder_forward

    torch.backends.cudnn.allow_tf32, allowed = False, torch.backends.cudnn.allow_tf32
    try:
        cfg = df.DebertaAttentionConfig(hidden_size=hidden, num_attention_heads=heads, attention_head_size=d, num_hidden_layers=2,
                                        intermediate_size=ffn, max_position_embeddings=512, position_buckets=64,
                                        norm_rel_ebd="layer_norm", conv_kernel_size=conv)
        reference, backbone = (hf_modules.Backbone(cfg, vocab_size=8).eval() for _ in range(2))
        for model in (reference, backbone):   # the harness ties the output block's width to hidden: give it the heads' width
            for layer in model.encoder.layer:
                layer.attention.output.dense = torch.nn.Linear(heads * d, hidden)
        hf_modules.initialize_parameters(reference, 12, std=0.05)
        backbone.load_state_dict(reference.state_dict())
        gen = torch.Generator().manual_seed(4)
        x = torch.randn(batch, length, hidden, generator=gen)
        mask = torch.arange(length)[None, :] < torch.randint(1, length + 1, (batch, 1), generator=gen)
        want = oracle_encoder_forward(reference.double(), cfg, x.double(), mask)
        df.optimize_deberta(backbone.to(dev), sequence_lengths=[length])
        encoder = backbone.encoder
        assert length in encoder._layer_loops
        with torch.inference_mode():
            got = encoder(x.to(dev), mask.to(dev)).last_hidden_state
            states = encoder(x.to(dev), mask.to(dev)).hidden_states
            encoder._layer_loops = {}
            for layer in encoder.layer:
                layer.attention.self._algo = 1   # the CUDA-core kernels
            plain = encoder(x.to(dev), mask.to(dev)).last_hidden_state
        encoder.check_device_status()
    finally:
        torch.backends.cudnn.allow_tf32 = allowed
    assert want.dtype == torch.float64 and len(states) == 3 and torch.equal(states[-1], got)
    error = (got.double().cpu() - want).norm() / want.norm()
    plain_error = (plain.double().cpu() - want).norm() / want.norm()
    assert error <= 1.25 * plain_error + 1e-7, (error.item(), plain_error.item())
