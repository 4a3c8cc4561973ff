"""FP32 attention at head dim 32 and lengths at which head dim 64 already reads its position scores from memory: one kernel computes
them there too, against the CUDA-core kernels."""

import pytest
import torch

pytestmark = pytest.mark.gpu
dev = "cuda"


@pytest.mark.parametrize("length", (3409, 3600, 8192))
def test_against_the_cuda_core_kernels(length):
    import disentangled_flash_b200 as df

    heads, d, buckets = 8, 32, 256
    cfg = df.DebertaAttentionConfig(hidden_size=heads * d, num_attention_heads=heads, attention_head_size=d,
                                    max_position_embeddings=512, position_buckets=buckets, norm_rel_ebd="none")
    module = df.DisentangledFlashAttention(cfg).eval()
    gen = torch.Generator().manual_seed(length)
    with torch.no_grad():
        for p in module.parameters():
            p.copy_(torch.empty(p.shape).normal_(0.0, 0.06, generator=gen))
    rel, hidden = torch.randn(2 * buckets, heads * d, generator=gen), torch.randn(1, length, heads * d, generator=gen)
    mask = (torch.arange(length)[None, :] < length - 70).to(dev)
    module = module.to(dev)
    with torch.no_grad():
        got, _ = module(hidden.to(dev), mask, rel_embeddings=rel.to(dev))
        module.check_device_status()
        module._algo = 1                     # the CUDA-core kernels
        module.clear_inference_cache()
        plain, _ = module(hidden.to(dev), mask, rel_embeddings=rel.to(dev))
    # both within some 4e-7 of fp64 in this norm at up to 600 positions; sums of `length` products of the same fp32 accumulation
    # grow no faster than its square root: 4e-7 * sqrt(8192 / 600) * 2 = 3e-6
    assert (got.double() - plain.double()).norm() <= 3e-6 * plain.double().norm()
    assert (got - plain).abs().max() <= 2e-5 * plain.abs().max().clamp(min=1.0)
