"""Infinities and NaN through the FP32 tensor-core path: the same elements come out infinite (and of which sign) or NaN as
from IEEE arithmetic, and the others are untouched."""

import pytest
import torch

import disentangled_flash_b200 as df
from disentangled_flash_b200 import _cabi as c

pytestmark = pytest.mark.gpu
dev = "cuda"
inf, nan = float("inf"), float("nan")


def pattern(x):
    return torch.where(x.isnan(), 3.0, torch.where(x.isinf(), x.sign() * 2, 0.0))


# one and two k-blocks and many (a split inner product), rows below and beyond a CTA's and a pair's tile
@pytest.mark.parametrize("m,k,heads", ((1, 256, 1), (33, 264, 3), (130, 768, 12), (700, 3072, 4), (4096, 512, 24)))
def test_projection_of_nonfinite_operands(m, k, heads):
    gen = torch.Generator().manual_seed(m)
    x, w = torch.randn(m, k, generator=gen), torch.randn(heads * 32, k, generator=gen)
    x[0, 3], x[m // 2, k - 1], x[m - 1, 65] = inf, -inf, inf
    w[5, 3], w[7, k - 1], w[9, 0], w[11, 65] = -inf, inf, inf, 0.0     # infinity by infinity, and by zero
    if m > 30:
        x[20, 9], x[21, 3], x[21, 4] = nan, inf, -inf                  # a row whose infinities are of both signs
    w[13, 2] = nan
    want = x.double() @ w.double().t()
    got = c.linear_heads_planes(x.to(dev), w.to(dev), None, heads=heads, head_dim=32)
    got = got.permute(1, 0, 2).reshape(m, heads * 32).double().cpu()
    assert torch.equal(pattern(got), pattern(want))
    finite = want.isfinite()
    assert want.isinf().any() and (got - want)[finite].norm() <= 1e-6 * want[finite].norm()


@pytest.mark.parametrize("head_dim,length", ((32, 40), (64, 300), (128, 70)))
def test_attention_with_nonfinite_values_matches_the_fp32_kernels(head_dim, length):
    heads = 256 // head_dim
    cfg = df.DebertaAttentionConfig(hidden_size=256, num_attention_heads=heads, attention_head_size=head_dim,
                                    max_position_embeddings=512, position_buckets=64, norm_rel_ebd="none")
    gen = torch.Generator().manual_seed(1)
    module = df.DisentangledFlashAttention(cfg).to(dev).eval()
    rel = torch.randn(128, 256, generator=gen).to(dev)
    with torch.no_grad():
        for p in module.parameters():
            p.copy_(torch.randn(p.shape, generator=gen) * 0.05)
        module.value_proj.bias[3], module.value_proj.bias[70] = inf, -inf   # every key: an infinite sum
        module.value_proj.bias[130] = nan
        module.prepare_for_inference(rel)
        plan = module.prepare_shape(length)
        hidden = torch.randn(2, length, 256, generator=gen).to(dev)
        mask = torch.ones(2, length, dtype=torch.bool, device=dev)
        got = module.forward_prepared(hidden, mask, plan)[0].cpu().double()
        module._algo = c.ALGO_SIMT
        want = module.forward_prepared(hidden, mask, plan)[0].cpu().double()
    assert torch.equal(pattern(got), pattern(want)) and want.isinf().any()
    finite = want.isfinite()
    assert (got - want)[finite].norm() <= 1e-5 * want[finite].norm()
