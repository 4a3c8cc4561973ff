"""FP32 attention keeps probabilities below 2^-126, at which FP32's normal numbers end, at every head dim."""

import math

import pytest
import torch

import disentangled_flash_b200 as df

pytestmark = pytest.mark.gpu
dev = "cuda"


@pytest.mark.parametrize("head_dim", (32, 64, 128))
@pytest.mark.parametrize("length", (64, 300))
@pytest.mark.parametrize("exponent", (-120, -127, -129, -131))
def test_a_probability_of_a_power_of_two(head_dim, length, exponent):
    heads, width, big = 256 // head_dim, 256, 120
    cfg = df.DebertaAttentionConfig(hidden_size=width, num_attention_heads=heads, attention_head_size=head_dim,
                                    max_position_embeddings=512, position_buckets=64, norm_rel_ebd="none")
    module = df.DisentangledFlashAttention(cfg).to(dev).eval()
    with torch.no_grad():
        for p in module.parameters():
            p.zero_()
        module.query_proj.bias[::head_dim] = 1.0          # q = (1, 0, ...), and the query projection of every position too
        module.key_proj.weight[::head_dim, 0] = 1.0       # k = (x[0], 0, ...)
        module.value_proj.weight[:, 1] = 1.0              # v = x[1] in every column
    hidden = torch.zeros(1, length, width)
    hidden[0, :, 0] = -1e6                                # no weight at all
    hidden[0, 0, 0] = 0.0                                 # the row's maximum, of value 0
    hidden[0, length - 1, 0] = exponent * math.log(2.0) * math.sqrt(3 * head_dim) / 2.0   # S and P2C are each k[0]
    hidden[0, length - 1, 1] = 2.0 ** big
    mask = torch.ones(1, length, dtype=torch.bool)
    rel = torch.zeros(128, width)
    with torch.no_grad():
        got, _ = module(hidden.to(dev), mask.to(dev), rel_embeddings=rel.to(dev))
        module.check_device_status()
    want = 2.0 ** (exponent + big)
    # the probability goes to the tensor core as three BF16 numbers, whose last step is 2^-133; the exponent (of at most 131) is off
    # by three FP32 roundings of 2^-24 each and as many of the projection and the score
    bound = want * 6 * 131 * 2.0 ** -24 + 2.0 ** (big - 134)
    assert (got.double() - want).abs().max() <= bound, (got.min().item(), got.max().item(), want)
