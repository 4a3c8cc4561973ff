"""FP32 attention with the position scores computed in the kernel (``attention_f32_rel.cu``): the FP32 module against an fp64
evaluation, next to the CUDA-core kernels' error, at sizes around the 128-row tiles and the 64-row pieces of their windows."""

import pytest
import torch

pytestmark = pytest.mark.gpu
dev = "cuda"


def _module(heads, d, terms, buckets, seed):
    import disentangled_flash_b200 as df

    cfg = df.DebertaAttentionConfig(hidden_size=heads * d, num_attention_heads=heads, attention_head_size=d, pos_att_type=terms,
                                    max_position_embeddings=512, position_buckets=buckets, norm_rel_ebd="none")
    module = df.DisentangledFlashAttention(cfg).eval()
    gen = torch.Generator().manual_seed(seed)
    with torch.no_grad():
        for p in module.parameters():
            p.copy_(torch.empty(p.shape).normal_(0.0, 0.06, generator=gen))
    return module, torch.randn(2 * buckets, heads * d, generator=gen), gen


def _reference(module, hidden, mask, rel, heads, terms, buckets):
    import oracle

    sd = {k: v.detach().double().cpu() for k, v in module.state_dict().items()}
    return oracle.attention_module_forward(
        hidden.double(), mask, wq=sd["query_proj.weight"], wk=sd["key_proj.weight"], wv=sd["value_proj.weight"],
        bq=sd["query_proj.bias"], bk=sd["key_proj.bias"], bv=sd["value_proj.bias"], rel_embeddings=rel.double(), num_heads=heads,
        pos_att_type=terms, position_buckets=buckets, max_relative_positions=512)


@pytest.mark.parametrize("d", (32, 64))
@pytest.mark.parametrize("terms", (("c2p", "p2c"), ("c2p",), ("p2c",)))
@pytest.mark.parametrize("length", (1, 17, 63, 64, 65, 127, 128, 129, 191, 192, 193, 256, 257, 400, 600))
def test_against_fp64(d, terms, length):
    heads, buckets, batch = 256 // d, 48, 2
    module, rel, gen = _module(heads, d, terms, buckets, length + d)
    hidden = torch.randn(batch, length, heads * d, generator=gen)
    mask = torch.arange(length)[None, :] < torch.tensor([[length], [(length + 1) // 2]])
    if length == 193:
        mask[1] = False                      # every query row attends to all keys alike
    if length == 129:
        mask[0, :70] = False                 # the first keys are padding
    want = _reference(module, hidden, mask, rel, heads, terms, buckets)
    module = module.to(dev)
    with torch.no_grad():
        got, _ = module(hidden.to(dev), mask.to(dev), rel_embeddings=rel.to(dev))
        again, _ = module(hidden.to(dev), mask.to(dev), rel_embeddings=rel.to(dev))
        module.check_device_status()
        module._algo = 1                     # the CUDA-core kernels
        module.clear_inference_cache()
        plain, _ = module(hidden.to(dev), mask.to(dev), rel_embeddings=rel.to(dev))
    assert torch.equal(got, again)
    error, plain_error = (got.cpu() - want).norm() / want.norm(), (plain.cpu() - want).norm() / want.norm()
    assert error <= 1.25 * plain_error + 1e-7, (error.item(), plain_error.item())
    # no single element far off: sums of up to 256 fp32 products, then a weighted mean of `length` values
    assert (got.cpu() - want).abs().max() <= 2e-5 * want.abs().max().clamp(min=1.0)


def test_long_sequences_and_the_kernels_that_read_scores_agree():
    """The longest table that fits shared memory (head dim 64), and the next length, which the score GEMMs serve."""
    heads, d, buckets = 4, 64, 256
    outs = []
    for length in (3400, 3600):
        module, rel, gen = _module(heads, d, ("c2p", "p2c"), buckets, 9)
        hidden = torch.randn(1, 3600, heads * d, generator=torch.Generator().manual_seed(1))[:, :length].contiguous()
        mask = torch.arange(length)[None, :] < 3300   # the same keys in both
        module = module.to(dev)
        with torch.no_grad():
            got, _ = module(hidden.to(dev), mask.to(dev), rel_embeddings=rel.to(dev))
            module.check_device_status()
        outs.append(got[:, :3300].double())
    assert (outs[0] - outs[1]).norm() / outs[1].norm() < 1e-6
