"""A prepared encoder reads the blocks around the attention as they are at the call: modules exchanged and parameters changed
after the preparation give what the encoder's Python loop, which calls them live, gives."""

import copy

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


def _by_data(w):
    w.data.copy_(torch.randn(w.shape, generator=torch.Generator().manual_seed(9)) * 0.05)


def _in_place(w):
    with torch.no_grad():
        w.mul_(-1.0)


@pytest.mark.parametrize("change", (_in_place, _by_data))
@pytest.mark.parametrize("which", ("attention.output", "intermediate", "output"))
@pytest.mark.parametrize("inference", (False, True))   # inference tensors count no changes
def test_fp32_weights_changed_in_place_are_used(which, change, inference):
    encoder, hidden, mask = prepared(torch.float32, 40, conv=3, inference=inference)
    before, _ = both(encoder, hidden, mask)
    with torch.inference_mode(inference):
        for layer in encoder.layer:
            change(layer.get_submodule(which).dense.weight)
    assert_follows(encoder, hidden, mask, before, torch.float32)


@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("length", (17, 64, 255))
def test_short_convolution_weights_changed_in_place_are_used(dtype, length):
    encoder, hidden, mask = prepared(dtype, length, conv=3)
    before, _ = both(encoder, hidden, mask)
    _by_data(encoder.conv.conv.weight)
    encoder.conv.conv.weight.data.mul_(4)
    assert_follows(encoder, hidden, mask, before, dtype)


@pytest.mark.parametrize("dtype,conv", ((torch.float32, 0), (torch.float16, 3)))
def test_a_captured_graph_reads_the_weights_as_they_are(dtype, conv):
    encoder, hidden, mask = prepared(dtype, 32, conv=conv)
    bucket = df.capture_deberta_buckets(encoder, 2)[32]
    before = bucket(hidden, mask).float().cpu()
    _in_place(encoder.conv.conv.weight if conv else encoder.layer[0].output.dense.weight)
    got = bucket(hidden, mask).float().cpu()
    with torch.inference_mode():
        want = encoder(hidden, mask).last_hidden_state.float().cpu()
    assert torch.equal(got, want) and (got - before).norm() / want.norm() > 0.05


def test_fp32_layers_of_every_width_use_their_own_weights():
    """Matrices of a few hundred to a few million elements, their planes one after the other in one workspace."""

    for hidden_size, heads, ffn, length in ((256, 4, 264, 3), (512, 8, 2048, 130), (1536, 24, 6144, 64)):
        cfg = df.DebertaAttentionConfig(hidden_size=hidden_size, num_attention_heads=heads, attention_head_size=64,
                                        num_hidden_layers=3, intermediate_size=ffn, max_position_embeddings=512,
                                        position_buckets=64, norm_rel_ebd="layer_norm", conv_kernel_size=0)
        backbone = hf_modules.Backbone(cfg, vocab_size=8).eval()
        hf_modules.initialize_parameters(backbone, 5, std=0.03)
        df.optimize_deberta(backbone.to(dev), sequence_lengths=[length])
        hidden = torch.randn(2, length, hidden_size, generator=torch.Generator().manual_seed(2)).to(dev)
        got, want = both(backbone.encoder, hidden, torch.ones(2, length, dtype=torch.bool, device=dev))
        assert (got - want).norm() / want.norm() < 5e-6


@pytest.mark.parametrize("dtype", (torch.float32, torch.float16))
def test_a_copy_of_a_prepared_encoder_has_weights_of_its_own(dtype):
    encoder, hidden, mask = prepared(dtype, 40)
    before, _ = both(encoder, hidden, mask)
    twin = copy.deepcopy(encoder)
    _in_place(twin.layer[1].output.dense.weight)
    with torch.inference_mode():
        twin(hidden, mask)   # the first call makes the copy's native loop
    assert 40 in twin._layer_loops
    assert_follows(twin, hidden, mask, before, dtype)
    assert torch.equal(both(encoder, hidden, mask)[0], before)


@pytest.mark.parametrize("dtype,length", ((torch.float32, 32), (torch.float16, 32), (torch.float16, 256)))
def test_a_captured_graph_outlives_the_preparation_it_was_captured_from(dtype, length):
    encoder, hidden, mask = prepared(dtype, length, conv=0 if dtype == torch.float32 else 3)
    bucket = df.capture_deberta_buckets(encoder, 2)[length]
    before = bucket(hidden, mask).clone()
    held = [t.data_ptr() for t in (*bucket.prepared[0][0][1:], *bucket.prepared[1][0]) if t is not None]
    encoder.prepare_for_inference([length + 1])
    fresh = {t.data_ptr() for plan in encoder._active_plans for t in plan[1:] if t is not None}
    assert held and not fresh & set(held)   # nothing new lies where the graph reads
    junk = [torch.full((n,), float("nan"), device=dev) for n in (1 << 10, 1 << 16, 1 << 18, 1 << 20) for _ in range(8)]
    assert torch.equal(bucket(hidden, mask), before) and junk
