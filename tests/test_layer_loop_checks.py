"""When the native layer loop may serve a call, and what it checks on the way: everything that needs no GPU.  The loops are
built over CPU modules whose prepared buffers are made by hand, and the native call is replaced by a recorder."""

import copy
import io

import pytest
import torch
from torch import nn

import hf_modules
import disentangled_flash_b200 as df
from disentangled_flash_b200 import _cabi, attention
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


LENGTH = 32


@pytest.fixture
def covered(monkeypatch):
    """``build(dtype, conv)`` -> the encoder, and whether its native loop covers a call now."""

    monkeypatch.setattr(_cabi.FollowingPlanes, "refresh", lambda self: None)

    def build(dtype=torch.float16, conv=0, bias=True, activation=None, misaligned=None):
        cfg = df.DebertaAttentionConfig(hidden_size=256, num_attention_heads=4, attention_head_size=64, num_hidden_layers=3,
                                        intermediate_size=512, max_position_embeddings=64, position_buckets=32,
                                        conv_kernel_size=conv)
        source = hf_modules.Encoder(cfg)
        for layer in source.layer:
            if not bias:
                layer.output.LayerNorm = nn.LayerNorm(256, cfg.layer_norm_eps, bias=False)
            if activation is not None:
                layer.intermediate.intermediate_act_fn = activation()
        encoder = df.DebertaV2InferenceEncoder(source, cfg).to(dtype).eval()
        if misaligned is not None:
            weight = encoder.get_submodule(misaligned).weight
            weight.data = torch.zeros(weight.numel() + 1, dtype=dtype)[1:].view_as(weight)
        f32, plans = dtype == torch.float32, []
        for layer in encoder.layer:
            module = layer.attention.self
            module._cached_qkv_weight, module._cached_qkv_bias = torch.zeros(768, 256, dtype=dtype), torch.zeros(768, dtype=dtype)
            module._cached_qkv_planes = torch.zeros(3, 768, 256, dtype=torch.bfloat16) if f32 else None
            plans.append(df.B200PreparedPositionPlan(LENGTH, torch.arange(9), torch.zeros(2 * LENGTH - 1, dtype=torch.int32),
                                                     torch.zeros(4, 9, 64, dtype=dtype), torch.zeros(4, 9, 64, dtype=dtype)))
        encoder._fused_output_blocks, encoder._fused_intermediates = [(True, True)] * 3, [not f32] * 3
        if conv:
            encoder._conv_fused = {LENGTH: False}
            encoder._conv_weight = encoder.conv.conv.weight.detach().permute(2, 0, 1).contiguous()
        plans = tuple(plans)
        loop = LayerLoop.build(encoder, LENGTH, plans, bool(conv))
        if loop is None:
            return encoder, None
        hidden, mask = torch.zeros(2, LENGTH, 256, dtype=dtype), torch.ones(2, LENGTH, dtype=torch.bool)

        encoder._layer_loops[LENGTH] = loop
        encoder._buckets.by_length[LENGTH] = plans
        encoder._buckets.select(LENGTH)
        encoder._conv_covered = {LENGTH: bool(conv)}

        def covers():
            with torch.no_grad():
                return loop.covers(encoder, plans, hidden, mask)

        return encoder, covers

    return build


def _linear(old):
    return nn.Linear(old.in_features, old.out_features, dtype=old.weight.dtype)


EXCHANGES = {
    "attention.output.dense": lambda e: setattr(e.layer[1].attention.output, "dense", _linear(e.layer[1].attention.output.dense)),
    "intermediate.dense": lambda e: setattr(e.layer[0].intermediate, "dense", _linear(e.layer[0].intermediate.dense)),
    "output.dense": lambda e: setattr(e.layer[2].output, "dense", _linear(e.layer[2].output.dense)),
    "LayerNorm": lambda e: setattr(e.layer[0].output, "LayerNorm", nn.LayerNorm(256, dtype=e.layer[0].output.LayerNorm.weight.dtype)),
    "attention.self": lambda e: setattr(e.layer[1].attention, "self", e.layer[2].attention.self),
    "attention.output": lambda e: setattr(e.layer[1].attention, "output", e.layer[2].attention.output),
    "output": lambda e: setattr(e.layer[1], "output", e.layer[2].output),
    "layer": lambda e: e.layer.__setitem__(1, e.layer[2]),
    "a layer less": lambda e: e.layer.__delitem__(2),
    "the list": lambda e: setattr(e, "layer", nn.ModuleList(e.layer)),
    "a parameter": lambda e: setattr(e.layer[2].output.dense, "weight", nn.Parameter(e.layer[2].output.dense.weight.clone())),
    "a parameter's data, transposed": lambda e: setattr(e.layer[0].attention.output.dense.weight, "data",
                                                        e.layer[0].attention.output.dense.weight.data.t()),
    "a parameter's type": lambda e: setattr(e.layer[0].output.dense.bias, "data",
                                            e.layer[0].output.dense.bias.data.view(torch.bfloat16)),
    "no bias": lambda e: setattr(e.layer[1].output.dense, "bias", None),
    "eps": lambda e: setattr(e.layer[1].output.LayerNorm, "eps", 1e-3),
    "activation": lambda e: setattr(e.layer[1].intermediate, "intermediate_act_fn", torch.relu),
    "terms": lambda e: setattr(e.layer[0].attention.self, "pos_att_type", ("c2p",)),
    "training": lambda e: e.layer[0].attention.self.train(),
    "kernel family": lambda e: setattr(e.layer[0].attention.self, "_algo", _cabi.ALGO_SIMT),
}


@pytest.mark.parametrize("dtype", (torch.float16, torch.float32))
@pytest.mark.parametrize("exchange", EXCHANGES)
def test_exchanged_modules_and_settings_are_not_read_at_their_old_place(covered, exchange, dtype):
    encoder, covers = covered(dtype)
    assert covers()
    EXCHANGES[exchange](encoder)
    assert not covers()


def test_a_parameter_that_appears_is_noticed(covered):
    encoder, covers = covered(bias=False)
    assert covers()
    encoder.layer[0].output.LayerNorm.bias = nn.Parameter(torch.ones(256, dtype=torch.float16))
    assert not covers()


def test_an_activation_module_is_compared_too(covered):
    encoder, covers = covered(activation=nn.GELU)
    assert covers()
    encoder.layer[0].intermediate.intermediate_act_fn.approximate = "tanh"
    assert not covers()


@pytest.mark.parametrize("change", (
    lambda e: setattr(e, "conv", None),
    lambda e: setattr(e, "conv", hf_modules.ConvLayer(df.DebertaAttentionConfig(hidden_size=256, conv_kernel_size=3)).half()),
    lambda e: setattr(e.conv, "conv", nn.Conv1d(256, 256, 3, padding=1).half()),
    lambda e: setattr(e.conv, "conv_act", "gelu"),
    lambda e: setattr(e.conv.LayerNorm, "eps", 1e-3),
    lambda e: e.conv.dropout.train(),
    lambda e: e.conv.register_forward_hook(lambda *a: None),
))
def test_a_changed_convolution_branch_is_noticed(covered, change):
    encoder, covers = covered(conv=3)
    assert covers()
    change(encoder)
    assert not covers()


def test_hooks_and_forwards_of_their_own_run_where_the_fp32_loop_would_skip_them(covered):
    for touch in (lambda block: block.register_forward_hook(lambda *a: None),
                  lambda block: block.dense.register_forward_pre_hook(lambda *a: None),
                  lambda block: setattr(block, "forward", lambda x: x)):
        encoder, covers = covered(torch.float32)
        assert covers()
        touch(encoder.layer[2].intermediate)
        assert not covers()


@pytest.mark.parametrize("dtype", (torch.float16, torch.float32))
@pytest.mark.parametrize("where", ("layer.0.attention.output.dense", "layer.2.output.dense"))
def test_misaligned_weights_are_left_to_the_python_loop(covered, where, dtype):
    assert covered(dtype, misaligned=where)[1] is None


def _saved_and_loaded(model):
    file = io.BytesIO()
    torch.save(model, file)
    file.seek(0)
    return torch.load(file, weights_only=False)


@pytest.mark.parametrize("dtype,conv", ((torch.float16, 0), (torch.bfloat16, 3), (torch.float32, 0)))
@pytest.mark.parametrize("duplicate", (copy.deepcopy, _saved_and_loaded))
def test_a_copy_of_a_prepared_encoder_makes_native_calls_of_its_own(covered, monkeypatch, dtype, conv, duplicate):
    encoder, covers = covered(dtype, conv=conv)
    with torch.no_grad():
        module = encoder.layer[0].attention.self
        module._layer_calls[LENGTH] = attention._LayerCall(module, encoder._active_plans[0])
        twin = duplicate(encoder)
        monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: True))
        loop = twin._layer_loop(torch.zeros(2, LENGTH, 256, dtype=dtype), torch.ones(2, LENGTH, dtype=torch.bool), twin._active_plans)
    assert covers() and not twin.layer[0].attention.self._layer_calls
    assert loop.layers[1].ffn_norm_w == twin.layer[1].output.LayerNorm.weight.data_ptr() != encoder.layer[1].output.LayerNorm.weight.data_ptr()
    if dtype == torch.float32:
        assert twin._weight_planes.addresses == [w for layer in twin.layer for w in (
            layer.attention.output.dense.weight.data_ptr(), layer.intermediate.dense.weight.data_ptr(), layer.output.dense.weight.data_ptr())]
    else:
        assert loop.layers[2].ffn_out_w == twin.layer[2].output.dense.weight.data_ptr()
