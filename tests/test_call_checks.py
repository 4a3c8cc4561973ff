"""What a call refuses before any address reaches the native code: the kernels cannot see widths, types or devices.  The
native call is replaced by a recorder and the module is built on the CPU, so nothing here needs a GPU ("meta" stands for
another device)."""

import pytest
import torch

import disentangled_flash_b200 as df
from disentangled_flash_b200 import _cabi, attention

LENGTH, HIDDEN, HEADS, HEAD_DIM = 16, 256, 4, 32


@pytest.fixture
def prepared(monkeypatch):
    """``(module, plan, calls)``: a module with the buffers ``prepare_for_inference`` leaves, and the native calls made."""

    def build(dtype=torch.float16):
        cfg = df.DebertaAttentionConfig(hidden_size=HIDDEN, num_attention_heads=HEADS, attention_head_size=HEAD_DIM,
                                        max_position_embeddings=64, position_buckets=32, norm_rel_ebd="none")
        module = df.DisentangledFlashAttention(cfg).to(dtype).eval()
        module._cached_qkv_weight = torch.cat([getattr(module, f"{n}_proj").weight.detach() for n in ("query", "key", "value")])
        module._cached_qkv_bias = torch.zeros(3 * HEADS * HEAD_DIM, dtype=dtype)
        distances, slots = 2 * LENGTH - 1, 24
        pos, rel = torch.zeros(HEADS, slots, HEAD_DIM, dtype=dtype), torch.zeros(HEADS, distances, HEAD_DIM, dtype=dtype)
        f32 = dtype == torch.float32
        planes = torch.zeros(3, *pos.shape, dtype=torch.bfloat16) if f32 else None
        if f32:
            module._cached_qkv_planes = torch.zeros(3, *module._cached_qkv_weight.shape, dtype=torch.bfloat16)
            rel = None
        plan = df.B200PreparedPositionPlan(LENGTH, torch.arange(slots), torch.zeros(distances, dtype=torch.int32), pos, pos.clone(),
                                           rel, None if f32 else rel.clone(), planes, planes)
        calls = []
        monkeypatch.setattr(module, "_validate_device_dtype", lambda tensor: None)
        monkeypatch.setattr(_cabi, "encoder_fwd", lambda p, *_: calls.append(("native", p.scale)))
        monkeypatch.setattr(attention, "_attention_forward", lambda *a: calls.append(("general", a)) or torch.empty(0))
        return module, plan, calls

    return build


def _inputs(dtype=torch.float16, width=HIDDEN):
    return torch.zeros(2, LENGTH, width, dtype=dtype), torch.ones(2, LENGTH, dtype=torch.bool)


@pytest.mark.parametrize("dtype", (torch.float16, torch.float32))
def test_a_fitting_call_reaches_the_native_code(prepared, dtype):
    module, plan, calls = prepared(dtype)
    with torch.no_grad():
        module.forward_prepared(*_inputs(dtype), plan)
    assert [kind for kind, _ in calls] == ["native"]


@pytest.mark.parametrize("algo", (_cabi.ALGO_AUTO, _cabi.ALGO_SIMT))
@pytest.mark.parametrize("case,error", (("narrow", ValueError), ("wide", ValueError), ("mask device", RuntimeError),
                                        ("hidden device", RuntimeError), ("dtype", TypeError), ("rank", ValueError)))
def test_wrong_inputs_are_refused_before_the_native_code(prepared, case, error, algo):
    module, plan, calls = prepared()
    module._algo = algo
    hidden, mask = _inputs()
    if case in ("narrow", "wide"):
        hidden = _inputs(width=HIDDEN // 2 if case == "narrow" else 2 * HIDDEN)[0]
    elif case == "mask device":
        mask = mask.to("meta")
    elif case == "hidden device":
        hidden, mask = hidden.to("meta"), mask.to("meta")
    elif case == "dtype":
        hidden = hidden.float()
    else:
        hidden = torch.zeros(2, LENGTH, 3, HIDDEN, dtype=torch.float16)
    with torch.no_grad(), pytest.raises(error):
        module.forward_prepared(hidden, mask, plan)
    assert not calls


@pytest.mark.parametrize("field,table", (
    ("rel_key", torch.zeros(HEADS, 2 * LENGTH + 1, HEAD_DIM, dtype=torch.float16)),
    ("rel_query", torch.zeros(HEADS // 2, 2 * LENGTH - 1, HEAD_DIM, dtype=torch.float16)),
    ("pos_key", torch.zeros(HEADS, 24, 2 * HEAD_DIM, dtype=torch.float16)),
    ("pos_query", torch.zeros(HEADS, 24, HEAD_DIM, dtype=torch.bfloat16)),
    ("rel_key", torch.zeros(HEADS, HEAD_DIM, 2 * LENGTH - 1, dtype=torch.float16).transpose(1, 2)),
    ("rel_query", torch.zeros(HEADS, 2 * LENGTH - 1, HEAD_DIM, dtype=torch.float16, device="meta")),
    ("delta_to_local", torch.zeros(2 * LENGTH - 2, dtype=torch.int32)),
))
def test_plans_of_another_geometry_are_refused(prepared, field, table):
    module, plan, calls = prepared()
    with torch.no_grad(), pytest.raises(ValueError, match=field):
        module.forward_prepared(*_inputs(), plan._replace(**{field: table}))
    assert not calls


def test_an_fp32_plan_without_planes_keeps_its_terms(prepared):
    """Only the general path has the position tables of such a plan (the reference's five fields)."""

    module, plan, calls = prepared(torch.float32)
    with torch.no_grad():
        module.forward_prepared(*_inputs(torch.float32), df.B200PreparedPositionPlan(*plan[:5]))
    assert [kind for kind, _ in calls] == ["general"]


def test_terms_and_scale_are_the_modules_present_ones(prepared):
    module, plan, calls = prepared()
    with torch.no_grad():
        module.forward_prepared(*_inputs(), plan)
        first = module._layer_calls[LENGTH]
        module.pos_att_type = ("c2p",)
        module.forward_prepared(*_inputs(), plan)
    assert calls[1][1] == pytest.approx(1 / (2 * HEAD_DIM) ** 0.5) and calls[0][1] == pytest.approx(1 / (3 * HEAD_DIM) ** 0.5)
    assert first.layers[0].rel_query and not module._layer_calls[LENGTH].layers[0].rel_query


@pytest.mark.parametrize("weight,bias", ((torch.float16, torch.float32), (torch.float32, torch.float16)))
def test_projection_refuses_operands_of_another_type(monkeypatch, weight, bias):
    monkeypatch.setattr(_cabi, "_require_cuda_contiguous", lambda name, t: None)
    with pytest.raises(TypeError):
        _cabi.linear_heads(torch.zeros(4, 64), torch.zeros(32, 64, dtype=weight), torch.zeros(32, dtype=bias), n_out=1, heads=1,
                           head_dim=32, rows_per_seq=4)
