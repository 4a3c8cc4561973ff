"""The negative tail of the GELU epilogues: an output is as exact, relative to itself, as its type's form (``csrc/dfl_common.cuh``),
also where BF16's exponent range holds results that FP16 rounds away."""

import math
import re
from pathlib import Path

import pytest
import torch

HEADER = Path(__file__).resolve().parent.parent / "disentangled_flash_b200" / "csrc" / "dfl_common.cuh"


def _exact(x: float) -> float:
    return 0.5 * x * math.erfc(-x / math.sqrt(2.0))


def _rational(x: float) -> float:
    """Abramowitz & Stegun 7.1.26 for x < 0."""
    z = -x / math.sqrt(2.0)
    t = 1.0 / (1.0 + 0.3275911 * z)
    q = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429))))
    return 0.5 * x * q * math.exp(-z * z)


def _polynomial(x: float) -> float:
    text = HEADER.read_text()
    start = text.index("void gelu_erf_pair(float& a, float& b)")
    p = 0.0
    for k in re.findall(r"k\((-?\d+\.\d+(?:e-?\d+)?)f\)", text[start:text.index("\n}", start)]):
        p = p * x + float(k)
    return x * 2.0 ** p


# rows: the tile kernel and the pair kernel
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("rows", (40, 16384))
def test_tail_of_the_epilogue(dtype, rows):
    from disentangled_flash_b200 import _cabi as c

    dev = torch.device("cuda", torch.cuda.current_device())
    values = torch.cat((-torch.arange(64, 104) / 8.0, -torch.arange(128, 256) / 32.0))   # -13 < x <= -4, exact in both types
    x, w = torch.zeros(rows, 64, device=dev, dtype=dtype), torch.zeros(values.numel(), 64, device=dev, dtype=dtype)
    bias = values.to(device=dev, dtype=dtype)
    assert torch.equal(bias.float().cpu(), values.float())
    got = c.dense(x, w, bias, activation=c.ACT_GELU)
    assert bool((got == got[:1]).all())
    form = torch.tensor([(_polynomial if dtype == torch.float16 else _rational)(v) for v in values.tolist()], dtype=torch.float64)
    # the form's exponent, up to 123, is an fp32 number of three roundings (3 x 123 x 2^-24 ln 2 = 1.6e-5), its two approximate
    # functions add 1e-6; what lies that near is rounded to the output's type, which keeps the order
    low, high = ((form * (1.0 + s)).to(dtype).double() for s in (3e-5, -3e-5))
    y = got[0].double().cpu()
    assert bool(((low <= y) & (y <= high)).all()), [(v, a, b) for v, a, b in zip(values.tolist(), y.tolist(), form.tolist()) if a != b][:4]
    # and the form itself: 1.5e-2 of the result down to -9 where the result is held
    if dtype == torch.bfloat16:
        for v, f in zip(values.tolist(), form.tolist()):
            assert v < -9.0 or abs(f - _exact(v)) <= 1.5e-2 * abs(_exact(v)), v
