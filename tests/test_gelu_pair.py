"""The GELU of the 16-bit GEMM epilogues, ``gelu_erf_pair`` (``csrc/dfl_common.cuh``): ``max(x, 0) - |x| 2^p(-|x|)`` with the
polynomial's constants read from the header, against ``math.erfc``; and both GEMM kernels' epilogues on the GPU at sizes around
their column chunks."""

import math
import re
from pathlib import Path

import pytest
import torch
import torch.nn.functional as F

HEADER = Path(__file__).resolve().parent.parent / "disentangled_flash_b200" / "csrc" / "dfl_common.cuh"


def _coefficients() -> list[float]:
    text = HEADER.read_text()
    start = text.index("void gelu_erf_pair(float& a, float& b)")
    body = text[start:text.index("\n}", start)]
    return [float(m) for m in re.findall(r"k\((-?\d+\.\d+(?:e-?\d+)?)f\)", body)]


def _gelu(x: float, c: list[float]) -> float:
    t = -abs(x)
    p = 0.0
    for k in c:
        p = p * t + k
    return t * 2.0 ** max(p, -2000.0) + max(x, 0.0)


def test_polynomial_against_erfc():
    c = _coefficients()
    assert len(c) == 9
    worst = tail = 0.0
    for i in range(-12000, 12001):
        x = i / 1000.0
        exact = 0.5 * x * math.erfc(-x / math.sqrt(2.0))
        err = abs(_gelu(x, c) - exact)
        worst = max(worst, err)
        if -4.5 <= x < 0.0:
            tail = max(tail, err / abs(exact))
    assert worst < 2.5e-7, worst
    assert tail < 5e-4, tail   # half an FP16 rounding step is 4.9e-4


def test_polynomial_keeps_falling():
    c = _coefficients()
    last = 0.0
    for i in range(0, 70000, 7):
        t, p = -i / 10.0, 0.0
        for k in c:
            p = p * t + k
        assert p <= last, i
        last = p


# rows: one tile kernel, one pair-kernel plan; columns: whole chunks, a ragged last chunk, a tile whose second warp has none
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("rows, n", [(40, 72), (40, 512), (16384, 768), (16384, 776), (16384, 1032), (16390, 320)])
def test_gelu_epilogue_columns(dtype, rows, n):
    from disentangled_flash_b200 import _cabi as c

    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(dev).manual_seed(rows + n)
    k = 64
    x = torch.randn(rows, k, generator=gen, device=dev).to(dtype)
    w = (torch.randn(n, k, generator=gen, device=dev) * 0.25).to(dtype)
    b = torch.randn(n, generator=gen, device=dev).to(dtype)
    x[3, :] = 0
    b[5:12] = torch.tensor([30.0, -30.0, 1000.0, -1000.0, 60000.0, -60000.0, float("nan")], device=dev).to(dtype)
    got = c.dense(x, w, b, activation=c.ACT_GELU).float()
    want = F.gelu(x.double() @ w.double().T + b.double()).float()
    assert torch.isnan(got[:, 11]).all()
    keep = torch.arange(n, device=dev) != 11
    got, want = got[:, keep], want[:, keep]
    # the output's rounding, and what an fp32 sum of 64 products of magnitude |b| + 2 can be off by
    ulp = 2.0 ** (-11 if dtype == torch.float16 else -8)
    bound = ulp * want.abs() + 1e-5 + 2.0 ** -22 * b[keep].abs().float()
    assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() - bound).max())
