"""add + LayerNorm on both sides of the row count at which the few-rows form ends, against PyTorch in fp32."""

import pytest
import torch
from torch.nn import functional as F

from helpers import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16, torch.float32))
@pytest.mark.parametrize("hidden", (64, 768, 1536, 2048))
@pytest.mark.parametrize("rows", (1, 9, 1184, 1185, 2368, 2369, 9000))
def test_row_counts(rows, hidden, dtype):
    from disentangled_flash_b200 import _cabi

    gen = torch.Generator("cuda").manual_seed(rows + hidden)
    x, residual = (torch.randn(rows, hidden, generator=gen, device="cuda").to(dtype) for _ in range(2))
    gamma, beta = (torch.randn(hidden, generator=gen, device="cuda").to(dtype) for _ in range(2))
    want = F.layer_norm(x.float() + residual.float(), (hidden,), gamma.float(), beta.float(), 1e-7)
    assert_close(_cabi.add_layernorm(x, residual, gamma, beta, 1e-7), want.cpu(), dtype, f"{rows} x {hidden}")
    want = F.layer_norm(x.float() + residual.float(), (hidden,), gamma.float(), None, 1e-7)
    assert_close(_cabi.add_layernorm(x, residual, gamma, None, 1e-7), want.cpu(), dtype, f"{rows} x {hidden} without bias")
