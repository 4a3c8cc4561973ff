"""Dense products of fewer than 128 rows, whose tiles load only the rows there are: row counts around a group of eight, one and
two 64-element pieces per k-block, inner products of one CTA and of several, after a product that leaves infinities in the
shared memory of the tiles' other rows, against fp64."""

import pytest
import torch

pytestmark = pytest.mark.gpu
dev = "cuda"


@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("n,k,activation", ((768, 768, 0), (3072, 768, 1), (768, 3072, 0), (72, 200, 0), (4608, 1536, 0)))
def test_few_rows(dtype, n, k, activation):
    from disentangled_flash_b200 import _cabi as c

    gen = torch.Generator().manual_seed(n + k)
    weight = (torch.randn(n, k, generator=gen) * k ** -0.5).to(dtype)
    bias = torch.randn(n, generator=gen).to(dtype)
    rows = torch.randn(127, k, generator=gen).to(dtype)
    full = rows.double() @ weight.double().T + bias.double()
    full = torch.nn.functional.gelu(full) if activation else full
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    poison = torch.full((127, k), float("inf"), dtype=dtype, device=dev)
    for m in (1, 7, 8, 9, 31, 33, 64, 100, 120, 121, 127):
        c.dense(poison, weight.to(dev), bias.to(dev), activation=activation)
        got = c.dense(rows[:m].to(dev), weight.to(dev), bias.to(dev), activation=activation)
        want = full[:m]
        # one rounding of the output, and fp32 sums
        assert ((got.double().cpu() - want).abs() <= eps * want.abs() + 1e-4).all(), (m, (got.double().cpu() - want).abs().max().item())
