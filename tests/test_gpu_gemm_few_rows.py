"""Products whose tiles of 128 rows load fewer: row counts around a group of eight, one and two 64-element pieces per k-block,
inner products of one CTA and of several, rows dealt out over CTA pairs and over several tiles, packed rows whose groups of 32 a
tile divides, after a product that leaves infinities in the shared memory of the tiles' other rows, against fp64."""

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


# Pairs of CTAs, their second one with few rows or none, rows dealt out over tiles, with and without a split inner product.
@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("n,k", ((768, 768), (2304, 768), (768, 3072), (72, 200), (6144, 1536), (1536, 6144)))
def test_ragged_pairs_and_several_tiles(dtype, n, k):
    from disentangled_flash_b200 import _cabi as c

    gen = torch.Generator().manual_seed(n * 2 + k)
    weight = (torch.randn(n, k, generator=gen) * k ** -0.5).to(dtype)
    bias = torch.randn(n, generator=gen).to(dtype)
    rows = torch.randn(600, k, generator=gen).to(dtype)
    full = rows.double() @ weight.double().T + bias.double()
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    weight, bias = weight.to(dev), bias.to(dev)
    poison = torch.full((768, k), float("inf"), dtype=dtype, device=dev)
    for m in (129, 130, 136, 137, 160, 200, 249, 255, 257, 264, 333, 385, 513, 600):
        c.dense(poison[:-(-m // 128) * 128], weight, bias)   # as many tiles, all of their rows
        got = c.dense(rows[:m].to(dev), weight, bias).double().cpu()
        # one rounding of the output, and fp32 sums
        assert ((got - full[:m]).abs() <= eps * full[:m].abs() + 1e-4).all(), (m, (got - full[:m]).abs().max().item())


@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("groups", (1, 3, 5, 7, 11, 17))
def test_packed_rows_whose_groups_a_tile_divides(dtype, groups):
    from disentangled_flash_b200 import _cabi as c

    heads, d, length = 12, 64, 96
    hidden, m = heads * d, 32 * groups
    gen = torch.Generator().manual_seed(groups)
    weight = (torch.randn(3 * hidden, hidden, generator=gen) * hidden ** -0.5).to(dtype)
    bias = torch.randn(3 * hidden, generator=gen).to(dtype)
    rows = torch.randn(m, hidden, generator=gen).to(dtype)
    slots = torch.randperm(18, generator=gen)[:groups]   # of the 32-row groups of six sequences of 96
    want = (rows.double() @ weight.double().T + bias.double()).view(m, 3, heads, d)
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    c.dense(torch.full((-(-m // 128) * 128, hidden), float("inf"), dtype=dtype, device=dev), weight.to(dev), bias.to(dev))
    outs = tuple(torch.full((6, heads, length, d), 7.0, dtype=dtype, device=dev) for _ in range(3))
    c.linear_heads(rows.to(dev), weight.to(dev), bias.to(dev), n_out=3, heads=heads, head_dim=d, rows_per_seq=length,
                   row_groups=(32 * slots).to(device=dev, dtype=torch.int32), outs=outs)
    for which, out in enumerate(outs):
        flat = out.double().cpu().transpose(1, 2).reshape(18, 32, heads, d)
        part = want[:, which].view(groups, 32, heads, d)
        assert ((flat[slots] - part).abs() <= eps * part.abs() + 1e-4).all(), which
        others = torch.ones(18, dtype=torch.bool).index_fill_(0, slots, False)
        assert (flat[others] == 7.0).all(), which
