"""The short-sequence form of the relative-table attention: row and key remainders of its four sizes, masks and single
terms, the packed output, and the batch size at which 65 .. 128 positions go to the other kernel."""

import pytest
import torch

from helpers import assert_close, make_core_case, oracle_core
from test_gpu_rel_attention import DTYPES, dev, expand, run_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype_name", sorted(DTYPES))
@pytest.mark.parametrize("d", (32, 64))
@pytest.mark.parametrize("batch,heads,length,mask,mode", (
    (1, 1, 1, "none", "both"), (3, 2, 15, "right", "c2p"), (2, 3, 16, "left", "p2c"), (3, 5, 17, "heavy", "both"),
    (2, 2, 31, "all", "both"), (40, 12, 33, "right", "both"), (3, 2, 48, "left", "c2p"), (2, 2, 63, "heavy", "p2c"),
    (3, 3, 81, "left", "both"), (2, 2, 113, "all", "p2c"), (12, 12, 127, "right", "both"), (16, 12, 127, "right", "both")))
def test_short_sequences(dtype_name, d, batch, heads, length, mask, mode):
    dtype = DTYPES[dtype_name]
    case = make_core_case(batch, heads, length, d, dtype, seed=length, mask=mask, mode=mode)
    got = run_rel(case)
    assert_close(got, oracle_core(case), dtype, f"L={length} d={d} mask={mask} mode={mode}")
    assert torch.equal(got, run_rel(case)), "two identical launches differ"


@pytest.mark.parametrize("length", (24, 64, 90))
def test_short_packed_output(length):
    from disentangled_flash_b200 import _cabi as c

    case = make_core_case(3, 2, length, 64, torch.float16, seed=7, mask="right")
    full = run_rel(case)
    counts = [min(length, -(-int(n) // 32) * 32) for n in case["mask"].sum(dim=1)]
    bases = [0, counts[0], counts[0] + counts[1]]
    rel_key, rel_query = expand(case)
    tables = tuple(torch.tensor(x, dtype=torch.int32, device=dev) for x in (bases, counts))
    packed = c.attention_rel_fwd(case["q"].to(dev), case["k"].to(dev), case["v"].to(dev), rel_key, rel_query,
                                 case["mask"].to(dev), case["scale"], packed_rows=(*tables, sum(counts)))
    for b in range(3):
        assert torch.equal(packed[bases[b]:bases[b] + counts[b]], full[b, :counts[b]]), b


# One CTA a head with more heads than SMs, two with fewer: a second CTA without rows (16 of 32 positions) and with one (33),
# uneven groups (six warps), and the numbers of heads at which 128 positions leave this kernel.
@pytest.mark.parametrize("dtype_name", sorted(DTYPES))
@pytest.mark.parametrize("batch,heads,length,d,mask,mode", (
    (2, 3, 16, 64, "none", "both"), (2, 3, 33, 32, "right", "both"), (2, 3, 49, 64, "left", "c2p"), (3, 2, 97, 64, "heavy", "p2c"),
    (12, 13, 17, 64, "right", "both"), (12, 13, 33, 64, "heavy", "c2p"), (12, 13, 64, 32, "left", "p2c"), (12, 13, 65, 64, "all", "both"),
    (12, 13, 96, 64, "right", "both"), (12, 13, 96, 32, "heavy", "both"), (13, 17, 128, 32, "right", "both"),
    (13, 18, 128, 32, "right", "both"), (12, 12, 128, 64, "heavy", "both")))
def test_one_and_two_ctas_per_head(dtype_name, batch, heads, length, d, mask, mode):
    dtype = DTYPES[dtype_name]
    case = make_core_case(batch, heads, length, d, dtype, seed=100 + length, mask=mask, mode=mode)
    got = run_rel(case)
    assert_close(got, oracle_core(case), dtype, f"L={length} d={d} heads={batch * heads} mask={mask} mode={mode}")
    assert torch.equal(got, run_rel(case)), "two identical launches differ"


# As many heads as SMs or fewer: two CTAs and two warps a row; one batch row more: one.  Scores, maxima and rounded probabilities are
# the same bits; row sums and P.V are added in fp32 in another order, 2 L roundings of 2^-24 each, before the output is rounded.
@pytest.mark.parametrize("dtype_name", sorted(DTYPES))
@pytest.mark.parametrize("length,d", ((24, 64), (33, 32), (64, 64), (64, 32), (96, 64), (96, 32)))
def test_one_cta_a_head_is_as_exact_as_two(dtype_name, length, d):
    dtype = DTYPES[dtype_name]
    heads = 12
    few = torch.cuda.get_device_properties(0).multi_processor_count // heads
    case = make_core_case(few + 1, heads, length, d, dtype, seed=300 + length, mask="heavy")
    one = run_rel(case)[:few].double().cpu()
    case.update({name: case[name][:few].contiguous() for name in ("q", "k", "v", "mask")})
    two = run_rel(case).double().cpu()
    want = oracle_core(case, compute=torch.float64)
    step = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7   # of the output type
    bound = step * torch.maximum(one.abs(), two.abs()) + 2 * length * 2.0 ** -24 * case["v"].abs().max().double()
    assert ((one - two).abs() <= bound).all(), ((one - two).abs() - bound).max().item()
    # output steps that fall the other way, at random: a few of 10^5 and more elements
    errors = [(got - want).norm().item() for got in (one, two)]
    assert max(errors) <= 1.01 * min(errors), errors
