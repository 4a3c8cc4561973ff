"""Relative-table attention, query tiles with kept and padded rows whose key tiles are not all walked: the padded rows' share of
the skipped keys is a column sum of V."""

import pytest
import torch

from helpers import assert_close, make_core_case, oracle_core
from test_gpu_rel_attention import DTYPES, run_rel

pytestmark = pytest.mark.gpu


# kept keys [first, last) per sequence: tiles skipped behind, before, on both sides; one kept key; a ragged last tile; none skipped
RANGES = ([(0, 130), (0, 1), (0, 300)], [(400, 640), (513, 514), (130, 640)], [(260, 380), (383, 385), (0, 640)])


@pytest.mark.parametrize("dtype_name", sorted(DTYPES))
@pytest.mark.parametrize("d", (32, 64, 128))
@pytest.mark.parametrize("mode", ("both", "c2p", "p2c"))
@pytest.mark.parametrize("ranges", range(len(RANGES)))
@pytest.mark.parametrize("length", (640, 601))
def test_padded_rows_attend_to_all_keys(dtype_name, d, mode, ranges, length):
    dtype = DTYPES[dtype_name]
    batch = 3 if mode != "both" else 60          # several items per CTA, folded ones among them
    case = make_core_case(batch, 3, length, d, dtype, seed=d + length, mask="none", mode=mode)
    position = torch.arange(length)
    mask = torch.stack([(position >= a) & (position < b) for a, b in RANGES[ranges]]).repeat(batch // 3, 1)
    case["mask"] = mask.to(case["mask"].dtype)
    got = run_rel(case)
    assert torch.equal(got, run_rel(case)), "two identical launches differ"
    if batch == 3:
        assert_close(got, oracle_core(case), dtype, f"d={d} L={length} mode={mode}")
    # a padded row is the mean of V over all keys: sums of `length` values of T in fp32, one rounding
    mean = case["v"].double().mean(2).reshape(batch, 1, -1)
    padded = got.double().cpu()[~mask.unsqueeze(-1).expand_as(got)].reshape(-1, mean.shape[-1])
    want = mean.expand_as(got)[~mask.unsqueeze(-1).expand_as(got)].reshape(-1, mean.shape[-1])
    ulp = 2.0 ** (-11 if dtype == torch.float16 else -8)
    assert bool(((padded - want).abs() <= ulp * want.abs() + 1e-5).all())
