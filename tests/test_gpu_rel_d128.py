"""The relative-table kernel at head dim 128, where table blocks and V come in 64-row pieces and K has one stage: key-tile
edges, single terms, mask patterns, items of padded rows only, and the packed output, against the fp32 oracle."""

import pytest
import torch

from helpers import assert_close, make_core_case, oracle_core
from test_gpu_rel_attention import DTYPES, run_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype_name", sorted(DTYPES))
@pytest.mark.parametrize("mode", ("both", "c2p", "p2c"))
@pytest.mark.parametrize("batch,heads,length,mask", ((3, 2, 97, "right"), (2, 2, 129, "right"), (1, 3, 191, "none"), (2, 2, 256, "left"),
                                                     (2, 2, 385, "heavy"), (9, 13, 512, "right"), (3, 2, 1100, "all")))
def test_head_dim_128(dtype_name, mode, batch, heads, length, mask):
    from disentangled_flash_b200 import _cabi

    dtype = DTYPES[dtype_name]
    assert _cabi.attention_rel_supported(dtype, length, 128, mode != "p2c", mode != "c2p")
    case = make_core_case(batch, heads, length, 128, dtype, seed=length, mask=mask, mode=mode)
    got = run_rel(case)
    assert_close(got, oracle_core(case), dtype, f"d=128 L={length} mask={mask} mode={mode}")
    assert torch.equal(got, run_rel(case)), "two identical launches differ"
