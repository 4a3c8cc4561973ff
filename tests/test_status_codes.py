"""The codes that expired device waits leave in the one status word of a forward tell the kernels apart."""

import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "disentangled_flash_b200" / "csrc"


def test_every_kernel_writes_codes_of_its_own_hundred():
    bases = dict(re.findall(r"(kWaits\w+) = (\d+)", (CSRC / "dfl_common.cuh").read_text()))
    assert len(set(bases.values())) == len(bases) == 6 and all(int(b) % 100 == 0 and int(b) > 0 for b in bases.values())
    used = []
    for source in sorted(CSRC.glob("*.cu")) + [CSRC / "attention_tc_common.cuh"]:
        text = source.read_text()
        used += re.findall(r"(?:kWaits = |atomicCAS\(status_word, 0, )(kWaits\w+)", text)
        for call in re.findall(r"ptx::mbar_wait\(([^;]*?)\)\)?(?:;| &&|\) )", text):
            assert re.search(r"(kWaits \+ \d+|, code)", call), (source.name, call)   # no bare number
    assert sorted(used) == sorted(bases)


def test_every_wait_of_the_relative_table_kernel_says_which_it_was():
    """A code below the hundred for every wait, and for every barrier that the PV and C2P issuer polls in turn."""
    text = (CSRC / "attention_rel_tc.cu").read_text()
    waits = [int(n) for n in re.findall(r"(?:wwait|load)\(.*?, (\d+)\)[;) &]", text)]
    polled = set(re.findall(r"complete\(&bars->(\w+).*?, (\d+)\)", text))
    assert len(polled) == len(dict(polled)) == len(set(re.findall(r"complete\(&bars->(\w+)", text))) == 9   # one code a barrier
    codes = waits + [int(code) for _, code in polled]
    for code in (5, 12, 17, 30, 41, 8, 13):   # of each way a wait is written
        assert code in codes
    assert len(set(codes)) == len(codes) and all(0 < n < 100 for n in codes), sorted(codes)


@pytest.mark.gpu
@pytest.mark.parametrize("code,kernel", ((107, "attention_tc_kernel"), (211, "gemm_tc_pair_kernel"), (324, "gemm_tile_kernel"),
                                         (418, "attention_rel_kernel"), (545, "gemm_f32_kernel"), (651, "attention_f32_kernel")))
def test_the_message_names_the_kernel(code, kernel):
    from disentangled_flash_b200 import _cabi as c

    word = torch.tensor([code], dtype=torch.int32, device="cuda")
    with pytest.raises(c.DflError, match=f"wait code {code}, {kernel}"):
        c.check_status(word)
    assert word.item() == 0
