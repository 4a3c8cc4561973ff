"""No two kernels share a hundred of wait codes, whatever a source calls its base, and every hundred names its kernel."""

import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "disentangled_flash_b200" / "csrc"


def _values() -> dict[str, int]:
    text = (CSRC / "dfl_common.cuh").read_text()
    body = text[text.index("enum WaitCodes {"):]
    values: dict[str, int] = {}
    for name, first, offset in re.findall(r"(kWaits\w+) = (\w+)(?: \+ (\d+))?", body[:body.index("};")]):
        values[name] = (values[first] if first in values else int(first)) + int(offset or 0)
    return values


def test_every_kernel_with_waits_has_a_hundred_of_its_own():
    values, bases = _values(), {}
    for source in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
        text = source.read_text()
        for name in set(re.findall(r"constexpr int \w+ = (kWaits\w+);|atomicCAS\(status_word, 0, (kWaits\w+)", text)):
            bases.setdefault(name[0] or name[1], []).append(source.name)
        if re.search(r"ptx::mbar_wait(?:_slow)?\(", text) and source.suffix == ".cu":
            assert re.search(r"constexpr int \w+ = kWaits\w+;|attention_tc_common.cuh", text), source.name
    assert sorted(bases) == sorted(values)
    assert all(len(where) == 1 for where in bases.values()), bases
    assert sorted(v // 100 for v in values.values()) == list(range(1, len(values) + 1)) and all(v % 100 == 0 for v in values.values())


def test_every_hundred_names_a_kernel_that_there_is():
    text = (CSRC / "dfl_common.cuh").read_text()
    names = dict(re.findall(r'case (kWaits\w+): return "(\w+)";', text))
    assert set(names) == set(_values()) and len(set(names.values())) == len(names)
    sources = "".join(p.read_text() for p in CSRC.glob("*.cu"))
    assert all(re.search(rf"\b{kernel}\(", sources) for kernel in names.values())


@pytest.mark.gpu
@pytest.mark.parametrize("code", (771, 791))
def test_the_message_names_the_kernel(code):
    from disentangled_flash_b200 import _cabi as c

    word = torch.tensor([code], dtype=torch.int32, device="cuda")
    with pytest.raises(c.DflError, match=f"wait code {code}, attention_f32_rel_kernel"):
        c.check_status(word)
    assert word.item() == 0
