"""Relative-table attention, several items a CTA: tiles whose padded rows take a column sum of V, plain tiles and tiles of padding follow
one another on the same barriers, exchange words and accumulator, and every row is what it is in a batch of its own."""

import math

import pytest
import torch

from helpers import make_core_case, tolerance
from test_gpu_rel_attention import DTYPES, run_rel

pytestmark = pytest.mark.gpu

# kept keys [first, last): key tiles skipped behind, before and on both sides, none; no kept key; one
RANGES = ((0, 130), (0, 640), (400, 640), (0, 0), (260, 380), (0, 500), (513, 514), (130, 640), (383, 385), (0, 1))


def _reference(case):
    """The attention in fp64 with position scores rounded to the type, [B, L, H*d], and sum_j p_j |v_j - out| of every output."""
    q, k, v, pk, pq = (case[n].double() for n in ("q", "k", "v", "pos_key", "pos_query"))
    dtype, (batch, heads, length, d) = case["q"].dtype, q.shape
    slot = case["lut"].long()[torch.arange(length)[:, None] - torch.arange(length)[None, :] + length - 1]   # [query, key]
    keep = case["mask"].bool()
    out, spread = torch.empty(2, batch, length, heads * d, dtype=torch.float64)
    for b in range(batch):
        for h in range(heads):
            c2p = torch.gather(q[b, h] @ pk[h].t(), 1, slot).to(dtype).double()
            p2c = torch.gather(k[b, h] @ pq[h].t(), 1, slot.t()).t().to(dtype).double()
            s = (q[b, h] @ k[b, h].t() + c2p + p2c) * case["scale"]
            s = torch.where(keep[b][:, None], s.masked_fill(~keep[b][None, :], -math.inf), torch.zeros_like(s))
            p = s.softmax(1)
            o = p @ v[b, h]
            out[b, :, h * d:(h + 1) * d] = o
            spread[b, :, h * d:(h + 1) * d] = torch.stack([(p * (v[b, h, :, c][None, :] - o[:, c][:, None]).abs()).sum(1) for c in range(d)], 1)
    return out, spread


@pytest.mark.parametrize("dtype_name", sorted(DTYPES))
@pytest.mark.parametrize("d", (32, 64, 128))
@pytest.mark.parametrize("length", (640, 601))
def test_every_item_is_what_it_is_alone(dtype_name, d, length):
    dtype, batch, group = DTYPES[dtype_name], 60, 3   # 900 items
    case = make_core_case(batch, 3, length, d, dtype, seed=3 * d + length, mask="none")
    position = torch.arange(length)
    order = torch.randint(len(RANGES), (batch,), generator=torch.Generator().manual_seed(d)).tolist()
    case["mask"] = torch.stack([(position >= RANGES[k][0]) & (position < RANGES[k][1]) for k in order]).to(case["mask"].dtype)
    together = run_rel(case)
    # a probability reaches the tensor core rounded to the type: by this much of itself, which moves an output by the sum below
    unit = 2.0 ** (-11 if dtype == torch.float16 else -8)
    for at in range(0, batch, group):
        few = dict(case, **{name: case[name][at:at + group] for name in ("q", "k", "v", "mask")})
        alone = run_rel(few)
        assert torch.equal(together[at:at + group], alone), f"sequences from {at}"
        want, spread = _reference(few)
        excess = (alone.double().cpu() - want).abs() - tolerance(dtype, want) - unit * spread
        assert excess.max() <= 0, (at, excess.max().item())
