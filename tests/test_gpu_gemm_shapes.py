"""The 16-bit GEMMs at the sizes where the choice of tile, of the split of the inner product and of the CTA pair changes
or a tile is ragged: single rows, one row past a tile, few columns with a long inner product, k-blocks with a remainder.
Reference: ``F.linear`` in fp32 on the rounded inputs; bound 2e-3 plus one rounding step of the output type."""

import pytest
import torch
from torch.nn import functional as F

pytestmark = pytest.mark.gpu
dev = "cuda"
ULP = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def _check(got, want, dtype, what):
    err = (got.float() - want).abs()
    assert torch.isfinite(got).all(), what
    assert bool((err <= 2e-3 + ULP[dtype] * want.abs()).all()), f"{what}: max abs error {err.max().item():.3e}"


@pytest.mark.parametrize("dtype", (torch.float16, torch.bfloat16))
@pytest.mark.parametrize("rows,n,k", (
    (1, 8, 8), (1, 768, 3072), (33, 72, 200), (128, 1024, 4096), (129, 768, 3072), (257, 1000, 264), (384, 1536, 6144),
    (1025, 3072, 768), (2331, 2304, 768), (2331, 768, 3072), (4100, 1032, 1024),
))
def test_dense_at_tile_and_split_edges(dtype, rows, n, k):
    from disentangled_flash_b200 import _cabi as c

    gen = torch.Generator(dev).manual_seed(rows + n + k)
    x = torch.randn(rows, k, generator=gen, device=dev).to(dtype)
    w = (torch.randn(n, k, generator=gen, device=dev) * (1.0 / k ** 0.5)).to(dtype)
    b = torch.randn(n, generator=gen, device=dev).mul_(0.5).to(dtype)
    want = F.linear(x.float().cpu(), w.float().cpu(), b.float().cpu()).to(dev)
    status = c.new_status_word(dev)
    for repeat in range(2):   # back to back: the second call's set-up overlaps the first one's tail
        got = c.dense(x, w, b, status=status)
    c.check_status(status)
    _check(got, want, dtype, f"dense {rows} x {n} x {k}")


@pytest.mark.parametrize("batch,length,heads,d", ((1, 1, 12, 64), (3, 43, 12, 64), (1, 32, 24, 32), (7, 333, 12, 64), (2, 65, 8, 128)))
def test_head_major_projection_at_ragged_lengths(batch, length, heads, d):
    from disentangled_flash_b200 import _cabi as c

    hid = heads * d
    gen = torch.Generator(dev).manual_seed(length)
    x = torch.randn(batch, length, hid, generator=gen, device=dev).half()
    w = (torch.randn(3 * hid, hid, generator=gen, device=dev) / hid ** 0.5).half()
    b = torch.randn(3 * hid, generator=gen, device=dev).half()
    want = F.linear(x.float().cpu(), w.float().cpu(), b.float().cpu()).to(dev)
    status = c.new_status_word(dev)
    outs = c.linear_heads(x, w, b, n_out=3, heads=heads, head_dim=d, rows_per_seq=length, status=status)
    c.check_status(status)
    for i, out in enumerate(outs):
        part = want[..., i * hid:(i + 1) * hid].reshape(batch, length, heads, d).transpose(1, 2)
        _check(out, part, torch.float16, f"output {i}")
