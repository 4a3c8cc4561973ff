"""The tiles that ``bench.py`` counts as attention work are the ones that the relative-table kernel walks (``tile_range`` in
``csrc/attention_rel_tc.cu``): the key tiles between the first and the last kept key for every query tile with a kept row."""

import inspect

import pytest
import torch

from test_bench_helpers import _bench


def _mask(length, *valid):
    return torch.arange(length)[None, :] < torch.tensor(valid)[:, None]


@pytest.mark.parametrize("mask,tiles", (
    (_mask(512, 512), 16 / 16),
    (_mask(512, 384), 9 / 16),             # three full query tiles x three key tiles, one tile of padding
    (_mask(512, 300), 9 / 16),             # two full and one mixed query tile x three key tiles
    (_mask(512, 1), 1 / 16),               # one mixed query tile x one key tile
    (_mask(512, 512, 384), 25 / 32),
    (~_mask(512, 200), 9 / 16),            # kept keys 200..511: query tile 1 is mixed
    (_mask(512, 0), 0.0),
    (_mask(300, 140), 4 / 9),              # a ragged last tile
    (_mask(333, 333), 1.0),
))
def test_walked_tiles(mask, tiles):
    assert _bench().executed_tile_fraction(mask, folded=True) == tiles


def test_the_roofline_counts_walked_tiles():
    bench = _bench()
    source = inspect.getsource(bench)
    assert source.count("executed_tile_fraction(m, folded=True)") == 1 and "executed_tile_fraction(m)" not in source
