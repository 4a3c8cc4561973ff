"""When the native layer loop may serve a call, and what it checks on the way: everything that needs no GPU.  The loops are
built over CPU modules whose prepared buffers are made by hand, and the native call is replaced by a recorder."""

import pytest
import torch
from torch import nn

import hf_modules
import disentangled_flash_b200 as df
from disentangled_flash_b200 import _cabi
from disentangled_flash_b200.layer_loop import LayerLoop


@pytest.mark.parametrize("wrong", (lambda x: x[:, :-1], lambda x: x.half(), lambda x: x.to("meta"), lambda x: x[..., :8]))
def test_a_convolution_branch_that_changes_the_state_is_refused(monkeypatch, wrong):
    loop = LayerLoop()
    loop.dtype, loop.device, loop.n_layers = torch.float32, torch.device("cpu"), 2
    runs = []
    monkeypatch.setattr(loop, "_run", lambda hidden, *a: runs.append(a[-2:]) or hidden)
    hidden, mask = torch.zeros(2, 4, 16), torch.ones(2, 4, dtype=torch.bool)
    with pytest.raises(ValueError, match="convolution branch"):
        loop.run(hidden, mask, None, None, lambda x, state, mask: wrong(state))
    assert runs == [(0, 1)]
    loop.run(hidden, mask, None, None, lambda x, state, mask: state)
    assert runs[1:] == [(0, 1), (1, 2)]
