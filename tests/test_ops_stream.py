"""The operators' way to the current stream: torch's short one where this build of it has one, else the public one.  No GPU is needed."""
import types

import pytest
import torch

from my_nn_engine_b200 import ops


@pytest.mark.parametrize("raw,device", [(None, lambda: 0), (lambda d: 1, None)])
def test_public_way_where_the_short_one_is_missing(monkeypatch, raw, device):
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=4321))
    monkeypatch.setattr(ops, "_raw_stream", raw)
    monkeypatch.setattr(ops, "_device", device)
    assert ops._stream() == 4321


def test_short_way_takes_the_current_device(monkeypatch):
    monkeypatch.setattr(ops, "_raw_stream", lambda d: 100 + d)
    monkeypatch.setattr(ops, "_device", lambda: 3)
    assert ops._stream() == 103
