"""The current stream's address with and without torch's private call."""
import types

import torch

from gpugraphs import core


def test_public_call_serves_where_the_private_one_is_absent(monkeypatch):
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream",
                        lambda device: types.SimpleNamespace(cuda_stream=4096 + device))
    assert core._raw_stream_of()(3) == 4099


def test_private_call_is_taken_where_it_is(monkeypatch):
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 7 + device, raising=False)
    assert core._raw_stream_of()(1) == 8
