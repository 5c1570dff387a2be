"""The stream that the binding passes on: the one given, else torch's current one,
also where this torch lacks the private call for its handle."""
import types

import pytest


def test_given_and_current_without_the_private_call(nmg, monkeypatch):
    import torch
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(cuda_stream=0x1234))
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert nmg._stream(None).value == 0x1234
    assert nmg._stream(types.SimpleNamespace(cuda_stream=0x77)).value == 0x77


@pytest.mark.gpu
def test_current_stream(nmg):
    import torch
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        assert nmg._stream(None).value == s.cuda_stream == torch.cuda.current_stream().cuda_stream
    assert (nmg._stream(None).value or 0) == torch.cuda.current_stream().cuda_stream
