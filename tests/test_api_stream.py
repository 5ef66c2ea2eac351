"""The stream argument of every call: the current stream's handle, also with a
torch that has no internal functions for it."""
import importlib.util
import types

import pytest
import torch

from gprt_b200 import api


def _copy_of_api():
    spec = importlib.util.spec_from_file_location("gprt_b200.api_copy", api.__file__)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


@pytest.mark.parametrize("missing", ["_cuda_getCurrentRawStream", "_cuda_getDevice"])
def test_stream_without_torch_internals(monkeypatch, missing):
    monkeypatch.delattr(torch._C, missing, raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=1234))
    assert _copy_of_api()._stream() == 1234


@pytest.mark.gpu
def test_stream_is_the_current_one(cuda):
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        assert api._stream() == s.cuda_stream
    assert api._stream() == torch.cuda.current_stream().cuda_stream
