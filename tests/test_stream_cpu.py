"""The current stream's handle: read directly where torch offers it, through the public calls where not."""

import types

import pytest

from nbody import lib


@pytest.fixture
def fresh(monkeypatch):
    monkeypatch.setattr(lib, "_current_stream", None, raising=False)
    return monkeypatch


def test_without_the_direct_calls(fresh):
    import torch
    for name in ("_cuda_getDevice", "_cuda_getCurrentRawStream"):
        if hasattr(torch._C, name):
            fresh.delattr(torch._C, name)
    fresh.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=1234))
    assert lib.stream_ptr() == 1234


def test_direct_calls_and_a_given_stream(fresh):
    import torch
    fresh.setattr(torch._C, "_cuda_getDevice", lambda: 3, raising=False)
    fresh.setattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 100 + d, raising=False)
    fresh.setattr(torch.cuda, "is_initialized", lambda: True)
    assert lib.stream_ptr() == 103
    assert lib.stream_ptr(types.SimpleNamespace(cuda_stream=7)) == 7
