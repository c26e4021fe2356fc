"""The stream that calls run on: torch's current one, by its raw handle or through its Stream object."""

import types

import pytest


@pytest.mark.parametrize("raw", [True, False])
def test_handle(fg, monkeypatch, raw):
    private = {"_cuda_getCurrentRawStream": lambda device: 1000 + device} if raw else {}
    cuda = types.SimpleNamespace(current_device=lambda: 3, current_stream=lambda: types.SimpleNamespace(cuda_stream=77))
    fake = types.SimpleNamespace(_C=types.SimpleNamespace(**private), cuda=cuda)
    monkeypatch.setattr(fg, "_torch", lambda: fake)
    assert fg._stream() == (1003 if raw else 77)


@pytest.mark.gpu
def test_handle_is_the_current_stream(fg, cuda):
    torch = cuda
    assert fg._stream() == torch.cuda.current_stream().cuda_stream
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert fg._stream() == side.cuda_stream
    assert fg._stream() == torch.cuda.current_stream().cuda_stream
