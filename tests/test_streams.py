"""Which stream a call without one gets: torch's current stream, whatever of torch's
private lookups there is."""
from __future__ import annotations

import sys
import types

import pytest


def _torch(initialized=True, private=("_cuda_getCurrentRawStream", "_cuda_getDevice")):
    lookups = {"_cuda_getCurrentRawStream": lambda dev: 0x100 + dev, "_cuda_getDevice": lambda: 2}
    return types.SimpleNamespace(
        cuda=types.SimpleNamespace(is_initialized=lambda: initialized,
                                   current_stream=lambda: types.SimpleNamespace(cuda_stream=0x102)),
        _C=types.SimpleNamespace(**{k: lookups[k] for k in private}))


@pytest.mark.parametrize("private", [("_cuda_getCurrentRawStream", "_cuda_getDevice"), ("_cuda_getDevice",),
                                     ("_cuda_getCurrentRawStream",), ()])
def test_the_current_torch_stream_is_found(monkeypatch, private):
    import beamforming_gb300 as bf

    monkeypatch.setitem(sys.modules, "torch", _torch(private=private))
    assert bf._stream_handle(None) == 0x102


def test_a_failing_lookup_is_not_the_default_stream(monkeypatch):
    import beamforming_gb300 as bf

    torch = _torch()
    torch._C._cuda_getCurrentRawStream = lambda: 0  # other arguments than it had
    monkeypatch.setitem(sys.modules, "torch", torch)
    with pytest.raises(TypeError):
        bf._stream_handle(None)


def test_without_torch_on_the_device(monkeypatch):
    import beamforming_gb300 as bf

    monkeypatch.setitem(sys.modules, "torch", _torch(initialized=False))
    assert bf._stream_handle(None) is None
    monkeypatch.delitem(sys.modules, "torch")
    assert bf._stream_handle(None) is None
    assert bf._stream_handle(7) == 7
