"""The stream of a call without one: torch's current stream, whichever of torch's own shortcuts this torch has."""
import types

import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("have", [("_cuda_getCurrentRawStream", "_cuda_getDevice"), ("_cuda_getCurrentRawStream",),
                                  ("_cuda_getDevice",), ()])
def test_current_stream_with_and_without_the_shortcuts(monkeypatch, have):
    import gpusnarks_gb300 as g
    shortcuts = {"_cuda_getCurrentRawStream": lambda device: 100 + device, "_cuda_getDevice": lambda: 3}
    monkeypatch.setattr(torch, "_C", types.SimpleNamespace(**{k: shortcuts[k] for k in have}))
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=103))
    assert g._stream_handle(None) == 103
    assert g._stream_handle(7) == 7
    assert g._stream_handle(types.SimpleNamespace(cuda_stream=9)) == 9
