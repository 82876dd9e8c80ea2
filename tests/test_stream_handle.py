"""The current stream's handle, also from a torch that does not hand it out
without a Stream object."""
import types

import pytest

torch = pytest.importorskip("torch")

from prismplan_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("handle,want", [(0, None), (7, 7)])
@pytest.mark.parametrize("raw", [True, False])
def test_current_stream(monkeypatch, handle, want, raw):
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(cuda_stream=handle))
    if raw:
        monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda dev: handle, raising=False)
    else:
        monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert _lib.stream_handle(None) == want


def test_given_stream():
    assert _lib.stream_handle(types.SimpleNamespace(cuda_stream=9)) == 9
