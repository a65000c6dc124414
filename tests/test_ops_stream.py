"""Where operator calls take torch's current stream from (no GPU needed)."""
import types

from cera_b200 import ops


def test_raw_handle_of_the_current_device(monkeypatch):
    monkeypatch.setattr(ops, "_device", lambda: 3)
    monkeypatch.setattr(ops, "_raw_stream", lambda device: 0x1000 + device)
    assert ops._stream().value == 0x1003


def test_a_torch_without_the_raw_handle(monkeypatch):
    monkeypatch.setattr(ops, "_raw_stream", None)
    monkeypatch.setattr(ops.torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=0x2000))
    assert ops._stream().value == 0x2000
