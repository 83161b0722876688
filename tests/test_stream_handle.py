"""The stream that native work is ordered on, with and without torch's private call."""

from types import SimpleNamespace

from pyturb_gb300 import backend


def fake_torch(raw):
    cuda = SimpleNamespace(current_device=lambda: 3,
                           current_stream=lambda: SimpleNamespace(cuda_stream=0x77))
    return SimpleNamespace(_C=SimpleNamespace(**raw), cuda=cuda)


def test_raw_handle_of_the_current_device(monkeypatch):
    torch = fake_torch({"_cuda_getCurrentRawStream": lambda device: 0x40 + device})
    monkeypatch.setattr(backend, "torch_module", lambda: torch)
    assert backend.stream_handle() == 0x43


def test_public_stream_where_torch_lacks_the_private_call(monkeypatch):
    torch = fake_torch({})
    monkeypatch.setattr(backend, "torch_module", lambda: torch)
    assert backend.stream_handle() == 0x77
