"""The stream handle with and without torch's private raw-stream call (host only: the
CUDA side is a stand-in)."""
import pytest

from flint_gb300 import native

torch = pytest.importorskip("torch")


@pytest.fixture
def cuda(monkeypatch):
    monkeypatch.setattr(native, "_raw_stream", None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: type("S", (), {"cuda_stream": 1000 + dev}))
    return monkeypatch


def test_raw_call(cuda):
    cuda.setattr(torch._C, "_cuda_getCurrentRawStream", lambda dev: 2000 + dev, raising=False)
    assert native.current_stream().value == 2003


def test_public_call_where_the_raw_one_is_missing(cuda):
    cuda.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    assert native.current_stream().value == 1003
