"""The current stream's handle comes from torch's raw query where torch has it, else from the public call."""
import types

import pytest

from seq_vp_3d_b200 import device


def test_public_call_without_the_raw_query(monkeypatch):
    monkeypatch.setattr(device.torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=0x1234))
    for missing in ("_raw_stream", "_device"):
        with monkeypatch.context() as m:
            m.setattr(device, missing, None)
            assert device.stream_ptr().value == 0x1234
    assert device.stream_ptr(types.SimpleNamespace(cuda_stream=0x55)).value == 0x55


def test_import_without_the_raw_query(monkeypatch):
    import importlib
    monkeypatch.delattr(device.torch._C, "_cuda_getCurrentRawStream", raising=False)
    monkeypatch.setattr(device.torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=0x77))
    spec = importlib.util.spec_from_file_location("seq_vp_3d_b200.device_without_raw", device.__file__)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    assert module.stream_ptr().value == 0x77


@pytest.mark.gpu
def test_raw_query_is_the_current_stream():
    import torch
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            assert (device.stream_ptr().value or 0) == torch.cuda.current_stream().cuda_stream
