"""Which workspace a call gets, with the devices' current streams made up (no GPU needed)."""

import pytest
import torch

from fdk import native


@pytest.fixture
def two_devices(monkeypatch):
    """Device 0 is current; `streams` holds each device's current stream."""
    streams = {0: 1000, 1: 1001}
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: streams[index], raising=False)
    return streams


def test_workspace_is_that_of_the_stream_the_kernel_is_launched_on(two_devices, monkeypatch):
    buffers = {(0, 1000): torch.zeros(1), (1, 1001): torch.zeros(1), (1, 1002): torch.zeros(1)}
    monkeypatch.setattr(native, "_workspaces", buffers)
    assert native.workspace(torch.device("cuda", 0)) is buffers[0, 1000]
    assert native.workspace(torch.device("cuda")) is buffers[0, 1000]
    assert native.workspace(torch.device("cuda", 1)) is buffers[1, 1001]
    two_devices[1] = 1002
    assert native.workspace(torch.device("cuda", 1)) is buffers[1, 1002]


def test_bound_host_calls_use_the_stream_of_the_weights_device(two_devices, monkeypatch):
    buffers = {(1, 1001): torch.zeros(4)}
    monkeypatch.setattr(native, "_workspaces", buffers)
    calls = []

    class Library:
        fdk_linear_lut_host = staticmethod(lambda *args: calls.append(args) or native.OK)

    class OnDeviceOne:
        device = torch.device("cuda", 1)
        is_cuda = True

        def data_ptr(self):
            return 256

        def numel(self):
            return 64

    monkeypatch.setattr(native, "lib", lambda: Library)
    t = OnDeviceOne()
    call = native.prepare_linear_lut_host(t, t, b"", t, t, 1, 64, 64, 4, torch.bfloat16)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    call(0, 0)
    assert calls[0][-1] == 1001 and buffers[1, 1001].data_ptr() in calls[0]
