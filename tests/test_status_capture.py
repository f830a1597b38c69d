"""No status word is posted from a graph: what counts is the stream of the call's own device, whichever is current."""

import contextlib
import types

import pytest
import torch

from rbf_attention_b200 import _lib, ops


@pytest.fixture
def rings(monkeypatch):
    """Rings of two devices; ``capturing`` holds the devices whose stream is being captured, device 0 is the current one."""
    capturing, entered = set(), []

    @contextlib.contextmanager
    def on_device(device):
        entered.append(device.index)
        yield
        entered.pop()

    library = types.SimpleNamespace(rbf_b200_map_status_slots=lambda *a: 0, rbf_b200_last_error=lambda: b"refused",
                                    rbf_b200_post_device_status=lambda ws, slot, stream: posted.append((entered[-1], slot)) or 0)
    posted = []
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t: t)
    monkeypatch.setattr(ops, "_OnDevice", on_device)
    monkeypatch.setattr(ops, "_stream_ptr", lambda device: 0)
    monkeypatch.setattr(ops._lib, "load", lambda: library)
    monkeypatch.setattr(ops._lib, "host", lambda: types.SimpleNamespace(capturing=lambda index: index in capturing))
    monkeypatch.setattr(torch._C, "_cuda_isCurrentStreamCapturing", lambda: 0 in capturing, raising=False)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: 0 in capturing)
    rings = [ops._StatusMonitor(torch.device("cuda", i)) for i in range(2)]
    for ring in rings:
        ring.mapped = 1 << 20
    return rings, capturing, posted


@pytest.mark.parametrize("captured", [0, 1])
def test_the_calls_own_device_decides(rings, captured):
    rings, capturing, posted = rings
    capturing.add(captured)
    for device, ring in enumerate(rings):
        slots = []
        ring.launch("call", lambda slot: slots.append(slot) or 0)
        ring.record(torch.zeros(4), "call")
        if device == captured:
            assert slots == [0] and not ring.pending and not posted
        else:
            assert slots[0] >= ring.mapped and len(ring.pending) == 2
            assert [on for on, _ in posted] == [device]
        posted.clear()


def test_the_extension_asks_a_devices_stream(built_library):
    host = _lib.host()
    if not torch.cuda.is_available():
        assert host.capturing(0) is False and host.capturing(3) is False
    with pytest.raises(TypeError):
        host.capturing("cuda")


@pytest.mark.gpu
def test_the_extension_sees_a_capture():
    host = _lib.host()
    assert not host.capturing(0)
    x = torch.zeros(8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert host.capturing(0)
        x += 1
    assert not host.capturing(0)
    del graph
