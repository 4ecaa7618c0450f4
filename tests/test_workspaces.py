"""Workspaces are one device's: the default stream's handle is the same number on
every device, so the handle alone does not tell them apart (host-side, faked
device and stream)."""

import pytest

torch = pytest.importorskip("torch")


def test_workspace_of_each_device_and_stream(monkeypatch):
    from jaxfun_gb300 import device

    now = {"device": 0, "stream": 0}
    monkeypatch.setattr(device, "_WORKSPACES", {})
    monkeypatch.setattr(device, "device", lambda: torch.device("cpu"))
    monkeypatch.setattr(device, "stream_handle", lambda stream=None: now["stream"])
    monkeypatch.setattr(torch.cuda, "current_device", lambda: now["device"])
    seen = {}
    for now["device"] in (0, 1):
        for now["stream"] in (0, 7):
            for slot in (0, 1):
                buf = device.workspace(1000, slot)
                assert all(buf is not other for other in seen.values())
                assert device.workspace(500, slot) is buf
                seen[now["device"], now["stream"], slot] = buf
    now.update(device=0, stream=0)
    assert device.workspace(1000) is seen[0, 0, 0]
