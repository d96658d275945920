"""The workspace sizes that the Python layer keeps (bulk_b200/algorithms.py) are
kept by device, and asked for with that device current: a reduce's workspace
grows with the SMs of its device.  Runs on the host, with stand-ins for the
devices and the library."""
from __future__ import annotations

import contextlib

import pytest
import torch

from bulk_b200 import algorithms


@pytest.fixture
def two_devices(monkeypatch):
    current = [0]
    asked = []

    @contextlib.contextmanager
    def device(index):
        was, current[0] = current[0], index if isinstance(index, int) else index.index
        try:
            yield
        finally:
            current[0] = was

    def workspace_bytes(algo, key, value, n):
        asked.append((current[0], algo, n))
        return 256 + 1000 * (current[0] + 1)

    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: current[0])
    monkeypatch.setattr(algorithms, "workspace_bytes", workspace_bytes)
    algorithms._need_bytes.cache_clear()
    yield asked
    algorithms._need_bytes.cache_clear()


def test_sizes_are_those_of_the_calls_device(two_devices):
    first, second = torch.device("cuda", 0), torch.device("cuda", 1)
    for _ in range(2):
        assert algorithms._need(first, "reduce", "f32", None, 1000) == 1256
        assert algorithms._need(second, "reduce", "f32", None, 1000) == 2256
    assert two_devices == [(0, "reduce", 1000), (1, "reduce", 1000)]  # each asked once
