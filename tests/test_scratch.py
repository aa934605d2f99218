"""The scratch and staging buffers of the host path around CUDA graphs, with the device calls replaced: which buffer a call gets, when it
is cleared, and that no buffer a graph may write goes back to the allocator.  CPU only."""
import gc
import weakref

import pytest
import torch

from gguf_jax_b200 import _backend, _lib

MB = 1 << 20


class Device:
    """Allocations, the running capture (0: none) and the buffers the native call path was given."""

    def __init__(self):
        self.capture, self.cleared, self.native_scratch = 0, [], {}

    def zeros(self, n, **_):
        t = torch.ones(n, dtype=torch.uint8)
        self.cleared.append((t.data_ptr(), self.capture))
        return t

    def set_scratch(self, dev, stream, t):
        self.native_scratch[dev, stream] = t

    def capture_id(self, stream):
        return self.capture


@pytest.fixture
def device(monkeypatch):
    d = Device()
    empty = torch.empty
    monkeypatch.setattr(_lib, "native", lambda: d)
    monkeypatch.setattr(torch, "zeros", d.zeros)
    monkeypatch.setattr(torch, "empty", lambda n, **_: empty(n, dtype=torch.uint8))
    monkeypatch.setattr(_backend, "_workspaces", _backend._Buffers(1 << 20, zeroed=True, publish=True))
    monkeypatch.setattr(_backend, "_stagings", _backend._Buffers(1 << 16, zeroed=False, publish=False))
    return d


def test_scratch_first_taken_by_a_capture_belongs_to_that_capture(device):
    device.capture = 7
    a = _backend.workspace(0, 5 * MB, 11, 5 * MB)
    assert (a.data_ptr(), 7) in device.cleared                       # cleared on every replay, before its first use
    assert _backend.workspace(0, 5 * MB, 11, 5 * MB) is a            # and once only
    device.capture = 8                                               # another graph, captured before the first has run
    b = _backend.workspace(0, 5 * MB, 11, 5 * MB)
    assert b is not a and (b.data_ptr(), 8) in device.cleared
    device.capture = 0                                               # and a call outside any
    c = _backend.workspace(0, 5 * MB, 11, 5 * MB)
    assert c is not a and c is not b and (c.data_ptr(), 0) in device.cleared
    assert device.native_scratch == {(0, 11): c}


def test_a_capture_uses_the_streams_scratch_where_it_is_large_enough(device):
    a = _backend.workspace(0, 5 * MB, 11, 5 * MB)
    device.capture = 7
    assert _backend.workspace(0, 2 * MB, 11, 2 * MB) is a
    assert _backend.workspace(0, 9 * MB, 11, 4 * MB) is a            # the least that will do
    assert _backend.workspace(0, 9 * MB, 12, 0) is None              # or nothing
    big = _backend.workspace(0, 9 * MB, 11)
    assert big.numel() >= 9 * MB and _backend.workspace(0, 9 * MB, 11, 1 * MB) is big
    assert len(device.cleared) == 2


@pytest.mark.parametrize("get", [lambda n: _backend.workspace(0, n, 11, n), lambda n: _backend.staging(0, n, 11)], ids=["workspace", "staging"])
def test_a_buffer_a_graph_uses_outlives_its_replacement(device, get):
    first = weakref.ref(get(2 * MB))
    get(3 * MB)
    gc.collect()
    device.native_scratch.clear()
    assert first() is None                                            # no graph knows it
    seen, size = [], 4 * MB
    for capture in range(1, 41):
        device.capture = capture
        buf = get(size)
        seen.append(weakref.ref(buf))
        device.capture = 0
        size += 1 * MB
        buf = get(size)
    del buf
    device.native_scratch.clear()
    gc.collect()
    current = get(1)
    in_graphs = [r() for r in seen[1:]]                               # (the first was the capture's own)
    assert all(t is not None for t in in_graphs)
    kept = {t.data_ptr(): t.numel() for t in in_graphs if t is not current}
    assert 0 < sum(kept.values()) < current.numel()                   # bounded by the size of the current one


def test_staging_first_taken_by_a_capture_is_not_used_outside(device):
    device.capture = 7
    a = _backend.staging(0, 1 * MB, 11)
    device.capture = 0
    assert _backend.staging(0, 1 * MB, 11) is not a
