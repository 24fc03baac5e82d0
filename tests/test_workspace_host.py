"""Which scratch buffer a call gets, and how long buffers live (host logic; buffers are host memory here)."""

import contextlib
import gc
import types
import weakref

import pytest
import torch

from ternel_b200 import ops

MIB = 1 << 20


@pytest.fixture
def host(monkeypatch):
    """ops with empty tables, host buffers, and a stream and a capture state that the test sets."""
    state = types.SimpleNamespace(stream=0, capturing=False, table={})
    zeros = torch.zeros

    def set_workspace(index, *rest):
        stream, buf = rest if len(rest) == 2 else (0, rest[0])
        state.table[stream] = buf

    monkeypatch.setattr(torch, "zeros", lambda *a, device=None, **k: zeros(*a, **k))
    monkeypatch.setattr(torch.cuda, "current_stream",
                        lambda *a: types.SimpleNamespace(cuda_stream=state.stream, synchronize=lambda: None))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state.capturing)
    for context in ("device", "stream"):
        monkeypatch.setattr(torch.cuda, context, lambda *a: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "default_stream", lambda *a: None)
    monkeypatch.setattr(ops._native, "binding", lambda: types.SimpleNamespace(set_workspace=set_workspace))
    for name in ("_workspaces", "_stream_workspaces", "_replaced"):
        if hasattr(ops, name):
            monkeypatch.setattr(ops, name, type(getattr(ops, name))())
    return state


def get(nbytes):
    return ops._workspace(torch.device("cuda", 0), nbytes)


def test_a_replaced_buffer_stays_alive(host):
    """Graphs hold the addresses they were captured with, so growing must not give a buffer back. What is kept is less
    than what is in use."""
    alive, sizes = [], []
    for nbytes in (1000, 3 * MIB, 17 * MIB, 20 * MIB, 55 * MIB, 40 * MIB):
        buf = get(nbytes)
        assert buf.numel() >= nbytes and not buf.any()
        if buf.numel() not in sizes:
            alive.append(weakref.ref(buf))
            sizes.append(buf.numel())
        del buf
    gc.collect()
    assert all(ref() is not None for ref in alive)
    assert sum(sizes[:-1]) < sizes[-1]
    assert get(0) is None


def test_a_captured_call_that_needs_more_brings_its_own_buffer(host):
    """Its zero-fill is a part of the graph, so nothing outside of the graph may take the buffer for zeroed."""
    first = get(2 * MIB)
    host.capturing, host.stream = True, 7
    assert get(MIB) is first
    own = get(40 * MIB)
    assert own is not first and own.numel() >= 40 * MIB
    host.capturing, host.stream = False, 0
    assert get(2 * MIB) is first


def test_every_stream_has_a_buffer_of_its_own(host):
    """Calls on two streams may overlap. Captured calls take the default stream's buffer, however the streams were warmed up,
    and only the last few streams keep one."""
    shared = get(2 * MIB)
    host.stream = 11
    side = get(2 * MIB)
    assert side is not shared and get(MIB) is side
    larger = get(20 * MIB)                              # a warm-up on a side stream
    assert larger is not side
    host.capturing = True
    captured = get(20 * MIB)
    assert captured is not larger and captured.numel() >= 20 * MIB
    host.capturing, host.stream = False, 0
    assert get(20 * MIB) is captured
    assert host.table[0] is captured and host.table[11] is larger
    for stream in range(100, 100 + 3 * ops.MAX_STREAM_WORKSPACES):
        host.stream = stream
        get(MIB)
        host.stream = 11
        assert get(20 * MIB) is larger                  # in use all along, so it is kept
    assert len(ops._stream_workspaces) == ops.MAX_STREAM_WORKSPACES
    assert host.table[100] is None                      # let go, also where the short call path looks
    assert len([buf for buf in host.table.values() if buf is not None]) == ops.MAX_STREAM_WORKSPACES + 1
