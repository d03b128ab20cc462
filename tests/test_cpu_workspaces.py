"""Whose a workspace is: its counters are at zero between launches only for launches that come one after the other."""
import threading

import pytest
import torch

from proxy_inference_engine_b200 import ops

CPU = torch.device("cpu")


@pytest.fixture
def at(monkeypatch):
    """The stream and the capture that a call finds itself on."""
    now = threading.local()
    monkeypatch.setattr(ops, "_raw_stream", lambda index: getattr(now, "stream", 0))
    monkeypatch.setattr(ops, "_capturing", lambda: getattr(now, "capture", 0) != 0)
    monkeypatch.setattr(ops, "_capture_id", lambda: getattr(now, "capture", 0))

    def move(stream=0, capture=0):
        now.stream, now.capture = stream, capture
    return move


def test_a_stream_has_its_own(at):
    w = ops._Workspaces()
    first = w.get("attn", 1000, CPU)
    assert w.get("attn", 1000, CPU) is first and w.get("qmv", 1000, CPU) is not first
    at(stream=1)
    other = w.get("attn", 1000, CPU)
    assert other is not first and not other.any()
    at(stream=0)
    assert w.get("attn", 500, CPU) is first


def test_a_thread_has_its_own(at):
    w, got = ops._Workspaces(), []
    first = w.get("attn", 1000, CPU)
    t = threading.Thread(target=lambda: got.append(w.get("attn", 1000, CPU)))
    t.start()
    t.join()
    assert got[0] is not first


def test_a_capture_has_its_own(at):
    """An eager call never sees a buffer whose zeros are only recorded, and a graph never one that a larger eager call replaces."""
    w = ops._Workspaces()
    eager = w.get("attn", 1000, CPU)
    at(stream=3, capture=7)
    captured = w.get("attn", 1000, CPU)
    new = w.get("first in a capture", 1000, CPU)
    assert captured is not eager and w.get("attn", 1000, CPU) is captured
    at()
    assert w.get("attn", 1000, CPU) is eager and w.get("first in a capture", 1000, CPU) is not new
    at(stream=3, capture=8)
    assert w.get("attn", 1000, CPU) is not captured


def test_they_are_bounded(at):
    w = ops._Workspaces()
    for i in range(3 * w.KEEP):
        w.get(i, 256, CPU)
    assert len(w.mine.eager) == w.KEEP
    last = w.get(3 * w.KEEP - 1, 256, CPU)
    assert w.get(3 * w.KEEP - 1, 256, CPU) is last and w.get(3 * w.KEEP - 1, 512, CPU).numel() == 512 and len(w.mine.eager) == w.KEEP
