"""Status words that binning calls leave in page-locked memory."""

import threading
import time

import pytest
import torch

from diffsoup_b200 import tiles


def test_threads_share_one_ring(monkeypatch):
    """Four threads that make the first call together: one ring, which every one of them gets."""
    made, seen, full = [], [], torch.full

    def slow_full(*args, pin_memory, **kw):
        time.sleep(0.05)
        made.append(full(*args, **kw))
        return made[-1]

    monkeypatch.setattr(tiles, "_slots", [])
    monkeypatch.setattr(torch, "full", slow_full)
    start = threading.Barrier(4)

    def first_call():
        start.wait()
        seen.append(tiles._status_slots()[0].data_ptr())

    threads = [threading.Thread(target=first_call) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(made) == 1 and set(seen) == {made[0].data_ptr()}
