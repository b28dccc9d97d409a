"""Status words that binning calls leave in page-locked memory."""

import threading
import time

import pytest
import torch

import diffsoup_b200 as ds
from diffsoup_b200 import scenes, tiles, viewer


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


@pytest.mark.gpu
def test_a_frame_reads_its_own_status():
    """render() takes no word of the ring, which other threads' calls may come round to while it waits, and grows
    on an overflow of its own alone."""
    vi = scenes.make_viewer_inputs(2, seed=5, level=3, num_tris=500, num_views=1, resolution=(64, 80))
    (W1, b1), (W2, b2), (W3, b3) = vi.mlp
    r = viewer.Renderer(vi.verts, vi.faces, vi.lut0, vi.lut1, W1, b1, W2, b2, W3, b3, level=vi.level)
    want = r.render(vi.mvps, 64, 80)
    frame = r._frame(1, 64, 80)
    capacity, words = frame.capacity, tiles._status_slots()[1]
    words[:] = [77] * len(words)
    assert torch.equal(r.render(vi.mvps, 64, 80), want) and frame.capacity == capacity
    frame.capacity = 8
    frame._alloc()
    assert torch.equal(r.render(vi.mvps, 64, 80), want) and frame.capacity == 16
    assert set(words) == {77}


@pytest.mark.gpu
def test_replays_leave_the_ring_alone():
    """A captured call's replays write into no word of the ring, which later calls have by then."""
    sc = scenes.make_scene(2, seed=2, num_tris=300, num_views=1, resolution=(48, 64), with_targets=False)
    pos = torch.from_numpy(sc.clip_positions()).cuda()
    tri, alpha = torch.from_numpy(sc.tri).cuda(), torch.rand(sc.T, 15, 1, device="cuda")
    call = lambda: ds.rasterize_multires_triangle_alpha((48, 64), pos, tri, 2, alpha, stochastic=False)  # noqa: E731
    want = call()
    graph = torch.cuda.CUDAGraph()
    tiles._last = None
    with torch.cuda.graph(graph):
        got = call()
    words = tiles._status_slots()[1]
    words[:] = [77] * len(words)
    got.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and set(words) == {77}
    call()
