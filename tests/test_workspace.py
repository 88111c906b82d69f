"""What a workspace keeps alive: outgrown buffers only where a captured graph may point at them."""
import weakref

import pytest
import torch

from mini_sglang_b200.parts import Workspace


def test_outgrown_buffers_are_released_unless_captured(monkeypatch):
    ws, capturing = Workspace(torch.device("cpu")), [False]
    monkeypatch.setattr(ws, "_capturing", lambda: capturing[0])

    def get(n, name="a", dtype=torch.float32):
        t = ws.get(name, n, dtype)
        assert t.numel() == n and t.dtype == dtype
        return weakref.ref(ws._bufs[name])

    first = get(100)
    assert get(50) is not None and first() is ws._bufs["a"]               # smaller requests: the same buffer
    second = get(200)
    assert first() is None and second() is not None                       # outgrown, never captured
    capturing[0] = True
    get(20)
    capturing[0] = False
    third = get(300)
    assert second() is not None and third() is not None                   # a graph holds the address of the second
    assert get(400) is not None and third() is None                       # ... and not of the third
    fourth = weakref.ref(ws._bufs["a"])
    capturing[0] = True
    fifth = get(500)                                                      # outgrown inside a capture: both stay
    capturing[0] = False
    get(600, dtype=torch.float16)
    assert fourth() is not None and fifth() is not None and second() is not None


@pytest.mark.gpu
def test_steps_of_growing_sizes_hold_the_largest_ones_scratch():
    ws = Workspace(torch.device("cuda"))
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    for n in range(1, 9):
        ws.get("a", n << 20, torch.float32)
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() - before <= (8 << 22) + (1 << 21)
    kept = ws.get("a", 4, torch.float32)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        ws.get("a", 4, torch.float32).fill_(3.0)
    torch.cuda.current_stream().wait_stream(side)
    ws.get("a", 16 << 20, torch.float32).zero_()
    kept.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert kept.tolist() == [3.0] * 4                                     # the graph's buffer is still the workspace's
