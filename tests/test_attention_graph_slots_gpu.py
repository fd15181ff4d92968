"""Persistent attention in a captured graph: its replays share no work queue with calls that other streams make meanwhile."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D, S", [(128, 300), (64, 700)])
def test_replay_beside_calls(lib, D, S):
    from kernl_b200.implementations.attention import attention_forward

    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn((6, 16, S, D), generator=g, device="cuda").half() for _ in range(3))
    expected = attention_forward(q, k, v, torch.empty_like(q), D ** -0.5, True, None)
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    o = torch.empty_like(q)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        attention_forward(q, k, v, o, D ** -0.5, True, None)
    outs = [torch.empty_like(q) for _ in range(4)]
    torch.cuda.synchronize()
    for i in range(1200):  # more calls than eager launches have queues
        if i % 8 == 0:
            with torch.cuda.stream(side):
                graph.replay()
        with torch.cuda.stream(other):
            attention_forward(q, k, v, outs[i % 4], D ** -0.5, True, None)
    torch.cuda.synchronize()
    assert torch.equal(o, expected) and all(torch.equal(t, expected) for t in outs)


def _captured(call, times, stream):
    graph = torch.cuda.CUDAGraph()
    slots = []
    with torch.cuda.graph(graph, stream=stream):
        for _ in range(times):
            slots.append(call())
    return graph, slots


def _wait_for(condition):
    import time

    end = time.monotonic() + 10.0
    while not condition() and time.monotonic() < end:  # (a graph's slots come back on a thread of the CUDA runtime)
        time.sleep(0.01)
    return condition()


@pytest.mark.parametrize("D, S", [(128, 300), (64, 700)])
def test_captured_launches_own_their_slots(lib, D, S):
    """A captured launch has a slot of its own, which no eager launch and no other live graph takes, and which comes back with its graph.
    Where all are owned a launch takes the form that needs none."""
    from kernl_b200.implementations.attention import attention_forward

    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn((6, 16, S, D), generator=g, device="cuda").half() for _ in range(3))
    few = [t[:1, :4].contiguous() for t in (q, k, v)]  # no more tiles than CTAs: nothing to draw

    def call(o=None, args=(q, k, v)):
        attention_forward(*args, torch.empty_like(args[0]) if o is None else o, D ** -0.5, True, None)
        return lib.kb_debug_attention_slots(0, 0)

    expected = torch.empty_like(q)
    eager = [call(expected) for _ in range(1030)]  # once around the eager ring
    assert all(0 <= s < 1024 and s == (eager[0] + i) % 1024 for i, s in enumerate(eager))
    assert call(None, few) == eager[-1]  # took none
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    torch.cuda.synchronize()
    before = lib.kb_debug_attention_slots(1, 0)
    first, a = _captured(call, 40, side)
    second, b = _captured(call, 40, side)
    assert all(s >= 1024 for s in a + b) and len(set(a + b)) == 80 and lib.kb_debug_attention_slots(1, 0) == before + 80
    first.replay()
    second.replay()
    torch.cuda.synchronize()
    del first
    assert _wait_for(lambda: lib.kb_debug_attention_slots(1, 0) == before + 40)
    third, c = _captured(call, 60, side)  # (those of the first graph are free again)
    assert not set(c) & set(b) and len(set(c)) == 60
    del second, third
    assert _wait_for(lambda: lib.kb_debug_attention_slots(1, 0) == before)
    try:
        lib.kb_debug_attention_slots(2, 0)
        o = torch.empty_like(q)
        graph, d = _captured(lambda: call(o), 1, side)
        assert d == [c[-1]] and lib.kb_debug_attention_slots(1, 0) == before  # took none
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(o, expected)
    finally:
        lib.kb_debug_attention_slots(2, -1)
