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
