"""CTA-pair GEMM: results that leave through bulk tensor stores, at the edges of boxes, tiles and rounds of tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("width", [192, 256])
@pytest.mark.parametrize("M, K, N, act, bias", [(129, 256, 136, "gelu", True), (257, 264, 200, "", False), (300, 320, 264, "relu", True),
                                                (513, 256, 1000, "tanh", True), (250, 520, 272, "swiglu", True), (385, 256, 1040, "swiglu", False),
                                                (2600, 256, 1928, "gelu", True)])
def test_linear_pair_stores(lib, M, K, N, act, bias, width, dtype):
    """The products are added in the order of the single-CTA kernel, so the results are the same bits, and a box that reaches
    beyond the last row or column stores nothing there (y is a column slice of a wider tensor)."""
    from kernl_b200.implementations.linear_layer import linear_layer

    g = torch.Generator().manual_seed(M + N)
    x, w = torch.randn((M, K), generator=g).to(dtype).cuda(), (torch.randn((N, K), generator=g) * K ** -0.5).to(dtype).cuda()
    b = torch.randn((N,), generator=g).to(dtype).cuda() if bias else None
    n_out = N // 2 if act == "swiglu" else N
    around = torch.full((M + 2, n_out + 16), 7.0, dtype=dtype, device="cuda")
    y = around[1:M + 1, 8:8 + n_out]
    try:
        lib.kb_debug_linear_pair(0)
        lib.kb_debug_force_bn(128)
        expected = linear_layer(x, w, b, act)
        lib.kb_debug_force_bn(0)
        lib.kb_debug_linear_pair(width)
        linear_layer(x, w, b, act, out=y)
    finally:
        lib.kb_debug_force_bn(0)
        lib.kb_debug_linear_pair(1)
    assert torch.equal(y, expected)
    y.fill_(7.0)
    assert torch.equal(around, torch.full_like(around, 7.0))


@pytest.mark.parametrize("off", [1, 4])
@pytest.mark.parametrize("width, M, K, N, act", [(192, 300, 256, 200, "gelu"), (256, 300, 256, 200, ""), (256, 257, 264, 272, "swiglu"),
                                                 (192, 2000, 768, 3072, ""), (256, 2000, 768, 3072, "")])
def test_bias_that_begins_anywhere(lib, width, M, K, N, act, off):
    """A bias that does not lie at a whole 16 bytes (a slice of a longer one, through the C ABI): the same bits, and no slower stores."""
    from kernl_b200 import _lib

    g = torch.Generator().manual_seed(M + N)
    x, w = torch.randn((M, K), generator=g).half().cuda(), (torch.randn((N, K), generator=g) * K ** -0.5).half().cuda()
    b = torch.randn((N,), generator=g).half().cuda()
    shifted = torch.zeros(N + 8, dtype=torch.float16, device="cuda")
    shifted[off:off + N] = b
    n_out = N // 2 if act == "swiglu" else N
    outs = [torch.full((M, n_out), 7.0, dtype=torch.float16, device="cuda") for _ in range(2)]
    side = torch.cuda.Stream()
    graphs = []
    try:
        lib.kb_debug_linear_pair(width)
        for out, bias in zip(outs, (b.data_ptr(), shifted.data_ptr() + 2 * off)):
            p = _lib.LinearParams(x=x.data_ptr(), w=w.data_ptr(), bias=bias, y=out.data_ptr(), M=M, N=N, K=K, x_row_stride=K,
                                  y_row_stride=n_out, activation=_lib.ACTIVATIONS[act], dtype=_lib.KB_F16)
            assert lib.kb_linear_fwd(p, _lib.current_stream(x.device)) == 0
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                for _ in range(20):
                    assert lib.kb_linear_fwd(p, side.cuda_stream) == 0
            graphs.append(graph)
    finally:
        lib.kb_debug_linear_pair(1)
    assert torch.equal(outs[0], outs[1])
    if M < 2000:
        return
    best = [1e9, 1e9]  # least of several: what else the box does only adds
    for _ in range(20):
        for i, graph in enumerate(graphs):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            graph.replay()
            end.record()
            end.synchronize()
            best[i] = min(best[i], start.elapsed_time(end))
    assert best[1] < 1.25 * best[0], best  # (stores by the threads: 1.5 to 1.6 times)


@pytest.mark.parametrize("width", [192, 256])
@pytest.mark.parametrize("M, K, N, act, pre, gap", [(129, 256, 136, "gelu", True, 0), (300, 264, 1000, "relu", True, 0), (513, 256, 4000, "tanh", True, 0),
                                                    (300, 264, 1000, "gelu", False, 3), (513, 256, 131, "", False, 0), (520, 320, 4000, "relu", False, 1)])
def test_linear_pair_stored_by_threads(lib, M, K, N, act, pre, gap, width):
    """Results that bulk stores cannot take, which the narrow tile now serves too: pre-activation output, rows of y at odd places, ragged columns."""
    from kernl_b200.implementations.linear_layer import linear_layer

    g = torch.Generator().manual_seed(M + N)
    x, w = torch.randn((M, K), generator=g).half().cuda(), (torch.randn((N, K), generator=g) * K ** -0.5).half().cuda()
    b = torch.randn((N,), generator=g).half().cuda()

    def call():
        around = torch.full((M + 2, N + gap), 7.0, dtype=torch.float16, device="cuda")
        before = torch.full((M + 2, N), 7.0, dtype=torch.float16, device="cuda")
        linear_layer(x, w, b, act, act_inputs=before[1:M + 1] if pre else None, out=around[1:M + 1, :N])
        return around, before

    try:
        lib.kb_debug_linear_pair(0)
        lib.kb_debug_force_bn(128)
        expected = call()
        lib.kb_debug_force_bn(0)
        lib.kb_debug_linear_pair(width)
        got = call()
    finally:
        lib.kb_debug_force_bn(0)
        lib.kb_debug_linear_pair(1)
    for a, e in zip(got, expected):
        assert torch.equal(a, e)
