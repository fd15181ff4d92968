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
