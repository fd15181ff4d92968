"""The front-ends' direct path (csrc/host_ops.cpp): plain operands go straight to the kernel, everything
that needs a copy, a conversion or an error message is left to the general path; both agree."""
import pytest
import torch

from oracle import kernl_oracle as O

pytestmark = pytest.mark.gpu


def _rand(shape, std=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(1)) * std).half().cuda()


@pytest.mark.parametrize("rows, k, shift, direct", [(5, 64, 0, True), (5, 60, 0, False), (5, 64, 4, False), (5, 64, 8, True)])
def test_linear_direct_or_general(lib, rows, k, shift, direct):
    from kernl_b200 import _lib
    from kernl_b200.implementations.linear_layer import linear_layer

    x = _rand((rows * k + shift,))[shift:].view(rows, k)  # `shift` elements off a 16-byte boundary
    w, b = _rand((48, k), 0.1), _rand((48,))
    y = _lib.native().linear(x, w, b, _lib.ACTIVATIONS["relu"], None, None)
    assert (y is not None) == direct
    O.assert_parity(linear_layer(x, w, b, "relu"), O.linear(x.cpu(), w.cpu(), b.cpu(), "relu"), what="linear")


@pytest.mark.parametrize("layout", ["contiguous", "column_major", "autocast"])
def test_attention_direct_or_general(lib, layout):
    from kernl_b200 import _lib
    from kernl_b200.implementations.attention import attention_forward

    q, k, v = (_rand((1, 2, 40, 64)) for _ in range(3))
    if layout == "column_major":
        q = q.transpose(2, 3).contiguous().transpose(2, 3)
    expected = O.attention(q.cpu(), k.cpu(), v.cpu(), 0.125)
    with torch.autocast("cuda", dtype=torch.float16, enabled=layout == "autocast"):
        direct = _lib.native().attention(q, k, v, torch.empty_like(k), 0.125, False, None)
        assert (direct is not None) == (layout == "contiguous")
        O.assert_parity(attention_forward(q, k, v, torch.empty_like(k), 0.125), expected, what=layout)
