"""Single-CTA GEMM with 32-column tiles: its epilogue's 16 columns per warp at ragged edges, odd alignments and every output form."""
import pytest
import torch

from oracle import kernl_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M, K, N, act, bias_at", [(1, 64, 16, "", 0), (128, 768, 96, "gelu", 0), (129, 72, 40, "relu", 0), (130, 136, 47, "tanh", 0), (65, 200, 129, "silu", 0),
                                                   (300, 64, 80, "fast_gelu", 1), (128, 264, 48, "swiglu", 0), (33, 128, 80, "swiglu", None), (257, 320, 5000, "gelu", None)])
def test_linear_narrow_tiles(lib, M, K, N, act, bias_at, dtype):
    """`bias_at`: elements between a 16-byte boundary and the bias (through the C ABI), None without one."""
    from kernl_b200 import _lib

    g = torch.Generator().manual_seed(M + N)
    x, w = torch.randn((M, K), generator=g).to(dtype), (torch.randn((N, K), generator=g) * K ** -0.5).to(dtype)
    b = None if bias_at is None else torch.randn((N,), generator=g).to(dtype)
    xc, wc = x.cuda(), w.cuda()
    bc = None if b is None else torch.cat((torch.zeros(8 + bias_at, dtype=dtype), b)).cuda()[8 + bias_at:]
    n_out = N // 2 if act == "swiglu" else N
    around = torch.full((M, n_out + 9), 7.0, dtype=dtype, device="cuda")
    pre = torch.empty((M, N), dtype=dtype, device="cuda") if act != "swiglu" else None
    for stride, y in ((n_out + 9, around), (n_out, torch.empty((M, n_out), dtype=dtype, device="cuda"))):
        pre_out = pre if stride == n_out else None  # (it shares the row stride)
        p = _lib.LinearParams(x=xc.data_ptr(), w=wc.data_ptr(), bias=None if bc is None else bc.data_ptr(), y=y.data_ptr(),
                              act_inputs=None if pre_out is None else pre_out.data_ptr(), M=M, N=N, K=K, x_row_stride=K, y_row_stride=stride,
                              activation=_lib.ACTIVATIONS[act], dtype=_lib.dtype_code(dtype))
        try:
            lib.kb_debug_force_bn(32)
            _lib.check(_lib.load().kb_linear_fwd(p, _lib.current_stream(xc.device)), "linear")
        finally:
            lib.kb_debug_force_bn(0)
        if act == "swiglu":
            z = O.linear(x, w, b, "").reshape(M, N // 16, 2, 8)
            expected = (torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]).reshape(M, n_out)
        else:
            expected = O.linear(x, w, b, act)
        atol = (1e-2 if dtype == torch.float16 else 8e-2)  # results of up to about 8: one rounding of eleven or eight bits
        O.assert_parity(y[:, :n_out], expected, max_abs=atol, what="narrow tiles")
        if pre_out is not None:
            O.assert_parity(pre, O.linear(x, w, b, ""), max_abs=atol, what="pre-activation")
    assert (around[:, n_out:] == 7.0).all()
