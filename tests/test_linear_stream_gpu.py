"""The few-row linear kernel (M <= 32): tile heights, K pieces, ragged edges, the gated epilogue."""
import pytest
import torch

from oracle import kernl_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32, 33])
@pytest.mark.parametrize("K, N, act", [(8, 1, ""), (72, 50, "relu"), (200, 4736, "gelu"), (256, 7105, ""), (520, 14000, "tanh"),
                                       (64, 4752, "swiglu"), (448, 11024, "swiglu")])
def test_few_row_linear(lib, dtype, M, K, N, act):
    from kernl_b200.implementations.linear_layer import interleave_gate_up, linear_layer

    g = torch.Generator().manual_seed(M * 7 + K)
    x = torch.randn((M, K), generator=g).to(dtype)
    w = (torch.randn((N, K), generator=g) * K ** -0.5).to(dtype)
    b = torch.randn((N,), generator=g).to(dtype)
    if act == "swiglu":
        wg, wu, bg, bu = w[: N // 2], w[N // 2:], b[: N // 2], b[N // 2:]
        out = linear_layer(x.cuda(), interleave_gate_up(wg, wu).cuda(), interleave_gate_up(bg, bu).cuda(), act)
        gate = torch.nn.functional.linear(x.float(), wg.float(), bg.float())
        expected = torch.nn.functional.silu(gate) * torch.nn.functional.linear(x.float(), wu.float(), bu.float())
    else:
        pre = torch.empty((M, N), dtype=dtype, device="cuda")
        out = linear_layer(x.cuda(), w.cuda(), b.cuda(), act, act_inputs=pre)
        expected = O.linear(x, w, b, act)
        O.assert_parity(pre, O.linear(x, w, b, ""), max_abs=1e-2 if dtype == torch.float16 else 6e-2, what="pre-activation")
    # bf16: half an ulp of the largest value is 2^-9 of it
    O.assert_parity(out, expected, max_abs=max(1e-2, 0.0 if dtype == torch.float16 else float(expected.abs().max()) / 200), what="few-row linear")
