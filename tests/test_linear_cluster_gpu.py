"""GEMM with K divided among the CTAs of a cluster: tile edges, divisions of K, the gated epilogue."""
import pytest
import torch

from oracle import kernl_oracle as O

pytestmark = pytest.mark.gpu


# bf16 keeps three bits less than fp16: eight times the bound of fp16
ATOL = {torch.float16: 1.0, torch.bfloat16: 8.0}


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("splits", [2, 3, 7, 16])
@pytest.mark.parametrize("bn", [32, 64, 0])
@pytest.mark.parametrize("M, K, N, act", [(17, 200, 129, "relu"), (65, 1032, 250, "gelu"), (130, 64, 128, ""), (128, 776, 1000, "tanh"), (250, 520, 272, "swiglu")])
def test_linear_cluster(lib, M, K, N, act, bn, splits, dtype):
    from kernl_b200.implementations.linear_layer import linear_layer

    g = torch.Generator().manual_seed(M + K)
    x = torch.randn((M, K), generator=g).to(dtype)
    w, b = (torch.randn((N, K), generator=g) * K ** -0.5).to(dtype), torch.randn((N,), generator=g).to(dtype)
    pre = None if act == "swiglu" else torch.empty((M, N), dtype=dtype, device="cuda")
    try:
        lib.kb_debug_force_splits(splits)
        lib.kb_debug_force_bn(bn)
        out, again = (linear_layer(x.cuda(), w.cuda(), b.cuda(), act, act_inputs=pre) for _ in range(2))
    finally:
        lib.kb_debug_force_splits(0)
        lib.kb_debug_force_bn(0)
    assert torch.equal(out, again)  # the parts are added in a fixed order
    z = O.linear(x, w, b, "")
    if act == "swiglu":
        z = z.reshape(M, N // 16, 2, 8)
        expected = (torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]).reshape(M, N // 2)
    else:
        expected = O.linear(x, w, b, act)
        O.assert_parity(pre, z, max_abs=1e-2 * ATOL[dtype], what="pre-activation")
    O.assert_parity(out, expected, max_abs=2e-2 * ATOL[dtype], what="cluster GEMM")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M", [33, 100, 300, 1000])
@pytest.mark.parametrize("K, N", [(72, 40), (768, 768), (1000, 504), (3072, 768), (4096, 1024)])
def test_linear_dispatch_by_size(lib, M, K, N, dtype):
    from kernl_b200.implementations.linear_layer import linear_layer

    g = torch.Generator().manual_seed(M * K)
    x, w = torch.randn((M, K), generator=g).to(dtype), (torch.randn((N, K), generator=g) * K ** -0.5).to(dtype)
    b = torch.randn((N,), generator=g).to(dtype)
    O.assert_parity(linear_layer(x.cuda(), w.cuda(), b.cuda(), "gelu"), O.linear(x, w, b, "gelu"), max_abs=1e-2 * ATOL[dtype], what="linear")
