"""The mma.sync attention kernel for short key ranges: tile and block edges, head dimensions, masks, GQA."""
import pytest
import torch

from oracle import kernl_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("mask", ["none", "pad", "row_bias", "bias", "causal"])
@pytest.mark.parametrize("M, N, D, group", [(1, 1, 64, 1), (63, 64, 64, 1), (65, 129, 64, 3), (200, 191, 40, 1), (128, 256, 128, 2), (70, 333, 80, 1),
                                            (256, 100, 16, 1), (500, 520, 64, 1), (130, 640, 112, 1)])
def test_attention_short(lib, dtype, mask, M, N, D, group):
    from kernl_b200.implementations.attention import attention_forward

    g = torch.Generator().manual_seed(M + N)
    B, HK = 2, 2
    q = torch.randn((B, M, HK * group, D), generator=g).to(dtype).transpose(1, 2)
    k, v = (torch.randn((B, HK, N, D), generator=g).to(dtype) for _ in range(2))
    m = None
    if mask == "pad":
        valid = torch.tensor([N, max(1, N // 3)])
        m = torch.where(valid[:, None] > torch.arange(N)[None, :], 0.0, float("-inf")).reshape(B, 1, 1, N).to(dtype)
    elif mask == "row_bias":
        m = torch.randn((B, HK * group, 1, N), generator=g).float()
    elif mask == "bias":
        m = torch.randn((1, HK * group, M, N), generator=g).to(dtype)
    lib.kb_debug_attention_short(1)
    try:
        out = attention_forward(q.cuda(), k.cuda(), v.cuda(), torch.empty_like(q, device="cuda"), D ** -0.5, mask == "causal",
                                m.cuda() if m is not None else None)
    finally:
        lib.kb_debug_attention_short(-1)
    kr, vr = (t.repeat_interleave(group, dim=1) for t in (k, v))
    expected = O.attention(q, kr, vr, D ** -0.5, mask == "causal", m)
    O.assert_parity(out, expected, max_abs=1e-2 if dtype == torch.float16 else 4e-2, what=f"short attention {mask}")


@pytest.mark.parametrize("M, N, D", [(300, 520, 128), (129, 1300, 80), (40, 128, 128)])
@pytest.mark.parametrize("causal", [False, True])
def test_attention_wide_heads_skip_padding(lib, M, N, D, causal):
    """Head dimensions above 64: key blocks behind a padding mask are not visited, a fully masked sequence and
    causal rows see all of them."""
    from kernl_b200.implementations.attention import attention_forward

    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn((4, 3, s, D), generator=g).half() for s in (M, N, N))
    live = torch.arange(N)[None, :] < torch.tensor([N, 1, N // 2, 0])[:, None]
    live[2, : min(130, N // 4)] = False  # masked in front too
    m = torch.where(live, 0.0, float("-inf")).reshape(4, 1, 1, N).half()
    lib.kb_debug_attention_short(0)
    try:
        out = attention_forward(q.cuda(), k.cuda(), v.cuda(), torch.empty_like(q, device="cuda"), D ** -0.5, causal, m.cuda())
    finally:
        lib.kb_debug_attention_short(-1)
    O.assert_parity(out, O.attention(q, k, v, D ** -0.5, causal, m), what="padding, wide heads")
