"""Persistent attention: several query tiles (head dimensions above 64: pairs of them) per CTA, drawn from a device-side counter."""
import pytest
import torch

from oracle import kernl_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("layout", ["heads_first", "heads_last", "odd_rows"])  # odd_rows: no bulk stores
@pytest.mark.parametrize("B, H, HK, M, N, D, causal", [(5, 16, 16, 700, 700, 128, True), (3, 52, 13, 129, 257, 128, False), (38, 8, 2, 128, 64, 72, False),
                                                       (7, 12, 12, 513, 300, 104, True), (75, 4, 4, 385, 640, 128, False),
                                                       (5, 16, 16, 700, 700, 64, True), (30, 12, 3, 200, 130, 64, False), (25, 12, 12, 129, 77, 40, False),
                                                       (40, 8, 8, 127, 65, 24, False)])
def test_items(B, H, HK, M, N, D, causal, layout, dtype):
    from kernl_b200.implementations.attention import attention_forward

    g = torch.Generator().manual_seed(M + N)
    q, k, v = (torch.randn(s, generator=g).to(dtype) for s in ((B, H, M, D), (B, HK, N, D), (B, HK, N, D)))
    if layout == "heads_last":
        around = torch.full((B, M + 1, H, D), 7.0, dtype=dtype, device="cuda")
        o = around[:, :M].transpose(1, 2)
    else:
        around = torch.full((B, H, M + 1, D + (3 if layout == "odd_rows" else 8)), 7.0, dtype=dtype, device="cuda")
        o = around[:, :, :M, :D]
    attention_forward(q.cuda(), k.cuda(), v.cuda(), o, D ** -0.5, causal, None)
    again = attention_forward(q.cuda(), k.cuda(), v.cuda(), torch.empty((B, H, M, D), dtype=dtype, device="cuda"), D ** -0.5, causal, None)
    assert torch.equal(o, again)  # whoever draws an item, and however it is stored
    expected = O.attention(q, k, v, D ** -0.5, causal, None)
    O.assert_parity(o, expected, max_abs=1e-2 if dtype == torch.float16 else 4e-2, what="attention")
    o.fill_(7.0)
    assert torch.equal(around, torch.full_like(around, 7.0))


@pytest.mark.parametrize("layout", ["bulk", "odd_rows"])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [72, 128])
@pytest.mark.parametrize("more", [-1, 0, 1])
def test_as_many_items_as_sms(lib, more, D, causal, layout):
    """One item per CTA up to as many as there are SMs, CTAs that stay above: the same bits for the heads that both launches have."""
    from kernl_b200.implementations.attention import attention_forward

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    H = sms // 2 + more  # two pairs of tiles per head
    g = torch.Generator(device="cuda").manual_seed(D + more)
    q, k, v = (torch.randn((1, H + 40, 300, D), generator=g, device="cuda").half() for _ in range(3))

    def call(heads):
        o = torch.full((1, heads, 301, D + (3 if layout == "odd_rows" else 8)), 7.0, dtype=torch.float16, device="cuda")
        attention_forward(q[:, :heads], k[:, :heads], v[:, :heads], o[:, :, :300, :D], D ** -0.5, causal, None)
        return o

    few, many = call(H), call(H + 40)
    assert torch.equal(few, many[:, :H])
    assert bool((few[:, :, 300] == 7.0).all()) and bool((few[:, :, :, D:] == 7.0).all())
    O.assert_parity(few[:, :3, :300, :D], O.attention(q[:, :3].cpu(), k[:, :3].cpu(), v[:, :3].cpu(), D ** -0.5, causal, None), what="attention")
