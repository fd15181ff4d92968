"""Decode attention with the query heads of a group in one CTA: piece edges, key shares, group sizes."""
import pytest
import torch

from oracle import kernl_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D, group, N, live, masked", [
    (64, 1, 1, 1, False), (64, 4, 31, 31, True), (64, 8, 128, 33, False), (64, 12, 1100, 1100, True), (64, 1, 5000, 4097, False),
    (128, 1, 16, 15, True), (128, 4, 3000, 2999, False), (128, 9, 65, 64, False), (128, 16, 777, 777, True), (128, 20, 300, 17, False),
    (256, 1, 200, 130, False), (256, 12, 1000, 999, True),
])
def test_decode_groups(lib, dtype, D, group, N, live, masked):
    from kernl_b200.implementations.attention_skinny import skinny_attention_forward

    g = torch.Generator().manual_seed(D + N)
    B, HK = 2, 2
    q = torch.randn((B, HK * group, 1, D), generator=g).to(dtype)
    k, v = (torch.randn((B, HK, N, D), generator=g).to(dtype) for _ in range(2))
    mask = torch.randn((1, HK * group, 1, N), generator=g).to(dtype) if masked else None
    kv_len = torch.tensor([live], device="cuda")
    out = skinny_attention_forward(q.cuda(), k.cuda(), v.cuda(), torch.empty_like(q, device="cuda"), D ** -0.5, False,
                                   mask.cuda() if masked else None, kv_len=kv_len)
    kr, vr = (t[:, :, :live].repeat_interleave(group, dim=1) for t in (k, v))
    expected = O.attention(q, kr, vr, D ** -0.5, False, mask[..., :live] if masked else None)
    O.assert_parity(out, expected, max_abs=1e-2 if dtype == torch.float16 else 4e-2, what="decode groups")
