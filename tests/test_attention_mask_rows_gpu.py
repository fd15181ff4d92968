"""Per-row masks at head dimension 64, staged row by row: where a row starts and ends in its 16-byte chunks."""
import pytest
import torch

from oracle import kernl_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shift", range(8))
@pytest.mark.parametrize("M, N, gap", [(130, 333, 0), (128, 64, 8), (9, 65, 3), (257, 455, 1)])
def test_staged_mask_rows(lib, dtype, shift, M, N, gap):
    """The mask is a view into a larger buffer that holds NaN everywhere else, `shift` elements off a 16-byte boundary
    and with `gap` elements between its rows."""
    from kernl_b200.implementations.attention import attention_forward

    g = torch.Generator().manual_seed(M + shift)
    H, row = 2, N + gap
    q, k, v = (torch.randn((2, H, s, 64), generator=g).to(dtype) for s in (M, N, N))
    buffer = torch.full((16 + H * M * row + 16,), float("nan"), dtype=dtype)
    strides = (0, M * row, row, 1)
    values = torch.randn((1, H, M, N), generator=g).to(dtype)
    values[:, :, :, N // 2] = float("-inf")
    buffer.as_strided((1, H, M, N), strides, 8 + shift).copy_(values)
    on_gpu = buffer.cuda()
    mask = on_gpu.as_strided((1, H, M, N), strides, 8 + shift)
    lib.kb_debug_attention_short(0)
    try:
        out = attention_forward(q.cuda(), k.cuda(), v.cuda(), torch.empty_like(q, device="cuda"), 0.125, False, mask)
    finally:
        lib.kb_debug_attention_short(-1)
    O.assert_parity(out, O.attention(q, k, v, 0.125, False, values), max_abs=1e-2 if dtype == torch.float16 else 3e-2, what="staged mask")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kind, B, H, M, N", [("float32", 13, 12, 257, 130), ("apart", 13, 12, 257, 130), ("float32", 2, 3, 130, 333), ("apart", 2, 3, 130, 65),
                                              ("negative", 13, 12, 257, 130), ("negative", 1, 2, 130, 200), ("row", 1, 2, 140, 8200), ("row32", 1, 2, 300, 8257)])
@pytest.mark.parametrize("persistent", [-1, 0, 1])
def test_masks_that_are_not_staged(lib, dtype, kind, B, H, M, N, persistent):
    """32-bit values, values that are not side by side, a scale that is not positive, rows of more than 8192 keys: in launches of
    few tiles and of many, with a CTA per tile and with CTAs that draw their tiles."""
    from kernl_b200.implementations.attention import attention_forward

    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn((B, H, s, 64), generator=g).to(dtype) for s in (M, N, N))
    scale = -0.125 if kind == "negative" else 0.125
    mask = None
    if kind in ("float32", "apart"):
        mask = torch.randn((1, H, M, 2 * N if kind == "apart" else N), generator=g).to(dtype if kind == "apart" else torch.float32)
        mask[..., 7] = float("-inf")
    elif kind != "negative":
        mask = torch.where(torch.arange(N) < N - 300, 0.0, float("-inf")).reshape(1, 1, 1, N).to(torch.float32 if kind == "row32" else dtype)
    on_gpu = mask.cuda() if mask is not None else None
    if kind == "apart":
        mask, on_gpu = mask[..., ::2], on_gpu[..., ::2]
    lib.kb_debug_attention_short(0)
    lib.kb_debug_attention_persistent(persistent)
    try:
        out = attention_forward(q.cuda(), k.cuda(), v.cuda(), torch.empty_like(q, device="cuda"), scale, False, on_gpu)
    finally:
        lib.kb_debug_attention_short(-1)
        lib.kb_debug_attention_persistent(-1)
    O.assert_parity(out, O.attention(q, k, v, scale, False, mask), max_abs=1e-2 if dtype == torch.float16 else 3e-2, what=kind)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B, M, N, D, causal, wide", [(2, 130, 7168, 128, False, False), (2, 130, 7169, 128, False, False), (2, 300, 7300, 80, False, True),
                                                      (1, 20, 9000, 128, False, True), (1, 400, 7200, 128, True, False)])
def test_long_row_masks_at_wide_heads(lib, dtype, B, M, N, D, causal, wide):
    """Row masks up to what fits in shared memory and beyond, one tile and two per CTA, the last key block cut; a sequence
    of which every key is masked."""
    from kernl_b200.implementations.attention import attention_forward

    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn((B, 2, s, D), generator=g).to(dtype) for s in (M, N, N))
    live = torch.arange(N)[None, :] < torch.tensor([N - 200, 0])[:B, None]
    mask = torch.where(live, torch.randn((B, N), generator=g), torch.tensor(float("-inf"))).reshape(B, 1, 1, N).to(torch.float16 if not wide else torch.float32)
    if mask.dtype != torch.float16:
        mask[B - 1, 0, 0, :9] = 0.0  # (the lowest 32-bit value leaves nothing of the scores it is added to)
    lib.kb_debug_attention_short(0)
    try:
        out = attention_forward(q.cuda(), k.cuda(), v.cuda(), torch.empty_like(q, device="cuda"), D ** -0.5, causal, mask.cuda())
    finally:
        lib.kb_debug_attention_short(-1)
    O.assert_parity(out, O.attention(q, k, v, D ** -0.5, causal, mask), max_abs=1e-2 if dtype == torch.float16 else 4e-2, what="long row mask")
