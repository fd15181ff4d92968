"""q/k/v projection with the rotary embedding and the cache write in its epilogue, against the projection and the kernel behind it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("on_device", [False, True])
@pytest.mark.parametrize("pair", [0, 1, 256])
@pytest.mark.parametrize("B, S, H, D, K, start, max_seq", [
    (8, 1, 4, 128, 512, 37, 40), (13, 1, 3, 40, 200, 0, 8), (1, 16, 2, 64, 264, 30, 40), (33, 1, 4, 96, 320, 7, 8),  # few rows: two launches; (1, 16): past the end
    (3, 100, 4, 128, 256, 0, 100), (5, 64, 2, 96, 264, 3, 70), (2, 300, 3, 64, 512, 0, 320), (4, 33, 4, 40, 256, 0, 40),  # rows of two sequences in a box
    (1, 640, 8, 128, 256, 10, 700)])
def test_linear_rope_kv_write(lib, B, S, H, D, K, start, max_seq, pair, on_device, dtype):
    from kernl_b200.implementations.linear_layer import linear_layer
    from kernl_b200.implementations.rope import linear_rope_kv_write, rope_kv_write

    g = torch.Generator().manual_seed(B * S + D)
    x = torch.randn((B * S, K), generator=g).to(dtype).cuda()
    w = (torch.randn((3 * H * D, K), generator=g) * K ** -0.5).to(dtype).cuda()
    ang = torch.rand((max_seq, D // 2), generator=g) * 6.28
    cos, sin = torch.cos(ang).cuda(), torch.sin(ang).cuda()
    pos = torch.tensor([start], device="cuda") if on_device else start
    caches = [torch.full((B, H, max_seq, D), 7.0, dtype=dtype, device="cuda") for _ in range(4)]
    try:
        lib.kb_debug_linear_pair(pair)
        expected = rope_kv_write(linear_layer(x, w, None), caches[0], caches[1], cos, sin, pos, B, S)
        q = linear_rope_kv_write(x, w, caches[2], caches[3], cos, sin, pos, B, S)
    finally:
        lib.kb_debug_linear_pair(1)
    n = min(S, max_seq - start)  # positions beyond the cache are left out
    assert torch.equal(q[:, :n], expected[:, :n]) and torch.equal(caches[2], caches[0]) and torch.equal(caches[3], caches[1])
    assert (caches[2][:, :, :start] == 7.0).all() and (caches[3][:, :, start + n:] == 7.0).all()
