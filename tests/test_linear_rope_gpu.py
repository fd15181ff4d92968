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


@pytest.mark.parametrize("on_device", [False, True])
@pytest.mark.parametrize("B, S, H, D, start, max_seq", [
    (1, 320, 4, 128, 250, 400), (1, 320, 4, 128, 272, 400),  # the end of the cache inside a box of 32 rows, and at its edge
    (1, 300, 3, 64, -40, 400), (1, 300, 3, 64, -64, 400), (1, 300, 2, 96, -10, 200),  # the beginning; both ends
    (3, 100, 4, 128, -10, 80), (5, 64, 2, 96, 30, 70), (2, 160, 2, 64, 500, 400),  # boxes of two sequences; nothing inside
    (1, 160, 2, 64, 2 ** 32, 400), (1, 160, 2, 64, 2 ** 32 + 70, 400), (1, 160, 2, 64, 2 ** 62, 400), (1, 160, 2, 64, 2 ** 31, 400),
    (1, 160, 2, 64, 2 ** 31 - 80, 400), (1, 160, 2, 64, -2 ** 32, 400)])  # positions beyond 32 bits
def test_positions_outside_the_cache(lib, B, S, H, D, start, max_seq, on_device):
    """The fused launch leaves out the rows that the two launches leave out: of the caches and of q."""
    from kernl_b200 import _lib

    K, dtype = 256, torch.float16
    g = torch.Generator().manual_seed(S + D)
    x = torch.randn((B * S, K), generator=g).to(dtype).cuda()
    w = (torch.randn((3 * H * D, K), generator=g) * K ** -0.5).to(dtype).cuda()
    ang = torch.rand((max_seq, D // 2), generator=g) * 6.28
    cos, sin = torch.cos(ang).cuda(), torch.sin(ang).cuda()
    pos = torch.tensor([start], device="cuda")
    stream = _lib.current_stream(x.device)

    def call(fused):
        y = torch.full((B * S, 3 * H * D), 7.0, dtype=dtype, device="cuda")
        q = torch.full((B, S, H, D), 7.0, dtype=dtype, device="cuda")
        k, v = (torch.full((B, H, max_seq, D), 7.0, dtype=dtype, device="cuda") for _ in range(2))
        lin = _lib.LinearParams(x=x.data_ptr(), w=w.data_ptr(), y=y.data_ptr(), M=B * S, N=3 * H * D, K=K, x_row_stride=K, y_row_stride=3 * H * D,
                                dtype=_lib.KB_F16)
        rope = _lib.RopeParams(qkv=y.data_ptr(), q_out=q.data_ptr(), k_cache=k.data_ptr(), v_cache=v.data_ptr(), cos=cos.data_ptr(),
                               sin=sin.data_ptr(), pos_dev=pos.data_ptr() if on_device else None, pos_host=0 if on_device else start, B=B, S=S,
                               H=H, D=D, max_seq=max_seq, dtype=_lib.KB_F16)
        if fused:
            assert lib.kb_linear_rope_kv_write(lin, rope, stream) == 0
            assert bool((y == 7.0).all())  # (in one launch indeed)
        else:
            assert lib.kb_linear_fwd(lin, stream) == 0 and lib.kb_rope_kv_write(rope, stream) == 0
        return q, k, v

    try:
        lib.kb_debug_linear_pair(256)
        expected, got = call(False), call(True)
    finally:
        lib.kb_debug_linear_pair(1)
    first, last = min(max(-start, 0), S), max(min(max_seq - start, S), 0)  # the rows inside
    assert bool((got[0][:, :first] == 7.0).all()) and bool((got[0][:, max(last, first):] == 7.0).all())
    for a, b in zip(got, expected):
        assert torch.equal(a, b)
