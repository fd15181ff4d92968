"""A bounded device-side wait that runs out: the kernel gives up, records it, and returns.

One GPU, one kernel, no fault: rank 0 of a two-rank all-reduce is launched alone with a wait limit
of a few thousand cycles, so the flag that its (absent) peer would set never arrives and the wait
expires. The kernel neither traps nor hangs; the host finds KB_ERR_TIMEOUT in the status word,
kernels launched before the word is read do no work, and after the read everything works again.
"""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _params(bufs, flags, residual, out, rank=0):
    from kernl_b200 import _lib

    p = _lib.AllReduceParams()
    for r in range(2):
        p.partials[r] = bufs[r].data_ptr()
        p.flags[r] = flags[r].data_ptr()
    p.residual, p.out, p.count = residual.data_ptr(), out.data_ptr(), out.numel()
    p.rank, p.world, p.dtype = rank, 2, _lib.KB_BF16
    return p


def test_expired_wait_sets_the_status_word_and_the_library_recovers(lib):
    from kernl_b200 import _lib
    from kernl_b200.implementations.attention import attention_forward
    from oracle import kernl_oracle as O

    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(0)
    bufs = [torch.randn(4096, generator=g).bfloat16().to(dev) for _ in range(2)]
    flags = [torch.zeros(64, dtype=torch.int32, device=dev) for _ in range(2)]  # "rank 1" is just more memory here
    residual = torch.randn(4096, generator=g).bfloat16().to(dev)
    out = torch.zeros(4096, dtype=torch.bfloat16, device=dev)
    stream = _lib.current_stream(dev)
    _lib.device_status()
    assert lib.kb_debug_wait_limit(20000, 20000) == 0
    try:
        # rank 0 alone: nobody sets its "ready" flag, the wait of ~20 000 cycles runs out
        assert lib.kb_allreduce_residual_fwd(_params(bufs, flags, residual, out), stream) == 0
        # a kernel launched while the word is set skips its work
        q = torch.randn((1, 2, 128, 64), generator=g).half().to(dev)
        sentinel = torch.full_like(q, 7.0)
        attention_forward(q, q, q, sentinel, 0.125, False, None)
        with pytest.raises(RuntimeError, match="wait expired") as info:
            _lib.device_status()
        word = [int(x) for x in info.value.args[0].split("word = ")[1].strip("[]").split(",")]
        assert word[0] == 1 and 500 <= word[1] < 600, word  # the all-reduce's flag waits are sites 500..579
        assert torch.equal(sentinel, torch.full_like(q, 7.0)), "a kernel ran although a wait had expired"
    finally:
        assert lib.kb_debug_wait_limit(0, 0) == 0  # defaults back
    assert _lib.device_status()[0] == 0
    # after the read: ordinary kernels work again ...
    fresh = attention_forward(q, q, q, torch.empty_like(q), 0.125, False, None)
    O.assert_parity(fresh, O.attention(q.cpu(), q.cpu(), q.cpu(), 0.125))
    # ... and so does the all-reduce once its peer's flags arrive. The peer is played by the host:
    # the call that gave up closed epoch 1, so the next one waits for 2 in "ready" and "done".
    assert int(flags[0][16]) == 1
    flags[0][1] = 2
    flags[0][8 + 1] = 2
    torch.cuda.synchronize()
    assert lib.kb_allreduce_residual_fwd(_params(bufs, flags, residual, out), stream) == 0
    assert _lib.device_status()[0] == 0
    want = (bufs[0].float() + bufs[1].float() + residual.float()).bfloat16()
    assert torch.equal(out, want)


@pytest.mark.parametrize("kernel", ["gemm_single", "gemm_pair", "gemm_cluster", "attn_d128", "attn_split", "attn_persistent", "attn_short"])
def test_kernels_with_waits_store_nothing_after_an_expiry(lib, kernel):
    from kernl_b200 import _lib
    from kernl_b200.implementations.attention import attention_forward
    from kernl_b200.implementations.linear_layer import linear_layer

    dev = torch.device("cuda", 0)
    bufs = [torch.zeros(4096, dtype=torch.bfloat16, device=dev) for _ in range(2)]
    flags = [torch.zeros(64, dtype=torch.int32, device=dev) for _ in range(2)]
    out = torch.zeros(4096, dtype=torch.bfloat16, device=dev)
    if kernel.startswith("gemm"):
        x, w = torch.randn((600, 256), device=dev).half(), torch.randn((512, 256), device=dev).half()
        result = torch.full((600, 512), 7.0, dtype=torch.float16, device=dev)
        call = lambda: linear_layer(x, w, None, "", out=result)
    else:
        q = torch.randn((2, 2, 300, 128 if kernel == "attn_d128" else 64), device=dev).half()
        result = torch.full_like(q, 7.0)
        call = lambda: attention_forward(q, q, q, result, 0.1)
    hooks = {"gemm_single": [(lib.kb_debug_force_bn, 64, 0)], "gemm_pair": [(lib.kb_debug_linear_pair, 256, 1)],
             "gemm_cluster": [(lib.kb_debug_force_splits, 2, 0)], "attn_persistent": [(lib.kb_debug_attention_persistent, 1, -1)],
             "attn_short": [(lib.kb_debug_attention_short, 1, -1)], "attn_d128": [(lib.kb_debug_attention_short, 0, -1)],
             "attn_split": [(lib.kb_debug_attention_short, 0, -1), (lib.kb_debug_attention_persistent, 0, -1)]}[kernel]
    _lib.device_status()
    for hook, on, _ in hooks:
        hook(on)
    try:
        call()  # (the kernel's one-time set-up is not part of the test)
        result.fill_(7.0)
        assert lib.kb_debug_wait_limit(0, 20000) == 0
        assert lib.kb_allreduce_residual_fwd(_params(bufs, flags, out, out), _lib.current_stream(dev)) == 0
        call()
        with pytest.raises(RuntimeError, match="wait expired"):
            _lib.device_status()
        assert bool((result == 7.0).all())
        call()
        assert _lib.device_status()[0] == 0 and not bool((result == 7.0).all())
    finally:
        assert lib.kb_debug_wait_limit(0, 0) == 0
        for hook, _, off in hooks:
            hook(off)


@pytest.mark.parametrize("D, shape", [(128, (10, 16, 300)), (64, (6, 16, 700))])
def test_queues_are_clean_after_an_expiry(lib, D, shape):
    """Launches that draw their tiles from a counter put it back also when they skip their work: every slot of the ring serves a full
    launch afterwards."""
    from kernl_b200 import _lib
    from kernl_b200.implementations.attention import attention_forward

    dev = torch.device("cuda", 0)
    bufs = [torch.zeros(4096, dtype=torch.bfloat16, device=dev) for _ in range(2)]
    flags = [torch.zeros(64, dtype=torch.int32, device=dev) for _ in range(2)]
    out = torch.zeros(4096, dtype=torch.bfloat16, device=dev)
    g = torch.Generator(device="cuda").manual_seed(D)
    B, H, S = shape
    q = torch.randn((B, H, S, D), generator=g, device=dev).half()
    expected = attention_forward(q, q, q, torch.empty_like(q), D ** -0.5, True, None)
    skipped = torch.full_like(q, 7.0)
    _lib.device_status()
    try:
        assert lib.kb_debug_wait_limit(0, 20000) == 0
        assert lib.kb_allreduce_residual_fwd(_params(bufs, flags, out, out), _lib.current_stream(dev)) == 0
        for _ in range(3):
            attention_forward(q, q, q, skipped, D ** -0.5, True, None)
        slot = lib.kb_debug_attention_slots(0, 0)
        with pytest.raises(RuntimeError, match="wait expired"):
            _lib.device_status()
    finally:
        assert lib.kb_debug_wait_limit(0, 0) == 0
    assert bool((skipped == 7.0).all())
    slots = set()
    for _ in range(1030):
        got = attention_forward(q, q, q, torch.zeros_like(q), D ** -0.5, True, None)
        slots.add(lib.kb_debug_attention_slots(0, 0))
        assert torch.equal(got, expected)
    assert slot in slots and len(slots) == 1024
