"""The front-ends called from several threads."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["attention", "linear"])
def test_first_cuda_call_of_a_thread(lib, op):
    """A thread that has made no CUDA call yet has no current context; the first one may be a kernel of this library."""
    import threading

    import torch

    from kernl_b200 import _lib
    from kernl_b200.implementations.attention import attention_forward
    from kernl_b200.implementations.linear_layer import linear_layer

    q = torch.randn((1, 2, 200, 64), device="cuda").half()
    w = torch.randn((256, 64), device="cuda").half()
    results = {}

    def call(name):
        out = torch.empty((1, 2, 200, 64) if op == "attention" else (400, 256), device="cuda", dtype=torch.float16) if name == "here" else outs[name]
        try:
            results[name] = attention_forward(q, q, q, out, 0.125) if op == "attention" else linear_layer(q.view(400, 64), w, None, "", out=out)
        except RuntimeError as e:
            results[name] = e

    outs = {"there": torch.empty((1, 2, 200, 64) if op == "attention" else (400, 256), device="cuda", dtype=torch.float16)}
    call("here")
    thread = threading.Thread(target=call, args=("there",))
    thread.start()
    thread.join()
    assert _lib.device_status()[0] == 0
    assert isinstance(results["there"], torch.Tensor), results["there"]
    assert torch.equal(results["here"], results["there"])


def test_a_blocked_launch_leaves_python_to_other_threads(lib):
    """Launches into a full queue wait for the GPU; the other threads of the process go on meanwhile."""
    import threading
    import time

    import torch

    from kernl_b200.implementations.layer_norm import layer_norm

    x = torch.randn((4, 64), device="cuda").half()
    w = torch.ones(64, device="cuda").half()
    layer_norm(x, w, None, 1e-5, use_rms_norm=True)
    torch.cuda.synchronize()
    took = []

    def launcher():
        begin = time.perf_counter()
        torch.cuda._sleep(2_000_000_000)  # about a second of GPU time ahead of the launches
        for _ in range(4000):  # more than a stream queues
            layer_norm(x, w, None, 1e-5, use_rms_norm=True)
        took.append(time.perf_counter() - begin)

    thread = threading.Thread(target=launcher)
    thread.start()
    longest, last = 0.0, time.perf_counter()
    while thread.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        longest, last = max(longest, now - last), now
    torch.cuda.synchronize()
    assert took[0] > 0.5, "the queue never filled: nothing was tested"
    assert longest < 0.25 * took[0], f"this thread stood still for {longest:.2f} s of {took[0]:.2f}"
