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
