"""Kernels that are launched programmatically and wait on the device: how they read the status word.

Such a kernel may set itself up while the kernel ahead of it still runs, and a wait of that one may yet expire. So it has to
read the status word behind pdl_wait() before it stores, and must not return ahead of pdl_wait(): the kernel behind
it would find it complete while the kernel ahead is not. Neither can be shown on a GPU without a wait that runs
out inside a kernel in flight, so the order is read from the source.
"""
import os
import re

import pytest

from kernl_b200 import build


def _kernels():
    found = {}
    for name in build.HEADERS:
        with open(os.path.join(build.CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__", text):
            begin = text.index("{", text.index(")", text.index("_kernel(", m.start())))
            depth, end = 0, begin
            while True:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
                if depth == 0:
                    break
            kernel = re.search(r"(\w+_kernel)\(", text[m.start():]).group(1)
            found[kernel] = text[begin:end]
    return found


KERNELS = _kernels()
# a bounded wait of the kernel's own, and a programmatic launch
WAITING = sorted(k for k, body in KERNELS.items() if "mbar_wait(" in body and "pdl_wait()" in body)


def test_the_kernels_are_found():
    assert {"linear_tc_kernel", "linear_pair_kernel", "linear_cluster_kernel", "attention_tc_kernel", "attention_split_kernel",
            "attention_persist_kernel"} <= set(WAITING)


@pytest.mark.parametrize("kernel", WAITING)
def test_status_is_read_behind_the_wait_for_the_kernel_ahead(kernel):
    body = KERNELS[kernel]
    wait = body.rindex("pdl_wait();")
    assert re.search(r"status_word\(\)|g_device_status", body[wait:]), "the status word is read ahead of pdl_wait() only"


@pytest.mark.parametrize("kernel", sorted(k for k, body in KERNELS.items() if "pdl_wait()" in body))
def test_no_return_ahead_of_the_wait_for_the_kernel_ahead(kernel):
    body = KERNELS[kernel]
    assert "return;" not in body[: body.index("pdl_wait();")]


@pytest.mark.parametrize("kernel", WAITING)
def test_one_thread_decides_whether_the_work_is_skipped(kernel):
    """What is read during set-up decides whether copies are issued and whether the CTA leaves: threads that read the word
    at different times may differ."""
    body = KERNELS[kernel]
    early = [m.start() for m in re.finditer(r"status_word\(\)|g_device_status", body[: body.rindex("pdl_wait();")])]
    assert len(early) <= 1
    for at in early:
        condition = body[body.rindex("if (", 0, at): at].split("\n")[0]
        assert re.match(r"if \(threadIdx\.x == [\d *]+\)", condition), condition
