"""Set-up that a kernel needs once per device (its shared-memory attribute), with several threads: nobody launches before it is done."""
import os
import shutil
import subprocess

from kernl_b200 import build

PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
#include <cuda_runtime.h>
static cudaError_t device_zero(int* dev) { *dev = 0; return cudaSuccess; }  // no GPU here
#define cudaGetDevice device_zero
#include "common.cuh"
int main() {
    kb::PerDeviceOnce once;
    std::atomic<int> sets{0}, finished{0}, early{0};
    std::vector<std::thread> threads;
    for (int i = 0; i < 8; ++i)
        threads.emplace_back([&] {
            const bool ok = once.run([&] {
                std::this_thread::sleep_for(std::chrono::milliseconds(sets++ == 0 ? 100 : 0));
                ++finished;
                return true;
            });
            if (!ok || finished == 0) ++early;
        });
    for (auto& t : threads) t.join();
    kb::PerDeviceOnce failing;
    int tries = 0;
    for (int i = 0; i < 3; ++i) failing.run([&] { return ++tries == 2; });
    printf("sets %d early %d tries %d\n", sets.load(), early.load(), tries);
}
"""


def test_nobody_launches_before_the_attribute_is_set(tmp_path):
    source, program = tmp_path / "once.cu", tmp_path / "once"
    source.write_text(PROGRAM)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-arch=sm_100a", "-I", build.CSRC, "-o", str(program), str(source)], check=True, cwd=os.path.dirname(build.CSRC))
    out = subprocess.run([str(program)], capture_output=True, text=True, check=True).stdout
    assert out == "sets 1 early 0 tries 2\n"
