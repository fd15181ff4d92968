"""Builds the CUDA library of kernl_b200 in-tree with nvcc for sm_100a, and the CPython module that
calls it from tensors.

`python -m kernl_b200.build` writes kernl_b200/libkernl_b200.so and kernl_b200/_host_ops.so next to
this file. nvcc cross-compiles without a GPU, so this runs on any box that has the CUDA toolkit.
"""
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_PATH = os.path.join(HERE, "libkernl_b200.so")
SOURCES = ["kernl_b200.cu"]
HEADERS = ["common.cuh", "norm.cuh", "linear.cuh", "linear_pair.cuh", "linear_cluster.cuh", "linear_stream.cuh", "attention.cuh", "attention_split.cuh", "attention_persist.cuh", "attention_short.cuh", "attention_decode.cuh", "allreduce.cuh", "rope.cuh"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17", "--shared",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: the kernl_b200 CUDA library cannot be built")
    return exe


HASH_PATH = LIB_PATH + ".srchash"
PUBLIC_HEADERS = [os.path.join(HERE, "..", "include", h) for h in ("kernl_b200.h", "kernl_b200_debug.h")]
HOST_PATH = os.path.join(HERE, "_host_ops.so")
HOST_SOURCE = os.path.join(CSRC, "host_ops.cpp")
HOST_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared"]


def _hash(deps, *words) -> str:
    h = hashlib.sha256(" ".join(words).encode())
    for d in deps:
        with open(d, "rb") as f:
            h.update(f.read())
    return h.hexdigest()


def _source_hash() -> str:
    """Hash of everything the library is built from (sources, headers, flags)."""
    return _hash([os.path.join(CSRC, f) for f in SOURCES + HEADERS] + PUBLIC_HEADERS, *NVCC_FLAGS)


def _host_hash() -> str:
    """The same for the CPython module, which is also bound to this torch and this Python."""
    import torch

    return _hash([HOST_SOURCE] + PUBLIC_HEADERS, *HOST_FLAGS, torch.__version__, sys.version)


def _differs(path, current_hash) -> bool:
    """A binary is rebuilt when it is missing or was built from other sources. By content, not by
    modification time: a copy of the tree to another machine keeps the contents, not the times."""
    if not os.path.exists(path) or not os.path.exists(path + ".srchash"):
        return True
    try:
        with open(path + ".srchash") as f:
            return f.read().strip() != current_hash
    except OSError:
        return True


def is_stale() -> bool:
    return _differs(LIB_PATH, _source_hash()) or _differs(HOST_PATH, _host_hash())


def _compile(cmd, path, source_hash, verbose=False) -> None:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n" + proc.stdout + proc.stderr)
    if verbose:
        print(proc.stderr)
    with open(path + ".srchash", "w") as f:
        f.write(source_hash + "\n")


def _build_host() -> None:
    import torch

    root = os.path.dirname(torch.__file__)
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    libs = ["torch_python", "torch_cuda", "torch_cpu", "torch", "c10_cuda", "c10"]
    cmd = [shutil.which("g++") or "g++", *HOST_FLAGS, *(f"-I{i}" for i in include), "-o", HOST_PATH, HOST_SOURCE,
           f"-L{HERE}", "-l:" + os.path.basename(LIB_PATH), "-L" + os.path.join(root, "lib"), *(f"-l{x}" for x in libs), "-Wl,-rpath,$ORIGIN"]
    _compile(cmd, HOST_PATH, _host_hash())


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile csrc/*.cu into libkernl_b200.so and csrc/host_ops.cpp into _host_ops.so (each skipped
    when up to date). Returns the library's path."""
    if force or _differs(LIB_PATH, _source_hash()):
        cmd = [_nvcc(), *NVCC_FLAGS]
        if verbose:
            cmd += ["-Xptxas", "-v"]
        cmd += ["-o", LIB_PATH] + [os.path.join(CSRC, s) for s in SOURCES]
        _compile(cmd, LIB_PATH, _source_hash(), verbose)
    if force or _differs(HOST_PATH, _host_hash()):
        _build_host()
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
