"""Build ``liboxq.so`` in-tree with nvcc for sm_100a.

Usage: ``python -m oxydllm_b200.build [--force] [--verbose]``.
"""
from __future__ import annotations

import fcntl
import glob
import os
import subprocess
import sys
import sysconfig

_HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(_HERE, "csrc")
LIB = os.path.join(_HERE, "liboxq.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--compiler-options", "-fPIC,-fvisibility=hidden", "-shared",
]


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(_HERE, "..", "include", "*.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every ``csrc/*.cu`` into one shared library; returns its path."""
    if not force and not _stale():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    extra = os.environ.get("OXQ_NVCC_FLAGS", "").split()  # extra defines for experiments
    # One builder at a time, and the library appears under its name only when complete: processes that start
    # together (test workers, ranks of a multi-GPU launch) never load a half-written file.
    with open(LIB + ".lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        if not force and not _stale():
            return LIB  # another process built it while this one waited
        tmp = f"{LIB}.{os.getpid()}.tmp"
        cmd = [nvcc, *NVCC_FLAGS, *extra, *(["-Xptxas", "-v"] if verbose else []), "-o", tmp, *sources()]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or res.returncode:
            sys.stderr.write(res.stdout + res.stderr)
        if res.returncode:
            if os.path.exists(tmp):
                os.remove(tmp)
            raise RuntimeError("nvcc failed building liboxq.so")
        os.replace(tmp, LIB)
    return LIB


def host_path() -> str:
    return os.path.join(_HERE, "_host" + sysconfig.get_config_var("EXT_SUFFIX"))


def build_host(force: bool = False) -> str:
    """Compile ``csrc/host_ops.cpp`` against the installed torch into the extension module ``_host``; returns its path."""
    import torch
    src, out = os.path.join(CSRC, "host_ops.cpp"), host_path()
    header = os.path.join(_HERE, "..", "include", "oxq.h")
    fresh = lambda: os.path.exists(out) and os.path.getmtime(out) >= max(os.path.getmtime(src), os.path.getmtime(header))  # noqa: E731
    if not force and fresh():
        return out
    root = os.path.dirname(torch.__file__)
    with open(out + ".lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        if not force and fresh():
            return out
        tmp = f"{out}.{os.getpid()}.tmp"
        cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", "-I" + os.path.join(root, "include"),
               "-I" + sysconfig.get_paths()["include"], "-I/usr/local/cuda/include", "-o", tmp, src, "-L" + os.path.join(root, "lib"),
               "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode:
            if os.path.exists(tmp):
                os.remove(tmp)
            raise RuntimeError("g++ failed building the host extension:\n" + res.stderr[-4000:])
        os.replace(tmp, out)
    return out


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
    print(build_host(force="--force" in sys.argv))
