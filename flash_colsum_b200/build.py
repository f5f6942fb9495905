"""Compile the CUDA library in-tree for B200 (sm_100a), and the PyTorch binding over it.

    python -m flash_colsum_b200.build [--force]

Both shared libraries land in ``flash_colsum_b200/_lib/`` next to the sources; they are
loaded from there and never installed into site-packages.  nvcc cross-compiles,
so this works on a machine without a GPU.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "_lib")
LIB_PATH = os.path.join(LIB_DIR, "libflash_colsum_b200.so")
SOURCES = [os.path.join(CSRC, "flash_colsum_sm100.cu")]
HEADERS = [os.path.join(CSRC, "sm100_ptx.cuh"), os.path.join(CSRC, "schedule.h"),
           os.path.join(CSRC, "colsum_small_q.cuh"), os.path.join(CSRC, "colsum_few_rows.cuh"),
           os.path.join(CSRC, "round_fp32.cuh"), os.path.join(CSRC, "colsum_math.cuh"),
           os.path.join(CSRC, "colsum_single_pass.cuh"), os.path.join(CSRC, "select_topk.cuh"),
           os.path.join(CSRC, "colsum_fused_short.cuh"), os.path.join(CSRC, "host_api.h"),
           os.path.join(os.path.dirname(PKG), "include", "flash_colsum_b200.h")]

# the operator's host path for PyTorch callers: a CPython extension module over the library above
BINDING_NAME = "_fcs_torch"
BINDING_PATH = os.path.join(LIB_DIR, BINDING_NAME + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
BINDING_SOURCE = os.path.join(CSRC, "torch_binding.cpp")
BINDING_HEADERS = [os.path.join(CSRC, "host_api.h"),
                   os.path.join(os.path.dirname(PKG), "include", "flash_colsum_b200.h")]

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-shared", "-Xcompiler", "-fPIC"]


def find_nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def _older(target: str, sources) -> bool:
    if not os.path.exists(target):
        return True
    built = os.path.getmtime(target)
    return any(os.path.getmtime(f) > built for f in sources)


def is_stale() -> bool:
    return _older(LIB_PATH, SOURCES + HEADERS) or _older(BINDING_PATH, [BINDING_SOURCE] + BINDING_HEADERS)


def _compile(cmd, target: str, verbose: bool) -> None:
    """Run a compiler into a file of its own and rename it over `target` when complete."""
    tmp = f"{target}.{os.getpid()}.tmp"
    res = subprocess.run(cmd + ["-o", tmp], capture_output=True, text=True)
    if res.returncode != 0:
        if os.path.exists(tmp):
            os.remove(tmp)
        raise RuntimeError("compiling failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    os.replace(tmp, target)
    if verbose:
        print(res.stderr)


def _build_library(verbose: bool) -> None:
    _compile([find_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + SOURCES, LIB_PATH, verbose)


def _build_binding(verbose: bool) -> None:
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(find_nvcc()))
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    cmd += ["-I" + d for d in include] + [BINDING_SOURCE, "-L" + os.path.join(root, "lib"), "-ltorch_python",
                                          "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]
    _compile(cmd, BINDING_PATH, verbose)


def build(force: bool = False, verbose: bool = False) -> str:
    """Build what is missing or older than its sources; returns the CUDA library's path."""
    if not force and not is_stale():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    # Several processes may get here at once (one rank per GPU): one of them builds, into
    # files of its own that are renamed over the libraries when complete, the others wait for
    # the lock and find them fresh.  Nobody can open a half-written file.
    import fcntl
    with open(os.path.join(LIB_DIR, ".build.lock"), "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if force or _older(LIB_PATH, SOURCES + HEADERS):
                _build_library(verbose)
            if force or _older(BINDING_PATH, [BINDING_SOURCE] + BINDING_HEADERS):
                _build_binding(verbose)
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
