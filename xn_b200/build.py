"""Builds, in-tree, ``libxnq.so`` (the C-ABI CUDA library; nvcc alone, for sm_100a only) and ``_xnq_torch.so`` (the torch side of a linear's call; the host
compiler, and the headers of the torch that is installed).

Usage: ``python -m xn_b200.build [--force] [--library]``.  No other architecture, no PTX fallback.  ``--library``: ``libxnq.so`` alone.
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libxnq.so")
TORCH_MODULE = os.path.join(HERE, "_xnq_torch.so")
TORCH_STAMP = os.path.join(HERE, "build", "torch_module.txt")

EXTRA = os.environ.get("XNQ_EXTRA_NVCC_FLAGS", "").split()
if os.environ.get("XNQ_LIB_NAME"):
    LIB = os.path.join(HERE, os.environ["XNQ_LIB_NAME"])
    OBJ = os.path.join(HERE, "build_" + os.environ["XNQ_LIB_NAME"].replace(".", "_"))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", *EXTRA,
]


def _nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; the xnq library can only be built with the CUDA toolkit")
    return nvcc


def sources() -> list[str]:
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps() -> list[str]:
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h", ".hpp"))]
    hdrs.append(os.path.join(HERE, "..", "include", "xnq.h"))
    return hdrs


def is_stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(p) > t for p in sources() + _deps())


def _torch_stamp() -> str:
    """What the module is compiled against: it uses torch's own layouts, so another torch or Python needs another build."""
    import torch
    return f"torch {torch.__version__} {torch.version.git_version} python {sys.version}"


def torch_module_is_stale() -> bool:
    src = os.path.join(CSRC, "torch_linear.cpp")
    if not os.path.exists(TORCH_MODULE) or os.path.getmtime(TORCH_MODULE) < os.path.getmtime(src):
        return True
    try:
        with open(TORCH_STAMP) as f:
            return f.read() != _torch_stamp()
    except OSError:
        return True


def build_torch_module(force: bool = False) -> str:
    if not force and not torch_module_is_stale():
        return TORCH_MODULE
    src = os.path.join(CSRC, "torch_linear.cpp")
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [*include_paths(), sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-I{p}" for p in inc), src, "-o", TORCH_MODULE, *(f"-L{p}" for p in library_paths()),
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-ltorch"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"the host compiler failed on {src}:\n{r.stdout}\n{r.stderr}")
    os.makedirs(os.path.dirname(TORCH_STAMP), exist_ok=True)
    with open(TORCH_STAMP, "w") as f:
        f.write(_torch_stamp())
    return TORCH_MODULE


def build_library(force: bool = False, verbose: bool = False) -> str:
    if not force and not is_stale():
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    newest_hdr = max(os.path.getmtime(p) for p in _deps())

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if not force and os.path.exists(obj) and os.path.getmtime(obj) > max(os.path.getmtime(src), newest_hdr):
            return obj
        cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj] + (["-Xptxas", "-v"] if verbose else [])
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(compile_one, sources()))
    r = subprocess.run([nvcc, "-shared", "-o", LIB, *objs], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
    if "--library" not in sys.argv:
        print(build_torch_module(force="--force" in sys.argv))
