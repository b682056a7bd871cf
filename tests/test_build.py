"""What the build needs: the C library nvcc alone, the torch module the torch that is installed."""
import os
import subprocess
import sys

import pytest

from xn_b200 import build as B


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """A build that compiles nothing: sources of one line, compilers that write an empty result and are remembered."""
    csrc = tmp_path / "csrc"
    csrc.mkdir()
    for name in ("a.cu", "torch_linear.cpp", "a.cuh"):
        (csrc / name).write_text("// nothing\n")
    for name, path in (("CSRC", csrc), ("OBJ", tmp_path / "build"), ("LIB", tmp_path / "lib.so"), ("TORCH_MODULE", tmp_path / "_t.so"),
                       ("TORCH_STAMP", tmp_path / "build" / "torch_module.txt")):
        monkeypatch.setattr(B, name, str(path))
    ran = []

    def run(cmd, **_):
        ran.append(os.path.basename(cmd[0]))
        open(cmd[cmd.index("-o") + 1], "w").close()
        return subprocess.CompletedProcess(cmd, 0, "", "")
    monkeypatch.setattr(B.subprocess, "run", run)
    monkeypatch.setattr(B, "_nvcc", lambda: "/usr/local/cuda/bin/nvcc")
    return ran


def test_the_library_needs_nvcc_alone(tree, monkeypatch):
    monkeypatch.setitem(sys.modules, "torch", None)   # an import of it raises
    B.build_library()
    assert tree == ["nvcc", "nvcc"] and not os.path.exists(B.TORCH_MODULE)


def test_the_module_follows_torch(tree, monkeypatch):
    import torch
    B.build_torch_module()
    assert len(tree) == 1
    B.build_torch_module()
    assert len(tree) == 1                            # up to date
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    B.build_torch_module()
    assert len(tree) == 2                            # compiled against another torch
    os.remove(B.TORCH_STAMP)
    B.build_torch_module()
    assert len(tree) == 3                            # against nobody knows what
