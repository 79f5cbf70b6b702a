"""Builds libncn_b200.so (nvcc, sm_100a; csrc/Makefile) and the extension module with the autograd nodes
(csrc/ncn_torch.cpp, against the installed torch) in-tree."""
from __future__ import annotations

import os
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libncn_b200.so")


def _torch_flags():
    """(compiler flags, linker flags) of an extension of the installed torch, for make."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    inc = cpp_extension.include_paths("cuda") + [sysconfig.get_paths()["include"]]
    flags = [f"-isystem {p}" for p in inc]
    flags.append(f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}")
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    return " ".join(flags), f"-L{lib} -lc10 -lc10_cuda -ltorch -ltorch_cpu -ltorch_python"


def build(verbose: bool = False, jobs: int | None = None) -> str:
    """Compile every kernel for sm_100a, link the shared library and the extension module; returns the library's path."""
    jobs = jobs or max(1, (os.cpu_count() or 2))
    cflags, ldflags = _torch_flags()
    cmd = ["make", "-C", CSRC, f"-j{jobs}", f"TORCH_CFLAGS={cflags}", f"TORCH_LDFLAGS={ldflags}", f"PYTHON={sys.executable}"]
    res = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if verbose or res.returncode != 0:
        print(res.stdout)
    if res.returncode != 0:
        raise RuntimeError("building libncn_b200.so failed (see the compiler output above)")
    return LIB_PATH


if __name__ == "__main__":
    print(build(verbose=True))
