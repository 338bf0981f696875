"""Builds csrc/libtriebwerk_b200.so in-tree with nvcc for sm_100a and, beside the package, the extension that Python
calls it through (``python -m triebwerk_b200.build``)."""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig

_HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(_HERE, "csrc")
LIB = os.path.join(CSRC, "libtriebwerk_b200.so")
HOSTCALL = os.path.join(_HERE, "_hostcall" + sysconfig.get_config_var("EXT_SUFFIX"))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-shared", "-Xcompiler",
         "-fPIC"]
_HEADER = os.path.join(os.path.dirname(_HERE), "include", "triebwerk_b200.h")


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))) + [_HEADER]


def _stale(target, deps) -> bool:
    return not os.path.exists(target) or os.path.getmtime(target) < max(os.path.getmtime(d) for d in deps)


def build_hostcall(force: bool = False) -> str:
    src = os.path.join(CSRC, "hostcall.cpp")
    if not force and not _stale(HOSTCALL, [src, _HEADER]):
        return HOSTCALL
    from torch.utils import cpp_extension as ce
    cmd = [os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-shared", "-fPIC", "-o", HOSTCALL, src]
    cmd += ["-I" + p for p in ce.include_paths("cuda")] + ["-I" + sysconfig.get_paths()["include"]]
    cmd += ["-L" + p for p in ce.library_paths("cuda")] + ["-L" + CSRC, "-Wl,-rpath,$ORIGIN/csrc"]
    cmd += ["-ltriebwerk_b200", "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    subprocess.check_call(cmd)
    return HOSTCALL


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile whatever is missing or older than its sources.  Returns the library's path."""
    if force or _stale(LIB, sources()):
        cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-o", LIB, os.path.join(CSRC, "tq_capi.cu")]
        subprocess.check_call(cmd)
    build_hostcall(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
