"""Builds libkiln_w4a16.so in-tree with nvcc for sm_100a (cross-compiles without a GPU), and _native.so, the extension
module that runs the Python entry points' host path, with g++ against the installed torch.

Usage: python -m kiln_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libkiln_w4a16.so")
SOURCES = ["api.cu", "decode_w4a16.cu", "epilogue_w4a16.cu", "pair_w4a16_umma.cu", "prefill_w4a16_umma.cu", "repack.cu", "smallm_w4a16_tmem.cu"]
NATIVE = os.path.join(HERE, "_native.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = [
    "-std=c++17", "-O3", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-pthread", "--expt-relaxed-constexpr",
]


def _native_command() -> list:
    import sysconfig

    import torch

    t = os.path.dirname(torch.__file__)
    cuda = os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")
    inc = [os.path.join(t, "include"), os.path.join(t, "include", "torch", "csrc", "api", "include"), cuda, sysconfig.get_paths()["include"]]
    return [os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            f'-DKILN_NATIVE_KEY="{_native_key()}"',
            *(f"-I{d}" for d in inc), os.path.join(CSRC, "host.cpp"), "-o", NATIVE, "-L" + os.path.join(t, "lib"), "-lc10", "-lc10_cuda",
            "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]


def _stale() -> bool:
    if not (os.path.exists(LIB) and os.path.exists(NATIVE)):
        return True
    t = min(os.path.getmtime(LIB), os.path.getmtime(NATIVE))
    # (sources only: the objects lie beside them, and the last of them is younger than _native.so, which is compiled meanwhile)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".cpp", ".h"))]
    deps.append(os.path.join(HERE, "..", "include", "kiln_w4a16.h"))
    return any(os.path.getmtime(d) > t for d in deps) or not _built_for_this_torch()


def _native_key() -> str:
    """What _native.so depends on besides its source; compiled into it (csrc/host.cpp)."""
    import torch

    return f"kiln_b200 native: python {sys.version_info[0]}.{sys.version_info[1]}, torch {torch.__version__}, abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)};"


def _built_for_this_torch() -> bool:
    with open(NATIVE, "rb") as f:
        return _native_key().encode() in f.read()


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return LIB
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(CSRC, src.replace(".cu", ".o"))
        cmd = [NVCC, *FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    obj = os.path.join(CSRC, "pack_host.o")
    procs.append(("pack_host.cpp", subprocess.Popen([os.environ.get("CXX", "g++"), "-std=c++17", "-O3", "-fPIC", "-c", os.path.join(CSRC, "pack_host.cpp"),
                                                     "-o", obj], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    objs.append(obj)
    procs.append(("host.cpp", subprocess.Popen(_native_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(f"--- {src}\n{out}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("compilation failed")
    subprocess.check_call([NVCC, "-shared", "-o", LIB, *objs, "-lcudart_static", "-lpthread", "-ldl", "-lrt"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
