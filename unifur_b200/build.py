"""Builds libnf4b200.so (the C-ABI CUDA library) and _host.so (the Python mirror's host path) in-tree.

    python -m unifur_b200.build [--force] [--verbose]

Each .cu under csrc/ is compiled to an object file beside the library and the objects
are linked into unifur_b200/libnf4b200.so (nvcc, sm_100a; cross-compiles without a GPU);
csrc/host/host.cpp becomes the extension module unifur_b200/_host.so against the installed torch.
"""
from __future__ import annotations

import concurrent.futures
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
HOST = os.path.join(CSRC, "host", "host.cpp")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libnf4b200.so")
HOST_LIB = os.path.join(HERE, "_host.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

# No -use_fast_math and no -ftz: quantize/dequantize must stay IEEE bit-exact.
FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--fmad=true",
    "-Xptxas", "-v",
]


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps_mtime():
    newest = 0.0
    for root, _, files in os.walk(CSRC):
        if root != CSRC:
            continue
        for f in files:
            if f.endswith((".cu", ".cuh", ".inc", ".h")):
                newest = max(newest, os.path.getmtime(os.path.join(root, f)))
    newest = max(newest, os.path.getmtime(os.path.join(HERE, "..", "include", "nf4_b200.h")))
    return newest


def _compile(src: str, verbose: bool) -> str:
    obj = os.path.join(OBJ, src[:-3] + ".o")
    cmd = [NVCC, *FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}")
    with open(obj + ".log", "w") as f:
        f.write(r.stderr)
    return obj


def _build_host(verbose: bool) -> None:
    """The Python extension ``_host`` (host path of the mirror), against the installed torch."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    inc = [*cpp_extension.include_paths(), sysconfig.get_paths()["include"],
           os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")]
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           "-Wall", "-Wextra", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *[a for d in inc for a in ("-isystem", d)], HOST,
           "-o", HOST_LIB, f"-L{HERE}", "-l:libnf4b200.so", f"-L{libs}", "-lc10", "-lc10_cuda", "-ltorch_cpu",
           "-ltorch_cuda", "-ltorch_python", f"-L{os.path.join(os.path.dirname(os.path.dirname(NVCC)), 'lib64')}",
           "-lcudart_static", "-ldl", "-lrt", "-lpthread", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0 or r.stderr:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode != 0:
        raise RuntimeError("building the host extension failed")


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    if force or not os.path.exists(LIB) or os.path.getmtime(LIB) < _deps_mtime():
        srcs = _sources()
        with concurrent.futures.ThreadPoolExecutor(max_workers=len(srcs)) as ex:
            objs = list(ex.map(lambda s: _compile(s, verbose), srcs))
        cmd = [NVCC, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a",
               "-Xcompiler", "-fPIC", "-lcudart_static", "-Xlinker", "-soname=libnf4b200.so"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            raise RuntimeError("link failed")
    header = os.path.join(HERE, "..", "include", "nf4_b200.h")
    if force or not os.path.exists(HOST_LIB) or os.path.getmtime(HOST_LIB) < max(os.path.getmtime(HOST), os.path.getmtime(header)):
        _build_host(verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
