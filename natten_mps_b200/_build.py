"""Build the native code in-tree: ``natten_mps_b200/libnatten_b200.so`` (the CUDA library behind the C ABI, no
torch in it) and ``natten_mps_b200/_native.so`` (the PyTorch operators on top of it, host code only).

nvcc cross-compiles for sm_100a without a GPU.  Each ``.cu`` file is compiled to
an object in ``csrc/build/`` (in parallel, skipped when the object is newer than
every source and header) and the objects are linked into one shared library.
"""
from __future__ import annotations

import concurrent.futures
import glob
import os
import subprocess

_PKG = os.path.dirname(os.path.abspath(__file__))
_CSRC = os.path.join(_PKG, "csrc")
LIB_PATH = os.path.join(_PKG, "libnatten_b200.so")
NATIVE_PATH = os.path.join(_PKG, "_native.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def build_native(headers, force: bool = False) -> str:
    """Compile csrc/torch_ops.cpp against the running interpreter's torch and link it to the CUDA library."""
    import sysconfig

    import torch

    src = os.path.join(_CSRC, "torch_ops.cpp")
    newest = max([os.path.getmtime(src)] + [os.path.getmtime(h) for h in headers if h.endswith(".h")])
    if not force and os.path.exists(NATIVE_PATH) and os.path.getmtime(NATIVE_PATH) >= newest:
        return NATIVE_PATH
    troot = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    subprocess.check_call([
        "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
        *[f"-I{d}" for d in (os.path.join(troot, "include"), os.path.join(troot, "include", "torch", "csrc", "api", "include"),
                             os.path.join(cuda, "include"), sysconfig.get_paths()["include"])],
        src, "-o", NATIVE_PATH, f"-L{_PKG}", "-l:libnatten_b200.so", "-Wl,-rpath,$ORIGIN",
        f"-L{os.path.join(troot, 'lib')}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"])
    return NATIVE_PATH


def build(force: bool = False, verbose: bool = False) -> str:
    sources = sorted(glob.glob(os.path.join(_CSRC, "*.cu")))
    headers = glob.glob(os.path.join(_CSRC, "*.cuh")) + glob.glob(
        os.path.join(os.path.dirname(_PKG), "include", "*.h"))
    newest_header = max((os.path.getmtime(h) for h in headers), default=0.0)
    objdir = os.path.join(_CSRC, "build")
    os.makedirs(objdir, exist_ok=True)
    flags = list(NVCC_FLAGS)
    if verbose:
        flags = flags + ["-Xptxas", "-v"]

    def compile_one(src: str) -> str:
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        stale = force or not os.path.exists(obj) or os.path.getmtime(obj) < max(
            os.path.getmtime(src), newest_header)
        if stale:
            subprocess.check_call([_nvcc(), *flags, "-c", src, "-o", obj])
        return obj

    with concurrent.futures.ThreadPoolExecutor(max_workers=max(1, min(8, len(sources)))) as pool:
        objects = list(pool.map(compile_one, sources))
    if force or not os.path.exists(LIB_PATH) or any(
            os.path.getmtime(o) > os.path.getmtime(LIB_PATH) for o in objects):
        subprocess.check_call([_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared",
                               "-o", LIB_PATH, *objects, "-lcuda"])
    build_native(headers, force)
    return LIB_PATH


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
