"""Build recipe for the lig_b200 CUDA library (sm_100a only).

Compiles every ``lig_b200/csrc/*.cu`` with nvcc for ``sm_100a`` into
``lig_b200/_build/*.o`` (in parallel, skipping up-to-date objects) and links
``lig_b200/liblig_b200.so``, which ``lig_b200._lib`` loads through ctypes; then
compiles ``lig_b200/csrc/host.cpp`` with g++ against torch's headers into
``lig_b200/_host.so``, the native half of ``lig_b200.ops``.
Run it as a script (``python lig_b200/build.py``): importing the package
loads the library, which must exist first.

Flags: ``-O3 --use_fast_math`` matches the reference's setup.py
(gsplat2d/setup.py:65-77), which the bit-exact tile counts and alpha-threshold
decisions depend on; ``-lineinfo`` keeps source correlation for ncu.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
HOST_SRC = os.path.join(CSRC, "host.cpp")
HOST_LIB = os.path.join(PKG, "_host.so")
BUILD = os.path.join(PKG, "_build")
HOST_STAMP = os.path.join(BUILD, "host.stamp")  # what _host.so was built against
LIB = os.path.join(PKG, "liblig_b200.so")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-O3", "--use_fast_math", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC",
              "--expt-relaxed-constexpr", "-I", INCLUDE]


def nvcc() -> str:
    path = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(path):
        raise RuntimeError("nvcc not found: the lig_b200 CUDA library cannot be built")
    return path


def _deps(src: str):
    return [src] + glob.glob(os.path.join(CSRC, "*.cuh")) + [os.path.join(INCLUDE, "lig_b200.h")]


def _stale(obj: str, deps) -> bool:
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(src: str, extra) -> str:
    obj = os.path.join(BUILD, os.path.basename(src)[:-3] + ".o")
    if _stale(obj, _deps(src)):
        cmd = [nvcc(), *ARCH, *NVCC_FLAGS, *extra, "-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        if r.stderr.strip():
            sys.stderr.write(r.stderr)
    return obj


def _run_host(cmd) -> None:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {HOST_SRC}:\n{r.stdout}\n{r.stderr}")


def _build_host() -> None:
    """Compile the native half of ops.py (a Python module on torch's headers,
    linked against the CUDA library beside it), unless it is newer than its
    source and was built against this Python and this torch."""
    import sysconfig

    import torch

    against = f"python {sys.version}\ntorch {torch.__version__}\n"
    try:
        with open(HOST_STAMP) as f:
            same = f.read() == against
    except OSError:
        same = False
    if same and not _stale(HOST_LIB, [HOST_SRC, os.path.join(INCLUDE, "lig_b200.h")]):
        return
    from torch.utils import cpp_extension as tx

    cuda = os.path.dirname(os.path.dirname(nvcc()))
    inc = [sysconfig.get_paths()["include"], os.path.join(cuda, "include"), *tx.include_paths()]
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-DTORCH_EXTENSION_NAME=_host", *[f for i in inc for f in ("-isystem", i)], HOST_SRC,
           "-o", HOST_LIB, "-L", PKG, "-l:liblig_b200.so", "-L", lib, "-lc10", "-lc10_cuda",
           "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python",
           "-L", os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath,$ORIGIN",
           f"-Wl,-rpath,{lib}"]
    _run_host(cmd)
    with open(HOST_STAMP, "w") as f:
        f.write(against)


def build(verbose: bool = False, extra=()) -> str:
    """Compile (incrementally) and link liblig_b200.so; returns its path."""
    os.makedirs(BUILD, exist_ok=True)
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(lambda s: _compile(s, list(extra)), srcs))
    if _stale(LIB, objs):
        cmd = [nvcc(), *ARCH, "-shared", "-o", LIB, *objs, "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_host()
    if verbose:
        print(f"built {LIB}, {HOST_LIB}")
    return LIB


if __name__ == "__main__":
    build(verbose=True, extra=sys.argv[1:])
