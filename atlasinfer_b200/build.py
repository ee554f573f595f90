"""Builds ``libatlas_b200.so`` (the C-ABI library) in-tree with nvcc for sm_100a.

    python -m atlasinfer_b200.build [--force] [--verbose]

The library is compiled from ``csrc/*.cu`` against ``include/atlas_b200.h`` and
written to ``atlasinfer_b200/lib/``, and beside it the module ``csrc/native.cpp``
(the host path of the Python surface, which calls the library).  nvcc
cross-compiles without a GPU.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libatlas_b200.so")

SOURCES = ["capi.cu", "quantize.cu", "dequant_repack.cu", "gemv.cu", "stream.cu", "peer.cu", "gemm.cu", "gemm_tile.cu"]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "-shared", "-cudart", "static",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; the atlas_b200 library cannot be built")


def _inputs():
    files = [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    deps = files + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    deps.append(os.path.join(ROOT, "include", "atlas_b200.h"))
    return files, deps


NATIVE_NAME = "_atlas_native"
NATIVE_SRC = os.path.join(CSRC, "native.cpp")


def native_path() -> str:
    """Where the host path belongs: its name carries the torch version and the interpreter it was compiled for, since
    it is tied to the C++ interfaces of both."""
    import torch

    abi = "" if torch.compiled_with_cxx11_abi() else "-oldabi"
    return os.path.join(LIB_DIR, f"{NATIVE_NAME}-torch{torch.__version__}{abi}" + sysconfig.get_config_var("EXT_SUFFIX"))


def _stale(target: str, sources) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in sources)


def build_native(force: bool = False, verbose: bool = False) -> str:
    """Compile the host path (``csrc/native.cpp``, against torch's headers) if it is missing or old; return its path."""
    header = os.path.join(ROOT, "include", "atlas_b200.h")
    target = native_path()
    if not force and not _stale(target, [NATIVE_SRC, header]):
        return target
    import torch
    from torch.utils import cpp_extension

    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    dirs = [*cpp_extension.include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"],
            os.path.join(ROOT, "include")]
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else (shutil.which("g++") or "c++")
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-DTORCH_EXTENSION_NAME={NATIVE_NAME}",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", *(f"-I{d}" for d in dirs), NATIVE_SRC,
           "-o", target, f"-L{LIB_DIR}", "-l:libatlas_b200.so", "-Wl,-rpath,$ORIGIN", f"-L{torch_lib}",
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("g++ failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stdout + res.stderr)
    return target


def is_stale() -> bool:
    return _stale(LIB_PATH, _inputs()[1])


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile what is missing or older than its sources: the C-ABI library and the host path on top of it.

    Returns the path of the C-ABI library."""
    build_library(force, verbose)
    build_native(force, verbose)
    return LIB_PATH


def build_library(force: bool = False, verbose: bool = False) -> str:
    if not force and not is_stale():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    files, _ = _inputs()
    cmd = [_nvcc(), *NVCC_FLAGS, "-I", os.path.join(ROOT, "include"), "-I", CSRC]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += ["-o", LIB_PATH, *files]
    env = dict(os.environ)
    # the image exports CC/CXX pointing at a compiler driver nvcc cannot use as host compiler
    cmd += ["-ccbin", "/usr/bin/g++"] if os.path.exists("/usr/bin/g++") else []
    res = subprocess.run(cmd, capture_output=True, text=True, env=env)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stdout + res.stderr)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
