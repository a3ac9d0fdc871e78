"""Build recipe for libtq_b200.so (hand-written CUDA for sm_100a behind a C ABI) and _tq_host.so (the host path of a
call, torch tensors to that ABI).

    python -m turboquant_plus_b200.build          # compile if sources are newer than the library

nvcc cross-compiles for sm_100a without a GPU.  The library is built in-tree, next to this
file, so that it travels with the source tree.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")
CSRC_HOST = os.path.join(PKG, "csrc_host")
LIB = os.path.join(PKG, "libtq_b200.so")
HOST_LIB = os.path.join(PKG, "_tq_host.so")
OBJ = os.path.join(PKG, "build")

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", f"-I{INCLUDE}", f"-I{CSRC}"]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found: libtq_b200.so cannot be built")
    return exe


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def host_sources():
    return sorted(os.path.join(CSRC_HOST, f) for f in os.listdir(CSRC_HOST) if f.endswith(".cpp"))


def _stale(lib: str, folder: str) -> bool:
    if not os.path.exists(lib):
        return True
    t = os.path.getmtime(lib)
    deps = [os.path.join(folder, f) for f in os.listdir(folder)] + [os.path.join(INCLUDE, "tq_b200.h")]
    return any(os.path.getmtime(p) > t for p in deps)


def _run(cmd, what: str, verbose: bool = False) -> None:
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")


def _object(src: str) -> str:
    return os.path.join(OBJ, os.path.basename(src).rsplit(".", 1)[0] + ".o")


def _build_cuda(ex, force: bool, verbose: bool) -> None:
    if not force and not _stale(LIB, CSRC):
        return
    nvcc = _nvcc()
    # an object file is kept while its source and every header are older than it
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")] + [os.path.join(INCLUDE, "tq_b200.h")]

    def fresh(src):
        obj = _object(src)
        return not force and os.path.exists(obj) and all(os.path.getmtime(p) < os.path.getmtime(obj) for p in [src, *headers])

    list(ex.map(lambda src: _run([nvcc, *NVCC_FLAGS, "-c", src, "-o", _object(src)], f"nvcc for {src}", verbose),
                [s for s in sources() if not fresh(s)]))
    _run([nvcc, "-shared", "-o", LIB, *map(_object, sources()), "-gencode", "arch=compute_100a,code=sm_100a"], "link")


def _build_host(verbose: bool) -> None:
    """The extension module is C++ against torch's headers and libtq_b200.so, which it finds beside itself."""
    import sysconfig
    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    inc = [INCLUDE, CSRC_HOST, os.path.join(base, "include"), os.path.join(base, "include/torch/csrc/api/include"),
           sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    _run(["g++", "-O3", "-pthread", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-w", *[f"-I{p}" for p in inc],
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *host_sources(), "-o", HOST_LIB,
          f"-L{os.path.join(base, 'lib')}", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-ltorch_python",
          f"-L{PKG}", "-l:libtq_b200.so", "-Wl,-rpath,$ORIGIN"], "g++ for _tq_host.so", verbose)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every csrc/*.cu for sm_100a, link libtq_b200.so and build _tq_host.so; returns the library's path."""
    os.makedirs(OBJ, exist_ok=True)
    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        _build_cuda(ex, force, verbose)
    if force or _stale(HOST_LIB, CSRC_HOST):
        _build_host(verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
