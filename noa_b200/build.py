"""Builds noa_b200's CUDA library, in tree: noa_b200/_lib/libnoa_b200.so (sm_100a only).

    python -m noa_b200.build [--verbose-ptxas]

Each .cu under noa_b200/csrc is compiled with nvcc for sm_100a (-gencode arch=compute_100a,code=sm_100a)
in parallel, then linked into one shared library with the CUDA runtime linked statically, so it loads
beside any PyTorch build; noa_b200/_lib/_marshal.<ABI tag>.so is the Python API's native marshalling, for the
Python that builds it. Rebuilds only what changed.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import importlib.machinery
import os
import shutil
import subprocess
import sys
import sysconfig
import warnings

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(ROOT, "include")
BUILD = os.path.join(PKG, "_build")
LIBDIR = os.path.join(PKG, "_lib")
LIB = os.path.join(LIBDIR, "libnoa_b200.so")
MARSHAL = "_marshal" + importlib.machinery.EXTENSION_SUFFIXES[0]

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
              "--expt-relaxed-constexpr", "-I", INCLUDE, "-I", CSRC] + ARCH


def nvcc() -> str:
    path = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(path):
        raise RuntimeError("nvcc not found: the CUDA toolkit is required to build noa_b200")
    return path


def _sources() -> list[str]:
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers() -> list[str]:
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h", ".hpp"))]
    inc = os.path.join(INCLUDE, "noa_b200")
    hs += [os.path.join(inc, f) for f in os.listdir(inc)]
    return hs


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(src: str, verbose_ptxas: bool) -> tuple[str, str]:
    obj = os.path.join(BUILD, os.path.basename(src)[:-3] + ".o")
    if not _stale(obj, [src] + _headers()):
        return obj, ""
    cmd = [nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose_ptxas else []) + ["-c", src, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
    return obj, r.stderr


def _build_marshal() -> None:
    """The Python API's native marshalling (csrc/marshal.c). It uses the whole CPython API, so its name carries
    the ABI tag of the Python it is built for and no other loads it. Without it (no Python headers, or it does
    not compile) the API marshals through ctypes instead."""
    src, out = os.path.join(CSRC, "marshal.c"), os.path.join(LIBDIR, MARSHAL)
    include = sysconfig.get_paths()["include"]
    if not os.path.exists(os.path.join(include, "Python.h")) or not _stale(out, [src] + _headers()):
        return
    cmd = [shutil.which("gcc") or "cc", "-O2", "-fPIC", "-shared", "-Wall", "-Wextra", "-I", INCLUDE, "-I", include,
           src, "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        warnings.warn(f"building {src} failed, calls will be marshalled through ctypes:\n{r.stdout}\n{r.stderr}",
                      RuntimeWarning)


def build(verbose_ptxas: bool = False, jobs: int | None = None) -> str:
    os.makedirs(BUILD, exist_ok=True)
    os.makedirs(LIBDIR, exist_ok=True)
    _build_marshal()
    srcs = _sources()
    with cf.ThreadPoolExecutor(max_workers=jobs or min(8, os.cpu_count() or 1)) as ex:
        results = list(ex.map(lambda s: _compile(s, verbose_ptxas), srcs))
    objs = [o for o, _ in results]
    if verbose_ptxas:
        for _, log in results:
            sys.stderr.write(log)
    if _stale(LIB, objs):
        cmd = [nvcc()] + ARCH + ["-shared", "-cudart", "static", "-o", LIB] + objs
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


def main() -> None:
    p = argparse.ArgumentParser()
    p.add_argument("--verbose-ptxas", action="store_true")
    args = p.parse_args()
    print(build(args.verbose_ptxas))


if __name__ == "__main__":
    main()
