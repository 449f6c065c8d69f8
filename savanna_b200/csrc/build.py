"""Builds the in-tree native libraries.

    python -m savanna_b200.csrc.build [--force]

  savanna_b200/libsavanna_b200.so    every CUDA kernel, compiled for sm_100a only
                                     (nvcc -gencode arch=compute_100a,code=sm_100a -lineinfo), C ABI
  savanna_b200/libsavanna_data.so    C++ dataset index builders, C ABI
  savanna_b200/_native.so            C++ autograd functions that call the CUDA library's entry points (PyTorch extension module)

The first two expose plain C symbols and are loaded with ctypes (ops/cuda_ops.py, data/helpers.py): the kernels include
no PyTorch header.  A content hash of the sources is stored next to each library; an up-to-date library is not rebuilt.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
BUILD = os.path.join(HERE, "build")
CUDA_LIB = os.path.join(PKG, "libsavanna_b200.so")
DATA_LIB = os.path.join(PKG, "libsavanna_data.so")
NATIVE_MODULE = os.path.join(PKG, "_native.so")
NATIVE_SOURCES = ("autograd_native.cpp",)
NATIVE_HEADERS = ("entries.h",)

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _sources(ext):
    return sorted(os.path.join(HERE, f) for f in os.listdir(HERE) if f.endswith(ext))


def _digest(files, extra=""):
    h = hashlib.sha256(extra.encode())
    for f in sorted(files):
        h.update(os.path.basename(f).encode())
        with open(f, "rb") as fh:
            h.update(fh.read())
    return h.hexdigest()


def _stamp(lib):
    return lib + ".hash"


def _fresh(lib, digest):
    try:
        return os.path.exists(lib) and open(_stamp(lib)).read().strip() == digest
    except OSError:
        return False


def _run(cmd, log):
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    log.append(" ".join(cmd) + "\n" + r.stdout)
    if r.returncode != 0:
        raise RuntimeError("command failed:\n" + " ".join(cmd) + "\n" + r.stdout)


def build_cuda(force=False, verbose=False):
    cus = _sources(".cu")
    headers = _sources(".cuh") + _sources(".h")
    digest = _digest(cus + headers, " ".join(NVCC_FLAGS))
    if not force and _fresh(CUDA_LIB, digest):
        return CUDA_LIB
    os.makedirs(BUILD, exist_ok=True)
    nvcc = _nvcc()
    log = []
    objs = [os.path.join(BUILD, os.path.basename(c)[:-3] + ".o") for c in cus]
    with cf.ThreadPoolExecutor(max_workers=min(8, len(cus))) as ex:
        futs = [ex.submit(_run, [nvcc] + NVCC_FLAGS + ["-c", c, "-o", o], log) for c, o in zip(cus, objs)]
        for f in futs:
            f.result()
    _run([nvcc, "-shared", "-o", CUDA_LIB] + objs + ["-lcudart"], log)
    with open(_stamp(CUDA_LIB), "w") as fh:
        fh.write(digest)
    with open(os.path.join(BUILD, "build.log"), "w") as fh:
        fh.write("\n".join(log))
    if verbose:
        print("\n".join(log))
    return CUDA_LIB


def build_data(force=False):
    cpps = [c for c in _sources(".cpp") if os.path.basename(c) not in NATIVE_SOURCES]
    digest = _digest(cpps)
    if not force and _fresh(DATA_LIB, digest):
        return DATA_LIB
    cxx = shutil.which("g++") or "g++"
    log = []
    _run([cxx, "-O3", "-std=c++17", "-shared", "-fPIC", "-o", DATA_LIB] + cpps, log)
    with open(_stamp(DATA_LIB), "w") as fh:
        fh.write(digest)
    return DATA_LIB


def build_native(force=False):
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    cpps = [os.path.join(HERE, c) for c in NATIVE_SOURCES]
    digest = _digest(cpps + [os.path.join(HERE, h) for h in NATIVE_HEADERS], f"{torch.__version__} {sys.version}")
    if not force and _fresh(NATIVE_MODULE, digest):
        return NATIVE_MODULE
    cxx = shutil.which("g++") or "g++"
    inc = cpp_extension.include_paths(device_type="cuda") + [sysconfig.get_paths()["include"]]
    log = []
    _run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_native", "-DTORCH_API_INCLUDE_EXTENSION_H",
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + ["-I" + i for i in inc] + cpps
         + ["-o", NATIVE_MODULE] + ["-L" + d for d in cpp_extension.library_paths()]
         + ["-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10", "-lc10_cuda", "-ltorch_cuda", "-ldl"], log)
    with open(_stamp(NATIVE_MODULE), "w") as fh:
        fh.write(digest)
    return NATIVE_MODULE


def build_all(force=False, verbose=False):
    with cf.ThreadPoolExecutor(max_workers=3) as ex:
        futs = [ex.submit(build_cuda, force, verbose), ex.submit(build_data, force), ex.submit(build_native, force)]
        return tuple(f.result() for f in futs)


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    libs = build_all(a.force, a.verbose)
    print("built:", *libs)
