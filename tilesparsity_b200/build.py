"""In-tree build of libtilesparse.so (sm_100a) and of the _tsfast extension.

`python tilesparsity_b200/build.py` compiles every .cu file under csrc/ with nvcc (cross-compiles
without a GPU) and links the shared library next to this file, where the loader looks for it; then
csrc/pyfast.cpp, the host path of the per-batch operators, with g++ against the installed torch.
"""
from __future__ import annotations

import importlib.metadata
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "obj")
LIB_PATH = os.path.join(HERE, "libtilesparse.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def extension_path(torch_version: str) -> str:
    """Where the extension built for this Python and that torch lies.  It is linked against torch's C++ ABI: another
    version's build has another name and is not loaded."""
    return os.path.join(HERE, f"_tsfast.{sysconfig.get_config_var('SOABI')}-torch{torch_version}.so")


def sources() -> list[str]:
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers() -> list[str]:
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))] + \
        [os.path.join(HERE, "..", "include", "tilesparse.h")]


def _older(path: str, deps: list[str]) -> bool:
    """Whether `path` is missing or older than one of `deps`."""
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; libtilesparse.so cannot be built")
    return nvcc


def _run(cmd: list[str]) -> str:
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(cmd[0] + " failed:\n" + proc.stdout + proc.stderr)
    return proc.stderr


def _build_library(force: bool, verbose: bool) -> None:
    os.makedirs(OBJ, exist_ok=True)
    nvcc, flags = find_nvcc(), NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else [])
    objects, todo = [], []
    for src in sources():
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        objects.append(obj)
        if force or _older(obj, [src] + _headers()):
            todo.append([nvcc, *flags, "-c", "-o", obj, src])
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 1) as pool:
        for err in pool.map(_run, todo):
            if verbose:
                sys.stderr.write(err)
    _run([nvcc, *NVCC_FLAGS, "-shared", "-o", LIB_PATH + ".tmp", *objects])
    os.replace(LIB_PATH + ".tmp", LIB_PATH)


def numpy_include() -> str:
    import numpy
    return numpy.get_include()


def _build_extension(path: str) -> None:
    root = os.path.dirname(importlib.util.find_spec("torch").origin)
    inc, lib = os.path.join(root, "include"), os.path.join(root, "lib")
    cuda = os.path.join(os.path.dirname(os.path.dirname(find_nvcc())), "include")
    _run([shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
          "-I" + inc, "-I" + os.path.join(inc, "torch", "csrc", "api", "include"), "-I" + cuda,
          "-I" + sysconfig.get_paths()["include"], "-I" + numpy_include(), "-o", path + ".tmp", os.path.join(CSRC, "pyfast.cpp"),
          "-L" + HERE, "-l:libtilesparse.so", "-Wl,-rpath,$ORIGIN", "-L" + lib, "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu",
          "-lc10_cuda", "-lc10"])
    os.replace(path + ".tmp", path)


def build(force: bool = False, verbose: bool = False) -> str:
    """Builds what is missing or older than its sources; returns the library's path."""
    if force or _older(LIB_PATH, sources() + _headers()):
        _build_library(force, verbose)
    ext = extension_path(importlib.metadata.version("torch"))
    if force or _older(ext, [os.path.join(CSRC, "pyfast.cpp"), os.path.join(HERE, "..", "include", "tilesparse.h")]):
        _build_extension(ext)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
