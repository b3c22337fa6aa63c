"""Builds libmimk.so (the C-ABI kernel library) in-tree with nvcc for sm_100a, and _native.so (the operators' calls from Python) with g++.

    python -m mimir_b200.build [--force] [--verbose]

nvcc cross-compiles without a GPU.  Objects go to mimir_b200/_build/, the library to mimir_b200/libmimk.so.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import importlib.metadata
import importlib.util
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libmimk.so")
NATIVE = os.path.join(HERE, "_native.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC or put it on PATH)")


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _native_for() -> str:
    """What the extension module is built against, found without importing torch."""
    return "\n".join([sys.version, importlib.metadata.version("torch"), importlib.util.find_spec("torch").origin])


def _build_native(force: bool, verbose: bool) -> None:
    """The extension module, against this interpreter's torch; it finds libmimk.so beside itself. Built anew for a newer source, and for another
    torch or interpreter than it was built for."""
    src, built_for = os.path.join(CSRC, "py_ops.cpp"), os.path.join(OBJ, "native_for.txt")
    if not force and not _stale(NATIVE, [src, os.path.join(ROOT, "include", "mimk.h")]) and os.path.exists(built_for):
        with open(built_for) as f:
            if f.read() == _native_for():
                return
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    includes = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include"), os.path.join(ROOT, "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           src, "-o", NATIVE, *(f"-I{i}" for i in includes), f"-L{lib}", f"-L{HERE}", "-l:libmimk.so", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu",
           "-ltorch", "-lc10_cuda", "-lc10", "-Wl,-rpath,$ORIGIN", f"-Wl,-rpath,{lib}"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode != 0:
        sys.stderr.write(f"--- py_ops.cpp\n{r.stdout}{r.stderr}\n")
    if r.returncode != 0:
        raise RuntimeError("g++ failed on py_ops.cpp")
    with open(built_for, "w") as f:
        f.write(_native_for())


def build(force: bool = False, verbose: bool = False) -> str:
    nvcc = _nvcc()
    os.makedirs(OBJ, exist_ok=True)
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(ROOT, "include", "*.h"))
    jobs = []
    for src in sources():
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
            jobs.append((src, cmd))

    def run(job):
        src, cmd = job
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r

    with cf.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for src, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(f"--- {os.path.basename(src)}\n{r.stdout}{r.stderr}\n")
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src}")
    objs = [os.path.join(OBJ, os.path.basename(s)[:-3] + ".o") for s in sources()]
    if force or jobs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    _build_native(force, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
