"""Build recipe for the CUDA library: nvcc, sm_100a only, one object per family, in-tree output.

``python -m better_benchmark_b200.build`` (or ``build_library()``) compiles every ``csrc/*.cu``
file to an object in ``csrc/_build/`` in parallel and links ``csrc/libb200_oracles.so``, and compiles
``csrc/calls.cpp``, the host side of the most frequent calls, to an extension module beside it that is named after the torch
and the Python it is compiled against (``native.calls_path()``).
Objects are rebuilt only when their source (or a shared header) is newer.
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys
from pathlib import Path

CSRC = Path(__file__).resolve().parent / "csrc"
BUILD_DIR = CSRC / "_build"
LIB_PATH = CSRC / "libb200_oracles.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    # a*b+c stays two rounded operations, as in the decomposed aten graphs; no fast-math anywhere
    "-fmad=false",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: set NVCC or put /usr/local/cuda/bin on PATH")


def _stale(obj: Path, src: Path, headers: list[Path]) -> bool:
    if not obj.exists():
        return True
    t = obj.stat().st_mtime
    return any(dep.stat().st_mtime > t for dep in [src, *headers, Path(__file__)])


def build_calls(force: bool = False) -> Path:
    """The extension module, against the torch that runs this. It holds no device code."""
    from .native import calls_path
    src, out = CSRC / "calls.cpp", calls_path()
    if not force and not _stale(out, src, [CSRC.parent.parent / "include" / "b200_oracles.h"]):
        return out
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include",
                Path(sysconfig.get_paths()["include"]), Path(_nvcc()).resolve().parent.parent / "include"]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *(f"-I{p}" for p in includes), str(src),
           "-o", str(out), f"-L{root / 'lib'}", "-ltorch_python", "-ltorch_cpu", "-lc10_cuda", "-lc10"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed on {src.name}:\n{res.stdout}\n{res.stderr}")
    return out


def build_library(force: bool = False, verbose: bool = False) -> Path:
    nvcc = _nvcc()
    BUILD_DIR.mkdir(exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    headers = sorted(CSRC.glob("*.cuh"))
    jobs = []
    for src in sources:
        obj = BUILD_DIR / (src.stem + ".o")
        if force or _stale(obj, src, headers):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc, *NVCC_FLAGS, "-Xptxas=-v", "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        obj.with_suffix(".ptxas").write_text(res.stderr)   # registers and spills of every kernel
        return src, res

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, 1 + len(jobs))) as pool:
        calls = pool.submit(build_calls, force)
        for src, res in pool.map(compile_one, jobs):
            if verbose and res.stderr:
                print(res.stderr, file=sys.stderr)
            if res.returncode != 0:
                raise RuntimeError(f"nvcc failed on {src.name}:\n{res.stdout}\n{res.stderr}")
        calls.result()

    objs = [BUILD_DIR / (s.stem + ".o") for s in sources]
    if force or jobs or not LIB_PATH.exists():
        cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a",
               "-o", str(LIB_PATH), *map(str, objs)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    return LIB_PATH


if __name__ == "__main__":
    path = build_library(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
