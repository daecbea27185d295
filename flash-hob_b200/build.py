"""Builds libfhob.so (the C-ABI library) in-tree with nvcc for sm_100a.

Usage: python flash-hob_b200/build.py [--force] [--verbose]
The library lands next to the Python host module (fhob/libfhob.so) so it
travels with the source tree; nothing is installed into site-packages.
fhob/_native.so, the host path of the Python package, is built beside it with g++.
Each source file is compiled to an object of its own (in parallel, and only
when it or a header changed), then the objects are linked.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
OBJ = HERE / "build"
OUT = HERE / "fhob" / "libfhob.so"
NATIVE = HERE / "fhob" / "_native.so"          # host path of the Python package, against torch's C++ API
NATIVE_SOURCE = "host_binding.cpp"
SOURCES = ["fhob_api.cu", "simt_kernels.cu", "tc_kernels.cu", "tc_forward.cu", "tc_backward.cu", "static_scratch.cu"]
HEADERS = ["fhob_common.cuh", "sm100_ptx.cuh", "tc_common.cuh", "../../include/fhob.h"]
FLAGS = ["-Xcompiler", "-fPIC", "-O3", "-std=c++17", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc_path() -> str:
    cuda_home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cand = Path(cuda_home) / "bin" / "nvcc"
    return str(cand) if cand.exists() else "nvcc"


def _newest_header() -> float:
    return max(p.stat().st_mtime for p in [(CSRC / h).resolve() for h in HEADERS] + [Path(__file__)])


def _native_stale() -> bool:
    deps = [CSRC / NATIVE_SOURCE, (CSRC / "../../include/fhob.h").resolve(), Path(__file__)]
    return not NATIVE.exists() or NATIVE.stat().st_mtime < max(p.stat().st_mtime for p in deps)


def _native_object(force: bool):
    """Compiles the binding (no link yet: it needs libfhob.so); None when it is up to date."""
    if not force and not _native_stale():
        return None
    import torch
    inc = Path(torch.__file__).parent / "include"
    cuda = Path(nvcc_path()).parent.parent / "include"
    obj = OBJ / "host_binding.o"
    subprocess.run(["g++", "-c", "-O2", "-std=c++17", "-fPIC", "-Wno-interference-size", f"-I{inc}",
                    f"-I{inc}/torch/csrc/api/include", f"-I{cuda}", f"-I{sysconfig.get_paths()['include']}",
                    str(CSRC / NATIVE_SOURCE), "-o", str(obj)], check=True)
    return obj


def _link_native(obj: Path) -> None:
    import torch
    subprocess.run(["g++", "-shared", str(obj), "-o", str(NATIVE), f"-L{Path(torch.__file__).parent / 'lib'}", "-lc10",
                    "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", f"-L{OUT.parent}", f"-l:{OUT.name}",
                    "-Wl,-rpath,$ORIGIN"], check=True)


def is_stale() -> bool:
    if not OUT.exists() or not NATIVE.exists() or _native_stale():
        return True
    t = OUT.stat().st_mtime
    return _newest_header() > t or any((CSRC / s).stat().st_mtime > t for s in SOURCES)


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not is_stale():
        return OUT
    OBJ.mkdir(exist_ok=True)
    nvcc, hdr = nvcc_path(), _newest_header()
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src: str) -> Path:
        obj = OBJ / (Path(src).stem + ".o")
        if (force or verbose or not obj.exists()
                or obj.stat().st_mtime < max(hdr, (CSRC / src).stat().st_mtime)):
            subprocess.run([nvcc, "-c", *FLAGS, *extra, "-o", str(obj), str(CSRC / src)], check=True)
        return obj

    with ThreadPoolExecutor(max_workers=len(SOURCES) + 1) as pool:
        native = pool.submit(_native_object, force)
        objs = list(pool.map(compile_one, SOURCES))
        native_obj = native.result()
    subprocess.run([nvcc, "-shared", *FLAGS, "-o", str(OUT)] + [str(o) for o in objs], check=True)
    if native_obj is not None:
        _link_native(native_obj)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
