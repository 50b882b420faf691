"""Build libokfcuda.so in-tree with nvcc for sm_100a.

    python -m chatokf_b200.build [--force] [--verbose]

The library links the CUDA runtime statically and exports only the C ABI of
include/okf_cuda.h.  Objects go to chatokf_b200/csrc/build/ (git-ignored); the
shared library sits beside this file so it travels with the package.  Beside it
goes _okfcall, the C module through which Python calls the library's hot entry
points, and for a torch with CUDA a library that reads this very torch's tensors.
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

from ._lib import tensor_path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = CSRC / "build"
LIB = PKG / "libokfcuda.so"
PYCALL = CSRC / "okf_pycall.c"
PYTENSOR = CSRC / "okf_pytensor.cpp"
PYMOD = PKG / ("_okfcall" + sysconfig.get_config_var("EXT_SUFFIX"))

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = [
    "-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC,-fvisibility=hidden",
    "--expt-relaxed-constexpr", "-Xptxas", "-warn-spills",
]


def nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found: libokfcuda.so cannot be built")
    return exe


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _headers_mtime() -> float:
    deps = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h"))
    deps.append(PKG.parent / "include" / "okf_cuda.h")
    return max(p.stat().st_mtime for p in deps)


def _stale(out: Path, src_mtime: float) -> bool:
    return not out.exists() or out.stat().st_mtime < max(src_mtime, _headers_mtime())


def _torch():
    try:
        import torch
    except ImportError:
        return None
    return torch


def needs_build() -> bool:
    tensor = tensor_path(_torch())
    return (_stale(LIB, max(p.stat().st_mtime for p in sources())) or _stale(PYMOD, PYCALL.stat().st_mtime)
            or (tensor is not None and _stale(tensor, PYTENSOR.stat().st_mtime)))


def _run(cmd: list[str], what: str) -> None:
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError(f"building {what} failed")


def build_pycall(force: bool = False) -> None:
    flags = ["-O2", "-Wall", "-fPIC", "-shared", "-fvisibility=hidden", "-I", sysconfig.get_paths()["include"]]
    _run([shutil.which("gcc") or "cc", *flags, str(PYCALL), "-o", str(PYMOD) + ".tmp"], PYMOD.name)
    os.replace(str(PYMOD) + ".tmp", PYMOD)
    torch = _torch()
    out = tensor_path(torch)
    if out is None or not (force or _stale(out, PYTENSOR.stat().st_mtime)):
        return
    root = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc()).resolve().parent.parent
    inc = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", cuda / "include"]
    libs = ["-L" + str(root / "lib"), "-Wl,-rpath," + str(root / "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    _run([shutil.which("g++") or "c++", *flags, "-std=c++17", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
          *(a for i in inc for a in ("-I", str(i))), str(PYTENSOR), *libs, "-o", str(out) + ".tmp"], out.name)
    os.replace(str(out) + ".tmp", out)


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not needs_build():
        return LIB
    OBJ.mkdir(exist_ok=True)
    cc = nvcc()
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src: Path) -> Path:
        obj = OBJ / (src.stem + ".o")
        if not force and not _stale(obj, src.stat().st_mtime):
            return obj
        cmd = [cc, *ARCH, *NVCC_FLAGS, *extra, "-c", str(src), "-o", str(obj)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode:
            sys.stderr.write(f"$ {' '.join(cmd)}\n{r.stdout}{r.stderr}")
        elif r.stderr.strip():
            sys.stderr.write(r.stderr)
        if r.returncode:
            raise RuntimeError(f"nvcc failed on {src.name}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_one, sources()))
    tmp = LIB.with_suffix(".so.tmp")
    cmd = [cc, *ARCH, "-shared", "-cudart", "static", "-o", str(tmp), *map(str, objs)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("link of libokfcuda.so failed")
    os.replace(tmp, LIB)
    build_pycall(force)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
