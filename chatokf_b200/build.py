"""Build libokfcuda.so in-tree with nvcc for sm_100a.

    python -m chatokf_b200.build [--force] [--verbose]

The library links the CUDA runtime statically and exports only the C ABI of
include/okf_cuda.h.  Objects go to chatokf_b200/csrc/build/ (git-ignored); the
shared library sits beside this file so it travels with the package.  Beside it
goes _okfcall, the C module through which Python calls the library's hot entry
points; it is linked against torch, whose tensors it reads.
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


def needs_build() -> bool:
    return (_stale(LIB, max(p.stat().st_mtime for p in sources()))
            or _stale(PYMOD, max(PYCALL.stat().st_mtime, PYTENSOR.stat().st_mtime)))


def build_pycall() -> None:
    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc()).resolve().parent.parent
    inc = ["-I", sysconfig.get_paths()["include"]]
    obj, tobj = OBJ / "okf_pycall.o", OBJ / "okf_pytensor.o"
    tcmd = ["-I", str(root / "include"), "-I", str(root / "include" / "torch" / "csrc" / "api" / "include"), "-I", str(cuda / "include"),
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    flags = ["-O2", "-Wall", "-fPIC", "-fvisibility=hidden"]
    libs = ["-L" + str(root / "lib"), "-Wl,-rpath," + str(root / "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    cxx = shutil.which("g++") or "c++"
    cmds = [[shutil.which("gcc") or "cc", *flags, *inc, "-c", str(PYCALL), "-o", str(obj)]]
    if not tobj.exists() or _stale(tobj, max(PYTENSOR.stat().st_mtime, Path(torch.__file__).stat().st_mtime)):
        cmds.append([cxx, *flags, "-std=c++17", *inc, *tcmd, "-c", str(PYTENSOR), "-o", str(tobj)])
    cmds.append([cxx, "-shared", str(obj), str(tobj), *libs, "-o", str(PYMOD) + ".tmp"])
    for cmd in cmds:
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError(f"building {PYMOD.name} failed")
    os.replace(str(PYMOD) + ".tmp", PYMOD)


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
    build_pycall()
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
