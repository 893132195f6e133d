"""Builds the native library in-tree with nvcc for sm_100a.

``python -m flagdnn_b200.build`` compiles ``csrc/*.cu`` into
``flagdnn_b200/libflagdnn_b200.so``.  nvcc cross-compiles without a GPU, so
this runs on build machines that have none.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
LIB_PATH = PKG_DIR / "libflagdnn_b200.so"
HOST_SOURCE = CSRC / "host" / "fastcall.cpp"
HOST_PATH = PKG_DIR / "_fastcall.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--threads", "4",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _stale() -> bool:
    if not LIB_PATH.exists():
        return True
    built = LIB_PATH.stat().st_mtime
    deps = [p for p in CSRC.glob("*") if p.is_file()] + [PKG_DIR.parent / "include" / "flagdnn_b200.h"]
    return any(p.stat().st_mtime > built for p in deps if p.exists())


def build(force: bool = False, verbose: bool = False, ptxas_info: bool = False) -> Path:
    """Compile the library if it is missing or older than its sources."""
    if not force and not _stale():
        return LIB_PATH
    cmd = [_nvcc(), *NVCC_FLAGS, "-shared", "-o", str(LIB_PATH)]
    if ptxas_info:
        cmd += ["-Xptxas", "-v"]
    cmd += [str(s) for s in sources()]
    if verbose:
        print(" ".join(cmd), file=sys.stderr)
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"nvcc failed ({proc.returncode}):\n{proc.stdout}\n{proc.stderr}")
    if verbose or ptxas_info:
        sys.stderr.write(proc.stdout + proc.stderr)
    return LIB_PATH


def host_tag() -> str:
    """What the host path must have been compiled against; the module carries it as ``built_for``."""
    import torch

    return f"flagdnn host path for torch {torch.__version__}"


def _host_stale() -> bool:
    """Missing, older than its source or the C ABI's header, or compiled against another torch."""
    header = PKG_DIR.parent / "include" / "flagdnn_b200.h"
    if not HOST_PATH.exists():
        return True
    built = HOST_PATH.stat().st_mtime
    if any(p.stat().st_mtime > built for p in (HOST_SOURCE, header) if p.exists()):
        return True
    return (host_tag() + "\0").encode() not in HOST_PATH.read_bytes()


def build_host(force: bool = False, verbose: bool = False) -> Path:
    """Compile the native host path of the eager operators (csrc/host/fastcall.cpp) against the installed torch."""
    if not force and not _host_stale():
        return HOST_PATH
    import sysconfig

    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parent.parent
    cxx = os.environ.get("CXX", "g++")
    if shutil.which(cxx) is None:
        raise RuntimeError(f"{cxx} not found; set CXX or put it on PATH")
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DFDNN_HOST_TAG="{host_tag()}"',
           f"-I{root / 'include'}", f"-I{root / 'include' / 'torch' / 'csrc' / 'api' / 'include'}",
           f"-I{sysconfig.get_paths()['include']}", f"-I{cuda / 'include'}",
           "-o", str(HOST_PATH), str(HOST_SOURCE), f"-L{root / 'lib'}",
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python", f"-Wl,-rpath,{root / 'lib'}"]
    if verbose:
        print(" ".join(cmd), file=sys.stderr)
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(f"{cxx} failed ({proc.returncode}):\n{proc.stdout}\n{proc.stderr}")
    return HOST_PATH


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True, ptxas_info="--ptxas-info" in sys.argv)
    build_host(force="--force" in sys.argv, verbose=True)   # the kernels do not wait for a host compiler
    print(LIB_PATH)
