"""In-tree build of the CUDA library (``cumm_b200/libcumm_b200.so``, sm_100a) and of the extension that reads
parameter records (``cumm_b200/_host.so``)."""
from __future__ import annotations

import os
import shutil
import subprocess
from pathlib import Path

_HERE = Path(__file__).resolve().parent
CSRC = _HERE / "csrc"
OUT = _HERE / "libcumm_b200.so"
HOST_OUT = _HERE / "_host.so"
SOURCES = ["api.cu"]
HOST_SOURCES = ["host_args.cpp"]
HEADERS = sorted(p.name for p in CSRC.glob("*.cuh"))


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found")
    return cand


def needs_build() -> bool:
    if not (OUT.exists() and HOST_OUT.exists()):
        return True
    t = min(OUT.stat().st_mtime, HOST_OUT.stat().st_mtime)
    deps = [CSRC / s for s in SOURCES + HOST_SOURCES + HEADERS] + [_HERE.parent / "include" / "cumm_b200.h"]
    return any(d.exists() and d.stat().st_mtime > t for d in deps)


def _build_host() -> None:
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    cxx = shutil.which("g++")
    if cxx is None:
        raise RuntimeError("g++ not found")
    cmd = [cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-o", str(HOST_OUT)]
    cmd += ["-I" + p for p in (sysconfig.get_paths()["include"], str(root / "include"),
                               str(root / "include" / "torch" / "csrc" / "api" / "include"))]
    cmd += [str(CSRC / s) for s in HOST_SOURCES]
    cmd += ["-L" + str(root / "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10"]
    subprocess.run(cmd, check=True, cwd=str(CSRC))


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not needs_build():
        return OUT
    cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
           "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-o", str(OUT)]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += [str(CSRC / s) for s in SOURCES]
    subprocess.run(cmd, check=True, cwd=str(CSRC))
    _build_host()
    return OUT


if __name__ == "__main__":
    print(build(force=True, verbose=bool(os.environ.get("VERBOSE"))))
