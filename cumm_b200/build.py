"""In-tree build of the CUDA library (``cumm_b200/libcumm_b200.so``, sm_100a) and of the extension that reads
parameter records (``_lib.host_path()``), which the library does without where it cannot be built."""
from __future__ import annotations

import os
import shutil
import subprocess
import warnings
from pathlib import Path

from ._lib import host_path, host_sources

_HERE = Path(__file__).resolve().parent
CSRC = _HERE / "csrc"
OUT = _HERE / "libcumm_b200.so"
SOURCES = ["api.cu"]
HOST_SOURCES = ["host_args.cpp"]
HEADERS = sorted(p.name for p in CSRC.glob("*.cuh"))


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found")
    return cand


def _stale(out: Path, sources) -> bool:
    deps = [CSRC / s for s in sources] + [_HERE.parent / "include" / "cumm_b200.h"]
    return not out.exists() or any(d.exists() and d.stat().st_mtime > out.stat().st_mtime for d in deps)


def needs_build() -> bool:
    return _stale(OUT, SOURCES + HEADERS) or _stale(host_path(), HOST_SOURCES)


def _build_host() -> None:
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    cxx = shutil.which("g++")
    if cxx is None:
        raise RuntimeError("g++ not found")
    cmd = [cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DCB2_HOST_SOURCES="{host_sources()}"', "-o", str(host_path())]
    cmd += ["-I" + p for p in (sysconfig.get_paths()["include"], str(root / "include"),
                               str(root / "include" / "torch" / "csrc" / "api" / "include"))]
    cmd += [str(CSRC / s) for s in HOST_SOURCES]
    cmd += ["-L" + str(root / "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10"]
    subprocess.run(cmd, check=True, cwd=str(CSRC))


def build(force: bool = False, verbose: bool = False) -> Path:
    if force or _stale(OUT, SOURCES + HEADERS):
        _build_library(verbose)
    if force or _stale(host_path(), HOST_SOURCES):
        try:
            _build_host()
        except (RuntimeError, OSError, subprocess.CalledProcessError) as e:
            warnings.warn(f"the native reader of parameter records was not built: {e}", RuntimeWarning, stacklevel=2)
    return OUT


def _build_library(verbose: bool) -> None:
    cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
           "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-o", str(OUT)]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    cmd += [str(CSRC / s) for s in SOURCES]
    subprocess.run(cmd, check=True, cwd=str(CSRC))


if __name__ == "__main__":
    print(build(force=True, verbose=bool(os.environ.get("VERBOSE"))))
