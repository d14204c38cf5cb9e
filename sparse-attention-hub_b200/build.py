"""Build the sm_100a shared library `lib/libsah_b200.so` from `csrc/*.cu`, and the host module
`lib/_sah_step.so` (CPython, against torch's headers) from `host/sah_step.cpp`.

    python sparse-attention-hub_b200/build.py [--force] [--verbose]

nvcc cross-compiles for sm_100a without a GPU.  The library exports only the
C ABI declared in `include/sah_b200.h`; it links the CUDA runtime dynamically so
that it shares the runtime instance of whatever process loads it.
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from importlib import metadata
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
REPO_DIR = PKG_DIR.parent
CSRC = PKG_DIR / "csrc"
LIB_DIR = PKG_DIR / "lib"
LIB_PATH = LIB_DIR / "libsah_b200.so"
OBJ_DIR = PKG_DIR / "build"
STEP_SRC = PKG_DIR / "host" / "sah_step.cpp"
STEP_PATH = LIB_DIR / "_sah_step.so"
STEP_STAMP = OBJ_DIR / "_sah_step.made_for"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-cudart", "shared",
    f"-I{REPO_DIR / 'include'}",
    f"-I{CSRC}",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the sm_100a library cannot be built")
    return exe


def _sources() -> list[Path]:
    return sorted(CSRC.glob("*.cu"))


def _deps_mtime() -> float:
    files = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + [REPO_DIR / "include" / "sah_b200.h"]
    return max(f.stat().st_mtime for f in files)


def is_stale() -> bool:
    return (not LIB_PATH.exists()) or LIB_PATH.stat().st_mtime < _deps_mtime()


def _step_made_for() -> str:
    """What the host module's binary interface depends on besides its sources."""
    return f"torch {metadata.version('torch')}, {sysconfig.get_config_var('SOABI')}"


def step_is_stale() -> bool:
    newest = max(f.stat().st_mtime for f in (STEP_SRC, REPO_DIR / "include" / "sah_b200.h"))
    return (not STEP_PATH.exists() or STEP_PATH.stat().st_mtime < newest
            or not STEP_STAMP.exists() or STEP_STAMP.read_text() != _step_made_for())


def build_step(force: bool = False, verbose: bool = False) -> Path:
    """Compile the host module; returns its path."""
    if not force and not step_is_stale():
        return STEP_PATH
    import torch
    from torch.utils import cpp_extension

    LIB_DIR.mkdir(exist_ok=True)
    tmp = STEP_PATH.with_suffix(".so.tmp")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           f"-I{REPO_DIR / 'include'}", f"-isystem{sysconfig.get_paths()['include']}",
           *(f"-isystem{d}" for d in cpp_extension.include_paths()), str(STEP_SRC), "-o", str(tmp),
           *(f"-L{d}" for d in cpp_extension.library_paths()), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed on {STEP_SRC.name}")
    os.replace(tmp, STEP_PATH)
    OBJ_DIR.mkdir(exist_ok=True)
    STEP_STAMP.write_text(_step_made_for())
    return STEP_PATH


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every kernel file and link the shared library, and build the host module; returns the
    library's path."""
    build_step(force, verbose)
    if not force and not is_stale():
        return LIB_PATH
    nvcc = _nvcc()
    OBJ_DIR.mkdir(exist_ok=True)
    LIB_DIR.mkdir(exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []

    def compile_one(src: Path) -> Path:
        obj = OBJ_DIR / (src.stem + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", str(src), "-o", str(obj)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or res.returncode != 0:
            sys.stderr.write(res.stdout + res.stderr)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_one, _sources()))
    tmp = LIB_PATH.with_suffix(".so.tmp")
    cmd = [nvcc, "-shared", "-cudart", "shared", "-gencode", "arch=compute_100a,code=sm_100a",
           "-o", str(tmp), *map(str, objs),
           "-Xlinker", "-rpath", "-Xlinker", "/usr/local/cuda/lib64"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("link of libsah_b200.so failed")
    os.replace(tmp, LIB_PATH)
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="--verbose" in sys.argv)
    print(path)
