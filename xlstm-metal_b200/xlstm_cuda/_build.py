"""Build ``libxlstm_cuda.so`` from ``csrc/`` with nvcc for sm_100a (in-tree, no JIT cache)."""
from __future__ import annotations

import os
import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG.parent / "csrc"
INCLUDE = PKG.parent.parent / "include"
OBJ = CSRC / "build"
LIB = PKG / "libxlstm_cuda.so"
HOST_SRC = CSRC / "host.cpp"     # tensor-level front end: a Python extension over the C ABI
HOST = PKG / "_host.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-I", str(INCLUDE), "-I", str(CSRC),
]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"
    return cand if Path(cand).exists() else "nvcc"


def sources():
    return sorted(CSRC.glob("*.cu"))


def needs_build() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h"))
    return any(d.stat().st_mtime > t for d in deps)


def build_host(force: bool = False) -> Path:
    """Compile the tensor-level front end against the installed torch."""
    deps = [HOST_SRC, *INCLUDE.glob("*.h")]
    if not force and HOST.exists() and all(d.stat().st_mtime <= HOST.stat().st_mtime for d in deps):
        return HOST
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_host",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-I{d}" for d in (*include_paths("cuda"), sysconfig.get_paths()["include"], INCLUDE)),
           str(HOST_SRC), "-o", str(HOST), *(f"-L{d}" for d in library_paths("cuda")),
           "-lc10", "-ltorch_cpu", "-lc10_cuda", "-ltorch_cuda", "-ltorch", "-ltorch_python",
           f"-L{PKG}", f"-l:{LIB.name}", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{HOST_SRC.name} failed to build:\n{r.stderr}")
    return HOST


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile every ``.cu`` to an object (in parallel) and link the shared library."""
    if not force and not needs_build():
        build_host()
        return LIB
    OBJ.mkdir(parents=True, exist_ok=True)
    nvcc = _nvcc()
    hdr_time = max(d.stat().st_mtime for d in list(CSRC.glob("*.cuh")) + list(INCLUDE.glob("*.h")))

    def compile_one(src: Path) -> Path:
        obj = OBJ / (src.stem + ".o")
        if not force and obj.exists() and obj.stat().st_mtime > max(src.stat().st_mtime, hdr_time):
            return obj
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose:
            print(r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stderr}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        objs = list(ex.map(compile_one, sources()))
    cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stderr}")
    build_host(force)
    return LIB


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
