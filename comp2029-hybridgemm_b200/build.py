"""Build the CUDA library in-tree for sm_100a: ``python build.py`` (nvcc and g++, no GPU needed)."""
from __future__ import annotations

import subprocess
import sys
import sysconfig
from pathlib import Path

HERE = Path(__file__).resolve().parent
CSRC = HERE / "csrc"
LIBRARY = HERE / "lib" / "libhygemm_b200.so"
TRACE_LIBRARY = HERE / "lib" / "libhygemm_b200_trace.so"   # same sources with -DHG_TRACE (per-CTA time stamps)
HOST_EXTENSION = HERE / "lib" / "_hygemm_host.so"          # host path of a layer call, against the installed torch
HOST_SOURCE = CSRC / "hg_host.cpp"
SOURCES = ["hg_quant.cu", "hg_gemm_simt.cu", "hg_gemm_tc.cu", "hg_gemm_cluster.cu", "hg_runtime.cu", "hg_tp.cu", "hg_clip.cu"]
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
         "-Xcompiler", "-fPIC", "-shared", "-cudart", "static"]


def stale(library: Path = LIBRARY) -> bool:
    if not library.exists():
        return True
    built = library.stat().st_mtime
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + [HERE.parent / "include" / "hygemm.h"]
    return any(d.stat().st_mtime > built for d in deps)


def build_host_extension(force: bool = False) -> Path:
    """Compile ``lib/_hygemm_host.so``; returns its path."""
    if not force and HOST_EXTENSION.exists() and HOST_EXTENSION.stat().st_mtime >= max(
            d.stat().st_mtime for d in (HOST_SOURCE, HERE.parent / "include" / "hygemm.h")):
        return HOST_EXTENSION
    from torch.utils.cpp_extension import include_paths, library_paths
    HOST_EXTENSION.parent.mkdir(exist_ok=True)
    cmd = ["g++", "-O2", "-std=c++20", "-fPIC", "-shared", "-Wall", "-I", sysconfig.get_paths()["include"],
           *[a for p in include_paths("cuda") for a in ("-isystem", p)], str(HOST_SOURCE), "-o", str(HOST_EXTENSION),
           *["-L" + p for p in library_paths("cuda")], "-lc10", "-lc10_cuda", "-lcudart", "-ltorch_cpu", "-ltorch_python"]
    result = subprocess.run(cmd, capture_output=True, text=True)
    if result.returncode:
        sys.stderr.write(result.stdout + result.stderr)
        raise RuntimeError(f"g++ failed building {HOST_EXTENSION.name}")
    return HOST_EXTENSION


def build_library(force: bool = False, verbose: bool = False, trace: bool = False) -> Path:
    """Compile every kernel into ``lib/libhygemm_b200.so`` (``trace``: the diagnostic twin
    ``lib/libhygemm_b200_trace.so``, whose GEMM kernel records per-CTA time stamps); returns its path.  Builds the host extension too."""
    build_host_extension(force)
    library = TRACE_LIBRARY if trace else LIBRARY
    if not force and not stale(library):
        return library
    library.parent.mkdir(exist_ok=True)
    cmd = ["nvcc", *FLAGS, "-t", "0", *(["-DHG_TRACE=1"] if trace else []), *(["-Xptxas", "-v"] if verbose else []),
           *[str(CSRC / s) for s in SOURCES], "-o", str(library)]
    result = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or result.returncode:
        sys.stderr.write(result.stdout + result.stderr)
    if result.returncode:
        raise RuntimeError(f"nvcc failed building {library.name}")
    return library


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv, trace="--trace" in sys.argv))
