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


def host_extension() -> Path:
    """Where the host path of a layer call is built.  It is C++ against torch and CPython, whose binary interfaces change with
    their versions, so it is named after both: after an upgrade another file is looked for and built."""
    import torch
    return HERE / "lib" / f"_hygemm_host.torch-{torch.__version__}.{sys.implementation.cache_tag}.so"


def build_host_extension(force: bool = False) -> Path:
    """Compile the host extension; returns its path."""
    extension = host_extension()
    if not force and extension.exists() and extension.stat().st_mtime >= max(
            d.stat().st_mtime for d in (HOST_SOURCE, HERE.parent / "include" / "hygemm.h")):
        return extension
    from torch.utils.cpp_extension import include_paths, library_paths
    extension.parent.mkdir(exist_ok=True)
    cmd = ["g++", "-O2", "-std=c++20", "-fPIC", "-shared", "-Wall", "-I", sysconfig.get_paths()["include"],
           *[a for p in include_paths("cuda") for a in ("-isystem", p)], str(HOST_SOURCE), "-o", str(extension),
           *["-L" + p for p in library_paths("cuda")], "-lc10", "-lc10_cuda", "-lcudart", "-ltorch_cpu", "-ltorch_python"]
    result = subprocess.run(cmd, capture_output=True, text=True)
    if result.returncode:
        sys.stderr.write(result.stdout + result.stderr)
        raise RuntimeError(f"g++ failed building {extension.name}")
    return extension


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
