"""Build ``libpe_gb300.so`` (the C-ABI library of sm_103a kernels) in-tree.

Each ``csrc/*.cu`` translation unit is compiled in parallel with nvcc for
``sm_103a`` only, then linked into ``panoptic_evaluator_gb300/libpe_gb300.so``.
Beside them ``csrc/host.cpp``, the evaluators' host path against torch's C++
API, becomes the extension module ``panoptic_evaluator_gb300/_host.so``, and
``_host.tag`` names the torch and Python it was built against; without it (no
torch headers) the evaluators take their Python host path. Objects go to
``_build/`` at the repository root. Rebuilds only when a source or header is
newer than the library, or when torch or Python is another.

    python -m panoptic_evaluator_gb300.build [--force] [--verbose]
"""

from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import warnings
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

from . import _native
from ._native import HOST_MODULE, HOST_TAG, host_tag

PACKAGE = Path(__file__).resolve().parent
CSRC = PACKAGE / "csrc"
ROOT = PACKAGE.parent
BUILD = ROOT / "_build"
LIBRARY = PACKAGE / "libpe_gb300.so"
HOST_SOURCE = CSRC / "host.cpp"
NOT_COMPILED = "\nnot compiled"  # in HOST_TAG: tried for this torch and Python without success
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC,-fvisibility=hidden",
         "-I", str(CSRC), "-I", str(ROOT / "include")]


def nvcc() -> str:
    for candidate in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if candidate and Path(candidate).exists():
            return candidate
    raise RuntimeError("nvcc not found; the CUDA toolkit is required to build libpe_gb300.so")


def sources():
    return sorted(CSRC.glob("*.cu"))


def stale() -> bool:
    if not LIBRARY.exists() or not HOST_TAG.exists():
        return True
    tag = HOST_TAG.read_text()
    if tag != host_tag() + NOT_COMPILED and (tag != host_tag() or not HOST_MODULE.exists()):
        return True
    built = min(LIBRARY.stat().st_mtime, HOST_TAG.stat().st_mtime)
    inputs = [*sources(), HOST_SOURCE, *CSRC.glob("*.cuh"), *CSRC.glob("*.h"), *(ROOT / "include").glob("*.h"),
              Path(__file__)]
    return any(path.stat().st_mtime > built for path in inputs)


def compile_host(verbose: bool = False) -> Path:
    """csrc/host.cpp -> _host.so, against the installed torch."""
    import sysconfig

    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc()).resolve().parent.parent
    include = [root / "include", root / "include/torch/csrc/api/include", sysconfig.get_paths()["include"],
               cuda / "include"]
    libraries = [root / "lib", cuda / "lib64"]
    tmp = HOST_MODULE.with_suffix(".so.tmp")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           "-Wall", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-isystem{p}" for p in include], f"-I{CSRC}", f"-I{ROOT / 'include'}", str(HOST_SOURCE), "-o", str(tmp),
           *[f"-L{p}" for p in libraries], "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-lcudart"]
    if verbose:
        print(" ".join(cmd), flush=True)
    result = subprocess.run(cmd, capture_output=True, text=True)
    if result.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed for {HOST_SOURCE.name}:\n{result.stdout}\n{result.stderr}")
    if verbose and (result.stdout or result.stderr):
        print(result.stdout + result.stderr, flush=True)
    os.replace(tmp, HOST_MODULE)
    return HOST_MODULE


def build_host(verbose: bool = False) -> None:
    """_host.so and its tag; a failure is a warning, since every evaluator has a Python host path as well."""
    HOST_TAG.unlink(missing_ok=True)
    try:
        compile_host(verbose)
        HOST_TAG.write_text(host_tag())
        if _native._host is False:  # looked for before it was there
            _native._host = None
    except (OSError, RuntimeError) as error:
        HOST_MODULE.unlink(missing_ok=True)
        HOST_TAG.write_text(host_tag() + NOT_COMPILED)
        warnings.warn(f"{HOST_MODULE.name} was not built: {error}", RuntimeWarning, stacklevel=2)


def build(force: bool = False, verbose: bool = False, extra: list[str] | None = None) -> Path:
    if not force and not stale():
        return LIBRARY
    compiler = nvcc()
    BUILD.mkdir(exist_ok=True)
    extra = list(extra or [])

    def compile_one(src: Path) -> Path:
        obj = BUILD / (src.stem + ".o")
        cmd = [compiler, *ARCH, *FLAGS, *extra, "-c", str(src), "-o", str(obj)]
        if verbose:
            print(" ".join(cmd), flush=True)
        result = subprocess.run(cmd, capture_output=True, text=True)
        if result.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src.name}:\n{result.stdout}\n{result.stderr}")
        if verbose and (result.stdout or result.stderr):
            print(result.stdout + result.stderr, flush=True)
        return obj

    with ThreadPoolExecutor(max_workers=min(9, os.cpu_count() or 1)) as pool:
        host = pool.submit(build_host, verbose)
        objects = list(pool.map(compile_one, sources()))
        host.result()
    tmp = LIBRARY.with_suffix(".so.tmp")
    cmd = [compiler, *ARCH, "-shared", "-o", str(tmp), *map(str, objects), "-lcudart"]
    result = subprocess.run(cmd, capture_output=True, text=True)
    if result.returncode != 0:
        raise RuntimeError(f"link failed:\n{result.stdout}\n{result.stderr}")
    os.replace(tmp, LIBRARY)
    return LIBRARY


def main(argv=None):
    parser = argparse.ArgumentParser(description=__doc__.splitlines()[0])
    parser.add_argument("--force", action="store_true")
    parser.add_argument("--verbose", action="store_true")
    parser.add_argument("--ptxas-info", action="store_true", help="print registers/spills per kernel")
    args = parser.parse_args(argv)
    extra = ["-Xptxas", "-v"] if args.ptxas_info else None
    path = build(force=args.force or args.ptxas_info, verbose=args.verbose or args.ptxas_info, extra=extra)
    print(path)


if __name__ == "__main__":
    sys.exit(main())
