"""Builds the native libraries in-tree with nvcc / g++ (seconds per file).

    python -m pfeife_b200.csrc.build [--force] [--verbose]

Outputs, next to the package's ``__init__.py``:
  * ``libpfeife_b200_kernels.so`` - every CUDA kernel, compiled for sm_100a only
  * ``libpfeife_b200_host.so``    - host-side C++ (planner evaluator, step executor helpers)
  * ``libpfeife_b200_calls.<abi>.so`` - the kernel library's entry points as a Python module, for the
    Python that builds it; left out where that has no headers (calls then go through ctypes)
  * ``libpfeife_b200_eager-<torch>.<abi>.so`` - eager calls of the ops with their autograd nodes, for the
    PyTorch that is installed, whose headers it takes half a minute over; left out where those are
    missing or other than it was written against (eager calls then go through Python)

Objects are cached under ``build/`` keyed by source mtime, so rebuilding after a one-file edit
recompiles one file.
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import hashlib
import importlib.metadata
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

CSRC = Path(__file__).resolve().parent
PKG = CSRC.parent
BUILD = PKG.parent / "build" / "pfeife_b200"

KERNEL_LIB = PKG / "libpfeife_b200_kernels.so"
HOST_LIB = PKG / "libpfeife_b200_host.so"
CALLS_LIB = PKG / ("libpfeife_b200_calls" + sysconfig.get_config_var("EXT_SUFFIX"))
CALLS_SRC = CSRC / "calls.cpp"
EAGER_SRC = CSRC / "eager.cpp"


def eager_lib() -> Path:
    """The name carries the PyTorch and the Python that the module is built for."""
    return PKG / (f"libpfeife_b200_eager-{importlib.metadata.version('torch')}"
                  + sysconfig.get_config_var("EXT_SUFFIX"))


def eager_sources() -> str:
    """What the module says that it was built from; the loader takes no module of other sources."""
    return hashlib.sha256(b"".join(p.read_bytes() for p in (EAGER_SRC, CSRC / "api.h"))).hexdigest()

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]
# Approximate division / square root / transcendentals are fine for activations and softmax,
# not for the optimizer update: those two files are bandwidth-bound and keep IEEE arithmetic.
FAST_MATH = ["--use_fast_math"]
PRECISE_SOURCES = {"optim.cu", "dp_fused.cu"}
CXX_FLAGS = ["-O3", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-pthread"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; set NVCC or install the CUDA toolkit")


def _stale(obj: Path, deps: list[Path]) -> bool:
    if not obj.exists():
        return True
    t = obj.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def _run(cmd: list[str], verbose: bool) -> None:
    if verbose:
        print(" ".join(cmd), flush=True)
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"build step failed:\n{' '.join(cmd)}\n{r.stdout}")
    if verbose and r.stdout.strip():
        print(r.stdout)


def build(force: bool = False, verbose: bool = False, ptxas_info: bool = False) -> None:
    BUILD.mkdir(parents=True, exist_ok=True)
    headers = sorted(CSRC.glob("*.h")) + sorted(CSRC.glob("*.cuh"))
    cu = sorted(CSRC.glob("*.cu"))
    cpp = [p for p in sorted(CSRC.glob("*.cpp")) if p not in (CALLS_SRC, EAGER_SRC)]
    nvcc = _nvcc()
    jobs = []
    objs_cu, objs_cpp = [], []
    for src in cu:
        obj = BUILD / (src.stem + ".cu.o")
        objs_cu.append(obj)
        if force or _stale(obj, [src] + headers):
            flags = list(NVCC_FLAGS) + ([] if src.name in PRECISE_SOURCES else FAST_MATH) + \
                (["-Xptxas", "-v"] if ptxas_info else [])
            jobs.append([nvcc, *flags, "-I", str(CSRC), "-c", str(src), "-o", str(obj)])
    for src in cpp:
        obj = BUILD / (src.stem + ".cpp.o")
        objs_cpp.append(obj)
        if force or _stale(obj, [src] + headers):
            jobs.append(["g++", *CXX_FLAGS, "-I", str(CSRC), "-c", str(src), "-o", str(obj)])
    include = Path(sysconfig.get_paths()["include"])
    with cf.ThreadPoolExecutor(max_workers=8) as ex:
        eager = ex.submit(_build_eager, include, force, verbose)       # the longest, and needs no other
        list(ex.map(lambda c: _run(c, verbose or ptxas_info), jobs))
        eager.result()
    if objs_cu and (force or jobs or _stale(KERNEL_LIB, objs_cu)):
        _run([nvcc, "-shared", "-o", str(KERNEL_LIB), *map(str, objs_cu),
              "-gencode", "arch=compute_100a,code=sm_100a"], verbose)
    if objs_cpp and (force or jobs or _stale(HOST_LIB, objs_cpp)):
        _run(["g++", "-shared", "-o", str(HOST_LIB), *map(str, objs_cpp), "-pthread"], verbose)
    if not (include / "Python.h").exists():
        CALLS_LIB.unlink(missing_ok=True)      # of another state of the sources, perhaps
        print(f"no Python.h in {include}: {CALLS_LIB.name} is not built, calls go through ctypes")
    elif force or _stale(CALLS_LIB, [CALLS_SRC, CSRC / "api.h"]):
        _run(["g++", *CXX_FLAGS, "-shared", "-I", str(include), "-I", str(CSRC),
              str(CALLS_SRC), "-o", str(CALLS_LIB)], verbose)


def _build_eager(include: Path, force: bool, verbose: bool) -> None:
    spec = importlib.util.find_spec("torch")
    torch_dir = Path(spec.origin).parent if spec and spec.origin else None
    cuda = Path(_nvcc()).resolve().parent.parent / "include"
    if torch_dir is None or not (torch_dir / "include" / "torch" / "extension.h").exists() \
            or not (include / "Python.h").exists():
        print("no headers of PyTorch or Python: eager calls go through Python")
        return
    lib = eager_lib()
    if not (force or _stale(lib, [EAGER_SRC, CSRC / "api.h"])):
        return
    inc = torch_dir / "include"
    try:
        _run(["g++", *[f if f != "-O3" else "-O2" for f in CXX_FLAGS], "-shared",
              f'-DPF_SOURCES="{eager_sources()}"', "-I", str(inc), "-I",
              str(inc / "torch" / "csrc" / "api" / "include"), "-I", str(cuda), "-I", str(include), "-I",
              str(CSRC), str(EAGER_SRC), "-o", str(lib), "-L", str(torch_dir / "lib"), "-ltorch",
              "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-ltorch_python"], verbose)
    except RuntimeError as e:              # another PyTorch's interfaces
        lib.unlink(missing_ok=True)
        print(f"{lib.name} is not built, eager calls go through Python:\n{str(e)[-2000:]}")


def main(argv=None) -> int:
    ap = argparse.ArgumentParser(description=__doc__)
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    ap.add_argument("--ptxas-info", action="store_true", help="print registers / spills / smem")
    a = ap.parse_args(argv)
    build(a.force, a.verbose, a.ptxas_info)
    print(f"built {KERNEL_LIB.name}" + (f" and {HOST_LIB.name}" if HOST_LIB.exists() else ""))
    return 0


if __name__ == "__main__":
    sys.exit(main())
