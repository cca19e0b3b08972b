"""ctypes loader for the in-tree sm_100a kernel library.

The library is built by ``python -m pfeife_b200.csrc.build`` into the package directory.  On a
machine with a CUDA device a missing library is an error (there is no silent eager fallback on
GPU); on a CPU-only machine ``lib()`` returns ``None`` and the ops use their PyTorch reference
implementations, which is what the CPU/gloo tests run.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import re
import sysconfig
import threading
from pathlib import Path
from typing import Optional

import torch

_PKG = Path(__file__).resolve().parent.parent
_KERNEL_LIB = _PKG / "libpfeife_b200_kernels.so"
_HOST_LIB = _PKG / "libpfeife_b200_host.so"

# built for one Python: the name carries its ABI
_CALLS_LIB = _PKG / ("libpfeife_b200_calls" + sysconfig.get_config_var("EXT_SUFFIX"))

_lib: Optional[ctypes.CDLL] = None
_calls = None
_eager = None
_eager_tried = False
_host: Optional[ctypes.CDLL] = None
_tried = False
_launches = 0  # kernels launched through this module (reported by bench.py)

PF_F32, PF_F16, PF_BF16 = 0, 1, 2
_tls = threading.local()
_DT = {torch.float32: PF_F32, torch.float16: PF_F16, torch.bfloat16: PF_BF16}


class KernelError(RuntimeError):
    pass


def dt(dtype: torch.dtype) -> int:
    try:
        return _DT[dtype]
    except KeyError:
        raise KernelError(f"unsupported dtype {dtype}") from None


def lib() -> Optional[ctypes.CDLL]:
    """The kernel library, or None on a machine without CUDA."""
    global _lib, _tried
    if _lib is not None:
        return _lib
    if not torch.cuda.is_available():
        return None
    if _tried:
        raise KernelError(f"{_KERNEL_LIB} failed to load earlier")
    _tried = True
    if not _KERNEL_LIB.exists():
        raise KernelError(
            f"{_KERNEL_LIB.name} is missing on a CUDA machine; run "
            "`python -m pfeife_b200.csrc.build` (GPU paths never fall back to eager PyTorch)")
    # make sure libcudart from torch is already mapped so the library binds to the same runtime
    torch.cuda.init()
    _lib = ctypes.CDLL(str(_KERNEL_LIB), mode=ctypes.RTLD_GLOBAL)
    return _lib


class _CtypesCalls:
    """The entry points of csrc/api.h with the arguments csrc/calls.cpp takes, through ctypes: for a
    Python without headers to build that module against.  A call costs some 5 us more."""

    def __init__(self, library: ctypes.CDLL):
        header = (_PKG / "csrc" / "api.h").read_text()
        for name, params in re.findall(r"PF_DECL int (pf_\w+)\(([^)]*)\)", header):
            kinds = [None if "*" in p else ctypes.c_longlong if "long long" in p
                     else ctypes.c_float if "float" in p else ctypes.c_int
                     for p in params.split(",") if p.strip()]
            setattr(self, name, self._entry(getattr(library, name), kinds))

    @staticmethod
    def _pointer(v):
        if v is None or isinstance(v, int):
            return ctypes.c_void_p(v)
        if isinstance(v, tuple):
            return (ctypes.c_longlong * len(v))(*v)
        return ctypes.c_void_p(v.data_ptr())

    def _entry(self, fn, kinds):
        def call(*args):
            if len(args) != len(kinds):
                raise TypeError(f"expected {len(kinds)} arguments, got {len(args)}")
            return fn(*(self._pointer(a) if k is None else k(a) for k, a in zip(kinds, args)))
        return call


def load_calls(library: ctypes.CDLL):
    """The Python module of the entry points of `library`, which is loaded with its symbols global."""
    if not _CALLS_LIB.exists():
        return _CtypesCalls(library)
    return _load("pfeife_b200_calls", _CALLS_LIB)


def _load(name: str, path: Path):
    loader = importlib.machinery.ExtensionFileLoader(name, str(path))
    spec = importlib.util.spec_from_loader(name, loader)
    module = importlib.util.module_from_spec(spec)
    loader.exec_module(module)
    return module


def calls():
    """The kernel library's entry points as a Python module, which takes tensors, None, numbers and
    tuples of strides as they are (csrc/calls.cpp); None on a machine without CUDA."""
    global _calls
    if _calls is None and lib() is not None:
        _calls = load_calls(_lib)
    return _calls


def eager():
    """Eager calls of the ops as a Python module (csrc/eager.cpp), or None: on a machine without CUDA, and
    where the module was not built for this PyTorch from these sources, or these are not there to tell
    (the calls then go through Python, which takes them 20 us longer in each direction)."""
    global _eager, _eager_tried
    if not _eager_tried and lib() is not None:
        _eager_tried = True
        from ..csrc import build
        path = build.eager_lib()
        if path.exists():
            try:
                sources = build.eager_sources()
            except FileNotFoundError:
                return None
            module = _load("pfeife_b200_eager", path)
            if module.SOURCES == sources:
                from . import kernels
                module.setup(kernels.status_word, check)
                _eager = module
    return _eager


def host_lib() -> Optional[ctypes.CDLL]:
    """Host-side C++ helpers (planner evaluator).  None when not built."""
    global _host
    if _host is None and _HOST_LIB.exists():
        _host = ctypes.CDLL(str(_HOST_LIB))
    return _host


def available() -> bool:
    return torch.cuda.is_available() and lib() is not None


def use_kernels(t: torch.Tensor) -> bool:
    """True when `t` lives on a CUDA device (then the native kernels must be used)."""
    return t.is_cuda


def ptr(t: Optional[torch.Tensor]):
    """Device pointer of `t` (NULL for None).  Also remembers, per thread, the device of the
    last tensor seen, which is the device ``stream()`` launches on: a thread's *current* torch
    device is not reliable (new Python threads start on device 0)."""
    if t is None:
        return ctypes.c_void_p(0)
    device = t.get_device()
    if device >= 0:
        _tls.op_device = device
    return ctypes.c_void_p(t.data_ptr())


def bind_thread(device_index: Optional[int] = None) -> None:
    """Makes sure the calling thread has the device's context bound inside the library's own
    CUDA runtime (threads created by PyTorch, such as autograd workers, arrive without one)."""
    idx = torch.cuda.current_device() if device_index is None else device_index
    code = calls().pf_bind_device(int(idx))          # remembers what the thread is bound to
    if code != 0:
        raise KernelError(f"pf_bind_device({idx}): CUDA error {code}")


def stream(device: Optional[int] = None) -> ctypes.c_void_p:
    """Handle of the torch stream that is current for the device of the operands (the device
    of the last tensor passed through ``ptr`` in this thread); binds the calling thread of the
    library's own CUDA runtime to that device."""
    if device is None:
        device = getattr(_tls, "op_device", None)
    if device is None:
        device = torch.cuda.current_device()
    bind_thread(device)
    return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(device))


def stream_of(t: torch.Tensor) -> int:
    """The torch stream that is current for the device of `t`, for ``calls()``; binds the calling
    thread to that device like ``stream``."""
    device = t.get_device()
    if device < 0:
        raise KernelError("a kernel was called on a tensor that is not on a CUDA device")
    bind_thread(device)
    return torch._C._cuda_getCurrentRawStream(device)


_sm_count_cache = {}


def sm_count(device=None) -> int:
    if type(device) is torch.device:
        idx = device.index
    else:
        idx = torch.cuda.current_device() if device is None else torch.device(device).index
    if idx not in _sm_count_cache:
        _sm_count_cache[idx] = torch.cuda.get_device_properties(idx).multi_processor_count
    return _sm_count_cache[idx]


def check(code: int, what: str) -> None:
    global _launches
    if code != 0:
        if code > 0:
            raise KernelError(f"{what}: CUDA error {code}")
        reasons = {-1: "unsupported dtype", -2: "misaligned pointer or pitch",
                   -3: "size beyond kernel limit", -100: "tensor-map encoder unavailable",
                   -101: "tensor-map encoding failed"}
        if code <= -1000:
            raise KernelError(f"{what}: tensor-map encoding failed (CUresult {-code - 1000})")
        raise KernelError(f"{what}: {reasons.get(code, code)}")
    _launches += 1


def launch_count() -> int:
    return _launches + (_eager.launches() if _eager is not None else 0)


def add_launches(n: int) -> None:
    """Accounts for kernels launched by replaying a captured CUDA graph."""
    global _launches
    _launches += n


def c_ll(v) -> ctypes.c_longlong:
    return ctypes.c_longlong(int(v))


def c_f(v) -> ctypes.c_float:
    return ctypes.c_float(float(v))
