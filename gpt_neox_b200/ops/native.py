"""ctypes binding of ``libneox_b200.so`` (CUDA kernels) and ``libneox_host.so`` (host C++).

The kernels expose a plain C ABI (raw device pointers + a stream handle), so no PyTorch headers are
needed at build time and a rebuild takes seconds.  ``lib()`` raises if the CUDA library cannot be
loaded: on a machine with a GPU a missing extension is an error, never a silent eager fallback.
"""
from __future__ import annotations

import ctypes
import os
from pathlib import Path

import torch
from torch.autograd import forward_ad

_LIBDIR = Path(__file__).resolve().parent / "_lib"
_cuda_lib = None
_host_lib = None

c_void_p, c_int, c_ll, c_float = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float

ERRORS = {1: "alignment", 2: "tensor-map encode", 3: "driver/alloc", 4: "launch", 5: "shape", 6: "too large"}


class NativeError(RuntimeError):
    pass


def _load(name: str, builder: str):
    path = _LIBDIR / name
    if not path.exists() and os.environ.get("NEOX_B200_NO_AUTOBUILD", "0") != "1":
        from . import build
        getattr(build, builder)()
    if not path.exists():
        raise NativeError(f"{path} is missing; run `python -m gpt_neox_b200.ops.build`")
    return ctypes.CDLL(str(path))


# The entry points of every linear layer, with their argument types declared: plain integers (addresses, strides) are then
# converted by ctypes itself, which is cheaper than wrapping each of some twenty in an object.
_GEMM_HEAD = [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_ll, c_ll, c_ll]
_GEMM_EPILOGUE = [c_int, c_void_p, c_void_p, c_ll, c_int, c_void_p, c_ll, c_void_p, c_ll, c_int, c_float]
_ARGTYPES = {
    "neox_gemm_skinny_16": [*_GEMM_HEAD, *_GEMM_EPILOGUE, c_int, c_void_p],
    "neox_gemm_16": [*_GEMM_HEAD, c_int, c_int, *_GEMM_EPILOGUE, c_void_p, c_int, c_void_p],
    "neox_gemm_splits": [c_int, c_int, c_int],
    "neox_gemm_accumulate_16": [*_GEMM_HEAD, c_int, c_int, c_float, c_int, c_void_p, c_int, c_void_p],
    "neox_gemm_16_2cta": [*_GEMM_HEAD, c_int, c_int, *_GEMM_EPILOGUE, c_int, c_void_p],
}

launch_count = 0   # number of kernel-launching library calls made by this process (see bench.py)


class _CountingLib:
    """Proxy over the CDLL that counts calls into kernel launchers (``neox_*`` entry points that take a
    stream); pure queries such as ``neox_read_status`` are not counted."""
    _NOT_LAUNCHES = {"neox_read_status", "neox_norm_bwd_blocks", "neox_sm_count_c", "neox_causal_conv_blocks",
                     "neox_gemm_splits"}

    def __init__(self, cdll):
        self._cdll = cdll
        self._cache = {}

    def __getattr__(self, name):
        fn = self._cache.get(name)
        if fn is None:
            raw = getattr(self._cdll, name)
            if name in _ARGTYPES:
                raw.argtypes = _ARGTYPES[name]
            if name in self._NOT_LAUNCHES:
                fn = raw
            else:
                def fn(*args, _raw=raw):
                    global launch_count
                    launch_count += 1
                    return _raw(*args)
            self._cache[name] = fn
        return fn

    def has(self, name):
        return hasattr(self._cdll, name)


def lib():
    """The CUDA kernel library (loaded once)."""
    global _cuda_lib
    if _cuda_lib is None:
        _cuda_lib = _CountingLib(_load("libneox_b200.so", "build_cuda"))
    return _cuda_lib


def host_lib():
    """The host-only C++ helper library (loaded once)."""
    global _host_lib
    if _host_lib is None:
        _host_lib = _load("libneox_host.so", "build_host")
    return _host_lib


_cuda_seen = False


def available() -> bool:
    """True when kernels can run: a CUDA device is visible (the library itself must then load).  Asked on every call of every
    operator, and the driver query behind it takes 4 us: once a device has been seen it is not asked again."""
    global _cuda_seen
    if not _cuda_seen:
        _cuda_seen = torch.cuda.is_available()
    return _cuda_seen


def stream_ptr() -> int:
    """Handle of the current stream of the current device, without the Stream object that ``torch.cuda.current_stream()``
    builds around it (15 us)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def plain_call(*tensors) -> bool:
    """May an operator compute its values directly instead of going through ``torch.autograd.Function`` (20 us of a decoding
    step's launch)?  Only where that makes no difference: nothing records gradients, and nothing else watches the call."""
    return not torch.is_grad_enabled() and untransformed(*tensors)


def untransformed(*tensors) -> bool:
    """No functorch transform, forward-mode level or tracer is active, and the arguments are plain tensors: nothing sees more
    of an operator than its values and its gradients."""
    if torch._C._functorch.peek_interpreter_stack() is not None or forward_ad._current_level >= 0 \
            or torch._C._get_tracing_state() is not None:
        return False
    for t in tensors:
        if t is not None and type(t) is not torch.Tensor and type(t) is not torch.nn.Parameter:
            return False
    return True


def ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def check(rc: int, what: str):
    if rc != 0:
        raise NativeError(f"{what} failed: {ERRORS.get(rc, rc)}")


def read_status() -> int:
    """Synchronise and return (then clear) the device status word; non-zero = a bounded wait expired."""
    return int(lib().neox_read_status())
