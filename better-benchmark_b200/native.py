"""ctypes binding of the C ABI in ``include/b200_oracles.h``.

The shared library is built in-tree (``csrc/libb200_oracles.so``) by ``build.py``. There is no
fallback of any kind: if the library is missing or a symbol cannot be resolved, loading raises
``NativeLibraryError`` and every kernel wrapper fails with it.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import sys
import threading
import warnings
from ctypes import c_char_p, c_double, c_int32, c_int64, c_void_p
from pathlib import Path

import os

# B200_ORACLES_LIB names another build of the library (a measurement variant); default: the in-tree one
LIB_PATH = Path(os.environ.get("B200_ORACLES_LIB") or Path(__file__).resolve().parent / "csrc" / "libb200_oracles.so")


def calls_path() -> Path:
    """The host side of the most frequent calls (csrc/calls.cpp), an extension module that works on the library loaded here. It is compiled
    against the C++ headers of one torch and one Python, and looks into their objects: a build for others has another name."""
    import torch
    build = f"{sys.implementation.cache_tag}.torch-{torch.__version__}.abi{int(torch._C._GLIBCXX_USE_CXX11_ABI)}"
    return Path(__file__).resolve().parent / "csrc" / f"b200_calls.{build}.so"

# dtype codes shared with csrc/common.cuh
F32, BF16, F16 = 0, 1, 2

# status codes shared with csrc/common.cuh
OK = 0
ERR_INVALID, ERR_UNSUPPORTED, ERR_ALIGNMENT, ERR_WORKSPACE, ERR_DEVICE_WAIT = -1, -2, -3, -4, -5


class NativeLibraryError(RuntimeError):
    """The CUDA library is not built or does not export the expected C ABI."""


class KernelArgumentError(ValueError):
    """An entry point rejected its arguments before launching anything (negative status)."""


class KernelLaunchError(RuntimeError):
    """A CUDA launch was rejected (positive status = cudaError_t). The text names CUDA so that
    sweep workers treat it as a device failure and restart."""


_P64 = ctypes.POINTER(c_int64)
_PF = c_void_p  # float* passed as raw address

# name -> (restype, argtypes); mirrors include/b200_oracles.h declaration by declaration
SIGNATURES = {
    "b200_last_error": (c_char_p, []),
    "b200_version": (c_int32, []),
    "b200_sm_count": (c_int32, []),
    "b200_l2_bytes": (c_int32, []),
    "b200_launch_count": (c_int64, []),
    "b200_last_kernel": (c_char_p, []),
    "b200_check_status": (c_int32, [c_void_p, c_void_p]),
    "b200_row_reduce": (c_int32, [c_void_p, c_void_p, c_int64, c_int64, c_int64, c_int64, _P64,
                                  c_int64, c_int32, c_int32, c_int32, c_void_p]),
    "b200_softmax": (c_int32, [c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_int64, c_int64,
                               _P64, _P64, _P64, c_int32, c_int32, c_double, c_int32, c_void_p]),
    "b200_norm_fwd": (c_int32, [c_void_p, c_void_p, c_void_p, c_void_p, _PF, _PF, _PF, c_int64,
                                c_int64, c_int64, c_int64, c_int32, c_int32, c_int32, c_double,
                                c_double, c_int32, c_void_p]),
    "b200_norm_fwd_residual": (c_int32, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, _PF, _PF, _PF,
                                         c_int64, c_int64, c_int64, c_int64, c_int32, c_int32, c_int32, c_double,
                                         c_double, c_int32, c_void_p]),
    "b200_norm_fwd_wait_timeouts": (c_int64, []),
    "b200_norm_bwd_wait_timeouts": (c_int64, []),
    "b200_norm_bwd_scratch_bytes": (c_int64, [c_int64]),
    "b200_norm_bwd": (c_int32, [c_void_p, c_void_p, c_void_p, _PF, _PF, c_void_p, _PF, _PF, c_int64,
                                c_int64, c_int64, c_int64, c_int32, c_int32, c_int32, c_int64,
                                c_int64, c_int64, c_int64, c_int64, c_void_p, c_int64, c_int32,
                                c_void_p]),
    "b200_batch_norm_wait_timeouts": (c_int64, []),
    "b200_batch_norm_scratch_bytes": (c_int64, [c_int64]),
    "b200_batch_norm_fwd": (c_int32, [c_void_p, c_void_p, c_void_p, c_void_p, _PF, _PF, _PF, _PF,
                                      c_int64, c_int64, c_int64, c_int64, c_int64, c_int64, c_int32,
                                      c_int32, c_double, c_double, c_int32, c_void_p, c_int64,
                                      c_void_p]),
    "b200_batch_norm_fwd_ex": (c_int32, [c_void_p, c_void_p, c_void_p, c_void_p, _PF, _PF, _PF, _PF,
                                         c_int64, c_int64, c_int64, c_int64, c_int64, c_int64, c_int32,
                                         c_int32, c_double, c_double, c_double, c_int32, c_void_p, c_int64,
                                         c_void_p]),
    "b200_batch_norm_bwd_ex": (c_int32, [c_void_p] * 9 + [c_int64] * 6 + [c_int32, c_int32, c_double, c_double,
                                                                          c_void_p, c_int64, c_void_p]),
    "b200_batch_norm_fwd_static_scratch": (c_int32, [c_void_p, c_void_p, c_void_p, c_void_p, _PF, _PF, _PF,
                                                     _PF, c_int64, c_int64, c_int64, c_int64, c_int64,
                                                     c_int64, c_int32, c_int32, c_double, c_double, c_int32,
                                                     c_void_p]),
    "b200_batch_norm_bwd_scratch_bytes": (c_int64, [c_int64]),
    "b200_batch_norm_bwd": (c_int32, [c_void_p] * 9 + [c_int64] * 6 + [c_int32, c_int32, c_double, c_void_p,
                                                                       c_int64, c_void_p]),
    "b200_col_reduce": (c_int32, [c_void_p, c_void_p, c_int64, c_int64, c_int64, c_int64, c_int64, c_int64,
                                  c_int32, c_int32, c_int32, c_void_p, c_int64, c_void_p]),
    "b200_permute_copy": (c_int32, [c_void_p, c_void_p, _P64, _P64, c_int32, c_int32, c_double, c_int32,
                                    c_void_p]),
    "b200_transpose_copy": (c_int32, [c_void_p, c_void_p, c_int64, c_int64, c_int64, c_int64, c_int64,
                                      c_int32, c_int32, c_double, c_int32, c_void_p]),
    "b200_cast_scale": (c_int32, [c_void_p, c_void_p, c_int64, c_int32, c_int32, c_double, c_int32, c_void_p]),
    "b200_dropout_rms_norm": (c_int32, [c_void_p, c_void_p, c_void_p, c_void_p, c_int32, c_int32, c_double,
                                        c_double, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int64,
                                        c_int64, c_int32, c_void_p]),
    "b200_softmax_dropout": (c_int32, [c_void_p, c_void_p, c_int64, c_int64, c_int64, c_int64, c_int64, c_int64,
                                       c_int64, c_int64, c_void_p, c_int32, c_double, c_void_p, c_void_p, c_void_p,
                                       c_void_p, c_void_p, c_int32, c_void_p]),
    "b200_dropout_add": (c_int32, [c_void_p, c_void_p, c_void_p, c_int32, c_double, c_void_p, c_void_p, c_int64,
                                   c_int32, c_void_p]),
    "b200_dropout_layer_norm": (c_int32, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int32, c_double,
                                          c_double, c_void_p, c_void_p, c_void_p, c_void_p, c_int64, c_int64,
                                          c_int32, c_void_p]),
}

_lib = None
_lock = threading.Lock()


def load() -> ctypes.CDLL:
    """Load the library once per process and bind every declared symbol."""
    global _lib
    if _lib is not None:
        return _lib
    with _lock:
        if _lib is not None:
            return _lib
        if not LIB_PATH.exists():
            raise NativeLibraryError(
                f"{LIB_PATH} is not built. Run `python -m better_benchmark_b200.build` "
                "(needs nvcc with sm_100a support). There is no CPU or eager fallback.")
        try:
            lib = ctypes.CDLL(str(LIB_PATH))
        except OSError as e:
            raise NativeLibraryError(f"cannot load {LIB_PATH}: {e}") from e
        for name, (restype, argtypes) in SIGNATURES.items():
            try:
                fn = getattr(lib, name)
            except AttributeError as e:
                raise NativeLibraryError(f"{LIB_PATH} does not export {name}") from e
            fn.restype = restype
            fn.argtypes = argtypes
        _lib = lib
        return lib


_calls = None
_BOUND = ("b200_row_reduce", "b200_softmax", "b200_norm_fwd_residual", "b200_norm_bwd", "b200_norm_bwd_scratch_bytes",
          "b200_batch_norm_fwd_ex", "b200_batch_norm_scratch_bytes", "b200_batch_norm_bwd_ex",
          "b200_batch_norm_bwd_scratch_bytes", "b200_transpose_copy", "b200_permute_copy", "b200_cast_scale")


class _LeftToPython:
    """Stands in for the module where it is not built: every call is left to the Python code of the wrappers."""

    def __getattr__(self, name):
        return lambda *args: None


def load_calls(scratch_by_device: dict, required: bool = False):
    """Load csrc/calls.cpp's module once per process and hand it the library's entry points. Where it is not built for this torch and this
    Python the wrappers' Python code takes every call, which it can, at two to four times the host time; with ``required`` that is an error."""
    global _calls
    lib = load()
    with _lock:
        if _calls is None:
            path = calls_path()
            if path.exists():
                try:
                    loader = importlib.machinery.ExtensionFileLoader("b200_calls", str(path))
                    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("b200_calls", loader))
                    loader.exec_module(module)
                except ImportError as e:
                    raise NativeLibraryError(f"cannot load {path}: {e}") from e
                module.bind({name: ctypes.cast(getattr(lib, name), c_void_p).value for name in _BOUND}, check, scratch_by_device)
                _calls = module
            elif not required:
                warnings.warn(f"{path} is not built, so every call takes the longer way through Python. "
                              "Run `python -m better_benchmark_b200.build`.", RuntimeWarning, stacklevel=2)
                _calls = _LeftToPython()
        if required and (_calls is None or isinstance(_calls, _LeftToPython)):
            raise NativeLibraryError(f"{calls_path()} is not built. Run `python -m better_benchmark_b200.build`.")
        return _calls


def last_error() -> str:
    msg = load().b200_last_error()
    return msg.decode("utf-8", "replace") if msg else ""


def check(status: int, what: str) -> None:
    """Turn an entry point's status into a Python exception."""
    if status == 0:
        return
    text = last_error()
    if status < 0:
        raise KernelArgumentError(f"{what}: status {status}: {text}")
    raise KernelLaunchError(f"{what}: CUDA error {status}: {text}")


_I64_ARRAYS = {n: c_int64 * n for n in (3, 4)}   # building an array type costs more than filling it


def i64_array(values) -> ctypes.Array:
    vals = [int(v) for v in values]
    kind = _I64_ARRAYS.get(len(vals)) or c_int64 * len(vals)
    return kind(*vals)
