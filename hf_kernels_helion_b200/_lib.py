"""ctypes binding of libb200fp8.so (C ABI: include/b200fp8.h).

There is deliberately no fallback: if the shared library is missing or a call
returns a non-zero status, a RuntimeError is raised.
"""
from __future__ import annotations

import ctypes
import sys
import warnings
from ctypes import c_char_p, c_int, c_int64, c_size_t, c_void_p
from pathlib import Path

LIB_PATH = Path(__file__).resolve().parent / "libb200fp8.so"
NATIVE_PATH = LIB_PATH.with_name("_torch_call.so")

OUT_BF16, OUT_FP32 = 0, 1
VARIANT_AUTO, VARIANT_TILE128, VARIANT_TILE256, VARIANT_STREAMK, VARIANT_TILE256_SK = 0, 1, 2, 3, 4
VARIANT_PAIR256, VARIANT_PAIR256_SPLIT = 5, 6
VARIANT_NAMES = {"auto": 0, "tile128": 1, "tile256": 2, "streamk": 3, "tile256_sk": 4, "pair256": 5, "pair256_split": 6,
                 "pair256_split_sk": 7}
CALL_ONE, CALL_ROWSCALE, CALL_SEVERAL, CALL_MULTICAST = 0, 1, 2, 3

# name -> (restype, argtypes); mirrors include/b200fp8.h one to one
SIGNATURES = {
    "b200fp8_version": (c_int, []),
    "b200fp8_strerror": (c_char_p, [c_int]),
    "b200fp8_quant_act": (c_int, [c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_int64, c_int64, c_int64, c_void_p]),
    "b200fp8_quant_weight": (c_int, [c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_int64, c_int64, c_int64,
                                     c_void_p]),
    "b200fp8_gemm": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_int64, c_int64,
                             c_int64, c_int64, c_int64, c_int64, c_int, c_int, c_void_p, c_size_t, c_void_p,
                             c_void_p]),
    "b200fp8_gemm_rowscale": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_int64,
                                      c_int64, c_int64, c_int64, c_int64, c_int64, c_int, c_void_p, c_size_t, c_void_p,
                                      c_void_p]),
    "b200fp8_gemm_rowscale_workspace_bytes": (c_int64, [c_int64, c_int64, c_int64]),
    "b200fp8_linear": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_int64, c_int64, c_int64,
                               c_int64, c_int64, c_int, c_int, c_void_p, c_size_t, c_void_p, c_void_p]),
    "b200fp8_linear_workspace_bytes": (c_int64, [c_int64, c_int64, c_int64, c_int]),
    "b200fp8_gemm_multicast": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_int64,
                                       c_int64, c_int64, c_int64, c_int64, c_int64, c_int, c_int, c_void_p, c_size_t,
                                       c_void_p, c_void_p]),
    "b200fp8_gemm_scatter": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_int64, c_int64,
                                     c_int64, c_int64, c_int64, c_int64, c_int64, c_int, c_int, c_void_p, c_size_t,
                                     c_void_p, c_void_p]),
    "b200fp8_peer_barrier": (c_int, [c_void_p, c_int, c_int, ctypes.c_uint32, c_void_p, c_void_p]),
    "b200fp8_peer_barrier_limited": (c_int, [c_void_p, c_int, c_int, ctypes.c_uint32, c_int64, c_void_p, c_void_p]),
    "b200fp8_ipc_export": (c_int, [c_void_p, c_void_p, c_void_p]),
    "b200fp8_ipc_open": (c_int, [c_void_p, c_void_p]),
    "b200fp8_ipc_close": (c_int, [c_void_p]),
    "b200fp8_gemm_workspace_bytes": (c_int64, [c_int64, c_int64, c_int64, c_int]),
    "b200fp8_gemm_auto_form": (c_int, [c_int64, c_int64, c_int64, c_int, c_void_p]),
    "b200fp8_gemm_pick_variant": (c_int, [c_int64, c_int64, c_int64]),
    "b200fp8_gemm_pair_clusters": (c_int, []),
    "b200fp8_gemm_decode_static": (c_int, [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_int64, c_int64, c_int64,
                                           c_int64, c_int64, c_int64, c_int64, c_int64, c_int, c_void_p, c_void_p]),
    "b200fp8_streamk_first_unit": (c_int64, [c_int64, c_int64, c_int64]),
    "b200fp8_streamk_owner": (c_int64, [c_int64, c_int64, c_int64]),
    "b200fp8_streamk_grid": (c_int64, [c_int64, c_int64, c_int64]),
}

_lib = None


def is_built() -> bool:
    return _lib is not None or LIB_PATH.exists()


def load():
    """Load the library once; raise if it has not been built."""
    global _lib
    if _lib is None:
        if not is_built():
            raise RuntimeError(
                f"{LIB_PATH} is missing: build it with `python -m hf_kernels_helion_b200.build` "
                "(there is no non-CUDA fallback)")
        lib = ctypes.CDLL(str(LIB_PATH))
        for name, (restype, argtypes) in SIGNATURES.items():
            fn = getattr(lib, name)
            fn.restype = restype
            fn.argtypes = argtypes
        _lib = lib
    return _lib


def native_tag() -> str:
    """The torch and the Python of this process, as the native call module names those it was built for."""
    import torch

    return f"torch {torch.__version__}, Python {sys.version_info.major}.{sys.version_info.minor}"


def load_native():
    """The module built from csrc/torch_call.cpp, bound to the library. None, with a warning, where it has not been
    built or was built for another torch or Python: every call then takes the way through the registered ops, which
    launches the same kernels and needs only the library. Raises if the library itself is missing."""
    lib = load()
    try:
        from . import _torch_call
        built_for = getattr(_torch_call, "built_for", "an unnamed torch and Python")
        why = None if built_for == native_tag() else f"was built for {built_for}"
    except ImportError as e:
        why = f"does not load ({e})"
    if why is not None:
        warnings.warn(f"{NATIVE_PATH} {why}; this is {native_tag()}. Calls go through the registered torch ops, at 30-50 us "
                      "of host time each. Build it with `python -m hf_kernels_helion_b200.build`", RuntimeWarning, stacklevel=2)
        return None
    _torch_call.bind(*(ctypes.cast(getattr(lib, name), c_void_p).value for name in (
        "b200fp8_gemm", "b200fp8_gemm_workspace_bytes", "b200fp8_gemm_rowscale", "b200fp8_gemm_rowscale_workspace_bytes",
        "b200fp8_linear", "b200fp8_linear_workspace_bytes", "b200fp8_quant_act", "b200fp8_quant_weight")))
    return _torch_call


def strerror(status: int) -> str:
    return load().b200fp8_strerror(int(status)).decode()


def check(status: int, what: str) -> None:
    if status != 0:
        raise RuntimeError(f"{what} failed: b200fp8 status {status} ({strerror(status)})")
