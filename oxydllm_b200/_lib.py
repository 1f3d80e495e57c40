"""ctypes binding of ``liboxq.so`` (the C ABI declared in ``include/oxq.h``).

The library is mandatory: there is no CPU or PyTorch fallback. If it is
missing it is built in-tree with nvcc; if that fails, importing raises.
"""
from __future__ import annotations

import ctypes
import importlib.util
import os
import warnings

from . import build as _build

OXQ_F32, OXQ_F16, OXQ_BF16 = 0, 1, 2

_vp, _i, _sz = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t

#: name -> argtypes; every entry returns an int status unless listed in _RESTYPE.
SIGNATURES = {
    "oxq_status_string": [_i],
    "oxq_last_error": [],
    "oxq_version": [],
    "oxq_awq_dequant": [_vp, _vp, _vp, _i, _vp, _i, _i, _i, _i, _vp],
    "oxq_awq_gemv": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _vp, _i, _i, _i, _i, _i, _vp],
    "oxq_awq_gemv_max_m": [_i, _i, _i],
    "oxq_decode_max_m": [],
    "oxq_decode_workspace_bytes": [_i, _i, _i],
    "oxq_awq_decode_matmul": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _vp, _i, _i, _i, _i, _i, _vp, _sz, _vp],
    "oxq_awq_ffn_gate_up": [_vp, _i, _vp, _vp, _vp, _i, _i, _vp, _i, _i, _i, _i, _vp, ctypes.c_size_t, _vp],
    "oxq_gptq_gemv": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _vp, _i, _i, _i, _i, _i, _i, _i, _vp],
    "oxq_w8a16_gemv": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _vp, _i, _i, _i, _i, _i, _vp],
    "oxq_w8a16_dequant": [_vp, _vp, _vp, _i, _vp, _i, _i, _i, _i, _vp],
    "oxq_w8a16_gemm": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _vp, _i, _i, _i, _i, _i, _vp, _sz, _vp],
    "oxq_gptq_dequant": [_vp, _vp, _vp, _i, _vp, _i, _i, _i, _i, _i, _i, _vp],
    "oxq_gguf_dequant": [_i, _vp, _vp, _i, _i, _i, _vp],
    "oxq_gguf_gemv": [_i, _vp, _i, _vp, _vp, _i, _vp, _i, _i, _i, _i, _vp],
    "oxq_gguf_scratch_bytes": [_i, _i, _i, _i],
    "oxq_gguf_matmul": [_i, _vp, _i, _vp, _vp, _i, _vp, _i, _i, _i, _i, _vp, _vp, _sz, _vp],
    "oxq_fp8_dequant": [_vp, _vp, _i, _i, _vp, _i, _i, _i, _vp],
    "oxq_fp8_gemv": [_vp, _i, _vp, _vp, _i, _i, _vp, _i, _vp, _i, _i, _i, _i, _vp],
    "oxq_mxfp4_dequant": [_vp, _vp, _vp, _i, _i, _i, _vp],
    "oxq_mxfp4_gemv": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _i, _i, _i, _vp],
    "oxq_gemm_workspace_bytes": [_i, _i],
    "oxq_gemm_check": [_vp, _vp],
    "oxq_selftest_wait_expiry": [_vp, ctypes.c_int, _vp],
    "oxq_selftest_gemm_wait_expiry": [_vp, ctypes.c_size_t, ctypes.c_int, _vp],
    "oxq_selftest_moe_wait_expiry": [_vp, ctypes.c_size_t, _vp],
    "oxq_selftest_moe_mx_wait_expiry": [_vp, ctypes.c_size_t, _vp],
    "oxq_selftest_packed_mx_wait_expiry": [_vp, ctypes.c_size_t, _vp],
    "oxq_selftest_group_wait_expiry": [_vp, ctypes.c_size_t, _vp],
    "oxq_selftest_q6k_wait_expiry": [_vp, ctypes.c_size_t, _vp],
    "oxq_awq_gemv_check": [_vp],
    "oxq_gemm_workspace_init": [_vp, _vp],
    "oxq_awq_gemm": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _vp, _i, _i, _i, _i, _i, _vp, _sz, _vp],
    "oxq_packed4_max_m": [_i, _i, _i],
    "oxq_packed4_streams": [_i, _i, _i, _i, _i],
    "oxq_packed4_scratch_bytes": [_i, _i],
    "oxq_packed4_full_scratch_bytes": [_i, _i, _i, _i, _i],
    "oxq_packed4_matmul": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _vp, _i, _i, _i, _i, _i, _i, _i, _vp, _vp, _sz, _vp],
    "oxq_awq_gemm_tp": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _i, _vp, _sz, _vp],
    "oxq_gptq_gemm": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _vp, _i, _i, _i, _i, _i, _i, _i, _vp, _sz, _vp],
    "oxq_gguf_gemm": [_i, _vp, _i, _vp, _vp, _i, _vp, _i, _i, _i, _i, _vp, _sz, _vp],
    "oxq_fp8_gemm": [_vp, _i, _vp, _vp, _i, _i, _vp, _i, _vp, _i, _i, _i, _i, _vp, _sz, _vp],
    "oxq_fp8_scratch_bytes": [_i, _i, _i, _i, _i],
    "oxq_fp8_matmul": [_vp, _i, _vp, _vp, _i, _i, _vp, _i, _vp, _i, _i, _i, _i, _vp, _vp, _sz, _vp],
    "oxq_mxfp4_gemm": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _i, _i, _i, _vp, _sz, _vp],
    "oxq_gptoss_moe_workspace_bytes": [_i, _i, _i, _i, _i],
    "oxq_gptoss_moe_forward": [_vp, _i, _vp, _i, _i, _i, _i, _i, _i, _vp, _vp, _vp, _vp, _vp, _vp, _i, ctypes.c_float,
                               _i, _i, _vp, _i, _vp, _sz, _vp],
    "oxq_gptoss_moe_forward_logits": [_vp, _i, _vp, _i, _i, _i, _i, _i, _i, _i, _vp, _vp, _vp, _vp, _vp, _vp, _i, ctypes.c_float,
                                      _i, _i, _vp, _i, _vp, _sz, _vp],
    "oxq_gptoss_experts_forward": [_vp, _i, _vp, _i, _i, _i, _i, _vp, _vp, _vp, _vp, _vp, _vp, _i, ctypes.c_float, _i, _i,
                                   _vp, _i, _vp, _sz, _vp],
    "oxq_moe_combine": [_vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp, _i, _vp],
    "oxq_moe_dispatch_plan": [_vp, _i, _i, _vp, _vp, _vp, _vp, _vp],
    "oxq_moe_gather_rows": [_vp, _vp, _i, _i, _i, _vp, _vp],
    "oxq_moe_expand_ids": [_vp, _i, _i, _i, _vp, _vp],
    "oxq_moe_route": [_vp, _i, _i, _i, _i, _vp, _vp, _vp],
    "oxq_awq_gemm_noalloc_max_k": [],
    "oxq_awq_gemm_noalloc": [_vp, _i, _vp, _vp, _vp, _i, _vp, _i, _vp, _i, _i, _i, _i, _i, _vp],
    "oxq_awq_gemm_noalloc_check": [_vp],
}
_RESTYPE = {"oxq_status_string": ctypes.c_char_p, "oxq_last_error": ctypes.c_char_p,
            "oxq_gemm_workspace_bytes": ctypes.c_size_t, "oxq_packed4_scratch_bytes": ctypes.c_size_t, "oxq_packed4_full_scratch_bytes": ctypes.c_size_t, "oxq_fp8_scratch_bytes": ctypes.c_size_t, "oxq_gguf_scratch_bytes": ctypes.c_size_t, "oxq_decode_workspace_bytes": ctypes.c_size_t, "oxq_gptoss_moe_workspace_bytes": ctypes.c_size_t, "oxq_awq_gemm_noalloc_max_k": ctypes.c_size_t}

_lib = None


class OxqError(RuntimeError):
    """A C-ABI call returned a non-zero status."""

    def __init__(self, fn: str, status: int, message: str):
        super().__init__(f"{fn}: {message} (status {status})")
        self.status = status
        self.message = message


def lib_path() -> str:
    return _build.LIB


def load() -> ctypes.CDLL:
    """Load (building if needed) the shared library and declare its prototypes."""
    global _lib
    if _lib is None:
        path = _build.build()
        if not os.path.exists(path):
            raise ImportError(f"{path} is missing and could not be built; the CUDA library is required")
        lib = ctypes.CDLL(path)
        for name, argtypes in SIGNATURES.items():
            fn = getattr(lib, name)
            fn.argtypes = argtypes
            fn.restype = _RESTYPE.get(name, _i)
        _lib = lib
    return _lib


_entries: dict = {}


def entry(name: str):
    """The entry point itself, for callers that make the same call again and again (``fail`` if it returns non-zero)."""
    fn = _entries.get(name)
    if fn is None:
        fn = _entries[name] = getattr(load(), name)
    return fn


def fail(name: str, rc: int) -> None:
    lib = load()
    raise OxqError(name, rc, lib.oxq_last_error().decode() or lib.oxq_status_string(rc).decode())


def call(name: str, *args) -> None:
    """Call an entry point; raise :class:`OxqError` with the library's message on failure."""
    rc = entry(name)(*args)
    if rc != 0:
        fail(name, rc)


_host = None


def host():
    """The native host side of decode calls (``csrc/host_ops.cpp``), or None where it cannot be built: the callers' Python code does the same."""
    global _host
    if _host is None:
        try:
            path = _build.build_host()
            spec = importlib.util.spec_from_file_location("oxydllm_b200._host", path)
            mod = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(mod)
            lib = load()
            mod.bind({name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in SIGNATURES})
            _host = mod
        except (RuntimeError, OSError, ImportError, KeyError) as e:
            warnings.warn(f"oxydllm_b200: calls take a few microseconds longer without the host extension ({e})")
            _host = False
    return _host or None
