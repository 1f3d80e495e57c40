"""Prefill-sized (m > 32) matmuls of the quantized linears on the tensor cores.

Thin callers of the ``oxq_*_gemm`` entry points. The dequantization slab
workspace is caller-owned device memory: one cached ``torch`` buffer per
device and size, shared by stream-ordered calls.
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib

_DT = {torch.float32: _lib.OXQ_F32, torch.float16: _lib.OXQ_F16, torch.bfloat16: _lib.OXQ_BF16}


def _dt(t: torch.dtype) -> int:
    try:
        return _DT[t]
    except KeyError:
        raise ValueError(f"unsupported dtype {t}") from None

_workspaces: dict = {}
_native = None


def native():
    """The host extension with this module's buffers in its hands, or None without it."""
    global _native
    if _native is None:
        _native = _lib.host() or False
        if _native:
            for kind, bufs in enumerate((_flags, _workspaces)):
                for buf in bufs.values():
                    _native.keep(kind, buf)
    return _native or None


def workspace_bytes(n: int, k: int) -> int:
    return int(_lib.entry("oxq_gemm_workspace_bytes")(n, k))


def workspace(n: int, k: int, device) -> torch.Tensor:
    """A device buffer large enough for ``oxq_*_gemm`` on an ``[n, k]`` weight (grown on demand, reused)."""
    need = workspace_bytes(n, k)
    key = _dev_index(device)
    buf = _workspaces.get(key)
    if buf is None or buf.numel() < need:
        buf = torch.zeros(need, dtype=torch.uint8, device=device)
        _workspaces[key] = buf
        if _native:
            _native.keep(1, buf)
    return buf


_decode_ws: dict = {}


def _dev_index(device) -> int:
    idx = (device if isinstance(device, torch.device) else torch.device(device)).index
    return torch.cuda.current_device() if idx is None else idx


def decode_workspace(m: int, k: int, n: int, device) -> torch.Tensor:
    """Workspace of ``oxq_awq_decode_matmul`` for this device (grown on demand, zero-filled, reused)."""
    need = int(_lib.load().oxq_decode_workspace_bytes(m, k, n))
    key = _dev_index(device)
    buf = _decode_ws.get(key)
    if buf is None or buf.numel() < need:
        buf = torch.zeros(need, dtype=torch.uint8, device=torch.device("cuda", key))
        _decode_ws[key] = buf
    return buf


def awq_decode_matmul(lin, x2, y):
    """``y = x2 . deq(W)`` for decode-sized batches on the tensor cores (``oxq_awq_decode_matmul``)."""
    ws = decode_workspace(x2.shape[0], lin.in_features, lin.out_features, x2.device)
    bp, bd = _bias(lin.bias)
    _lib.call("oxq_awq_decode_matmul", _p(x2), _dt(x2.dtype), _p(lin.qweight), _p(lin.qzeros), _p(lin.scales),
              _dt(lin.scales.dtype), bp, bd, _p(y), _dt(y.dtype), x2.shape[0], lin.in_features, lin.out_features,
              lin.group_size, _p(ws), ws.numel(), _st())


_flags: dict = {}


def _flag_words(device) -> torch.Tensor:
    """What ``oxq_packed4_matmul`` reports through on this device: a header of its own, which no larger layer ever replaces (a captured
    graph keeps its address) and which costs no slab."""
    key = _dev_index(device)
    buf = _flags.get(key)
    if buf is None:
        buf = _flags[key] = torch.zeros(256, dtype=torch.uint8, device=torch.device("cuda", key))
        if _native:
            _native.keep(0, buf)
    return buf


def check(ws: torch.Tensor) -> None:
    """Synchronise and raise if a tensor-core kernel recorded a timed-out wait in ``ws`` or in its device's flag words."""
    for buf in (ws, _flags.get(ws.device.index)):
        if buf is not None:
            _lib.call("oxq_gemm_check", ctypes.c_void_p(buf.data_ptr()),
                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))


def _p(t) -> int:
    return 0 if t is None else t.data_ptr()


def _st() -> int:
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _bias(b):
    return _p(b), (_dt(b.dtype) if b is not None else 0)


def awq_matmul(lin, x2, y):
    ws = workspace(lin.out_features, lin.in_features, x2.device)
    bp, bd = _bias(lin.bias)
    _lib.call("oxq_awq_gemm", _p(x2), _dt(x2.dtype), _p(lin.qweight), _p(lin.qzeros), _p(lin.scales),
              _dt(lin.scales.dtype), bp, bd, _p(y), _dt(y.dtype), x2.shape[0], lin.in_features, lin.out_features,
              lin.group_size, _p(ws), ws.numel(), _st())


def packed4_matmul(lin, x2, y, tensors=None):
    """``y = x2 . deq(W) (+ bias)`` for the 4-bit layouts by the grouped unpack + tcgen05 kernel (``oxq_packed4_matmul``). The
    scratch is this call's own, so calls on several streams do not meet."""
    m, n = x2.shape[0], lin.out_features
    flag = _flags.get(x2.device.index)
    if flag is None:
        flag = _flag_words(x2.device)
    need = lin._scratch_bytes.get(m)
    if need is None:
        need = lin._scratch_bytes[m] = int(_lib.load().oxq_packed4_full_scratch_bytes(m, lin.in_features, n, lin.group_size,
                                                                                                int(lin.pack_dim == "in")))
    scratch = torch.empty(need, dtype=torch.uint8, device=x2.device)
    qw, qz, sc, sc_dt, b, b_dt = tensors or lin._tensors()
    _lib.call("oxq_packed4_matmul", x2.data_ptr(), _dt(x2.dtype), qw, qz, sc, sc_dt, b, b_dt, y.data_ptr(), _dt(y.dtype), m,
              lin.in_features, n, lin.group_size, int(lin.pack_dim == "in"), int(lin.sym), flag.data_ptr(), scratch.data_ptr(), need,
              _st())


def w8a16_matmul(lin, x2, y):
    """``y = x2 . deq(W)^T (+ bias)`` for the 8-bit AWQ layout (``oxq_w8a16_gemm``)."""
    ws = workspace(lin.out_features, lin.in_features, x2.device)
    bp, bd = _bias(lin.bias)
    _lib.call("oxq_w8a16_gemm", _p(x2), _dt(x2.dtype), _p(lin.qweight), _p(lin.qzeros), _p(lin.scales),
              _dt(lin.scales.dtype), bp, bd, _p(y), _dt(y.dtype), x2.shape[0], lin.in_features, lin.out_features,
              lin.group_size, _p(ws), ws.numel(), _st())


def gptq_matmul(raw, x2, y, bias=None):
    """``y = x2 . deq(W)^T (+ bias)`` for a GPTQ-packed ``QuantWeight`` or ``PackedQuantLinear`` (4 or 8 bit,
    ``oxq_gptq_gemm``)."""
    from .linear import _as_u32_words, _dt
    feat = lambda v: v() if callable(v) else v
    k, n, g = feat(raw.in_features), feat(raw.out_features), feat(raw.group_size)
    ws = workspace(n, k, x2.device)
    qw, sc = _as_u32_words(raw.qweight), raw.scales.contiguous()
    qz = None if raw.qzeros is None else _as_u32_words(raw.qzeros)
    sym = raw.qzeros is None or raw.zero_point == "symmetric"
    bp, bd = _bias(bias)
    _lib.call("oxq_gptq_gemm", _p(x2), _dt(x2.dtype), _p(qw), _p(qz), _p(sc), _dt(sc.dtype), bp, bd, _p(y), _dt(y.dtype),
              x2.shape[0], k, n, g, raw.bits, int(sym), _p(ws), ws.numel(), _st())


def awq_ffn_gate_up(lin, x2, y, activation: int, tensors=None):
    """``y[m, inter] = act(x . W_gate^T) * (x . W_up^T)`` on the fused ``[gate | up]`` AWQ linear ``lin``."""
    ws = workspace(lin.out_features, lin.in_features, x2.device)
    _lib.call("oxq_awq_ffn_gate_up", x2.data_ptr(), _lib.OXQ_BF16, *(tensors or lin._tensors())[:4], activation, y.data_ptr(),
              x2.shape[0], lin.in_features, lin.out_features // 2, lin.group_size, _p(ws), ws.numel(), _st())


def fp8_matmul(lin, s, s_out, s_in, x2, y):
    m, k, n, w = x2.shape[0], lin.in_features, lin.out_features, lin.weight
    if not (x2.data_ptr() | w.data_ptr()) & 15:
        need = int(_lib.entry("oxq_fp8_scratch_bytes")(m, k, n, s_out, s_in))
        if need:  # scratch of this call's own: calls on several streams do not meet
            bp, bd = _bias(lin.bias)
            flag = _flag_words(x2.device)
            scratch = torch.empty(need, dtype=torch.uint8, device=x2.device)
            _lib.call("oxq_fp8_matmul", x2.data_ptr(), _dt(x2.dtype), w.data_ptr(), _p(s), s_out, s_in, bp, bd, y.data_ptr(), _dt(y.dtype),
                      m, k, n, flag.data_ptr(), scratch.data_ptr(), need, _st())
            return
    ws = workspace(lin.out_features, lin.in_features, x2.device)
    bp, bd = _bias(lin.bias)
    _lib.call("oxq_fp8_gemm", _p(x2), _dt(x2.dtype), _p(lin.weight), _p(s), s_out, s_in, bp, bd, _p(y), _dt(y.dtype),
              x2.shape[0], lin.in_features, lin.out_features, _p(ws), ws.numel(), _st())


def gguf_matmul(lin, x2, y):
    ws = workspace(lin.out_features, lin.in_features, x2.device)
    bp, bd = _bias(lin.bias)
    _lib.call("oxq_gguf_gemm", lin.ggml_type, _p(x2), _dt(x2.dtype), _p(lin.blocks), bp, bd, _p(y), _dt(y.dtype),
              x2.shape[0], lin.in_features, lin.out_features, _p(ws), ws.numel(), _st())


def gguf_stream_matmul(lin, x2, y) -> bool:
    """``y = x2 . deq(W)^T (+ bias)`` by the stream kernel (``oxq_gguf_matmul``) with scratch of the call's own; False where another
    kernel is the better one."""
    m = x2.shape[0]
    need = int(_lib.entry("oxq_gguf_scratch_bytes")(lin.ggml_type, m, lin.in_features, lin.out_features))
    if not need:
        return False
    flag = _flag_words(x2.device)
    scratch = torch.empty(need, dtype=torch.uint8, device=x2.device)
    bp, bd = _bias(lin.bias)
    _lib.call("oxq_gguf_matmul", lin.ggml_type, x2.data_ptr(), _dt(x2.dtype), lin.blocks.data_ptr(), bp, bd, y.data_ptr(), _dt(y.dtype),
              m, lin.in_features, lin.out_features, flag.data_ptr(), scratch.data_ptr(), need, _st())
    return True


def mxfp4_matmul(lin, x2, y):
    ws = workspace(lin.out_features, lin.in_features, x2.device)
    bp, bd = _bias(lin.bias)
    _lib.call("oxq_mxfp4_gemm", _p(x2), _dt(x2.dtype), _p(lin.blocks), _p(lin.scales), bp, bd, _p(y), _dt(y.dtype),
              x2.shape[0], lin.in_features, lin.out_features, _p(ws), ws.numel(), _st())
