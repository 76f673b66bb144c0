"""Python entry points of the tcgen05 flash-attention kernels (csrc/kernels/attention_sm100.cuh)."""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from ._lib import ptr

_P, _I, _L, _F = ctypes.c_void_p, ctypes.c_int32, ctypes.c_int64, ctypes.c_float


def _fn(name, argtypes):
    f = getattr(_lib.lib(), name)
    f.restype = _I
    f.argtypes = argtypes
    return f


def flash_fwd(qkv: torch.Tensor, H: int, KV: int, hd: int, out: torch.Tensor | None = None, n_seq: int = 1):
    """Causal GQA attention over the fused projection buffer. Returns ``(out [rows, H*hd], lse [n_seq * H, T])``: ``n_seq``
    sequences of ``T`` rows one after the other."""
    rows = qkv.shape[0]
    T = rows // n_seq
    if T * n_seq != rows:
        raise ValueError("the rows are not sequences of equal length")
    if out is None:
        out = torch.empty(rows, H * hd, dtype=torch.bfloat16, device=qkv.device)
    lse = torch.empty(n_seq * H, T, dtype=torch.float32, device=qkv.device)
    f = _fn("opk_attn_fwd", [_P, _P, _P, _I, _I, _I, _I, _I, _L, _L, _F, _P, _P])
    rc = f(ptr(qkv), ptr(out), ptr(lse), T, H, KV, hd, n_seq, qkv.stride(0), out.stride(0), hd**-0.5,
           _lib.err_word(qkv.device).data_ptr(), _lib.stream_ptr(qkv.device))
    _lib.check(rc, "opk_attn_fwd")
    return out, lse


def flash_bwd(dout, qkv, out, lse, H: int, KV: int, hd: int, dqkv: torch.Tensor, split_heads: bool = True, n_seq: int = 1):
    """Gradient with respect to the fused projection buffer (dQ, dK, dV written into ``dqkv``)."""
    T = qkv.shape[0] // n_seq
    t64 = (T + 63) // 64 * 64
    dsum = torch.empty(2, n_seq * H, t64, dtype=torch.float32, device=qkv.device)   # rowsum(dO*O), then -lse*log2(e)
    part = None
    if H > KV and split_heads:
        part = torch.empty(n_seq * 2 * (H // KV) * T * KV * hd, dtype=torch.float32, device=qkv.device)
    f = _fn("opk_attn_bwd", [_P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _L, _L, _F, _P, _P])
    rc = f(ptr(qkv), ptr(out), ptr(dout), ptr(lse), ptr(dsum), ptr(dqkv),
           ptr(part), T, H, KV, hd, n_seq,
           qkv.stride(0), out.stride(0), hd**-0.5, _lib.err_word(qkv.device).data_ptr(), _lib.stream_ptr(qkv.device))
    _lib.check(rc, "opk_attn_bwd")
    return dqkv
