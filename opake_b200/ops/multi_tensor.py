"""Multi-tensor kernels of the functional API (csrc/kernels/multi_tensor.cu): one launch for all leaves of a tree.

``usable`` decides whether a list of tensors may take them; everything else keeps the leaf-by-leaf torch formulas, whose
products and sums the kernels round in the same places (square root and quotient of the Adam update: correctly rounded,
within an ulp of the library's). The leaves' addresses are packed per call into the kernel's parameters:
nothing is cached between calls.
"""
from __future__ import annotations

import functools
import struct
from ctypes import c_float

import torch

from . import _lib, _protos

_LEAF = struct.Struct(_protos.MT_LEAF)
_DTYPES = (torch.float32, torch.bfloat16)
_PLAIN = (torch.Tensor, torch.nn.Parameter)


def usable(*groups) -> bool:
    """All tensors are plain dense contiguous fp32 / bf16 CUDA tensors on one device, tensors at the same position of the
    groups have the same shape, and nothing watches the computation (autograd, functorch, forward-mode, dispatch modes,
    tracing): the kernels are invisible to all of these."""
    first = groups[0]
    if not first or not all(len(g) == len(first) for g in groups):
        return False
    if (torch._C._functorch.maybe_current_level() is not None or torch._C._len_torch_dispatch_stack() > 0
            or torch._C._len_torch_function_stack() > 0 or torch.autograd.forward_ad._current_level >= 0
            or torch.jit.is_tracing() or torch.compiler.is_compiling()):
        return False
    t0 = first[0]
    if not isinstance(t0, torch.Tensor) or not t0.is_cuda:
        return False
    dev, grad = t0.device, torch.is_grad_enabled()
    for row in zip(*groups):
        shape = None
        for t in row:
            if type(t) not in _PLAIN or t.device != dev or t.dtype not in _DTYPES or t.layout is not torch.strided:
                return False
            if not t.is_contiguous() or t.is_conj() or t.is_neg() or (grad and t.requires_grad):
                return False
            if shape is None:
                shape = t.shape
            elif t.shape != shape:
                return False
    return True


def _pack(rows) -> bytes:
    """``rows``: (buffers (at most six, ``None`` allowed), elements, aux, scalar)."""
    out = bytearray()
    for bufs, n, aux, s in rows:
        ptrs, mask = [0] * 6, 0
        for i, t in enumerate(bufs):
            if t is not None:
                ptrs[i] = _lib.ptr(t)
                if t.dtype is torch.bfloat16:
                    mask |= 1 << i
        # c_float rounds and overflows to infinity like a scalar next to an fp32 tensor; struct refuses what is out of range
        out += _LEAF.pack(*ptrs, n, aux, c_float(s).value, mask)
    return bytes(out)


def _call(name: str, device, *args) -> None:
    with torch.cuda.device(device):
        _lib.check(getattr(_lib.lib(), name)(*args, _lib.stream_ptr(device)), name)


@functools.cache
def _clip_tiles() -> tuple[int, int]:
    """Elements per entry of the kernels' partial sums before and after clipping: constants of the library."""
    lib = _lib.lib()
    return lib.opk_mt_sumsq_tile(), lib.opk_mt_apply_tile()


def clip_and_sum(leaves, clip: float, guards, outs, *, prev=None, scale: float = 1.0, with_postsq: bool = False):
    """``outs[i] = (prev[i] + sum_b stored(leaves[i][b] * factor_b)) * scale``; ``leaves[i]``: ``[B, ...]`` contiguous.
    ``guards``: ``(keep, tiny)`` of the clip factor for bf16 and for fp32 storage. Returns ``(norms fp64, clipped mask,
    squared norms after clipping or None)``, each ``[B]``."""
    dev, B = leaves[0].device, leaves[0].shape[0]
    n = [l[0].numel() for l in leaves]
    blob = _pack([((l, o, None if prev is None else prev[i]), n[i], 0, 0.0) for i, (l, o) in enumerate(zip(leaves, outs))])
    t_sq, t_ap = _clip_tiles()
    n_sq, n_ap = sum((k + t_sq - 1) // t_sq for k in n), sum((k + t_ap - 1) // t_ap for k in n)
    partial = torch.empty(B, max(n_sq, 1), dtype=torch.float64, device=dev)
    factors = torch.empty(2, B, dtype=torch.float32, device=dev)
    norms = torch.empty(B, dtype=torch.float64, device=dev)
    clipped = torch.empty(B, dtype=torch.bool, device=dev)
    post = torch.empty(B, n_ap, dtype=torch.float64, device=dev) if with_postsq else None
    _call("opk_mt_sumsq_partial", dev, blob, len(leaves), B, n_sq, _lib.ptr(partial))
    (kb, tb), (kf, tf) = guards
    _call("opk_mt_clip_factors", dev, _lib.ptr(partial), n_sq, B, clip, kb, tb, kf, tf, factors[0].data_ptr(), factors[1].data_ptr(),
          _lib.ptr(norms), _lib.ptr(clipped))
    _call("opk_mt_apply_sum", dev, blob, len(leaves), B, n_ap, factors[0].data_ptr(), factors[1].data_ptr(), scale, _lib.ptr(post))
    return norms, clipped, (None if post is None else post.sum(1))


def add_gaussian(centers, stds, offsets, seed: int):
    """``center + std * z`` per leaf; ``offsets``: position of the leaf's first element in the flattened tree (multiple of 4)."""
    outs = [torch.empty_like(c) for c in centers]
    blob = _pack([((c, o), c.numel(), off // 4, s) for c, o, s, off in zip(centers, outs, stds, offsets)])
    _call("opk_mt_gaussian", centers[0].device, blob, len(centers), seed & (2**64 - 1))
    return outs


def adam(grads, mu, nu, *, b1: float, b2: float, bc1: float, bc2: float, eps: float, phi_hat=None):
    """New ``(updates, mu, nu)``; ``phi_hat``: per leaf, what the noise bias correction subtracts (``None``: off)."""
    outs = [(torch.empty_like(g), torch.empty_like(m), torch.empty_like(v)) for g, m, v in zip(grads, mu, nu)]
    blob = _pack([((g, m, v, *o), g.numel(), 0, 0.0 if phi_hat is None else phi_hat[i])
                  for i, (g, m, v, o) in enumerate(zip(grads, mu, nu, outs))])
    _call("opk_mt_adam", grads[0].device, blob, len(grads), b1, 1 - b1, b2, 1 - b2, bc1, bc2, eps, int(phi_hat is not None))
    return [o[0] for o in outs], [o[1] for o in outs], [o[2] for o in outs]


def finish_update(updates, step: float, params=None, decay: float = 0.0):
    """``(update + decay * param) * step`` per leaf (``params=None``: ``update * step``)."""
    outs = [torch.empty_like(u) for u in updates]
    blob = _pack([((u, None if params is None else params[i], o), u.numel(), 0, 0.0) for i, (u, o) in enumerate(zip(updates, outs))])
    _call("opk_mt_finish_update", updates[0].device, blob, len(updates), decay, step)
    return outs


def add_update(params, updates):
    """``param + update`` per leaf, the update rounded to the parameter's type first."""
    outs = [torch.empty_like(p) for p in params]
    blob = _pack([((p, u, o), p.numel(), 0, 0.0) for p, u, o in zip(params, updates, outs)])
    _call("opk_mt_add_update", params[0].device, blob, len(params))
    return outs
