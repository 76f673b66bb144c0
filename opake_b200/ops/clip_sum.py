"""Fused clip-and-sum of materialised per-example gradients (counterpart of ``fused_clip_sum``,
packages/opake-patches/src/opake/api/patches/kernels/_clip_sum.py:270-379).

``leaves`` are ``[B, ...]`` tensors (bf16 or fp32) as produced by ``vmap(grad)``. Three multi-tensor kernels (per-example
squared norms; clip factors; scaled, storage-rounded, summed gradients) do the work for the whole tree. The factors use
the formula of the portable path in the same precision (fp64), so both paths agree on them up to the order in which the
squared norms are summed, and to fp32 summation order on the sums. Non-finite entries count as zero.
"""
from __future__ import annotations

from typing import Sequence

import torch

from . import _lib, multi_tensor as MT

__all__ = ["fused_clip_sum", "supported"]

accumulates = True       # fused_clip_sum takes ``prev`` and ``scale``


def supported(leaves: Sequence[torch.Tensor]) -> bool:
    return bool(leaves) and all(l.is_cuda and l.dtype in (torch.bfloat16, torch.float32) and l.dim() >= 1 for l in leaves) \
        and leaves[0].shape[0] <= 65535


def _guard(store: torch.dtype, roundoff: float) -> tuple[float, float]:
    """``(keep, tiny)`` of ``engine.clipping.numerics.guard_factor`` for an fp32 multiply: ``ratio * keep - tiny``."""
    fs, fm = torch.finfo(store), torch.finfo(torch.float32)
    rounding = fs.eps if store == torch.float32 else fs.eps / 2 + fm.eps
    return 1.0 - rounding - 2.0 * roundoff, fs.smallest_normal * fs.eps


def fused_clip_sum(leaves: Sequence[torch.Tensor], clipping_norm: float, *, with_postsq: bool = False, out_dtypes=None, prev=None,
                   scale: float = 1.0):
    """Returns ``(sums, norms, clipped_mask, post_norms)``: per-leaf fp32 sums of the clipped examples, the ``[B]``
    pre-clip norms (fp64), which examples were clipped, and (``with_postsq``) the norms after clipping. ``prev``: fp32 sums
    of earlier micro-batches that this one is added to; ``scale`` multiplies the result."""
    from ..engine.clipping import numerics as N
    leaves = [l.contiguous() for l in leaves]
    prev = None if prev is None else [p.contiguous() for p in prev]       # the portable path may leave other strides
    dev = leaves[0].device
    B = leaves[0].shape[0]
    outs = [torch.empty(l.shape[1:], dtype=torch.float32, device=dev) for l in leaves]
    if B == 0:
        for i, o in enumerate(outs):
            o.zero_() if prev is None else o.copy_(prev[i])
            if scale != 1.0:
                o.mul_(scale)
        z = torch.zeros(0, dtype=torch.float64, device=dev)
        return outs, z, z.bool(), (z if with_postsq else None)
    ro = N.norm_roundoff(leaves, torch.float64)
    norms, mask, post = MT.clip_and_sum(leaves, max(float(clipping_norm), 0.0), (_guard(torch.bfloat16, ro), _guard(torch.float32, ro)),
                                        outs, prev=prev, scale=scale, with_postsq=with_postsq)
    if out_dtypes is not None:
        outs = [o.to(d) for o, d in zip(outs, out_dtypes)]
    return outs, norms, mask, (torch.sqrt(post) if with_postsq else None)
