"""vmap-safe autograd wrappers around the sm_100a row kernels (packages/opake-patches/src/opake/api/patches/kernels/
rms_norm.py:74-373, fused_add_rms_norm.py:68-134, swiglu.py:31-130, geglu.py:39-330, cross_entropy.py:29-236,629-704,
rope_embedding.py:50-215).

Every op is two dispatcher operators (``ops/nodes.py``), forward and backward, each with a ``vmap`` rule, so that
``vmap(grad(loss))`` and double vmap work. The kernels act on rows, so a vmapped batch is handled by folding the batch
dimension into the row dimension: ONE launch for the whole batch. Only parameter gradients differ under vmap: they
must stay per example, and are reduced per example instead of over all rows. Inputs that are not CUDA bf16 take the
plain-PyTorch formulas (same math, used on CPU and as the numerical reference in the tests).
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from ...ops.nodes import Operator, front

__all__ = ["opake_rms_norm", "opake_fused_add_rms_norm", "opake_swiglu", "opake_geglu", "opake_cross_entropy",
           "opake_selective_log_softmax", "opake_rope_qk", "native_rows"]


def native_rows(x: torch.Tensor) -> bool:
    return x.is_cuda and x.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0


# =============================================================================================== RMSNorm
def _rms_ref(x, w, eps, offset):
    xf = x.float()
    y = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps) * (w.float() + offset)
    return y.to(x.dtype)


def _rms_norm_bwd(dy, x, w, rstd, offset):
    from ...ops import kernels as K
    D = x.shape[-1]
    dw = torch.zeros(D, dtype=torch.float32, device=x.device)
    dx = K.rmsnorm_bwd(dy.reshape(-1, D).contiguous(), x.reshape(-1, D).contiguous(), w, rstd.reshape(-1), dw=dw, w_offset=offset)
    return dx.view(x.shape), dw.to(w.dtype)


def _rms_norm_bwd_vmap(B, in_dims, dy, x, w, rstd, offset):
    from ...ops import kernels as K
    if in_dims[2] is not None:
        raise NotImplementedError("per-example norm weights are not supported")
    dy, x, rstd = front(dy, in_dims[0], B), front(x, in_dims[1], B), front(rstd, in_dims[3], B)
    D = x.shape[-1]
    dy2, x2, r1 = dy.reshape(-1, D).contiguous(), x.reshape(-1, D).contiguous(), rstd.reshape(-1).contiguous()
    dx = K.rmsnorm_bwd(dy2, x2, w, r1, dw=None, w_offset=offset).view(x.shape)
    # the weight gradient stays per example: one reduction kernel over each example's rows
    # (packages/opake-patches/src/opake/api/patches/kernels/rms_norm.py:292-373)
    return (dx, K.rmsnorm_dw_per_example(dy2, x2, r1, B).to(w.dtype)), (0, 0)


def _rms_norm(x, w, eps, offset):
    from ...ops import kernels as K
    D = x.shape[-1]
    y, rstd = K.rmsnorm_fwd(x.reshape(-1, D).contiguous(), w, eps, offset)
    return y.view(x.shape), rstd.view(x.shape[:-1])


def _rms_norm_vmap(B, in_dims, x, w, eps, offset):
    if in_dims[1] is not None:
        raise NotImplementedError("per-example norm weights are not supported")
    return _RMSNorm(front(x, in_dims[0], B), w, eps, offset), (0, 0)


_RMSNormBwd = Operator("rms_norm_bwd", "(Tensor dy, Tensor x, Tensor w, Tensor rstd, float offset) -> (Tensor, Tensor)", _rms_norm_bwd,
                       _rms_norm_bwd_vmap).not_differentiable("double backward through the fused RMSNorm is not supported")
_RMSNorm = Operator("rms_norm", "(Tensor x, Tensor w, float eps, float offset) -> (Tensor, Tensor)", _rms_norm, _rms_norm_vmap)
_RMSNorm.differentiated_by(_RMSNormBwd, "g0 i0 i1 o1 i3", [0, 1, None, None], [True, False])


def opake_rms_norm(x: torch.Tensor, weight: torch.Tensor, eps: float = 1e-6, offset: float = 0.0) -> torch.Tensor:
    """``x * rsqrt(mean(x^2) + eps) * (weight + offset)`` over the last dimension (``offset = 1`` is the Gemma form)."""
    if native_rows(x) and weight.dtype == torch.bfloat16:
        return _RMSNorm(x, weight, float(eps), float(offset))[0]
    return _rms_ref(x, weight, eps, offset)


def _add_rms_norm_bwd(dy, ds, s, w, rstd, offset):
    """``d(x) = d(residual) = ds + d(rmsnorm)/d(sum)``: the residual gradient is added inside the norm-backward kernel."""
    from ...ops import kernels as K
    D = s.shape[-1]
    dw = torch.zeros(D, dtype=torch.float32, device=s.device)
    dx = K.rmsnorm_bwd(dy.reshape(-1, D).contiguous(), s.reshape(-1, D).contiguous(), w, rstd.reshape(-1),
                       dres=ds.reshape(-1, D).contiguous(), dw=dw, w_offset=offset)
    return dx.view(s.shape), dw.to(w.dtype)


def _add_rms_norm_bwd_vmap(B, in_dims, dy, ds, s, w, rstd, offset):
    from ...ops import kernels as K
    if in_dims[3] is not None:
        raise NotImplementedError("per-example norm weights are not supported")
    dy, ds, s, rstd = (front(t, d, B) for t, d in zip((dy, ds, s, rstd), (in_dims[0], in_dims[1], in_dims[2], in_dims[4])))
    D = s.shape[-1]
    dy2, s2, r1 = dy.reshape(-1, D).contiguous(), s.reshape(-1, D).contiguous(), rstd.reshape(-1).contiguous()
    dx = K.rmsnorm_bwd(dy2, s2, w, r1, dres=ds.reshape(-1, D).contiguous(), dw=None, w_offset=offset).view(s.shape)
    return (dx, K.rmsnorm_dw_per_example(dy2, s2, r1, B).to(w.dtype)), (0, 0)


def _add_rms_norm(x, residual, w, eps, offset):
    """``s = x + residual; y = rmsnorm(s)`` in one kernel (packages/opake-patches/src/opake/api/patches/kernels/
    fused_add_rms_norm.py:68-134); returns ``(y, s, rstd)``."""
    from ...ops import kernels as K
    D = x.shape[-1]
    s, y, rstd = K.add_rmsnorm_fwd(x.reshape(-1, D).contiguous(), residual.reshape(-1, D).contiguous(), w, eps, offset)
    return y.view(x.shape), s.view(x.shape), rstd.view(x.shape[:-1])


def _add_rms_norm_vmap(B, in_dims, x, residual, w, eps, offset):
    if in_dims[2] is not None:
        raise NotImplementedError("per-example norm weights are not supported")
    return _AddRMSNorm(front(x, in_dims[0], B), front(residual, in_dims[1], B), w, eps, offset), (0, 0, 0)


_AddRMSNormBwd = Operator("add_rms_norm_bwd", "(Tensor dy, Tensor ds, Tensor s, Tensor w, Tensor rstd, float offset) -> (Tensor, Tensor)",
                          _add_rms_norm_bwd, _add_rms_norm_bwd_vmap)
_AddRMSNormBwd.not_differentiable("double backward through the fused add + RMSNorm is not supported")
_AddRMSNorm = Operator("add_rms_norm", "(Tensor x, Tensor residual, Tensor w, float eps, float offset) -> (Tensor, Tensor, Tensor)",
                       _add_rms_norm, _add_rms_norm_vmap)
_AddRMSNorm.differentiated_by(_AddRMSNormBwd, "g0 g1 o1 i2 o2 i4", [0, 0, 1, None, None], [True, True, False])


def opake_fused_add_rms_norm(x, residual, weight, eps: float = 1e-6, offset: float = 0.0):
    """Returns ``(normed, new_residual)`` with ``new_residual = x + residual``; one kernel forward, and the residual
    gradient is folded into the norm's backward kernel."""
    if native_rows(x) and residual.dtype == x.dtype and residual.shape == x.shape and weight.dtype == torch.bfloat16:
        y, s, _ = _AddRMSNorm(x, residual, weight, float(eps), float(offset))
        return y, s
    s = x + residual
    return opake_rms_norm(s, weight, eps, offset), s


# =============================================================================================== gated activations
def _dense16(t: torch.Tensor) -> torch.Tensor:
    """Contiguous and on a 16-byte boundary (a contiguous slice of a larger buffer may start anywhere)."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _glu_bwd(dact, gate, up, kind):
    from ...ops import kernels as K
    return K.glu_split_bwd(_dense16(dact), _dense16(gate), _dense16(up), kind)


def _glu_bwd_vmap(B, in_dims, dact, gate, up, kind):
    return _GluBwd(*(front(t, d, B).contiguous() for t, d in zip((dact, gate, up), in_dims)), kind), (0, 0)


def _glu(gate, up, kind):
    """Element-wise on two buffers: gate and up are read where the projections left them (no interleaved copy), and saved as they
    are: editing one of them in place before the backward pass raises, as it does with the plain formula."""
    from ...ops import kernels as K
    return K.glu_split_fwd(_dense16(gate), _dense16(up), kind)


def _glu_vmap(B, in_dims, gate, up, kind):
    return _Glu(front(gate, in_dims[0], B).contiguous(), front(up, in_dims[1], B).contiguous(), kind), 0


_GluBwd = Operator("glu_bwd", "(Tensor dact, Tensor gate, Tensor up, int kind) -> (Tensor, Tensor)", _glu_bwd, _glu_bwd_vmap)
_GluBwd.not_differentiable("double backward through the fused gated activation is not supported")
_Glu = Operator("glu", "(Tensor gate, Tensor up, int kind) -> Tensor", _glu, _glu_vmap)
_Glu.differentiated_by(_GluBwd, "g0 i0 i1 i2", [0, 1, None], [True])


def _native_glu(gate: torch.Tensor, up: torch.Tensor) -> bool:
    return native_rows(gate) and gate.shape == up.shape and up.dtype == gate.dtype and up.device == gate.device


def opake_swiglu(gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    """``silu(gate) * up``."""
    if _native_glu(gate, up):
        return _Glu(gate, up, 0)
    return F.silu(gate) * up


def opake_geglu(gate: torch.Tensor, up: torch.Tensor, approximate: str = "tanh") -> torch.Tensor:
    """``gelu(gate) * up`` (exact or tanh approximation)."""
    if _native_glu(gate, up):
        return _Glu(gate, up, 2 if approximate == "tanh" else 1)
    return F.gelu(gate, approximate=approximate) * up


# =============================================================================================== cross entropy
def _cross_entropy_bwd(g, logits, labels, lse, scale, softcap):
    from ...ops import kernels as K
    V = logits.shape[-1]
    coef = g.reshape(-1).float().contiguous()          # the kernel drops the rows whose label is negative
    d = K.cross_entropy_bwd(logits.reshape(-1, V), labels.reshape(-1), lse.reshape(-1), coef, scale, softcap)
    return d.view(logits.shape)


def _cross_entropy_bwd_vmap(B, in_dims, g, logits, labels, lse, scale, softcap):
    args = [front(t, d, B).contiguous() for t, d in zip((g, logits, labels, lse), in_dims[:4])]
    return _CEBwd(*args, scale, softcap), 0


def _cross_entropy(logits, labels, scale, softcap):
    from ...ops import kernels as K
    V = logits.shape[-1]
    lab = labels.reshape(-1).to(torch.int32, copy=True).contiguous()      # kept for the backward pass: never the caller's buffer
    nll, lse = K.cross_entropy_fwd(logits.reshape(-1, V), lab, scale, softcap)
    return nll.view(labels.shape), lse.view(labels.shape), lab.view(labels.shape)


def _cross_entropy_vmap(B, in_dims, logits, labels, scale, softcap):
    return _CE(front(logits, in_dims[0], B).contiguous(), front(labels, in_dims[1], B).contiguous(), scale, softcap), (0, 0, 0)


_CEBwd = Operator("cross_entropy_bwd", "(Tensor g, Tensor logits, Tensor labels, Tensor lse, float scale, float softcap) -> Tensor",
                  _cross_entropy_bwd, _cross_entropy_bwd_vmap)
_CEBwd.not_differentiable("double backward through the fused cross-entropy is not supported")
_CE = Operator("cross_entropy", "(Tensor logits, Tensor labels, float scale, float softcap) -> (Tensor, Tensor, Tensor)", _cross_entropy,
               _cross_entropy_vmap)
_CE.differentiated_by(_CEBwd, "g0 i0 o2 o1 i2 i3", [0, None, None, None], [True, False, False])


def opake_cross_entropy(logits: torch.Tensor, labels: torch.Tensor, *, ignore_index: int = -100, logit_scale: float = 1.0,
                        logit_softcapping: float = 0.0) -> torch.Tensor:
    """Per-position NLL (fp32; zero where ``labels == ignore_index``) of row-wise softmax over the last dimension."""
    # every negative label is ignored further down: only an ignore_index outside [-2^31, 0) has to be replaced
    lab = labels if -(2**31) <= ignore_index < 0 else torch.where(labels == ignore_index, torch.full_like(labels, -1), labels)
    if logits.is_cuda and logits.dtype in (torch.bfloat16, torch.float32) and logits.stride(-1) == 1 and logits.is_contiguous():
        return _CE(logits, lab, float(logit_scale), float(logit_softcapping))[0]
    z = logits.float() * logit_scale
    if logit_softcapping:
        z = logit_softcapping * torch.tanh(z / logit_softcapping)
    nll = torch.logsumexp(z, -1) - z.gather(-1, lab.clamp(min=0).unsqueeze(-1)).squeeze(-1)
    return torch.where(lab >= 0, nll, torch.zeros_like(nll))


def opake_selective_log_softmax(logits: torch.Tensor, indices: torch.Tensor) -> torch.Tensor:
    """``log_softmax(logits)[..., indices]``: minus the cross entropy against ``indices``."""
    return -opake_cross_entropy(logits, indices, ignore_index=-(2**31))


# =============================================================================================== RoPE
def _rotated(qk, table, n_heads, head_dim, backward):
    from ...ops import kernels as K
    out = qk.clone(memory_format=torch.contiguous_format)
    # leading dimensions are sequences of shape[-2] positions each
    K.rope_(out.view(-1, out.shape[-1]), table, n_heads, head_dim, backward=backward, period=out.shape[-2] if out.dim() > 2 else 0)
    return out


def _rope_vmap(op):
    def rule(B, in_dims, qk, table, n_heads, head_dim):
        if in_dims[1] is not None:
            raise NotImplementedError("per-example rotary tables are not supported")
        return op()(front(qk, in_dims[0], B).contiguous(), table, n_heads, head_dim), 0          # [B, T, C]: the table indexes T

    return rule


# Rotation of the q and k heads of a fused [rows, (Hq + Hk) * hd] buffer (rotate-half) and its inverse, each the other's gradient.
_ROPE_SCHEMA = "(Tensor qk, Tensor table, int n_heads, int head_dim) -> Tensor"
_RopeQK = Operator("rope", _ROPE_SCHEMA, lambda *a: _rotated(*a, False), _rope_vmap(lambda: _RopeQK))
_RopeQKInverse = Operator("rope_inverse", _ROPE_SCHEMA, lambda *a: _rotated(*a, True), _rope_vmap(lambda: _RopeQKInverse))
_RopeQK.differentiated_by(_RopeQKInverse, "g0 i1 i2 i3", [0, None, None, None], [True])
_RopeQKInverse.differentiated_by(_RopeQK, "g0 i1 i2 i3", [0, None, None, None], [True])


def opake_rope_qk(qk: torch.Tensor, table: torch.Tensor, n_heads: int, head_dim: int) -> torch.Tensor:
    """``qk`` is ``[T, n_heads * head_dim (+ untouched columns)]``; ``table`` the ``[T, head_dim/2, 2]`` cos/sin table."""
    if native_rows(qk):
        return _RopeQK(qk.contiguous(), table, int(n_heads), int(head_dim))
    T = qk.shape[-2]
    x = qk[..., : n_heads * head_dim].reshape(*qk.shape[:-1], n_heads, head_dim)
    cos = torch.cat([table[:T, :, 0], table[:T, :, 0]], -1)[:, None, :].to(x.dtype)
    sin = torch.cat([table[:T, :, 1], table[:T, :, 1]], -1)[:, None, :].to(x.dtype)
    rot = torch.cat([-x[..., head_dim // 2:], x[..., : head_dim // 2]], -1)
    y = (x * cos + rot * sin).reshape(*qk.shape[:-1], n_heads * head_dim)
    return torch.cat([y, qk[..., n_heads * head_dim:]], -1)
