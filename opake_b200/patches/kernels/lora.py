"""Fused LoRA linear layers with explicit backward and vmap rules (packages/opake-patches/src/opake/api/patches/
kernels/lora.py:206,499,1063: ``Opake_LoRA_W``, ``_QKV``, ``_MLP``).

``y = x W^T + s (x A^T) B^T (+ bias)`` with frozen ``W`` and trainable ``A [r, in]``, ``B [out, r]``. The backward is
written out (instead of letting autograd trace five matmuls) so that under ``vmap`` only the two small adapter
gradients are materialised per example: ``dA_b = s (dy_b B)^T x_b`` and ``dB_b = s dy_b^T (x_b A^T)``; ``dx`` is one
flattened GEMM chain for the whole batch. ``lora_grad_sq_norms`` gives the per-example squared norms of ``dA`` and
``dB`` without forming them (Gram identity), for clipping LoRA-only fine-tuning without any per-example tensor.
On CUDA bf16 the large products run on the tcgen05 GEMM; everything else uses ``torch.matmul``.
"""
from __future__ import annotations

import torch

from ...ops.nodes import Operator, front

__all__ = ["lora_linear", "lora_qkv", "lora_mlp", "lora_grad_sq_norms"]


def _mm(a: torch.Tensor, b_nk: torch.Tensor) -> torch.Tensor:
    """``a [M, K] @ b_nk[N, K]^T``."""
    if a.is_cuda and a.dtype == torch.bfloat16 and b_nk.dtype == torch.bfloat16 and a.shape[-1] % 8 == 0 and b_nk.shape[0] % 8 == 0 \
            and a.shape[0] >= 128:
        from ...ops import gemm as G
        return G.gemm(a.contiguous(), b_nk.contiguous())
    return a @ b_nk.t()


def _mm_nn(a: torch.Tensor, b_kn: torch.Tensor) -> torch.Tensor:
    """``a [M, K] @ b_kn[K, N]``."""
    if a.is_cuda and a.dtype == torch.bfloat16 and b_kn.dtype == torch.bfloat16 and a.shape[-1] % 8 == 0 and b_kn.shape[1] % 8 == 0 \
            and a.shape[0] >= 128:
        from ...ops import gemm as G
        return G.gemm(a.contiguous(), b_kn.contiguous(), b_mn=True)
    return a @ b_kn


def _native_pair(a: torch.Tensor, b: torch.Tensor, n: int) -> bool:
    return a.is_cuda and a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and a.shape[-1] % 8 == 0 and n % 8 == 0 and a.shape[0] >= 128


def _adapted(x, W, xa, B, s):
    """``x W^T + s (xa B^T)``; on the tcgen05 GEMM the base product enters as the residual of the adapter's epilogue. The
    epilogue rounds where the formula does: whether a call has the rows and widths for the kernel does not show in its result."""
    y = _mm(x, W)
    if _native_pair(xa, B, B.shape[0]) and y.dtype == torch.bfloat16 and y.shape[1] % 8 == 0:
        from ...ops import gemm as G
        return G.gemm(xa.contiguous(), B.contiguous(), out=y, residual=y, alpha=s, stepwise=True)
    return y + s * _mm(xa, B)


def _adapted_nn(dy, W, dyB, A, s, dx=None):
    """``(dx +) dy W + s (dyB A)``, added from the left; ``dx`` may be overwritten."""
    if (_native_pair(dy, W, W.shape[1]) and _native_pair(dyB, A, A.shape[1]) and (dx is None or dx.dtype == torch.bfloat16)):
        from ...ops import gemm as G
        out = G.gemm(dy.contiguous(), W.contiguous(), b_mn=True, out=dx, residual=dx, stepwise=True)
        return G.gemm(dyB.contiguous(), A.contiguous(), b_mn=True, out=out, residual=out, alpha=s, stepwise=True)
    base = _mm_nn(dy, W)
    return (base if dx is None else dx + base) + s * _mm_nn(dyB, A)


def _lora_bwd(dy, x, xa, W, A, B, s):
    # dy [M, out], x [M, in], xa [M, r]
    dyB = _mm_nn(dy, B)                                  # [M, r]
    dx = _adapted_nn(dy, W, dyB, A, s)                   # [M, in]
    dA = s * (dyB.t() @ x)                               # [r, in]
    dB = s * (dy.t() @ xa)                               # [out, r]
    return dx, dA, dB


def _lora_bwd_vmap(n, in_dims, dy, x, xa, W, A, B, s):
    if any(d is not None for d in in_dims[3:6]):
        raise NotImplementedError("per-example LoRA weights are not supported")
    dy, x, xa = (front(t, d, n) for t, d in zip((dy, x, xa), in_dims[:3]))
    M = dy.shape[1]
    dyf = dy.reshape(n * M, -1)
    dyB = _mm_nn(dyf, B)
    dx = _adapted_nn(dyf, W, dyB, A, s).view(n, M, -1)
    dA = s * torch.bmm(dyB.view(n, M, -1).transpose(1, 2), x)        # [n, r, in]
    dB = s * torch.bmm(dy.transpose(1, 2), xa)                       # [n, out, r]
    return (dx, dA, dB), (0, 0, 0)


def _lora(x, W, A, B, s):
    xa = _mm(x, A)                                       # [M, r]
    return _adapted(x, W, xa, B, s), xa


def _lora_vmap(n, in_dims, x, W, A, B, s):
    if any(d is not None for d in in_dims[1:4]):
        raise NotImplementedError("per-example LoRA weights are not supported")
    x = front(x, in_dims[0], n)
    M = x.shape[1]
    y, xa = _LoRA(x.reshape(n * M, -1), W, A, B, s)
    return (y.view(n, M, -1), xa.view(n, M, -1)), (0, 0)


_LoRABwd = Operator("lora_bwd", "(Tensor dy, Tensor x, Tensor xa, Tensor W, Tensor A, Tensor B, float s) -> (Tensor, Tensor, Tensor)",
                    _lora_bwd, _lora_bwd_vmap).not_differentiable("double backward through the fused LoRA linear is not supported")
_LoRA = Operator("lora", "(Tensor x, Tensor W, Tensor A, Tensor B, float s) -> (Tensor, Tensor)", _lora, _lora_vmap)
_LoRA.differentiated_by(_LoRABwd, "g0 i0 o1 i1 i2 i3 i4", [0, None, 1, 2, None], [True, False])


def lora_linear(x, weight, lora_a, lora_b, scaling: float, bias=None):
    """``x [..., in]`` -> ``[..., out]``."""
    lead = x.shape[:-1]
    y = _LoRA(x.reshape(-1, x.shape[-1]), weight, lora_a, lora_b, float(scaling))[0]
    if bias is not None:
        y = y + bias
    return y.view(*lead, -1)


def _adapter_grads(dy, x, xa, A, B, s, n=None):
    """``(dy B, dA, dB)`` for one adapted projection; with ``n`` the row dimension is ``n`` examples of ``M`` rows and the
    adapter gradients stay per example."""
    dyB = _mm_nn(dy, B)
    if n is None:
        return dyB, s * (dyB.t() @ x), s * (dy.t() @ xa)
    M = dy.shape[0] // n
    dA = s * torch.bmm(dyB.view(n, M, -1).transpose(1, 2), x.view(n, M, -1))
    dB = s * torch.bmm(dy.view(n, M, -1).transpose(1, 2), xa.view(n, M, -1))
    return dyB, dA, dB


def _lora_qkv_grads(n, dq, dk, dv, x, xaq, xak, xav, Wq, Aq, Bq, Wk, Ak, Bk, Wv, Av, Bv, sq, sk, sv):
    """Backward of three adapted projections of ONE input: the input gradient is a single accumulated chain, the six
    adapter gradients are the only per-example tensors under vmap (``Opake_LoRA_QKV``, lora.py:499 of the reference)."""
    dx, grads = None, []
    for dy, xa, W, A, B, s in ((dq, xaq, Wq, Aq, Bq, sq), (dk, xak, Wk, Ak, Bk, sk), (dv, xav, Wv, Av, Bv, sv)):
        dyB, dA, dB = _adapter_grads(dy, x, xa, A, B, s, n)
        part = _adapted_nn(dy, W, dyB, A, s)
        dx = part if dx is None else dx + part
        grads += [dA, dB]
    return (dx, *grads)


def _lora_qkv_bwd_vmap(n, in_dims, *args):
    if any(d is not None for d in in_dims[7:16]):
        raise NotImplementedError("per-example LoRA weights are not supported")
    acts = [front(t, d, n) for t, d in zip(args[:7], in_dims[:7])]
    M = acts[0].shape[1]
    out = _lora_qkv_grads(n, *[t.reshape(n * M, -1) for t in acts], *args[7:])
    return (out[0].view(n, M, -1), *out[1:]), (0,) * 7


def _lora_qkv(x, Wq, Aq, Bq, Wk, Ak, Bk, Wv, Av, Bv, sq, sk, sv):
    outs, xas = [], []
    for W, A, B, s in ((Wq, Aq, Bq, sq), (Wk, Ak, Bk, sk), (Wv, Av, Bv, sv)):
        xa = _mm(x, A)
        outs.append(_adapted(x, W, xa, B, s))
        xas.append(xa)
    return (*outs, *xas)


def _lora_qkv_vmap(n, in_dims, x, *rest):
    if any(d is not None for d in in_dims[1:10]):
        raise NotImplementedError("per-example LoRA weights are not supported")
    x = front(x, in_dims[0], n)
    M = x.shape[1]
    return tuple(t.view(n, M, -1) for t in _LoRAQKV(x.reshape(n * M, -1), *rest)), (0,) * 6


_QKV_WEIGHTS = "Tensor Wq, Tensor Aq, Tensor Bq, Tensor Wk, Tensor Ak, Tensor Bk, Tensor Wv, Tensor Av, Tensor Bv, float sq, float sk, float sv"
_LoRAQKVBwd = Operator("lora_qkv_bwd", "(Tensor dq, Tensor dk, Tensor dv, Tensor x, Tensor xaq, Tensor xak, Tensor xav, " + _QKV_WEIGHTS
                       + ") -> (" + ", ".join(["Tensor"] * 7) + ")", lambda *args: _lora_qkv_grads(None, *args), _lora_qkv_bwd_vmap)
_LoRAQKVBwd.not_differentiable("double backward through the fused LoRA projections is not supported")
_LoRAQKV = Operator("lora_qkv", "(Tensor x, " + _QKV_WEIGHTS + ") -> (" + ", ".join(["Tensor"] * 6) + ")", _lora_qkv, _lora_qkv_vmap)
_LoRAQKV.differentiated_by(_LoRAQKVBwd, "g0 g1 g2 i0 o3 o4 o5 " + " ".join(f"i{j}" for j in range(1, 13)),
                           [0, None, 1, 2, None, 3, 4, None, 5, 6, None, None, None], [True] * 3 + [False] * 3)


def lora_qkv(x, q, k, v):
    """Three adapted projections of the same input in one autograd node; each of ``q, k, v`` is
    ``(weight, A, B, scaling, bias)``. The input is saved once and its gradient accumulated in one chain."""
    lead = x.shape[:-1]
    out = _LoRAQKV(x.reshape(-1, x.shape[-1]), q[0], q[1], q[2], k[0], k[1], k[2], v[0], v[1], v[2],
                   float(q[3]), float(k[3]), float(v[3]))[:3]
    res = []
    for y, p in zip(out, (q, k, v)):
        if len(p) > 4 and p[4] is not None:
            y = y + p[4]
        res.append(y.view(*lead, -1))
    return tuple(res)


def _native_act(*ts) -> bool:
    # equal shapes: the kernel walks all buffers by one index (projections of other widths broadcast or fail in the formula)
    return all(t.is_cuda and t.dtype == torch.bfloat16 and t.shape == ts[0].shape and t.is_contiguous() and t.data_ptr() % 16 == 0
               and t.numel() % 8 == 0 for t in ts)


def _act_fwd(g, u, act: str):
    if _native_act(g, u):
        from ...ops import kernels as K
        return K.glu_split_fwd(g, u, 3 if act == "silu" else 4)
    gf = g.float()
    a = torch.nn.functional.silu(gf) if act == "silu" else torch.nn.functional.gelu(gf, approximate="tanh")
    return (a * u.float()).to(g.dtype)


def _act_bwd(dh, g, u, act: str):
    if _native_act(dh, g, u):
        from ...ops import kernels as K
        return K.glu_split_bwd(dh, g, u, 3 if act == "silu" else 4)
    gf, uf, dhf = g.float(), u.float(), dh.float()
    if act == "silu":
        sig = torch.sigmoid(gf)
        a, da = gf * sig, sig * (1 + gf * (1 - sig))
    else:
        c = 0.7978845608028654
        t = torch.tanh(c * (gf + 0.044715 * gf ** 3))
        a = 0.5 * gf * (1 + t)
        da = 0.5 * (1 + t) + 0.5 * gf * (1 - t * t) * c * (1 + 3 * 0.044715 * gf * gf)
    return (dhf * uf * da).to(g.dtype), (dhf * a).to(g.dtype)


def _lora_mlp_grads(n, dy, x, g, u, xag, xau, had, Wg, Ag, Bg, Wu, Au, Bu, Wd, Ad, Bd, sg, su, sd, act):
    """Backward of the adapted gated MLP (``Opake_LoRA_MLP``, lora.py:1063 of the reference): the activation is
    recomputed from the saved pre-activations, the three adapted projections are differentiated by hand."""
    h = _act_fwd(g, u, act)
    dyB, dAd, dBd = _adapter_grads(dy, h, had, Ad, Bd, sd, n)
    dh = _adapted_nn(dy, Wd, dyB, Ad, sd)
    dg, du = _act_bwd(dh, g, u, act)
    dgB, dAg, dBg = _adapter_grads(dg, x, xag, Ag, Bg, sg, n)
    duB, dAu, dBu = _adapter_grads(du, x, xau, Au, Bu, su, n)
    dx = _adapted_nn(du, Wu, duB, Au, su, _adapted_nn(dg, Wg, dgB, Ag, sg))
    return dx, dAg, dBg, dAu, dBu, dAd, dBd


def _lora_mlp_bwd_vmap(n, in_dims, *args):
    if any(d is not None for d in in_dims[7:16]):
        raise NotImplementedError("per-example LoRA weights are not supported")
    acts = [front(t, d, n) for t, d in zip(args[:7], in_dims[:7])]
    M = acts[0].shape[1]
    out = _lora_mlp_grads(n, *[t.reshape(n * M, -1) for t in acts], *args[7:])
    return (out[0].view(n, M, -1), *out[1:]), (0,) * 7


def _lora_mlp(x, Wg, Ag, Bg, Wu, Au, Bu, Wd, Ad, Bd, sg, su, sd, act):
    xag, xau = _mm(x, Ag), _mm(x, Au)
    g, u = _adapted(x, Wg, xag, Bg, sg), _adapted(x, Wu, xau, Bu, su)
    h = _act_fwd(g, u, act)
    had = _mm(h, Ad)
    return _adapted(h, Wd, had, Bd, sd), g, u, xag, xau, had


def _lora_mlp_vmap(n, in_dims, x, *rest):
    if any(d is not None for d in in_dims[1:10]):
        raise NotImplementedError("per-example LoRA weights are not supported")
    x = front(x, in_dims[0], n)
    M = x.shape[1]
    return tuple(t.view(n, M, -1) for t in _LoRAMLP(x.reshape(n * M, -1), *rest)), (0,) * 6


_MLP_WEIGHTS = ("Tensor Wg, Tensor Ag, Tensor Bg, Tensor Wu, Tensor Au, Tensor Bu, Tensor Wd, Tensor Ad, Tensor Bd, float sg, float su, "
                "float sd, str act")
_LoRAMLPBwd = Operator("lora_mlp_bwd", "(Tensor dy, Tensor x, Tensor g, Tensor u, Tensor xag, Tensor xau, Tensor had, " + _MLP_WEIGHTS
                       + ") -> (" + ", ".join(["Tensor"] * 7) + ")", lambda *args: _lora_mlp_grads(None, *args), _lora_mlp_bwd_vmap)
_LoRAMLPBwd.not_differentiable("double backward through the fused LoRA MLP is not supported")
_LoRAMLP = Operator("lora_mlp", "(Tensor x, " + _MLP_WEIGHTS + ") -> (" + ", ".join(["Tensor"] * 6) + ")", _lora_mlp, _lora_mlp_vmap)
_LoRAMLP.differentiated_by(_LoRAMLPBwd, "g0 i0 o1 o2 o3 o4 o5 " + " ".join(f"i{j}" for j in range(1, 14)),
                           [0, None, 1, 2, None, 3, 4, None, 5, 6, None, None, None, None], [True] + [False] * 5)


def lora_mlp(x, gate, up, down, act: str = "silu"):
    """Gated MLP with adapters on all three projections in one autograd node (``act``: ``silu`` or ``gelu_tanh``); each
    of ``gate, up, down`` is ``(weight, A, B, scaling[, bias])``. Projection biases take the composed path."""
    if any(len(p) > 4 and p[4] is not None for p in (gate, up, down)):
        from .functions import opake_geglu, opake_swiglu
        g, u = lora_linear(x, *gate), lora_linear(x, *up)
        h = opake_swiglu(g, u) if act == "silu" else opake_geglu(g, u)
        return lora_linear(h, *down)
    lead = x.shape[:-1]
    y = _LoRAMLP(x.reshape(-1, x.shape[-1]), gate[0], gate[1], gate[2], up[0], up[1], up[2], down[0], down[1], down[2],
                 float(gate[3]), float(up[3]), float(down[3]), "silu" if act == "silu" else "gelu_tanh")[0]
    return y.view(*lead, -1)


def lora_grad_sq_norms(x, dy, lora_a, lora_b, scaling: float):
    """Per-example ``(||dA_b||^2, ||dB_b||^2)`` for ``x [n, T, in]``, ``dy [n, T, out]`` without materialising the
    gradients: ``||U^T V||_F^2 = sum((U U^T) * (V V^T))`` with T x T Gram matrices (cheap when ``T << in, out``)."""
    s2 = float(scaling) ** 2
    xf, dyf = x.float(), dy.float()
    dyB = dyf @ lora_b.float()                      # [n, T, r]
    xa = xf @ lora_a.float().t()                    # [n, T, r]
    gx = torch.bmm(xf, xf.transpose(1, 2))          # [n, T, T]
    gdy = torch.bmm(dyf, dyf.transpose(1, 2))
    na = s2 * (torch.bmm(dyB, dyB.transpose(1, 2)) * gx).sum((1, 2))
    nb = s2 * (gdy * torch.bmm(xa, xa.transpose(1, 2))).sum((1, 2))
    return na, nb
