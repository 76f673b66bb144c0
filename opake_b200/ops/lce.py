"""Fused linear + cross-entropy: per-token NLL of ``hidden @ weight.T`` without materialising fp32 logits.

Counterpart of ``opake_linear_cross_entropy_loss`` (packages/opake-patches/src/opake/api/patches/kernels/
linear_cross_entropy.py:1223-1276, kernels :101-247 and :292-528). The reference tiles the vocabulary inside a Triton
program and merges partial log-sum-exps under a spin lock; here the vocabulary GEMM runs on the tcgen05 kernel with
two epilogues: the forward epilogue reduces every 256-column tile to (max, sum-exp, target logit) per row, a tiny
finalize kernel merges the tiles, and the backward epilogue recomputes the logits tile and writes
``coef * (softmax - onehot)`` in bf16, from which dH and dW are two more GEMMs. Up to ``KEEP_BYTES`` of logits, over all losses
that wait for their backward pass, are left behind by the forward epilogue instead where memory is plenty (same bits, a pass
over memory in place of the product).

Both directions are dispatcher operators (``ops/nodes.py``) with ``vmap`` rules so that ``vmap(grad(loss))`` works: a
batch of examples sharing one weight is flattened into rows for the forward and dH; the per-example weight gradient
is one batched GEMM (packages/opake-patches/src/opake/api/patches/kernels/linear_cross_entropy.py:772-779 allocates
the same ``(B, V, D)`` result).
"""
from __future__ import annotations

import threading

import torch
from torch.multiprocessing.reductions import StorageWeakRef

from .nodes import Operator, front

IGNORE_INDEX = -100

# Logits that may wait for their backward passes at a time, over all losses on a device. They are twice the bf16 gradient that a
# backward pass writes anyway; beyond this size the second product is the smaller price.
KEEP_BYTES = 1 << 30
# Up to here nobody asks how much memory is left: the count takes 60 us on the host.
_UNASKED_BYTES = 256 << 20
_WAITING: list[tuple[torch.device, StorageWeakRef, int]] = []
_WAITING_LOCK = threading.Lock()
_TOP_HOOKS = getattr(torch._C._autograd, "_top_saved_tensors_default_hooks", None)       # without it nothing is kept


def _keep_logits(hidden, weight) -> bool:
    """Whether the forward pass leaves its logits for a backward pass: one is coming, and nobody is moving or replacing what
    autograd saves (offloading hooks would carry the logits around)."""
    return (torch.is_grad_enabled() and (hidden.requires_grad or weight.requires_grad)
            and _TOP_HOOKS is not None and _TOP_HOOKS(True) is None)


def native_available(hidden: torch.Tensor, weight: torch.Tensor) -> bool:
    return (hidden.is_cuda and hidden.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16
            and hidden.shape[-1] % 8 == 0)


# ------------------------------------------------------------------------------------------- plain-torch fallback
def _chunked_nll(hidden, weight, labels, logit_scale, softcap, chunk: int = 4096):
    """Per-token NLL in fp32, differentiable, ``chunk`` rows at a time (portable path, CPU included)."""
    out = []
    for s in range(0, hidden.shape[0], chunk):
        h = hidden[s:s + chunk]
        lab = labels[s:s + chunk]
        logits = (h.to(torch.float32) @ weight.to(torch.float32).t()) * logit_scale
        if softcap:
            logits = softcap * torch.tanh(logits / softcap)
        lse = torch.logsumexp(logits, dim=-1)
        tgt = logits.gather(-1, lab.clamp(min=0).unsqueeze(-1)).squeeze(-1)
        out.append(torch.where(lab >= 0, lse - tgt, torch.zeros_like(lse)))
    return torch.cat(out) if out else hidden.new_zeros(0, dtype=torch.float32)


# ------------------------------------------------------------------------------------------- native forward
def _logits_buffer(rows: int, vocab: int, dim: int, examples: int, device) -> torch.Tensor:
    """fp32 buffer in which the logits wait for their backward pass; empty where the losses that are waiting already leave no room for
    them, or the device would not have as much memory again as they and the backward pass take. (They stay through all of the backward
    pass: it may be asked for a second time.)"""
    from . import _lib, gemm as G
    n = G.lce_logits_floats(rows, vocab)
    # d logits, d hidden, d weight per example and its scaled copy
    needed = 4 * n + 2 * (n + rows * dim + 2 * examples * vocab * dim)
    with _WAITING_LOCK:
        _WAITING[:] = [w for w in _WAITING if not w[1].expired()]
        waiting = 4 * n + sum(size for dev, _, size in _WAITING if dev == device)
        if waiting <= KEEP_BYTES and (waiting <= _UNASKED_BYTES or 2 * needed <= _lib.free_bytes(device, plenty=16 * needed)):
            try:
                z = torch.empty(n, dtype=torch.float32, device=device)
                _WAITING.append((device, StorageWeakRef(z.untyped_storage()), 4 * n))
                return z
            except torch.cuda.OutOfMemoryError:
                pass
    return torch.empty(0, dtype=torch.float32, device=device)


def _native_fwd(hidden, weight, labels, logit_scale, softcap, keep, examples=1):
    """``(nll, lse, int32 labels, logits)``; the last one is empty unless ``keep`` and there is room for them."""
    from . import gemm as G, kernels as K
    T, V = hidden.shape[0], weight.shape[0]
    tiles = G.lce_tiles(V, parts=2 if softcap else 1)
    pmax = torch.empty(T, tiles, dtype=torch.float32, device=hidden.device)
    psum = torch.empty_like(pmax)
    tgt = torch.empty(T, dtype=torch.float32, device=hidden.device)
    lab = labels.to(torch.int32, copy=True).contiguous()      # kept for the backward pass: never the caller's buffer
    if keep and G.lce_keeps_logits(T, V, hidden.shape[1], softcap):
        z = _logits_buffer(T, V, hidden.shape[1], examples, hidden.device)
    else:
        z = torch.empty(0, dtype=torch.float32, device=hidden.device)
    G.gemm(hidden, weight, epilogue=G.EPI_LCE_FWD, labels=lab, pmax=pmax, psum=psum, tgt=tgt, alpha=logit_scale,
           softcap=softcap, z=z if z.numel() else None)
    lse, nll = K.lce_finalize(pmax, psum, tgt, lab)
    return nll, lse, lab, z


def _native_dlogits(hidden, weight, lab, lse, z, coef, logit_scale, softcap):
    from . import gemm as G
    T, V = hidden.shape[0], weight.shape[0]
    Vp = (V + 7) // 8 * 8
    dlog = torch.empty(T, Vp, dtype=torch.bfloat16, device=hidden.device)[:, :V]
    if z.numel():
        return G.lce_grad(z, lab, lse, coef.contiguous(), dlog, softcap)
    G.gemm(hidden, weight, out=dlog, epilogue=G.EPI_LCE_BWD, labels=lab, lse=lse, coef=coef.contiguous(),
           alpha=logit_scale, softcap=softcap)
    return dlog


def _linear_ce_bwd(grad_nll, hidden, weight, lab, lse, z, logit_scale, softcap):
    from . import gemm as G
    coef = (grad_nll.to(torch.float32) * (lab >= 0)).contiguous()
    dlog = _native_dlogits(hidden, weight, lab, lse, z, coef, logit_scale, softcap)
    # dlog is the gradient with respect to logit_scale * (hidden @ weight.T)
    d_hidden = G.gemm(dlog, weight, b_mn=True, alpha=logit_scale)
    d_weight = G.linear_wgrad(dlog, hidden)
    if logit_scale != 1.0:
        d_weight = d_weight * logit_scale
    return d_hidden, d_weight


def _linear_ce_bwd_vmap(B, in_dims, grad_nll, hidden, weight, lab, lse, z, logit_scale, softcap):
    from . import gemm as G
    if in_dims[2] is not None:
        raise NotImplementedError("fused linear cross-entropy under vmap needs one shared weight")
    g, h, lb, ls = (front(x, d, B) for x, d in zip((grad_nll, hidden, lab, lse), (in_dims[0], in_dims[1], in_dims[3], in_dims[4])))
    T, D = h.shape[1], h.shape[2]
    hf = h.reshape(B * T, D).contiguous()
    labf = lb.reshape(B * T).contiguous()
    coef = (g.to(torch.float32).reshape(B * T) * (labf >= 0)).contiguous()
    # the stored logits have the rows of the whole batch when the forward pass ran under this vmap, which shows in lse; with
    # a vmap over cotangents alone they are one example's
    zf = z if in_dims[4] is not None and in_dims[5] is None else z.new_empty(0)
    dlog = _native_dlogits(hf, weight, labf, ls.reshape(B * T).contiguous(), zf, coef, logit_scale, softcap)
    d_hidden = G.gemm(dlog, weight, b_mn=True, alpha=logit_scale).view(B, T, D)
    V = weight.shape[0]
    d_weight = torch.empty(B, V, D, dtype=torch.bfloat16, device=hidden.device)
    G.gemm(dlog.view(B, T, -1), hf.view(B, T, D), a_mn=True, b_mn=True, out=d_weight)
    if logit_scale != 1.0:
        d_weight = d_weight * logit_scale
    return (d_hidden, d_weight), (0, 0)


def _linear_ce(hidden, weight, labels, logit_scale, softcap, keep):
    return _native_fwd(hidden.contiguous(), weight, labels, logit_scale, softcap, keep)


def _linear_ce_vmap(B, in_dims, hidden, weight, labels, logit_scale, softcap, keep):
    if in_dims[1] is not None:
        raise NotImplementedError("fused linear cross-entropy under vmap needs one shared weight")
    h, lb = front(hidden, in_dims[0], B), front(labels, in_dims[2], B)
    T, D = h.shape[1], h.shape[2]
    nll, lse, lab, z = _native_fwd(h.reshape(B * T, D).contiguous(), weight, lb.reshape(B * T), logit_scale, softcap, keep, B)
    return (nll.view(B, T), lse.view(B, T), lab.view(B, T), z), (0, 0, 0, None)


# the backward pass is an operator of its own so that it can carry a vmap rule (per-example dW)
_LinearCEBackward = Operator("linear_ce_bwd", "(Tensor grad_nll, Tensor hidden, Tensor weight, Tensor lab, Tensor lse, Tensor z, "
                             "float logit_scale, float softcap) -> (Tensor, Tensor)", _linear_ce_bwd, _linear_ce_bwd_vmap)
_LinearCEBackward.not_differentiable("second-order differentiation of the fused linear cross-entropy is not supported")
_LinearCE = Operator("linear_ce", "(Tensor hidden, Tensor weight, Tensor labels, float logit_scale, float softcap, bool keep) -> "
                     "(Tensor, Tensor, Tensor, Tensor)", _linear_ce, _linear_ce_vmap)
_LinearCE.differentiated_by(_LinearCEBackward, "g0 i0 i1 o2 o1 o3 i3 i4", [0, 1, None, None, None, None], [True, False, False, False])


def linear_cross_entropy(hidden: torch.Tensor, weight: torch.Tensor, labels: torch.Tensor, *, logit_scale: float = 1.0,
                         logit_softcapping: float = 0.0, use_token_scaling: bool = False,
                         force_portable: bool = False) -> torch.Tensor:
    """Per-token NLL (fp32, zero where ``labels < 0``) of ``softmax(logit_scale * hidden @ weight.T)``.

    ``hidden`` is ``[T, D]``, ``weight`` ``[V, D]``, ``labels`` ``[T]`` already aligned with ``hidden`` (the caller
    shifts). ``use_token_scaling`` multiplies each token's loss by its detached target probability (the DFT
    objective, packages/opake-alignment/src/opake/api/alignment/sft/loss/_dft.py:43-88).
    """
    if hidden.dim() != 2:
        raise ValueError("hidden must be [T, D]; flatten leading dimensions first")
    if not force_portable and native_available(hidden, weight):
        nll = _LinearCE(hidden, weight, labels, float(logit_scale), float(logit_softcapping), _keep_logits(hidden, weight))[0]
    else:
        nll = _chunked_nll(hidden, weight, labels, float(logit_scale), float(logit_softcapping))
    if use_token_scaling:
        nll = nll * torch.exp(-nll).detach()
    return nll


def opake_linear_cross_entropy_loss(hidden_states, weight, labels, ignore_index: int = IGNORE_INDEX,
                                    logit_softcapping: float = 0, label_smoothing: float = 0.0,
                                    use_token_scaling: bool = False, logit_scale: float = 1.0) -> torch.Tensor:
    """Reference-shaped entry (packages/opake-patches/src/opake/api/patches/kernels/linear_cross_entropy.py:1223):
    ``hidden_states [..., L, D]`` and ``labels [..., L]`` in Hugging Face layout (position t predicts t+1); returns
    the per-sequence **sum** of token losses, shape ``[...]``."""
    if label_smoothing:
        raise NotImplementedError("label smoothing is not implemented in the fused linear cross-entropy")
    lead = hidden_states.shape[:-2]
    L, D = hidden_states.shape[-2:]
    h = hidden_states[..., :-1, :].reshape(-1, D)
    lab = labels[..., 1:]
    lab = torch.where(lab == ignore_index, torch.full_like(lab, -1), lab).reshape(-1)
    nll = linear_cross_entropy(h, weight, lab, logit_scale=logit_scale, logit_softcapping=logit_softcapping,
                               use_token_scaling=use_token_scaling)
    return nll.view(*lead, L - 1).sum(-1)
