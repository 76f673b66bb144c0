"""Functional wrappers over the bandwidth-bound sm_100a kernels (csrc/kernels/elementwise.cu, dp_step.cu).

They replace the reference's Triton kernels (packages/opake-patches/src/opake/api/patches/kernels/:
rms_norm.py, fused_add_rms_norm.py, rope_embedding.py, swiglu.py, geglu.py, cross_entropy.py, _clip_sum.py)
and the eager noise/optimizer math (opake-dpsgd noise/_gaussian.py, opake-optimizers _adam.py).
Every function launches on the current CUDA stream and returns without synchronising.
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from ._protos import DpStepArgs

_bf16 = torch.bfloat16


def _L():
    return _lib.lib()


def _s(t: torch.Tensor) -> int:
    return _lib.stream_ptr(t.device)


_p = _lib.ptr


def _chk(code: int, name: str) -> None:
    _lib.LAUNCHES[0] += 1
    if code != 0:
        raise _lib.KernelLibraryError(f"{name} failed with code {code}: {_L().opk_last_error().decode()}")


# ------------------------------------------------------------------------------------------------ norms
def rmsnorm_fwd(x, w, eps: float = 1e-6, w_offset: float = 0.0, out=None, copy=None):
    """``x``, ``out`` and ``copy`` may be column slices of wider row-major matrices (row pitch = ``stride(0)``). ``out`` may be
    ``x``; ``copy`` receives ``x``."""
    T, D = x.shape
    y = torch.empty_like(x) if out is None else out
    rstd = torch.empty(T, dtype=torch.float32, device=x.device)
    _chk(_L().opk_rmsnorm_fwd_ld(_p(x), x.stride(0), _p(w), _p(y), y.stride(0), _p(rstd), T, D, eps, w_offset, _p(copy),
                                   0 if copy is None else copy.stride(0), _s(x)), "rmsnorm_fwd")
    return y, rstd


def add_rmsnorm_fwd(x, r, w, eps: float = 1e-6, w_offset: float = 0.0):
    T, D = x.shape
    s, y = torch.empty_like(x), torch.empty_like(x)
    rstd = torch.empty(T, dtype=torch.float32, device=x.device)
    _chk(_L().opk_add_rmsnorm_fwd(_p(x), _p(r), _p(w), _p(s), _p(y), _p(rstd), T, D, eps, w_offset, _s(x)),
         "add_rmsnorm_fwd")
    return s, y, rstd


_RMS_WS: dict = {}
_RMS_WS_ROWS = 296


def _rms_workspace(device, floats: int) -> torch.Tensor:
    """Per-device scratch for the per-CTA partial weight gradients of the norm backward kernel. Calls on one device
    share it, so they must be ordered on one stream (the model runtimes issue every example on a single stream)."""
    key = device.index
    ws = _RMS_WS.get(key)
    if ws is None or ws.numel() < floats:
        ws = torch.empty(floats, dtype=torch.float32, device=device)
        _RMS_WS[key] = ws
    return ws


def _per_example(dw) -> tuple[int, int]:
    """Examples and pitch of a per-example fp32 output: ``[n]`` (one example) or ``[examples, n]``."""
    return (1, 0) if dw is None or dw.dim() == 1 else (dw.shape[0], dw.stride(0))


def rmsnorm_bwd_scratch(D: int, examples: int, device) -> torch.Tensor:
    """Scratch of :func:`rmsnorm_bwd` for a caller that keeps its own (one per stream, and one that a graph may hold on to)."""
    return torch.empty(_RMS_WS_ROWS * examples * D, dtype=torch.float32, device=device)


def rmsnorm_bwd(dy, x, w, rstd, dres=None, dw=None, w_offset: float = 0.0, out=None, scratch=None):
    """Returns ``dx`` (plus ``dres`` when given); accumulates the weight gradient into fp32 ``dw`` when given. ``dw``
    ``[examples, D]``: the rows are that many examples of equal length, one after the other."""
    T, D = x.shape
    n, pitch = _per_example(dw)
    dx = torch.empty_like(x) if out is None else out
    ws_rows = _RMS_WS_ROWS * n
    ws = None
    if dw is not None:
        ws = _rms_workspace(x.device, ws_rows * D) if scratch is None else scratch
        if ws.numel() < ws_rows * D:
            raise ValueError("scratch is too small")
    if dres is not None and dres.stride(0) != dx.stride(0):
        raise ValueError("dres must have the row pitch of the output")
    _chk(_L().opk_rmsnorm_bwd_ld(_p(dy), dy.stride(0), _p(x), x.stride(0), _p(w), _p(rstd), _p(dres), _p(dx), dx.stride(0),
                                 _p(dw), _p(ws), ws_rows, T // n, D, w_offset, n, pitch, _s(x)), "rmsnorm_bwd")
    return dx


def layernorm_fwd(x, w, b, eps: float = 1e-5, out=None):
    T, D = x.shape
    y = torch.empty_like(x) if out is None else out
    mean = torch.empty(T, dtype=torch.float32, device=x.device)
    rstd = torch.empty(T, dtype=torch.float32, device=x.device)
    _chk(_L().opk_layernorm_fwd(_p(x), _p(w), _p(b), _p(y), _p(mean), _p(rstd), T, D, eps, _s(x)), "layernorm_fwd")
    return y, mean, rstd


def layernorm_bwd(dy, x, w, mean, rstd, dres=None, dw=None, db=None, out=None):
    T, D = x.shape
    dx = torch.empty_like(x) if out is None else out
    n, pitch = _per_example(dw)
    if dw is not None and db is not None and _per_example(db) != (n, pitch):
        raise ValueError("dw and db must have one layout")
    _chk(_L().opk_layernorm_bwd(_p(dy), _p(x), _p(w), _p(mean), _p(rstd), _p(dres), _p(dx), _p(dw), _p(db), T // n, D, n, pitch,
                                _s(x)), "layernorm_bwd")
    return dx


# ------------------------------------------------------------------------------------------------ rope
def rope_table(seq_len: int, head_dim: int, theta: float = 10000.0, device=None, scaling: dict | None = None):
    """``[T, head_dim/2, 2]`` fp32 (cos, sin) table; ``scaling`` implements the Llama-3 frequency rescale."""
    inv = 1.0 / (theta ** (torch.arange(0, head_dim, 2, dtype=torch.float64) / head_dim))
    if scaling and scaling.get("rope_type", scaling.get("type")) == "llama3":
        factor = scaling["factor"]
        lo, hi = scaling["low_freq_factor"], scaling["high_freq_factor"]
        old = scaling["original_max_position_embeddings"]
        wavelen = 2 * torch.pi / inv
        smooth = ((old / wavelen) - lo) / (hi - lo)
        scaled = torch.where(wavelen > old / lo, inv / factor, inv)
        mid = (wavelen <= old / lo) & (wavelen >= old / hi)
        inv = torch.where(mid, (1 - smooth) * inv / factor + smooth * inv, scaled)
    ang = torch.arange(seq_len, dtype=torch.float64)[:, None] * inv[None, :]
    return torch.stack([ang.cos(), ang.sin()], dim=-1).to(torch.float32).to(device).contiguous()


class RopeTables:
    """The rotary tables of one model, longer ones as longer sequences come. None is dropped: a CUDA graph that was captured for shorter
    sequences reads the table of its time. Each is at least twice as long as the one before it, so all together are less than two of
    the longest."""

    def __init__(self, head_dim: int, theta: float, scaling: dict | None, rows: int):
        self.args, self.rows = (head_dim, theta), rows
        self.scaling = scaling
        self.tables: dict[str, list[torch.Tensor]] = {}

    def get(self, T: int, device) -> torch.Tensor:
        kept = self.tables.setdefault(str(device), [])
        if not kept or kept[-1].shape[0] < T:
            rows = max(T, 2 * kept[-1].shape[0] if kept else self.rows)
            kept.append(rope_table(rows, *self.args, device=device, scaling=self.scaling))
        return kept[-1]


def rope_(qk, table, n_heads: int, head_dim: int, pos=None, backward: bool = False, period: int = 0):
    """Rotate the first ``n_heads`` heads of every row of ``qk`` in place (rotate-half convention). Row ``t`` sits at
    position ``pos[t]``, else ``t % period`` (``period`` rows per sequence), else ``t``."""
    _chk(_L().opk_rope(_p(qk), _p(table), _p(pos), period, qk.shape[0], n_heads, head_dim, qk.stride(0),
                             -1.0 if backward else 1.0, _s(qk)), "rope")
    return qk


# ------------------------------------------------------------------------------------------------ activations
def swiglu_fwd(gu):
    T, F2 = gu.shape
    act = torch.empty(T, F2 // 2, dtype=_bf16, device=gu.device)
    _chk(_L().opk_swiglu_fwd(_p(gu), _p(act), T, F2 // 2, _s(gu)), "swiglu_fwd")
    return act


def swiglu_bwd(dact, gu, out=None):
    T, F = dact.shape
    dgu = torch.empty_like(gu) if out is None else out
    _chk(_L().opk_swiglu_bwd(_p(dact), _p(gu), _p(dgu), T, F, _s(gu)), "swiglu_bwd")
    return dgu


def geglu_fwd(gu, approximate: bool = True, out=None):
    T, F2 = gu.shape
    act = torch.empty(T, F2 // 2, dtype=_bf16, device=gu.device) if out is None else out
    _chk(_L().opk_geglu_fwd(_p(gu), _p(act), T, F2 // 2, int(approximate), _s(gu)), "geglu_fwd")
    return act


def geglu_bwd(dact, gu, approximate: bool = True, out=None):
    T, F = dact.shape
    dgu = torch.empty_like(gu) if out is None else out
    _chk(_L().opk_geglu_bwd(_p(dact), _p(gu), _p(dgu), T, F, int(approximate), _s(gu)), "geglu_bwd")
    return dgu


def glu_split_fwd(gate, up, kind: int):
    """``act(gate) * up`` of two contiguous bf16 buffers (a multiple of 8 elements); kind 0 SwiGLU, 1 GEGLU, 2 GEGLU tanh;
    3 and 4: 0 and 2 with every fp32 operation rounded by itself (library exponential)."""
    act = torch.empty_like(gate)
    _chk(_L().opk_glu_split_fwd(_p(gate), _p(up), _p(act), gate.numel(), kind, _s(gate)), "glu_split_fwd")
    return act


def glu_split_bwd(dact, gate, up, kind: int):
    dgate, dup = torch.empty_like(gate), torch.empty_like(up)
    _chk(_L().opk_glu_split_bwd(_p(dact), _p(gate), _p(up), _p(dgate), _p(dup), gate.numel(), kind, _s(gate)), "glu_split_bwd")
    return dgate, dup


def gelu_fwd(x, out=None):
    y = torch.empty_like(x) if out is None else out
    _chk(_L().opk_gelu_fwd(_p(x), _p(y), x.numel(), _s(x)), "gelu_fwd")
    return y


def gelu_bwd(dy, x, out=None):
    dx = torch.empty_like(x) if out is None else out
    _chk(_L().opk_gelu_bwd(_p(dy), _p(x), _p(dx), x.numel(), _s(x)), "gelu_bwd")
    return dx


# ------------------------------------------------------------------------------------------------ embedding
def embedding_fwd(tok, table, pos_table=None, out=None, period: int = 0):
    """``out[t] = table[tok[t]]`` (``+ pos_table[t]``; with ``period`` rows per sequence ``pos_table[t % period]``)."""
    T, D = tok.numel(), table.shape[1]
    if out is None:
        out = torch.empty(T, D, dtype=_bf16, device=table.device)
    _chk(_L().opk_embedding_fwd(_p(tok), _p(table), _p(pos_table), _p(out), T, D, table.shape[0], period, _s(table)), "embedding_fwd")
    return out


class EmbeddingGradWorkspace:
    """Scratch for the per-example compact embedding gradient (first-occurrence table, fp32 rows) of ``examples`` sequences."""

    def __init__(self, vocab: int, max_tokens: int, dim: int, device, examples: int = 1):
        self.vocab, self.max_tokens = vocab, max_tokens
        self.first_pos = torch.full((examples * vocab,), 2**31 - 1, dtype=torch.int32, device=device)
        self.rep = torch.empty(examples * max_tokens, dtype=torch.int32, device=device)
        self.gc = torch.empty(examples * max_tokens, dim, dtype=torch.float32, device=device)

    def examples(self, j: int, n: int) -> "EmbeddingGradWorkspace":
        """The scratch of examples ``j .. j+n-1`` as a workspace of its own (views)."""
        part = object.__new__(EmbeddingGradWorkspace)
        part.vocab, part.max_tokens = self.vocab, self.max_tokens
        part.first_pos = self.first_pos[j * self.vocab : (j + n) * self.vocab]
        part.rep = self.rep[j * self.max_tokens : (j + n) * self.max_tokens]
        part.gc = self.gc[j * self.max_tokens : (j + n) * self.max_tokens]
        return part


def embedding_bwd_compact(tok, dx, ws: EmbeddingGradWorkspace, sumsq, examples: int = 1):
    """``examples`` sequences of ``ws.max_tokens`` tokens one after the other (one sequence may be shorter)."""
    T, D = dx.shape
    if examples > 1 and (T != examples * ws.max_tokens or ws.first_pos.numel() < examples * ws.vocab):
        raise ValueError("the workspace holds sequences of another number or length")
    _chk(_L().opk_embedding_bwd_compact(_p(tok), _p(dx), _p(ws.first_pos), _p(ws.rep), _p(ws.gc), _p(sumsq), T // examples, D,
                                        ws.vocab, examples, _s(dx)), "embedding_bwd_compact")


def embedding_accumulate(tok, ws: EmbeddingGradWorkspace, scale, acc, T: int, shared: bool = False):
    """``acc[tok[t]] += bf16(gc[t] * scale)`` for representative rows. ``shared``: other GPUs add to the same rows at the
    same time (sharded sums; ``acc`` may alias the owner's shard on another GPU), so reductions are used."""
    D = acc.shape[1]
    fn = _L().opk_embedding_accumulate_shared if shared else _L().opk_embedding_accumulate
    _chk(fn(_p(tok), _p(ws.rep), _p(ws.gc), _p(scale), _p(acc), T, D, _s(tok)), "embedding_accumulate")


# ------------------------------------------------------------------------------------------------ losses
def lce_finalize(pmax, psum, tgt, labels):
    T, tiles = pmax.shape
    lse = torch.empty(T, dtype=torch.float32, device=pmax.device)
    nll = torch.empty(T, dtype=torch.float32, device=pmax.device)
    _chk(_L().opk_lce_finalize(_p(pmax), _p(psum), _p(tgt), _p(labels), _p(lse), _p(nll), T, tiles, _s(pmax)),
         "lce_finalize")
    return lse, nll


def rmsnorm_dw_per_example(dy, x, rstd, batch: int):
    """``[batch, D]`` fp32 RMSNorm weight gradients, one per example, of a batch folded into rows (``dy``, ``x``:
    ``[batch * rows, D]`` bf16 contiguous; ``rstd``: ``[batch * rows]``)."""
    D = x.shape[-1]
    rows = x.numel() // D // batch
    dw = torch.zeros(batch, D, dtype=torch.float32, device=x.device)
    _chk(_L().opk_rmsnorm_dw_per_example(_p(dy), _p(x), _p(rstd), _p(dw), batch, rows, D, _s(x)), "rmsnorm_dw_per_example")
    return dw


def loss_coef(labels, nll, coef, loss, ntok=None, weight=None):
    """Mean-over-supervised-tokens loss of one example and the per-token coefficients of its gradient:
    ``coef[t] = (labels[t] >= 0) / max(1, n_supervised)`` (times ``weight``), ``loss = sum(nll * coef)``. ``loss`` of several
    elements: that many examples of equal length, one after the other."""
    n = loss.numel()
    _chk(_L().opk_loss_coef(_p(labels), _p(nll), _p(weight), _p(coef), _p(loss), _p(ntok), labels.numel() // n, n, _s(nll)), "loss_coef")


def cross_entropy_fwd(logits, labels, scale: float = 1.0, softcap: float = 0.0):
    T, V = logits.shape
    nll = torch.empty(T, dtype=torch.float32, device=logits.device)
    lse = torch.empty(T, dtype=torch.float32, device=logits.device)
    _chk(_L().opk_cross_entropy_fwd(_p(logits), int(logits.dtype == torch.float32), _p(labels), _p(nll), _p(lse), T, V,
                                    logits.stride(0), scale, softcap, _s(logits)), "cross_entropy_fwd")
    return nll, lse


def cross_entropy_bwd(logits, labels, lse, coef, scale: float = 1.0, softcap: float = 0.0):
    T, V = logits.shape
    d = torch.empty_strided(logits.shape, logits.stride(), dtype=logits.dtype, device=logits.device)    # the kernel uses one row pitch
    _chk(_L().opk_cross_entropy_bwd(_p(logits), int(logits.dtype == torch.float32), _p(labels), _p(lse), _p(coef), _p(d),
                                    T, V, logits.stride(0), scale, softcap, _s(logits)), "cross_entropy_bwd")
    return d


# ------------------------------------------------------------------------------------------------ DP primitives
def sumsq_(x, out, round_bf16: bool = False):
    """``out (float64) += sum(x**2)``: one sum, or with ``out`` of several elements one for each ``x[j]`` (contiguous)."""
    n = out.numel()
    _chk(_L().opk_sumsq(_p(x), int(x.dtype == torch.float32), int(round_bf16), x.numel() // n, _p(out), n,
                        x.stride(0) if n > 1 else 0, _s(x)), "sumsq")


def scatter_rows_cast_sumsq(src, dst_base, offsets, sumsq, widths=None):
    """fp32 rows ``src[r]`` (their first ``widths[r]`` columns, int32, when given) -> bf16 at ``dst_base + offsets[r]``;
    ``sumsq += sum(stored**2)``. ``src [examples, R, D]`` and ``dst_base [examples, n]``: one destination and sum each."""
    R, D = src.shape[-2:]
    n = src.shape[0] if src.dim() == 3 else 1
    _chk(_L().opk_scatter_rows_cast_sumsq(_p(src), _p(dst_base), _p(offsets), _p(widths), R, D, _p(sumsq), n,
                                          dst_base.stride(0) if n > 1 else 0, _s(src)), "scatter_rows_cast_sumsq")


def colsum_(dy, out):
    """``out += dy.sum(0)``; ``out [examples, N]``: the rows are that many examples of equal length, one after the other."""
    T, N = dy.shape
    n, pitch = _per_example(out)
    _chk(_L().opk_colsum(_p(dy), _p(out), T // n, N, dy.stride(0), n, pitch, _s(dy)), "colsum")


def embedding_add_rows(tok, ws, dense, T: int):
    """``dense[tok[t]] += gc[t]``; ``dense [examples, V, D]``: ``T`` tokens of each example into a matrix of its own."""
    n = dense.shape[0] if dense.dim() == 3 else 1
    _chk(_L().opk_embedding_add_rows(_p(tok), _p(ws.rep), _p(ws.gc), _p(dense), T, dense.shape[-1], n,
                                     dense.stride(0) if n > 1 else 0, _s(dense)), "embedding_add_rows")


def clip_scale(sumsq, clip: float, *, scale_out, norm_out=None, counters=None, auto: bool = False, gamma: float = 0.01,
               n_leaves: int = 1, widest_leaf: int = 1, reset: bool = True, loss=None, loss_sum=None):
    """``sumsq`` of several elements: one factor (and norm) for each. ``loss_sum`` (fp32 scalar): ``loss``, one per sum, is added to it
    in order."""
    if loss_sum is not None and (loss is None or loss.numel() != sumsq.numel()):
        raise ValueError("one loss for each squared norm")
    _chk(_L().opk_clip_scale(_p(sumsq), clip, int(auto), gamma, n_leaves, widest_leaf, _p(scale_out), _p(norm_out),
                             _p(counters), int(reset), sumsq.numel(), _p(loss), _p(loss_sum), _s(sumsq)), "clip_scale")


def clip_accumulate(g, scale, acc, overwrite: bool = False):
    _chk(_L().opk_clip_accumulate2(_p(g), _p(scale), _p(acc), g.numel(), int(overwrite), _s(g)), "clip_accumulate")


def clip_accumulate_group(gs, scales, acc, overwrite: bool = False):
    """``acc (+)= sum_j stored(gs[j] * scales[j])`` for up to 8 examples in one pass over the fp32 sums."""
    import ctypes

    n = len(gs)
    if not 1 <= n <= 8 or len(scales) != n:
        raise ValueError("a group holds 1 to 8 gradient buffers with one scale each")
    gp = (ctypes.c_void_p * n)(*[_p(g) for g in gs])
    sp = (ctypes.c_void_p * n)(*[_p(t) for t in scales])
    _chk(_L().opk_clip_accumulate_group(gp, sp, n, _p(acc), gs[0].numel(), int(overwrite), _s(acc)), "clip_accumulate_group")


def clip_accumulate_group_push(gs, scales, acc_ptrs: list[int], bounds: list[int], rank: int, n: int):
    """Sharded sums: the group's clipped sum ``sum_j stored(gs[j] * scales[j])`` over the first ``n`` elements is added
    to the owners' shards with reductions (``acc_ptrs[o]`` = device address of owner ``o``'s fp32 shard, peer-mapped for
    remote owners; owner ``o`` holds the elements ``[bounds[o], bounds[o+1])``)."""
    import ctypes

    k = len(gs)
    if not 1 <= k <= 8 or len(scales) != k:
        raise ValueError("a group holds 1 to 8 gradient buffers with one scale each")
    gp = (ctypes.c_void_p * k)(*[_p(g) for g in gs])
    sp = (ctypes.c_void_p * k)(*[_p(t) for t in scales])
    ap = (ctypes.c_void_p * len(acc_ptrs))(*acc_ptrs)
    bp = (ctypes.c_int64 * len(bounds))(*bounds)
    _chk(_L().opk_clip_accumulate_group_push(gp, sp, k, ap, bp, len(acc_ptrs), rank, n, _s(gs[0])), "clip_accumulate_group_push")


def copy_bytes(dst_ptr: int, src_ptr: int, nbytes: int, device) -> None:
    """Copy with the library's own kernel; either address may be peer-mapped memory of another GPU."""
    _chk(_L().opk_copy_bytes(dst_ptr, src_ptr, nbytes, _lib.stream_ptr(device)), "copy_bytes")


def philox_normal_(out, seed: int, step: int, *, stream_id: int = 0, offset: int = 0, sigma: float = 1.0,
                   accumulate: bool = False):
    _chk(_L().opk_philox_normal(_p(out), out.numel(), seed & (2**64 - 1), stream_id, step, offset, sigma,
                                int(accumulate), _s(out)), "philox_normal")
    return out


def dp_step(*, grad_src: list[int], shard_begin: int, shard_len: int, inv_batch: float, sigma: float, seed: int,
            step: int, m, v, master, param_dst: list[int], param_src, lr: float, beta1: float, beta2: float, eps: float,
            weight_decay: float, bc1: float, bc2: float, phi_hat: float, stream_id: int = 0, zero_grad: bool = False,
            blt_state=None, blt_decay=None, blt_scale=None, toep_state=None, toep_coef=None, toep_pos: int = 0,
            sgd_mode: bool = False, device=None, group=(), group_scales=(), group_len: int = 0, skip_sum: bool = False):
    """Launch the fused reduce-scatter + noise + DP-AdamW(-BC) + all-gather kernel for this rank's shard.

    ``grad_src`` / ``param_dst`` are raw device addresses (this rank first, then its peers). ``group`` / ``group_scales``:
    per-example bf16 gradients (elements ``[0, group_len)`` of the flat vector) and clip factors that are not in the sums
    yet and are added by this kernel; ``skip_sum``: the sums hold nothing below ``group_len`` and are not read there.
    """
    a = DpStepArgs()
    gs = (ctypes.c_void_p * len(grad_src))(*grad_src)
    pd = (ctypes.c_void_p * max(1, len(param_dst)))(*param_dst)
    a.grad_src, a.n_src = gs, len(grad_src)
    a.shard_begin, a.shard_len = shard_begin, shard_len
    a.inv_batch, a.sigma = inv_batch, sigma
    a.seed, a.stream_id, a.step = seed & (2**64 - 1), stream_id, step & 0xFFFFFFFF
    a.m, a.v, a.master = _p(m), _p(v), _p(master)
    a.param_dst, a.n_dst, a.param_src = pd, len(param_dst), _p(param_src)
    a.lr, a.beta1, a.beta2, a.eps, a.weight_decay = lr, beta1, beta2, eps, weight_decay
    a.bc1, a.bc2, a.phi_hat, a.zero_grad = bc1, bc2, phi_hat, int(zero_grad)
    if blt_state is not None:
        a.blt_state, a.blt_nbuf = _p(blt_state), blt_state.shape[0]
        a.blt_decay, a.blt_scale = _p(blt_decay), _p(blt_scale)
    if toep_coef is not None:       # banded Toeplitz C^-1: ring of the last len(coef) - 1 outputs (none for one coefficient)
        a.toep_coef = _p(toep_coef)
        a.toep_nlag = 0 if toep_state is None else toep_state.shape[0]
        a.toep_state, a.toep_pos = _p(toep_state), toep_pos
        if toep_coef.numel() != a.toep_nlag + 1:
            raise ValueError("toep_coef holds one coefficient more than the ring has slots")
    a.sgd_mode = int(sgd_mode)
    if group:
        if len(group) != len(group_scales) or len(group) > 8 or any(g.numel() < group_len for g in group):
            raise ValueError("a group holds 1 to 8 gradient buffers of at least group_len elements with one scale each")
        a.group_g = (ctypes.c_void_p * len(group))(*[_p(g) for g in group])
        a.group_scale = (ctypes.c_void_p * len(group))(*[_p(t) for t in group_scales])
    a.n_group, a.group_len, a.skip_sum = len(group), group_len, int(skip_sum)
    dev = device if device is not None else (m.device if m is not None else torch.device("cuda"))
    _chk(_L().opk_dp_step(ctypes.byref(a), _lib.stream_ptr(dev)), "dp_step")


# ------------------------------------------------------------------------------------------------ mixture of experts
class MoePlan:
    """Device-side routing state of one MoE layer invocation (buffers are reused across examples). ``T`` tokens are those of
    ``examples`` sequences of equal length, one after the other; ``group_k [E, 2]``, or ``[examples, E, 2]`` for several."""

    def __init__(self, T: int, E: int, k: int, device, examples: int = 1):
        if examples > 1 and (T % examples or E * examples > 256):
            raise ValueError("examples of equal length, and at most 256 pairs of expert and example")
        self.T, self.E, self.k, self.examples = T, E, k, examples
        self.n = T * k
        self.R = _L().opk_moe_rows_capacity(self.n, E, examples)
        i32 = dict(dtype=torch.int32, device=device)
        self.idx = torch.empty(T, k, **i32)
        self.wts = torch.empty(T, k, dtype=torch.float32, device=device)
        self.probs = torch.empty(T, E, dtype=torch.float32, device=device)
        self.dest = torch.empty(T, k, **i32)
        self.src_entry = torch.empty(self.R, **i32)
        self.tile_group = torch.empty(self.R // 128, **i32)
        self.group_k = torch.empty(*(() if examples == 1 else (examples,)), E, 2, **i32)
        self.counts = torch.empty(E, **i32)

    def part(self, examples: int) -> "MoePlan":
        """Plan for the first ``examples`` sequences, in the same buffers."""
        p = object.__new__(MoePlan)
        p.T, p.E, p.k, p.examples = self.T // self.examples * examples, self.E, self.k, examples
        p.n = p.T * p.k
        p.R = _L().opk_moe_rows_capacity(p.n, p.E, examples)
        p.idx, p.wts, p.probs, p.dest = (t[: p.T] for t in (self.idx, self.wts, self.probs, self.dest))
        p.src_entry, p.tile_group, p.counts = self.src_entry[: p.R], self.tile_group[: p.R // 128], self.counts
        p.group_k = self.group_k[0] if examples == 1 else self.group_k[:examples]
        return p

    def build(self, idx: torch.Tensor) -> "MoePlan":
        """Row plan for expert ids chosen by the caller (``[T, k]`` int32). Ids outside ``[0, E)`` are dropped: their
        ``dest`` entry becomes -1 and the combine kernels skip them."""
        self.idx.copy_(idx.reshape(self.T, self.k))
        _chk(_L().opk_moe_plan(_p(self.idx), self.n, self.E, self.examples, self.R, _p(self.dest), _p(self.src_entry), _p(self.tile_group),
                               _p(self.group_k), _p(self.counts), _s(self.idx)), "moe_plan")
        return self


def moe_route(logits, plan: MoePlan, norm_topk: bool = False):
    T, E = logits.shape
    _chk(_L().opk_moe_route(_p(logits), logits.stride(0), T, E, plan.k, int(norm_topk), _p(plan.idx), _p(plan.wts), _p(plan.probs),
                            _s(logits)), "moe_route")
    _chk(_L().opk_moe_plan(_p(plan.idx), plan.n, E, plan.examples, plan.R, _p(plan.dest), _p(plan.src_entry), _p(plan.tile_group), _p(plan.group_k),
                           _p(plan.counts), _s(logits)), "moe_plan")
    return plan


def moe_route_bwd(plan: MoePlan, dwts, dlogits, norm_topk: bool = False):
    _chk(_L().opk_moe_route_bwd(_p(plan.probs), _p(plan.idx), _p(dwts), plan.T, plan.E, plan.k, int(norm_topk), _p(dlogits),
                                dlogits.stride(0), _s(dlogits)), "moe_route_bwd")
    return dlogits


def moe_gather(x, plan: MoePlan, out, entry_scale=None):
    _chk(_L().opk_moe_gather(_p(x), x.stride(0), _p(plan.src_entry), plan.k, _p(entry_scale), plan.R, x.shape[1], _p(out), _s(x)),
         "moe_gather")
    return out


def moe_combine(y, plan: MoePlan, out, wts=None, residual=None):
    _chk(_L().opk_moe_combine(_p(y), _p(plan.dest), _p(wts), plan.k, _p(residual), plan.T, y.shape[1], _p(out), _s(y)), "moe_combine")
    return out


def moe_combine_bwd(dy, y, plan: MoePlan, dwts):
    _chk(_L().opk_moe_combine_bwd(_p(dy), _p(y), _p(plan.dest), plan.n, plan.k, y.shape[1], _p(dwts), _s(y)), "moe_combine_bwd")
    return dwts
