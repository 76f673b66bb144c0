"""Differentiable operators whose autograd node lives in the dispatcher (csrc/host/nodes.cpp).

An operator is a function on tensors and a ``vmap`` rule, its gradient another operator. Under
``vmap(grad(...))`` torch runs a Python ``autograd.Function`` through Python bookkeeping at every transform level, 0.6 ms for a
forward and backward pass on the host whatever the tensors' size; these operators go through the dispatcher as torch's own do.
Saved tensors, version checks and saved-tensor hooks are those of torch's own operators; second-order and forward-mode
differentiation raise ``NotImplementedError``.
"""
from __future__ import annotations

import torch

from .._build import NODES_LIB, build_nodes

_LIB = torch.library.Library("opake_b200", "DEF")


def _native():
    import importlib.util
    import sys

    name = "opake_b200._C._opake_nodes"
    if name not in sys.modules:
        if not NODES_LIB.exists():
            build_nodes()
        spec = importlib.util.spec_from_file_location(name, NODES_LIB)
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        sys.modules[name] = module
    return sys.modules[name]


def front(t: torch.Tensor, dim: int | None, batch: int) -> torch.Tensor:
    """The batched dimension of a ``vmap`` rule's argument first; an unbatched argument is expanded."""
    return t.unsqueeze(0).expand(batch, *t.shape) if dim is None else t.movedim(dim, 0)


def plain(*args) -> bool:
    """No argument takes part in a transform or a graph, and nobody traces: the dispatcher can be passed by."""
    wrapped, record = torch._C._functorch.is_functorch_wrapped_tensor, torch.is_grad_enabled()
    for a in args:
        if isinstance(a, torch.Tensor) and (wrapped(a) or (record and a.requires_grad)):
            return False
    return torch.autograd.forward_ad._current_level < 0 and not torch.compiler.is_compiling() and not torch.jit.is_tracing()


_BELOW = torch._C.DispatchKeySet(torch._C.DispatchKey.FuncTorchBatched)


def _batched(call, rule):
    """Kernel of an operator at a ``vmap`` level: ``rule(batch size, dimensions, *values) -> (results, dimensions)`` on the values
    behind the batched tensors (torch's own way of registering a rule costs 50 us a call)."""
    F = torch._C._functorch

    def kernel(*args):
        with torch._C._ExcludeDispatchKeyGuard(_BELOW):
            level = F.maybe_current_level()
            values, dims, batch = [], [], None
            for a in args:
                d = None
                if isinstance(a, torch.Tensor) and F.is_batchedtensor(a) and F.maybe_get_level(a) == level:
                    a, d = F._unwrap_batched(a, level)
                    batch = a.shape[d]
                values.append(a)
                dims.append(d)
            if batch is None:
                return call(*args)
            out, out_dims = rule(batch, tuple(dims), *values)
            if isinstance(out, torch.Tensor):
                return F._add_batch_dim(out, out_dims, level)
            return tuple(t if d is None else F._add_batch_dim(t, d, level) for t, d in zip(out, out_dims))

    return kernel


class Operator:
    """``op(*args)``: the dispatcher operator, or its implementation ``forward`` where nothing would notice the difference."""

    def __init__(self, name: str, schema: str, forward, vmap):
        _LIB.define(name + schema)
        _LIB.impl(name, forward, "CompositeExplicitAutograd")
        self.name, self.forward = f"opake_b200::{name}", forward
        self.call = getattr(torch.ops.opake_b200, name).default
        _LIB.impl(name, _batched(self.call, vmap), "FuncTorchBatched")

    def __call__(self, *args):
        return self.forward(*args) if plain(*args) else self.call(*args)

    def differentiated_by(self, backward: "Operator", args: str, grads: list[int | None], outputs: list[bool]) -> "Operator":
        """``args``: what ``backward`` is called with, ``g0`` the gradient of output 0, ``i1`` input 1 and ``o2`` output 2 of the
        forward call. ``grads``: for each input the result of ``backward`` that is its gradient. ``outputs``: which outputs are
        differentiable."""
        plan = [("gio".index(a[0]), int(a[1:])) for a in args.split()]
        _native().register_differentiable(self.name, backward.name, plan, [-1 if g is None else g for g in grads], outputs)
        return self

    def not_differentiable(self, message: str) -> "Operator":
        _native().register_terminal(self.name, message)
        return self
