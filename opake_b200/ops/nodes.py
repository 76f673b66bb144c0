"""Differentiable operators whose autograd node lives in the dispatcher (csrc/host/nodes.cpp).

An operator is a function on tensors and a ``vmap`` rule, its gradient another operator. Under
``vmap(grad(...))`` torch runs a Python ``autograd.Function`` through Python bookkeeping at every transform level, 0.6 ms for a
forward and backward pass on the host whatever the tensors' size; these operators go through the dispatcher as torch's own do.
Saved tensors, version checks and saved-tensor hooks are those of torch's own operators; second-order and forward-mode
differentiation raise ``NotImplementedError``. Where the native nodes cannot be had (no built library and no compiler), the same
operators are Python ``autograd.Function`` objects.
"""
from __future__ import annotations

import threading
import warnings

import torch

from .._build import build_nodes, nodes_lib

_LIB = torch.library.Library("opake_b200", "DEF")

# Interfaces that torch keeps to itself. Where one of them is gone the operators take the supported, slower way (see _python_route).
_PRIVATE = (("DispatchKeySet",), ("DispatchKey", "FuncTorchBatched"), ("_ExcludeDispatchKeyGuard",), ("_functorch", "maybe_current_level"),
            ("_functorch", "is_functorch_wrapped_tensor"), ("_functorch", "is_batchedtensor"), ("_functorch", "maybe_get_level"),
            ("_functorch", "_unwrap_batched"), ("_functorch", "_add_batch_dim"))


def _private_interfaces() -> bool:
    for path in _PRIVATE:
        where = torch._C
        for name in path:
            where = getattr(where, name, None)
            if where is None:
                return False
    return hasattr(torch.autograd.forward_ad, "_current_level")


_HAVE_PRIVATE = _private_interfaces()
_NATIVE: bool | None = None          # whether the native nodes are in place; None: nothing has needed them yet
_NATIVE_LOCK = threading.RLock()
_OPERATORS: list["Operator"] = []


def _native():
    import importlib.util
    import sys

    name = "opake_b200._C._opake_nodes"
    if name not in sys.modules:
        path = nodes_lib()
        if not path.exists():
            build_nodes()
        spec = importlib.util.spec_from_file_location(name, path)
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        sys.modules[name] = module
    return sys.modules[name]


def _native_route() -> bool:
    """Whether calls that something follows go to the native nodes. The first such call loads (or compiles) them: importing the
    operators, and running them where nothing follows, needs neither the library nor a compiler."""
    global _NATIVE
    if _NATIVE is None:
        with _NATIVE_LOCK:
            if _NATIVE is None:
                try:
                    if not _HAVE_PRIVATE:
                        raise RuntimeError("this torch lacks an interface that they use")
                    native = _native()
                except (RuntimeError, OSError, ImportError) as exc:
                    warnings.warn(f"the native autograd nodes are not available, Python ones are used (slower under vmap): {exc}", stacklevel=3)
                    _NATIVE = False
                else:
                    for op in _OPERATORS:
                        op._register(native)
                    _NATIVE = True
    return _NATIVE


def front(t: torch.Tensor, dim: int | None, batch: int) -> torch.Tensor:
    """The batched dimension of a ``vmap`` rule's argument first; an unbatched argument is expanded."""
    return t.unsqueeze(0).expand(batch, *t.shape) if dim is None else t.movedim(dim, 0)


def plain(*args) -> bool:
    """No argument takes part in a transform or a graph, and nobody traces: the dispatcher can be passed by."""
    if not _HAVE_PRIVATE:
        return False
    wrapped, record = torch._C._functorch.is_functorch_wrapped_tensor, torch.is_grad_enabled()
    for a in args:
        if isinstance(a, torch.Tensor) and (wrapped(a) or (record and a.requires_grad)):
            return False
    return torch.autograd.forward_ad._current_level < 0 and not torch.compiler.is_compiling() and not torch.jit.is_tracing()


_BELOW = torch._C.DispatchKeySet(torch._C.DispatchKey.FuncTorchBatched) if _HAVE_PRIVATE else None


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


def _python_route(op: "Operator"):
    """The operator as a Python ``autograd.Function``: torch's supported way, for where the native nodes cannot be had."""
    tensor = object()

    def forward(*args):
        return op.forward(*args)

    def setup_context(ctx, inputs, output):
        if op.backward is None:
            return
        plan, _, differentiable = op.rule
        outputs = output if isinstance(output, tuple) else (output,)
        values = [(inputs if source == _INPUT else outputs)[i] for source, i in plan if source != _GRAD]
        ctx.constants = [tensor if isinstance(v, torch.Tensor) else v for v in values]
        ctx.save_for_backward(*(v for v in values if isinstance(v, torch.Tensor)))
        ctx.mark_non_differentiable(*(t for t, d in zip(outputs, differentiable) if not d))

    def backward(ctx, *grads):
        if op.backward is None:
            raise NotImplementedError(op.message)
        saved, constants, args = iter(ctx.saved_tensors), iter(ctx.constants), []
        for source, i in op.rule[0]:
            if source == _GRAD:
                args.append(grads[i])
            else:
                v = next(constants)
                args.append(next(saved) if v is tensor else v)
        out = op.backward(*args)
        out = out if isinstance(out, tuple) else (out,)
        return tuple(None if g is None else out[g] for g in op.rule[1])

    def jvp(ctx, *tangents):
        raise NotImplementedError(f"{op.name} has no forward-mode derivative")

    def vmap(info, in_dims, *args):
        return op.vmap(info.batch_size, in_dims, *args)

    return type(op.name.replace("::", "_"), (torch.autograd.Function,),
                {f.__name__: staticmethod(f) for f in (forward, setup_context, backward, jvp, vmap)})


_GRAD, _INPUT, _OUTPUT = range(3)        # as in csrc/host/nodes.cpp


class Operator:
    """``op(*args)``: the dispatcher operator, or its implementation ``forward`` where nothing would notice the difference."""

    def __init__(self, name: str, schema: str, forward, vmap):
        _LIB.define(name + schema)
        _LIB.impl(name, forward, "CompositeExplicitAutograd")
        self.name, self.forward, self.vmap = f"opake_b200::{name}", forward, vmap
        self.call = getattr(torch.ops.opake_b200, name).default
        if _HAVE_PRIVATE:
            _LIB.impl(name, _batched(self.call, vmap), "FuncTorchBatched")
        self.backward, self.rule, self.message = None, None, ""
        self._function = None

    def __call__(self, *args):
        if plain(*args):
            return self.forward(*args)
        if _native_route():
            return self.call(*args)
        if self._function is None:
            self._function = _python_route(self)
        return self._function.apply(*args)

    def differentiated_by(self, backward: "Operator", args: str, grads: list[int | None], outputs: list[bool]) -> "Operator":
        """``args``: what ``backward`` is called with, ``g0`` the gradient of output 0, ``i1`` input 1 and ``o2`` output 2 of the
        forward call. ``grads``: for each input the result of ``backward`` that is its gradient. ``outputs``: which outputs are
        differentiable."""
        self.backward, self.rule = backward, ([("gio".index(a[0]), int(a[1:])) for a in args.split()], grads, outputs)
        return self._declared()

    def not_differentiable(self, message: str) -> "Operator":
        self.message = message
        return self._declared()

    def _declared(self) -> "Operator":
        with _NATIVE_LOCK:
            _OPERATORS.append(self)
            if _NATIVE:
                self._register(_native())
        return self

    def _register(self, native) -> None:
        if self.backward is None:
            native.register_terminal(self.name, self.message)
        else:
            plan, grads, outputs = self.rule
            native.register_differentiable(self.name, self.backward.name, plan, [-1 if g is None else g for g in grads], outputs)
