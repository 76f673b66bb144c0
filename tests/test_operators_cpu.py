"""Dispatcher operators with native autograd nodes (ops/nodes.py) under autograd and the functorch transforms, on the LoRA
functions, whose formulas run on any device and in fp64."""
import pytest
import torch
from torch.func import grad, jacrev, jvp, vmap

from opake_b200.patches.kernels import lora_linear, lora_mlp, lora_qkv


def _t(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed), dtype=torch.float64) * 0.5


W, A, B = _t(6, 5, seed=1), _t(2, 5, seed=2), _t(6, 2, seed=3)
X = _t(3, 4, 5, seed=4)


def _fused(x, a, b):
    return lora_linear(torch.tanh(x), W, a, b, 0.7)


def _plain(x, a, b):
    h = torch.tanh(x)
    return h @ W.t() + 0.7 * (h @ a.t()) @ b.t()


def _loss(f):
    return lambda a, b, x: (f(x, a, b) ** 2).sum()


def _close(got, want):
    got, want = ([t] if isinstance(t, torch.Tensor) else list(t) for t in (got, want))
    assert len(got) == len(want) and all(torch.allclose(g, w, rtol=1e-12, atol=1e-12) for g, w in zip(got, want))


@pytest.mark.parametrize("transform", [
    lambda f: vmap(grad(_loss(f), (0, 1, 2)), (None, None, 0))(A, B, X),
    lambda f: vmap(vmap(grad(_loss(f), (0, 1)), (None, None, 0)), (None, None, 0))(A, B, X.reshape(3, 2, 2, 5)),
    lambda f: grad(lambda a: vmap(_loss(f), (None, None, 0))(a, B, X).sum())(A),
    lambda f: vmap(grad(_loss(f)), (None, None, 1))(A, B, X),
    lambda f: jacrev(lambda a: f(X[0], a, B))(A),
    lambda f: vmap(jacrev(lambda a, x: f(x, a, B)), (None, 0))(A, X),
], ids=["vmap(grad)", "vmap(vmap(grad))", "grad(vmap)", "inner batch dimension", "jacrev", "vmap(jacrev)"])
def test_transforms(transform):
    _close(transform(_fused), transform(_plain))


def test_vmap_of_leaves_that_autograd_follows():
    a = A.clone().requires_grad_()
    for f in (_fused, _plain):
        vmap(_loss(f), (None, None, 0))(a, B, X).sum().backward()
    assert torch.allclose(a.grad, 2 * grad(lambda t: vmap(_loss(_plain), (None, None, 0))(t, B, X).sum())(A))


def test_autograd_and_what_it_saves():
    leaves = [t.clone().requires_grad_() for t in (X[0], A, B)]
    _close(torch.autograd.grad((_fused(*leaves) ** 2).sum(), leaves), torch.autograd.grad((_plain(*leaves) ** 2).sum(), leaves))
    # only what depends on a leaf that wants it
    a = A.clone().requires_grad_()
    y = _fused(X[0], a, B)
    y.sum().backward(retain_graph=True)
    first = a.grad.clone()
    y.sum().backward()
    _close(a.grad, 2 * first)
    with pytest.raises(RuntimeError, match="second time"):
        y.sum().backward()
    with torch.no_grad():
        assert not _fused(*leaves).requires_grad
    assert not _fused(X[0], A, B).requires_grad and _fused(X[0], a, B).requires_grad
    # an edit in place between the passes, and hooks on saved tensors
    y = _fused(X[0], a, B)
    with torch.no_grad():
        a.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.shape), t)[1], lambda t: t):
        lora_linear(X[0], W, a, B, 0.7)
    assert sorted(map(tuple, seen)) == sorted([(4, 5), (4, 2), (6, 5), (2, 5), (6, 2)])


def test_refused():
    a = A.clone().requires_grad_()
    g, = torch.autograd.grad((_fused(X[0], a, B) ** 2).sum(), a, create_graph=True)
    with pytest.raises(NotImplementedError, match="double backward"):
        g.sum().backward()
    with pytest.raises(NotImplementedError, match="double backward"):
        grad(lambda a: grad(lambda a: (_fused(X[0], a, B) ** 2).sum())(a).sum())(A)
    with pytest.raises(NotImplementedError, match="forward-mode"):
        jvp(lambda a: _fused(X[0], a, B), (A,), (A,))
    with pytest.raises(NotImplementedError, match="per-example LoRA weights"):
        vmap(lambda a, x: _fused(x, a, B), (0, 0))(A.expand(3, 2, 5), X)


def test_outputs_that_the_loss_does_not_use():
    proj = [(_t(6, 5, seed=10 + i), _t(2, 5, seed=20 + i), _t(6, 2, seed=30 + i), 0.5) for i in range(3)]

    def q_only(a, x):
        return lora_qkv(x, (proj[0][0], a, *proj[0][2:]), *proj[1:])[0].pow(2).sum()

    def plain(a, x):
        return (x @ proj[0][0].t() + 0.5 * (x @ a.t()) @ proj[0][2].t()).pow(2).sum()

    for f in (lambda h: vmap(grad(h, (0, 1)), (None, 0))(proj[0][1], X),
              lambda h: torch.autograd.grad(h(a := proj[0][1].clone().requires_grad_(), X[0]), a)):
        _close(f(q_only), f(plain))


def test_text_argument_and_saved_outputs():
    p = [(_t(7, 5, seed=1), _t(2, 5, seed=2), _t(7, 2, seed=3), 0.5), (_t(7, 5, seed=4), _t(2, 5, seed=5), _t(7, 2, seed=6), 0.5),
         (_t(5, 7, seed=7), _t(2, 7, seed=8), _t(5, 2, seed=9), 0.5)]
    lin = lambda x, q, a: x @ q[0].t() + q[3] * (x @ a.t()) @ q[2].t()
    for act, fn in (("silu", torch.nn.functional.silu), ("gelu_tanh", lambda t: torch.nn.functional.gelu(t, approximate="tanh"))):
        fused = lambda a, x: lora_mlp(x, (p[0][0], a, *p[0][2:]), p[1], p[2], act=act).pow(2).sum()
        plain = lambda a, x: lin(fn(lin(x, p[0], a)) * lin(x, p[1], p[1][1]), p[2], p[2][1]).pow(2).sum()
        got, want = (vmap(grad(f, (0, 1)), (None, 0))(p[0][1], X) for f in (fused, plain))
        assert all((g - w).norm() <= 1e-5 * w.norm() for g, w in zip(got, want))        # the activation is formed in fp32


@pytest.mark.parametrize("through_dispatcher", [False, True])
def test_tensors_without_memory_are_refused(through_dispatcher):
    """Under a tracer's FakeTensorMode no kernel may be launched: a fake tensor has the address zero."""
    from torch._subclasses.fake_tensor import FakeTensorMode, UnsupportedOperatorException

    from opake_b200.ops import flash, gemm, lce
    from opake_b200.patches.kernels import functions as fns, lora

    run = (lambda op, *a: op.call(*a)) if through_dispatcher else (lambda op, *a: op(*a))
    with FakeTensorMode():
        x = torch.empty(128, 64, device="cuda", dtype=torch.bfloat16)
        label = torch.empty(128, device="cuda", dtype=torch.int64)
        for f in (lambda: run(fns._Glu, x, x, 0), lambda: run(fns._RMSNorm, x, x[0], 1e-5, 0.0), lambda: run(fns._AddRMSNorm, x, x, x[0], 1e-5, 0.0),
                  lambda: run(fns._CE, x, label, 1.0, 0.0), lambda: run(fns._RopeQK, x, x.float(), 1, 64),
                  lambda: run(lce._LinearCE, x, x, label, 1.0, 0.0, True), lambda: lora._LoRA(x, x[:64], x[:8], x[:64, :8], 1.0),
                  lambda: gemm.gemm(x, x), lambda: flash.flash_fwd(torch.empty(128, 192, device="cuda", dtype=torch.bfloat16), 1, 1, 64)):
            with pytest.raises((NotImplementedError, UnsupportedOperatorException)):
                f()
