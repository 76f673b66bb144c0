"""Vector forms of the row kernels at widths, offsets and row counts where vectors, heads and tails meet."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(shape, dev, scale=1.0):
    return (torch.randn(shape, device=dev, dtype=torch.float32) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("T,D", [(1, 8), (9, 256), (300, 264), (1021, 768), (40, 1024), (33, 1032)])
@pytest.mark.parametrize("res", [False, True])
def test_layernorm_backward(cuda, T, D, res):
    from opake_b200.ops import kernels as K

    x, dy, w, b = _rand((T, D), cuda), _rand((T, D), cuda), _rand((D,), cuda), _rand((D,), cuda)
    dres = _rand((T, D), cuda) if res else None
    _, mean, rstd = K.layernorm_fwd(x, w, b)
    dw, db = torch.ones(D, device=cuda), torch.ones(D, device=cuda)        # gradients are added
    dx = K.layernorm_bwd(dy, x, w, mean, rstd, dres=dres, dw=dw, db=db)
    xd = x.double().requires_grad_()
    wd, bd = w.double().requires_grad_(), b.double().requires_grad_()
    y = torch.nn.functional.layer_norm(xd, (D,), wd, bd, 1e-5)
    gx, gw, gb = torch.autograd.grad(y, (xd, wd, bd), dy.double())
    if res:
        gx = gx + dres.double()
    scale = gx.abs().max().clamp(min=1.0)
    assert bool(((dx.double() - gx).abs() <= gx.abs() * 2.0 ** -8 + 1e-4 * scale).all())
    tol = 1e-5 * T ** 0.5 * 16
    assert bool(((dw.double() - 1 - gw).abs() <= tol).all()) and bool(((db.double() - 1 - gb).abs() <= tol).all())


@pytest.mark.parametrize("T,N,pitch", [(1, 8, 8), (7, 264, 264), (1021, 768, 768), (300, 2304, 2304), (130, 256, 512), (50, 12, 12)])
def test_column_sums(cuda, T, N, pitch):
    from opake_b200.ops import kernels as K

    dy = _rand((T, pitch), cuda)[:, :N]
    out = torch.ones(N, device=cuda)
    K.colsum_(dy, out)
    assert bool(((out.double() - 1 - dy.double().sum(0)).abs() <= 1e-5 * T ** 0.5 * 8).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,off", [(1, 0), (7, 0), (4096, 0), (100_003, 0), (100_003, 1)])
def test_sum_of_squares(cuda, dtype, n, off):
    from opake_b200.ops import kernels as K

    x = torch.randn(n + off, device=cuda).to(dtype)[off:]
    out = torch.zeros(1, dtype=torch.float64, device=cuda)
    K.sumsq_(x, out)
    want = x.double().pow(2).sum().item()
    assert abs(out.item() - want) <= want * 64 * 2.0 ** -24


def test_ragged_rows_scatter(cuda):
    from opake_b200.ops import kernels as K

    src = torch.randn(4, 300, device=cuda)
    widths = torch.tensor([300, 1, 129, 256], dtype=torch.int32, device=cuda)
    offs = torch.tensor([0, 304, 312, 448], dtype=torch.int64, device=cuda)
    dst = torch.zeros(800, dtype=torch.bfloat16, device=cuda)
    ss = torch.zeros(1, dtype=torch.float64, device=cuda)
    K.scatter_rows_cast_sumsq(src, dst, offs, ss, widths)
    want = torch.zeros_like(dst)
    for r, (o, n) in enumerate(zip(offs.tolist(), widths.tolist())):
        want[o:o + n] = src[r, :n].to(torch.bfloat16)
    assert torch.equal(dst, want)
    ref = want.double().pow(2).sum().item()
    assert abs(ss.item() - ref) <= ref * 300 * 2.0 ** -24


@pytest.mark.parametrize("D", [8, 264, 2048, 2056, 4096, 8192, 8200])
def test_add_rmsnorm_widths(cuda, D):
    from opake_b200.ops import kernels as K

    x, r, w = _rand((5, D), cuda), _rand((5, D), cuda), _rand((D,), cuda)
    s, y, rstd = K.add_rmsnorm_fwd(x, r, w, 1e-5, 0.5)
    assert torch.equal(s, x + r)
    sd = s.double()
    rs = torch.rsqrt(sd.pow(2).mean(-1, keepdim=True) + 1e-5)
    ref = sd * rs * (w.double() + 0.5)
    assert bool(((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-6).all())
    assert bool(((rstd.double() - rs[:, 0]).abs() <= rs[:, 0] * 1e-5).all())


@pytest.mark.parametrize("kind", ["silu", "gelu", "gelu_tanh"])
@pytest.mark.parametrize("shape,offset", [((3, 8), 0), ((2, 5, 264), 0), ((7, 1000), 3)])
def test_gated_activation_split(cuda, kind, shape, offset):
    """Gate and up in separate buffers, also when their storage does not start on a 16-byte boundary; vmap agrees."""
    from opake_b200.patches.kernels import opake_geglu, opake_swiglu

    n = 1
    for v in shape:
        n *= v

    def make():
        return _rand((n + offset,), cuda)[offset:].view(shape)

    gate, up, d = make().requires_grad_(), make().requires_grad_(), make()
    fn = opake_swiglu if kind == "silu" else (lambda a, b: opake_geglu(a, b, "tanh" if kind == "gelu_tanh" else "none"))
    act = {"silu": torch.nn.functional.silu, "gelu": torch.nn.functional.gelu,
           "gelu_tanh": lambda t: torch.nn.functional.gelu(t, approximate="tanh")}[kind]
    out = fn(gate, up)
    got = torch.autograd.grad(out, (gate, up), d)
    gd, ud = gate.detach().double().requires_grad_(), up.detach().double().requires_grad_()
    ref = act(gd) * ud
    want = torch.autograd.grad(ref, (gd, ud), d.double())
    for a, b in zip((out, *got), (ref, *want)):
        assert bool(((a.double() - b).abs() <= b.abs() * 2.0 ** -7 + 1e-4).all())
    assert torch.equal(torch.func.vmap(fn)(gate.detach(), up.detach()), out.detach())
    assert torch.equal(torch.func.vmap(fn, in_dims=(0, None))(gate.detach(), up.detach()[0])[0], out.detach()[0])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V,softcap", [(1, 0.0), (7, 0.0), (37, 30.0), (4001, 0.0), (32000, 0.0), (5003, 30.0)])
def test_cross_entropy_rows(cuda, dtype, V, softcap):
    from opake_b200.patches.kernels import opake_cross_entropy

    logits = (torch.randn(9, V, device=cuda) * 3).to(dtype)
    if V > 4:
        logits[0, 1:4] = float("-inf")                    # masked entries
        logits[1, :-1] = torch.finfo(dtype).min           # the type's lowest value as a mask
    logits.requires_grad_()
    labels = torch.randint(0, V, (9,), device=cuda)
    labels[0], labels[1], labels[4] = 0, V - 1, -100
    c = torch.rand(9, device=cuda)
    nll = opake_cross_entropy(logits, labels, logit_softcapping=softcap)
    (g,) = torch.autograd.grad(nll, logits, c)
    ld = logits.detach().double().requires_grad_()
    z = softcap * torch.tanh(ld / softcap) if softcap else ld
    ref = torch.nn.functional.cross_entropy(z, labels, reduction="none", ignore_index=-100)
    (want,) = torch.autograd.grad(ref, ld, c.double())
    assert bool(((nll.double() - ref).abs() <= ref.abs() * 1e-5 + 2e-5).all())
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-5
    assert bool(((g.double() - want).abs() <= want.abs() * eps + 2e-6).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V", [7, 256, 4001, 32000, 50257])
@pytest.mark.parametrize("softcap", [0.0, 30.0])
def test_cross_entropy_keeps_nan(cuda, dtype, V, softcap):
    """A NaN anywhere in a row (before its first 16-byte boundary, in a vector, a whole vector, after the last vector, behind
    masked entries, everywhere) makes the row's loss and gradient NaN and touches no other row."""
    from opake_b200.patches.kernels import opake_cross_entropy

    base = torch.randn(12, V, device=cuda) * 3
    spots = [slice(0, 1), slice(V - 1, V), slice(V // 2, V // 2 + 1), slice(0, min(16, V)), slice(max(0, V - 16), V), slice(0, V)]
    rows = [1, 3, 5, 7, 9, 11]                       # odd rows of an odd width start off the 16-byte boundary
    for r, s in zip(rows, spots):
        base[r, s] = float("nan")
    if V > 20:
        base[3, : V - 1] = float("-inf")             # NaN after nothing but masked entries
        base[2, : V - 1] = float("-inf")             # one entry left: its loss is 0
    logits = base.to(dtype).requires_grad_()
    labels = torch.full((12,), V - 1, device=cuda)
    nll = opake_cross_entropy(logits, labels, logit_softcapping=softcap)
    (g,) = torch.autograd.grad(nll.sum(), logits)
    bad = torch.zeros(12, dtype=torch.bool, device=cuda)
    bad[rows] = True
    assert torch.equal(nll.isnan(), bad)
    assert torch.equal(g.isnan().any(1), bad)
    z = softcap * torch.tanh(logits.detach().double() / softcap) if softcap else logits.detach().double()
    ref = torch.nn.functional.cross_entropy(z, labels, reduction="none")
    assert bool(((nll.double() - ref).abs() <= ref.abs() * 1e-5 + 2e-5)[~bad].all())


def test_cross_entropy_label_buffer_may_be_refilled(cuda):
    from opake_b200.patches.kernels import opake_cross_entropy

    logits = torch.randn(9, 128, device=cuda).to(torch.bfloat16).requires_grad_()
    labels = torch.arange(9, dtype=torch.int32, device=cuda)
    (want,) = torch.autograd.grad(opake_cross_entropy(logits, labels.long()).sum(), logits)
    nll = opake_cross_entropy(logits, labels)
    labels.zero_()
    (got,) = torch.autograd.grad(nll.sum(), logits)
    assert torch.equal(got, want)
    f = torch.func.vmap(torch.func.grad(lambda z, l: opake_cross_entropy(z, l).sum()))
    assert torch.equal(f(logits.detach().view(3, 3, 128), torch.arange(9, dtype=torch.int32, device=cuda).view(3, 3)).view(9, 128), want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V", [512, 513, 2047, 2056, 4104, 8190, 12345])
def test_cross_entropy_row_forms(cuda, dtype, V):
    """Around the widths where rows change from single elements to vectors, and from one round of loads to several."""
    from opake_b200.patches.kernels import opake_cross_entropy

    logits = (torch.randn(5, V, device=cuda) * 3).to(dtype).requires_grad_()
    labels = torch.randint(0, V, (5,), device=cuda)
    c = torch.rand(5, device=cuda)
    nll = opake_cross_entropy(logits, labels)
    (g,) = torch.autograd.grad(nll, logits, c)
    ld = logits.detach().double().requires_grad_()
    ref = torch.nn.functional.cross_entropy(ld, labels, reduction="none")
    (want,) = torch.autograd.grad(ref, ld, c.double())
    assert bool(((nll.double() - ref).abs() <= ref.abs() * 1e-5 + 2e-5).all())
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-5
    assert bool(((g.double() - want).abs() <= want.abs() * eps + 2e-6).all())


@pytest.mark.parametrize("kind", ["silu", "gelu", "gelu_tanh"])
@pytest.mark.parametrize("n,offset", [(1, 0), (1000, 0), (1000, 1), (131072, 0), (131080, 0), (131073, 0), (200_000, 1), (12_582_920, 0)])
def test_interleaved_activation_forms(cuda, kind, n, offset):
    """One element per thread or eight, buffers on 16-byte and on 2-byte boundaries."""
    from opake_b200.ops import kernels as K

    gu = _rand((2 * n + offset,), cuda, 2.0)[offset:].view(1, 2 * n)
    d = _rand((n + offset,), cuda)[offset:].view(1, n)
    if kind == "silu":
        act, dgu = K.swiglu_fwd(gu), K.swiglu_bwd(d, gu)
    else:
        act, dgu = K.geglu_fwd(gu, kind == "gelu_tanh"), K.geglu_bwd(d, gu, kind == "gelu_tanh")
    g, u, dd = gu[0, 0::2].double().requires_grad_(), gu[0, 1::2].double().requires_grad_(), d[0].double()
    f = torch.nn.functional.silu(g) if kind == "silu" else torch.nn.functional.gelu(g, approximate="tanh" if kind == "gelu_tanh" else "none")
    dg, du = torch.autograd.grad(f * u, (g, u), dd)
    for a, b in ((act[0], (f * u).detach()), (dgu[0, 0::2], dg), (dgu[0, 1::2], du)):
        assert bool(((a.double() - b).abs() <= b.abs() * 2.0 ** -7 + 1e-4).all())


def test_cross_entropy_of_padded_rows(cuda):
    from opake_b200.ops import kernels as K

    wide = torch.randn(9, 520, device=cuda)
    lab, c = torch.arange(9, dtype=torch.int32, device=cuda), torch.rand(9, device=cuda)
    for V in (515, 37):
        z = wide[:, :V]
        nll, lse = K.cross_entropy_fwd(z, lab)
        d = K.cross_entropy_bwd(z, lab, lse, c)
        zc = z.contiguous()
        nll2, lse2 = K.cross_entropy_fwd(zc, lab)
        d2 = K.cross_entropy_bwd(zc, lab, lse2, c)
        assert torch.allclose(nll, nll2, rtol=1e-6, atol=1e-6) and torch.allclose(d, d2, rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("T,D", [(5, 64), (9, 1024), (33, 2048), (7, 4096), (3, 8200)])
def test_rmsnorm_in_place_leaves_a_copy_of_its_input(cuda, T, D):
    from opake_b200.ops import kernels as K

    wide = torch.randn(T, 2 * D + 16, device=cuda).to(torch.bfloat16)
    w = torch.randn(D, device=cuda).to(torch.bfloat16)
    want, rstd = K.rmsnorm_fwd(wide[:, 8 : D + 8].contiguous(), w)
    before, copies = wide.clone(), torch.zeros(T, D + 8, device=cuda, dtype=torch.bfloat16)
    x = wide[:, 8 : D + 8]
    _, again = K.rmsnorm_fwd(x, w, out=x, copy=copies[:, 8:])
    assert torch.equal(copies[:, 8:], before[:, 8 : D + 8]) and not copies[:, :8].any()
    assert torch.equal(x, want) and torch.equal(again, rstd)
    assert torch.equal(wide[:, :8], before[:, :8]) and torch.equal(wide[:, D + 8 :], before[:, D + 8 :])
