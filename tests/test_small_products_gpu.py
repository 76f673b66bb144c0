"""Products with few output tiles (narrow tiles, one per CTA) at the edges of tiles and reductions."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (M, N, K): one tile, one element past a tile, ragged everything, long reductions, narrow N, single rows
SHAPES = [(128, 128, 64), (129, 136, 72), (1, 8, 8), (317, 2048, 2048), (300, 264, 1032), (64, 2048, 2048), (1024, 768, 3072),
          (2048, 16, 520), (77, 50264, 64), (256, 40, 8192)]


def _rand(shape, dev, scale=1.0):
    return (torch.randn(shape, device=dev, dtype=torch.float32) * scale).to(torch.bfloat16)


def _check(out, a, b, extra=None):
    """fp64 product; bound: half an ulp of the bf16 store (2^-9 relative, twice for slack) plus fp32 summation of K terms."""
    ref = a.double() @ b.double()
    mag = (a.double().abs() @ b.double().abs()) * 2.0 ** -23 * (16 + a.shape[-1] ** 0.5)
    if extra is not None:
        ref = ref + extra.double()
    err = (out.double() - ref).abs()
    assert bool((err <= ref.abs() * 2.0 ** -8 + mag + 1e-30).all()), float((err - ref.abs() * 2.0 ** -8 - mag).max())


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_plain_products(cuda, M, N, K, layout):
    from opake_b200.ops import gemm as G
    from opake_b200.ops._lib import raise_if_device_error

    if layout == "tn":
        M = (M + 7) // 8 * 8                  # row pitch of the transposed operand
    a, b = _rand((M, K), cuda), _rand((K, N), cuda)
    A = a.t().contiguous() if layout == "tn" else a
    B = b.t().contiguous() if layout == "nt" else b
    out = G.gemm(A, B, a_mn=layout == "tn", b_mn=layout != "nt")
    raise_if_device_error(cuda)
    _check(out, a, b)
    again = G.gemm(A, B, a_mn=layout == "tn", b_mn=layout != "nt")
    assert torch.equal(out, again)


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (317, 2048, 2048), (130, 264, 1032), (2048, 16, 520)])
def test_bias_residual_and_batches(cuda, M, N, K):
    from opake_b200.ops import gemm as G
    from opake_b200.ops._lib import raise_if_device_error

    a, w, bias, res = _rand((M, K), cuda), _rand((N, K), cuda), _rand((N,), cuda), _rand((M, N), cuda)
    out = res.clone()
    G.gemm(a, w, out=out, residual=out, bias=bias)          # in place over the residual
    _check(out, a, w.t(), bias.float() + res.float())
    a3, w3 = _rand((4, M, K), cuda), _rand((2, N, K), cuda)
    out3 = G.gemm(a3, w3, b_batch_div=2)
    raise_if_device_error(cuda)
    for i in range(4):
        _check(out3[i], a3[i], w3[i // 2].t())


@pytest.mark.parametrize("T,N,K", [(8, 64, 64), (317, 3072, 2048), (100, 136, 72), (1024, 768, 768)])
def test_weight_gradient_norm(cuda, T, N, K):
    from opake_b200.ops import gemm as G
    from opake_b200.ops._lib import raise_if_device_error

    dy, x = _rand((T, N), cuda, 0.1), _rand((T, K), cuda)
    ss = torch.zeros(1, dtype=torch.float64, device=cuda)
    out = G.linear_wgrad(dy, x, sumsq=ss)
    raise_if_device_error(cuda)
    _check(out, dy.t(), x)
    want = out.double().pow(2).sum().item()
    assert abs(ss.item() - want) <= want * 264 * 2.0 ** -24      # 256 squares and a shuffle tree in fp32


@pytest.mark.parametrize("T,F,D", [(128, 512, 256), (300, 200, 1032), (317, 1408, 512), (100, 64, 72)])
def test_gated_epilogues(cuda, T, F, D):
    from opake_b200.ops import gemm as G
    from opake_b200.ops._lib import raise_if_device_error

    x, w = _rand((T, D), cuda), _rand((2 * F, D), cuda, D ** -0.5)
    act = torch.empty(T, F, dtype=torch.bfloat16, device=cuda)
    raw = G.gemm(x, w, epilogue=G.EPI_SWIGLU, act=act)
    _check(raw, x, w.t())
    g, u = raw.double()[:, 0::2], raw.double()[:, 1::2]
    want = torch.nn.functional.silu(g) * u
    assert bool(((act.double() - want).abs() <= want.abs() * 2.0 ** -7 + 1e-30).all())
    dy, wd = _rand((T, D), cuda), _rand((D, F), cuda, D ** -0.5)
    out = torch.empty_like(raw)
    G.swiglu_dgrad(dy, wd, raw, out=out)
    raise_if_device_error(cuda)
    dact, sg = dy.double() @ wd.double(), torch.sigmoid(g)
    ref = torch.stack([dact * u * sg * (1 + g * (1 - sg)), dact * g * sg], dim=-1).reshape(T, 2 * F)
    # d(act) is rounded to bf16 before the activation's derivative, the result once more: two roundings
    assert bool(((out.double() - ref).abs() <= ref.abs() * 2.0 ** -7 + 2e-3).all())
