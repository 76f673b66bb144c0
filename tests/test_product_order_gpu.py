"""One order of summation for every product: a row's result does not depend on how many rows are processed with it, although
the number of rows decides which GEMM kernel and tile width run."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = (1, 31, 40, 128, 129, 317, 640)       # few rows: narrow tiles; 1024 rows (the comparison): wider tiles, pairs of SMs


def _rand(shape, dev, scale=1.0):
    return (torch.randn(shape, device=dev, dtype=torch.float32) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("layout", ["nt", "nn"])
@pytest.mark.parametrize("N,K", [(64, 2048), (512, 8192), (2048, 2048), (768, 3072), (8192, 2048)])
def test_rows_of_plain_products(cuda, N, K, layout):
    from opake_b200.ops import gemm as G
    from opake_b200.ops._lib import raise_if_device_error

    x, w, res = _rand((1024, K), cuda), _rand((N, K) if layout == "nt" else (K, N), cuda), _rand((1024, N), cuda)
    whole = G.gemm(x, w, b_mn=layout == "nn", residual=res, out=torch.empty_like(res))
    for M in ROWS:
        part = G.gemm(x[:M], w, b_mn=layout == "nn", residual=res[:M], out=torch.empty(M, N, dtype=x.dtype, device=cuda))
        assert torch.equal(part, whole[:M]), M
    raise_if_device_error(cuda)


@pytest.mark.parametrize("F,D", [(512, 2048), (8192, 2048), (1408, 4096)])
def test_rows_of_gated_products(cuda, F, D):
    from opake_b200.ops import gemm as G
    from opake_b200.ops._lib import raise_if_device_error

    x, w, dy, wd = _rand((1024, D), cuda), _rand((2 * F, D), cuda, D ** -0.5), _rand((1024, D), cuda), _rand((D, F), cuda, D ** -0.5)
    act = torch.empty(1024, F, dtype=x.dtype, device=cuda)
    gu = G.gemm(x, w, epilogue=G.EPI_SWIGLU, act=act)
    dgu = G.swiglu_dgrad(dy, wd, gu, out=torch.empty_like(gu))
    for M in ROWS:
        a = torch.empty(M, F, dtype=x.dtype, device=cuda)
        g = G.gemm(x[:M], w, epilogue=G.EPI_SWIGLU, act=a)
        assert torch.equal(g, gu[:M]) and torch.equal(a, act[:M]), M
        assert torch.equal(G.swiglu_dgrad(dy[:M], wd, gu[:M], out=torch.empty_like(g)), dgu[:M]), M
    raise_if_device_error(cuda)


@pytest.mark.parametrize("N,K", [(64, 2048), (768, 3072), (2304, 768)])
def test_weight_gradient_with_and_without_norm(cuda, N, K):
    """Products over the rows: the weight gradient has the same bits with the norm (persistent kernels) and without."""
    from opake_b200.ops import gemm as G

    for T in (64, 317, 1024):
        dy, x = _rand((T, N), cuda), _rand((T, K), cuda)
        ss = torch.zeros(1, dtype=torch.float64, device=cuda)
        assert torch.equal(G.linear_wgrad(dy, x), G.linear_wgrad(dy, x, sumsq=ss))


@pytest.mark.parametrize("T,D,V", [(129, 512, 8192), (65, 256, 4000)])
def test_functional_gradients_do_not_depend_on_the_micro_batch(cuda, T, D, V):
    from torch.func import grad, vmap

    from opake_b200.ops.lce import opake_linear_cross_entropy_loss as lce

    h, w = _rand((8, T, D), cuda), _rand((V, D), cuda, 0.02)
    lab = torch.randint(0, V, (8, T), device=cuda)
    f = vmap(grad(lambda a, b, l: lce(a, b, l), argnums=(0, 1)), in_dims=(0, None, 0))
    dh, dw = f(h, w, lab)
    for lo, hi in ((0, 1), (1, 4), (4, 8)):
        ph, pw = f(h[lo:hi], w, lab[lo:hi])
        assert torch.equal(ph, dh[lo:hi]) and torch.equal(pw, dw[lo:hi])


@pytest.mark.parametrize("M,N,K", [(634, 2048, 8192), (600, 1992, 8200), (2048, 768, 6408), (3000, 760, 3072), (1021, 2048, 12296)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_pair_tiles_of_128_columns(cuda, M, N, K, b_mn):
    """Sizes that leave 256-wide pairs idle over a long reduction, with and without bias and residual: the bits of the single-CTA
    kernel (every product adds in one order), and those within the rounding of bf16 of the exact sum."""
    from opake_b200.ops import gemm as G

    a = torch.randn(M, K, device=cuda).to(torch.bfloat16)
    b = (torch.randn(K, N, device=cuda) if b_mn else torch.randn(N, K, device=cuda)).to(torch.bfloat16)
    r, bias = torch.randn(M, N, device=cuda).to(torch.bfloat16), torch.randn(N, device=cuda).to(torch.bfloat16)
    for kw in ({}, {"bias": bias, "residual": r}):
        out = torch.empty(M, N + 8, device=cuda, dtype=torch.bfloat16)[:, :N] if not kw else torch.empty(M, N, device=cuda, dtype=torch.bfloat16)
        G.gemm(a, b, b_mn=b_mn, out=out, **kw)
        before = G.pair_mode()
        try:
            G.set_pair_mode(False)
            single = G.gemm(a, b, b_mn=b_mn, out=torch.empty(M, N, device=cuda, dtype=torch.bfloat16), **kw)
        finally:
            G.set_pair_mode(before)
        assert torch.equal(out, single)
    exact = a.double() @ (b.double() if b_mn else b.double().t())
    got = G.gemm(a, b, b_mn=b_mn).double()
    bound = a.double().abs() @ (b.double().abs() if b_mn else b.double().abs().t())
    # one rounding to bf16 and K fp32 additions, each at most 2^-24 of the absolute sum
    assert ((got - exact).abs() <= exact.abs() * 2.0 ** -8 + bound * K * 2.0 ** -24).all()


def _norm_by_row_segments(c, width):
    """Squared norm of ``c [N, K]`` with the fp32 partial sums of the product's epilogue: ``width`` columns of a row one after the other
    (the squares of bf16 values are exact), 32 rows by halving; the segments in fp64."""
    N, Kd = c.shape
    sq = torch.zeros((N + 31) // 32 * 32, (Kd + width - 1) // width * width, device=c.device)
    sq[:N, :Kd] = c.float() ** 2
    sq = sq.view(sq.shape[0], -1, width)
    run = torch.zeros_like(sq[..., 0])
    for j in range(width):
        run = run + sq[..., j]
    run = run.view(-1, 32, run.shape[-1])
    while run.shape[1] > 1:
        run = run[:, : run.shape[1] // 2] + run[:, run.shape[1] // 2 :]
    return run.double().sum().item()


@pytest.mark.parametrize("N,K", [(256, 2048), (768, 768), (2304, 768), (2048, 2056), (4104, 2048)])      # one round of tiles, several
@pytest.mark.parametrize("T", [64, 317, 512, 513, 1024])
@pytest.mark.parametrize("batch", [1, 3])
def test_norm_of_a_weight_gradient_is_summed_in_one_way(cuda, N, K, T, batch):
    """Neither the rows of an example nor the examples of a launch choose the partial sums of its norm."""
    from opake_b200.ops import gemm as G
    from opake_b200.ops._lib import raise_if_device_error

    dy, x = _rand((batch, T, N), cuda), _rand((batch, T, K), cuda)
    sums = torch.zeros(batch, dtype=torch.float64, device=cuda)
    out = G.linear_wgrad(dy, x, sumsq=sums) if batch > 1 else G.linear_wgrad(dy[0], x[0], sumsq=sums)[None]
    raise_if_device_error(cuda)
    for j in range(batch):
        want = _norm_by_row_segments(out[j], 256)
        assert abs(sums[j].item() - want) <= 1e-13 * want           # some thousand additions in fp64
