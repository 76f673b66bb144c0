"""Column sums and weight gradients of one and of several examples: the edges of the loops that load eight rows ahead."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 8, 57, 63, 64, 65, 129, 1500])
@pytest.mark.parametrize("N", [8, 256, 264, 7])
@pytest.mark.parametrize("examples", [1, 3])
def test_column_sums(cuda, T, N, examples):
    """fp32 sums of T values in any order: at most T roundings of the sum of magnitudes each; nothing beside the columns is written."""
    from opake_b200.ops import kernels as K

    torch.manual_seed(T + N)
    dy = torch.randn(examples * T, N, device=cuda).to(torch.bfloat16)
    out = torch.full((examples, N + 8 - N % 4), 2.0, device=cuda)
    out[:, :N] = 0.5
    K.colsum_(dy, out[0, :N] if examples == 1 else out[:, :N])
    x = dy.double().view(examples, T, N)
    slack = (T + 1) * 2.0**-24 * (x.abs().sum(1) + 0.5)
    assert ((out[:, :N].double() - 0.5 - x.sum(1)).abs() <= slack).all() and bool((out[:, N:] == 2.0).all())


@pytest.mark.parametrize("T", [1, 63, 64, 65, 296, 311])           # rows of partial sums: up to 296 per example
@pytest.mark.parametrize("D", [8, 264, 4104])
def test_weight_gradient_of_several_examples_has_the_bits_of_single_ones(cuda, T, D):
    from opake_b200.ops import kernels as K

    torch.manual_seed(T + D)
    n = 3
    x, dy = (torch.randn(n * T, D, device=cuda).to(torch.bfloat16) for _ in range(2))
    w = torch.randn(D, device=cuda).to(torch.bfloat16)
    y, rstd = K.rmsnorm_fwd(x, w)
    copy = torch.empty_like(x)
    y2, rstd2 = K.rmsnorm_fwd(x, w, copy=copy)
    assert torch.equal(y, y2) and torch.equal(rstd, rstd2) and torch.equal(copy, x)
    dw = torch.zeros(n, D, device=cuda)
    dx = K.rmsnorm_bwd(dy, x, w, rstd, dw=dw)
    for j in range(n):
        r = slice(j * T, (j + 1) * T)
        one = torch.zeros(D, device=cuda)
        assert torch.equal(K.rmsnorm_bwd(dy[r], x[r], w, rstd[r], dw=one), dx[r]) and torch.equal(one, dw[j])


@pytest.mark.parametrize("n", [1, 7, 8, 2048, 100003])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_squared_sums_of_several_buffers(cuda, n, dtype):
    """Eight squares in fp32, then fp64: the same sum alone and in a batch; 8 * 2^-24 of it from the exact one."""
    from opake_b200.ops import kernels as K

    torch.manual_seed(n)
    pitch = (n + 7) // 8 * 8 + 8
    x = torch.randn(3, pitch, device=cuda).to(dtype)[:, :n]
    sums = torch.zeros(3, dtype=torch.float64, device=cuda)
    K.sumsq_(x, sums)
    for j in range(3):
        one = torch.zeros(1, dtype=torch.float64, device=cuda)
        K.sumsq_(x[j], one)
        exact = x[j].double().square().sum()
        assert abs(one.item() - sums[j].item()) <= 1e-12 * one.item() and abs(one.item() - exact.item()) <= 64 * 2.0**-24 * exact.item()
