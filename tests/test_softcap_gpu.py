"""Soft-capped logits in the epilogue of the fused linear cross-entropy."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [30.0, 50.0, 7.3, 1e35, 1e-6])
@pytest.mark.parametrize("parts", [1, 2])
def test_cap_is_divided_by(cuda, cap, parts):
    """One column and a one-hot reduction: the epilogue's running maximum is cap * tanh(z / cap) of a known z, bit for bit (the
    product with a 1 / cap rounded to 24 bits is off by an ulp of the quotient for many of them)."""
    from opake_b200.ops import gemm as G
    from opake_b200.ops._lib import raise_if_device_error

    T = 4096
    z = torch.linspace(-120, 120, T, device=cuda).to(torch.bfloat16)
    z[:4] = torch.tensor([float("inf"), float("-inf"), 3e38, 1e-38], device=cuda).to(torch.bfloat16)
    x = torch.zeros(T, 8, device=cuda, dtype=torch.bfloat16)
    x[:, 0] = z
    w = torch.zeros(1, 8, device=cuda, dtype=torch.bfloat16)
    w[0, 0] = 1.0
    tiles = G.lce_tiles(1, parts=parts)
    pmax, psum = (torch.empty(T, tiles, device=cuda) for _ in range(2))
    tgt, labels = torch.empty(T, device=cuda), torch.zeros(T, dtype=torch.int32, device=cuda)
    G.gemm(x, w, epilogue=G.EPI_LCE_FWD, labels=labels, pmax=pmax, psum=psum, tgt=tgt, softcap=cap)
    raise_if_device_error(cuda)
    c = torch.full((T,), cap, device=cuda)           # a tensor: dividing by a Python number multiplies with its reciprocal
    want = c * torch.tanh(z.float() / c)
    assert torch.equal(tgt, want) and torch.equal(pmax.max(1).values, want)
