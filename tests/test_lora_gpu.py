"""LoRA operators on the device against the composed formulas."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _proj(dev, n, k, r=16, s=2.0):
    bf = torch.bfloat16
    return (torch.randn(n, k, device=dev).mul(k ** -0.5).to(bf), torch.randn(r, k, device=dev).mul(k ** -0.5).to(bf),
            torch.randn(n, r, device=dev).mul(0.02).to(bf), s)


def test_gated_mlp_of_unequal_widths(cuda):
    """Widths that do not broadcast are refused, a single `up` column broadcasts."""
    from opake_b200.patches.kernels import lora_mlp

    x = torch.randn(256, 64, device=cuda).to(torch.bfloat16)
    gate, down = _proj(cuda, 128, 64), _proj(cuda, 64, 128)
    with pytest.raises(RuntimeError):
        lora_mlp(x, gate, _proj(cuda, 64, 64), down)
    up = _proj(cuda, 1, 64)
    wide = (up[0].expand(128, 64).contiguous(), up[1], up[2].expand(128, 16).contiguous(), up[3])
    out = lora_mlp(x, gate, up, down)
    assert out.shape == (256, 64)
    want = lora_mlp(x, gate, wide, down).float()
    # the single column comes from another matrix product (at most two bf16 roundings apart)
    assert float((out.float() - want).norm() / want.norm()) < 2.0 ** -7


@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_gated_activation_has_the_bits_of_the_formula(cuda, act):
    from opake_b200.patches.kernels import lora

    # all gate values of a normal distribution's range and the extremes, against random up and gradient values
    g = torch.randn(1 << 22, device=cuda).mul(4).to(torch.bfloat16)
    g[:8] = torch.tensor([0.0, -0.0, 88.0, -88.0, 120.0, -120.0, 1e-30, -1e-30], device=cuda).to(torch.bfloat16)
    u, dh = (torch.randn(1 << 22, device=cuda).to(torch.bfloat16) for _ in range(2))
    got = [lora._act_fwd(g, u, act), *lora._act_bwd(dh, g, u, act)]
    native, lora._native_act = lora._native_act, lambda *a: False
    try:
        want = [lora._act_fwd(g, u, act), *lora._act_bwd(dh, g, u, act)]
    finally:
        lora._native_act = native
    for a, b in zip(got, want):
        assert torch.equal(a, b), int((a != b).sum())


@pytest.mark.parametrize("rows,k,n,r,s", [(128, 64, 72, 8, 2.0), (640, 256, 512, 16, 0.7), (2048, 512, 256, 32, 1.0)])
def test_adapted_projection_rounds_like_the_formula(cuda, rows, k, n, r, s):
    """``round(x W^T) + round(s round(xa B^T))`` in bf16, forward and input gradient, also onto an earlier gradient."""
    from opake_b200.patches.kernels import lora

    torch.manual_seed(0)
    x, dy, dx0 = (torch.randn(rows, w, device=cuda).to(torch.bfloat16) for w in (k, n, k))
    W, A, B, _ = _proj(cuda, n, k, r)
    xa, dyB = lora._mm(x, A), lora._mm_nn(dy, B)
    assert torch.equal(lora._adapted(x, W, xa, B, s), lora._mm(x, W) + s * lora._mm(xa, B))
    assert torch.equal(lora._adapted_nn(dy, W, dyB, A, s), lora._mm_nn(dy, W) + s * lora._mm_nn(dyB, A))
    want = dx0 + lora._mm_nn(dy, W) + s * lora._mm_nn(dyB, A)
    assert torch.equal(lora._adapted_nn(dy, W, dyB, A, s, dx0.clone()), want)
