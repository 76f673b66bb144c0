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
