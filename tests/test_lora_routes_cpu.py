"""Which LoRA calls may take the fused kernels (decided on the host, no device needed)."""
import pytest
import torch

from opake_b200.patches.kernels import lora


class _Cuda:
    """What the route decision looks at, standing in for a CUDA bf16 tensor."""

    is_cuda, dtype = True, torch.bfloat16

    def __init__(self, *shape, address=0):
        self.shape, self._address = torch.Size(shape), address

    def is_contiguous(self):
        return True

    def data_ptr(self):
        return self._address

    def numel(self):
        return self.shape.numel()


def test_gated_activation_kernel_needs_equal_shapes():
    """The kernel reads `up` element by element next to `gate`: a narrower `up` would be read past its end."""
    assert lora._native_act(_Cuda(128, 64), _Cuda(128, 64))
    assert not lora._native_act(_Cuda(128, 64), _Cuda(128, 32))
    assert not lora._native_act(_Cuda(128, 64), _Cuda(128, 1))
    assert not lora._native_act(_Cuda(128, 64), _Cuda(128, 64), _Cuda(64, 64))
    assert not lora._native_act(_Cuda(128, 64), _Cuda(128, 64, address=8))


@pytest.mark.parametrize("up_width", [32, 1])
def test_projections_of_other_widths(up_width):
    """Refused (no broadcast exists) or broadcast, as the plain formula does."""
    torch.manual_seed(0)
    p = lambda n, k: (torch.randn(n, k), torch.randn(4, k), torch.randn(n, 4), 1.0)
    x, gate, up, down = torch.randn(16, 8), p(64, 8), p(up_width, 8), p(8, 64)
    if up_width == 1:
        lin = lambda t, w: t @ w[0].t() + t @ w[1].t() @ w[2].t()
        want = lin(torch.nn.functional.silu(lin(x, gate)) * lin(x, up), down)
        assert torch.allclose(lora.lora_mlp(x, gate, up, down), want, rtol=1e-4, atol=1e-4)
    else:
        with pytest.raises(RuntimeError):
            lora.lora_mlp(x, gate, up, down)
