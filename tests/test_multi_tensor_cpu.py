"""Host side of the multi-tensor kernels, no device needed."""
import math
import struct

import pytest
import torch

from opake_b200.ops import multi_tensor as MT


@pytest.mark.parametrize("value,want", [(1.5, 1.5), (1e39, math.inf), (-1e39, -math.inf), (math.inf, math.inf), (3.4028235e38, 3.4028234663852886e38),
                                        (1e-50, 0.0)])
def test_scalars_beyond_fp32_pack_as_infinity(value, want):
    """As in the formulas, where a Python number meets an fp32 tensor."""
    (s,) = struct.unpack_from("<f", MT._pack([((torch.zeros(4),), 4, 0, value)]), 6 * 8 + 2 * 8)
    assert s == want
    assert float(torch.ones(1) * value) == want


def test_earlier_sums_reach_the_clip_kernel_contiguous(monkeypatch):
    """The kernel reads the sums of earlier micro-batches by a running index. They come from the portable path when an earlier
    micro-batch was too large for the kernel, with whatever strides its reduction left."""
    from opake_b200.ops import clip_sum

    seen = {}

    def kernel(leaves, clip, guards, outs, *, prev=None, scale=1.0, with_postsq=False):
        seen["prev"] = prev
        return torch.zeros(2, dtype=torch.float64), torch.zeros(2, dtype=torch.bool), None

    monkeypatch.setattr(clip_sum.MT, "clip_and_sum", kernel)
    prev = [torch.arange(15.0).view(5, 3).t(), torch.ones(4)]
    clip_sum.fused_clip_sum([torch.ones(2, 3, 5), torch.ones(2, 4)], 1.0, prev=prev)
    assert all(p.is_contiguous() for p in seen["prev"])
    assert all(torch.equal(p, q) for p, q in zip(seen["prev"], prev))
