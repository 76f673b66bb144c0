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
