"""Host side of the patched row operators, no device needed."""
import torch


def test_cross_entropy_keeps_its_own_labels(monkeypatch):
    """The labels that the backward pass reads are a copy: a caller may refill an int32 label buffer in between."""
    from opake_b200.ops import kernels as K
    from opake_b200.patches.kernels.functions import _CE

    monkeypatch.setattr(K, "cross_entropy_fwd", lambda z, lab, scale, softcap: (torch.zeros(z.shape[0]), torch.zeros(z.shape[0])))
    for dtype in (torch.int32, torch.int64):
        for labels in (torch.arange(6, dtype=dtype), torch.arange(12, dtype=dtype)[::2], torch.ones(1, dtype=dtype).expand(6)):
            kept = _CE.forward(torch.zeros(6, 8), labels, 1.0, 0.0)[2]
            assert kept.dtype == torch.int32 and kept.is_contiguous() and torch.equal(kept, labels.int())
            assert kept.untyped_storage().data_ptr() != labels.untyped_storage().data_ptr()
