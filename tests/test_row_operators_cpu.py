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


def test_cross_entropy_gradient_of_padded_rows(monkeypatch):
    """The kernel writes the gradient with the row pitch of the logits: the buffer has to have that pitch too."""
    from opake_b200.ops import kernels as K

    seen = {}

    class Lib:
        @staticmethod
        def opk_cross_entropy_bwd(*a):
            seen["pitch"] = a[8]
            return 0

    monkeypatch.setattr(K, "_L", lambda: Lib)
    monkeypatch.setattr(K, "_chk", lambda *a: None)
    monkeypatch.setattr(K, "_s", lambda t: None)
    for logits in (torch.zeros(4, 16)[:, :11], torch.zeros(4, 11)):
        d = K.cross_entropy_bwd(logits, torch.zeros(4, dtype=torch.int32), torch.zeros(4), torch.zeros(4))
        assert d.shape == logits.shape and d.stride(0) == seen["pitch"] == logits.stride(0)
        assert d.untyped_storage().nbytes() >= 4 * (3 * logits.stride(0) + 11)
