"""Buffers of the one-rank engine over steps of different lengths: what graphs read stays, what is optional gives way."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(cuda, cfg=None, **kw):
    from opake_b200.models.config import tiny_llama
    from opake_b200.parallel.engine import EngineConfig, ShardedDPEngine

    return ShardedDPEngine(cfg or tiny_llama(), EngineConfig(**{**dict(logical_batch=4, noise_multiplier=0.1, accumulate_group=3, lr=1e-3), **kw}), cuda)


def _batch(cfg, B, T, seed):
    gen = torch.Generator().manual_seed(seed)
    # no token twice in an example: the rows of a repeated one are added by fp32 atomics
    tok = torch.rand(B, cfg.vocab_size, generator=gen).argsort(1)[:, :T].to(torch.int32).contiguous().pin_memory()
    lab = torch.roll(tok, -1, 1).clone()
    lab[:, -1] = -100
    return tok, lab


def _same(a, b):
    for x, y in ((a.params, b.params), (a.m, b.m), (a.v, b.v)):
        for p, q in zip(a.layout.views(x).values(), b.layout.views(y).values()):       # without the gaps between the tensors
            assert torch.equal(p, q)


def test_sequences_longer_than_the_rotary_table(cuda):
    """A step, a sequence beyond max_seq, the step's graphs again."""
    a, b = _engine(cuda), _engine(cuda)
    cfg = a.model_cfg
    for i in range(3):
        batch = _batch(cfg, 4, 64, i)
        la, lb = a.step(*batch), b.step(*batch)
        assert torch.equal(la, lb)
        a.runtime.logits(_batch(cfg, 1, (i + 2) * cfg.max_seq, i)[0][0].to(cuda))
        junk = [torch.full((1 << k,), float("nan"), device=cuda) for k in range(8, 20)]         # what was given back is taken again
        del junk
    _same(a, b)


def _kept_logits(eng):
    """Bytes of the distinct buffers in which workspaces leave logits."""
    zs = {ws["z"].untyped_storage().data_ptr(): ws["z"].untyped_storage().nbytes() for ws in eng.runtime._ws.values() if ws.get("z") is not None}
    return sum(zs.values())


@pytest.mark.parametrize("lengths", [(100, 90, 75, 61, 50, 41, 33), (33, 41, 50, 61, 75, 90, 100)])
def test_stored_logits_of_all_lengths_share_their_memory(cuda, lengths, monkeypatch):
    """Steps of many lengths, each twice (captured, replayed): at most four times what the longest needs, within the limit where memory is
    short, and the bits of an engine without stored logits."""
    from opake_b200.models.decoder import DecoderRuntime
    from opake_b200.ops import _lib, gemm as G

    a, b, c = _engine(cuda), _engine(cuda), _engine(cuda)
    vocab = a.model_cfg.vocab_size
    one = 4 * G.lce_logits_floats(3 * max(lengths), vocab)         # three examples go through the model together
    steps = [_batch(a.model_cfg, 4, T, T + i) for i in range(2) for T in lengths]
    for batch in steps:
        a.step(*batch)
    assert 0 < _kept_logits(a) <= 4 * one
    with monkeypatch.context() as m:
        m.setattr(_lib, "free_bytes", lambda device, plenty=None: 4 * one // 2)
        for batch in steps:
            b.step(*batch)
    assert 0 < _kept_logits(b) <= one // 2
    monkeypatch.setattr(DecoderRuntime, "_logits_buffer", lambda self, ws: None)
    for batch in steps:
        c.step(*batch)
    _same(a, c)
    _same(b, c)
