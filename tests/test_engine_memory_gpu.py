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
