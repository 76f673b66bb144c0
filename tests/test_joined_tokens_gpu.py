"""Several examples in one pass on ordinary text: tokens that repeat, models with biases, a step of one example before the others."""
from dataclasses import replace

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(name):
    from opake_b200.models.config import gpt2_small, tiny_llama

    return {"llama": tiny_llama(), "tied": tiny_llama(tie_embeddings=True), "biases": tiny_llama(qkv_bias=True, qk_norm=True),
            "gpt2": replace(gpt2_small(), vocab_size=515, d_model=192, n_layers=2, n_heads=3, n_kv_heads=3, ffn=768, max_seq=320)}[name]


def _runtime(cfg, cuda, n_slots):
    from opake_b200.models.decoder import DecoderRuntime, init_params_
    from opake_b200.models.flat import build_layout

    layout = build_layout(cfg)
    params = torch.empty(layout.total, dtype=torch.bfloat16, device=cuda)
    init_params_(cfg, params, layout, seed=3)
    return DecoderRuntime(cfg, params, layout=layout, n_slots=n_slots)


@pytest.mark.parametrize("name", ["llama", "tied", "biases", "gpt2"])
@pytest.mark.parametrize("T", [17, 130, 300])
def test_gradients_of_repeated_tokens(cuda, name, T):
    """Matrix gradients to the bit, those of vectors, which are fp32 sums over the rows, by a bf16 step. The rows of a repeated token are added by
    fp32 atomics: within the rounding of any order from the sum in fp64 of the gradients that were added."""
    cfg = replace(_model(name), max_seq=320)
    n, tied = 3, cfg.tie_embeddings
    gen = torch.Generator().manual_seed(T)
    tok = (torch.rand(n, T, generator=gen).pow(4) * 40).to(torch.int32).to(cuda)           # one token fills a third of an example
    lab = torch.roll(tok, -1, 1)
    lab[:, -1] = -100
    both, one = _runtime(cfg, cuda, n), _runtime(cfg, cuda, 1)
    ws = both.workspace(T, n)
    both.example_grad(tok.view(-1), lab.reshape(-1).contiguous(), ws=ws)
    for j in range(n):
        ws1 = one.workspace(T)
        one.sumsqs[0].zero_()
        one.example_grad(tok[j], lab[j].contiguous(), ws=ws1)
        dx = ws["dx"][j * T : (j + 1) * T]
        assert torch.equal(dx, ws1["dx"])
        count = torch.bincount(tok[j].long(), minlength=cfg.vocab_size)[:, None]
        exact, size = (torch.zeros(cfg.vocab_size, cfg.d_model, dtype=torch.float64, device=cuda).index_add_(0, tok[j].long(), v)
                       for v in (dx.double(), dx.double().abs()))
        slack = count * 2.0**-24 * size                              # fp32 sums of `count` terms in any order, at 1 / 2 ulp each
        for got in (ws["embs"][j], ws1["embs"][0]):
            rows = got.rep[:T] == torch.arange(T, device=cuda, dtype=torch.int32)
            ids = tok[j][rows].long()
            assert sorted(ids.tolist()) == sorted(set(tok[j].tolist()))
            assert ((got.gc[:T][rows].double() - exact[ids]).abs() <= slack[ids]).all()
        for key, g in one.gs[0].items():
            x, y = both.gs[j][key], g
            if key == "embed" and not tied:
                continue
            if key == "embed":                                       # bf16 of (bf16 head gradient + the row): a step, where the row differs
                assert ((x.double() - y.double()).abs() <= 2.0**-6 * y.double().abs() + 2 * slack).all()
            elif x.dim() == 1 and name in ("gpt2", "biases"):
                assert (x.double() - y.double()).norm() <= 2.0**-7 * y.double().norm()
            else:
                assert torch.equal(x, y), key
        a, b = both.sumsqs[j].item(), one.sumsqs[0].item()
        assert abs(a - b) <= 1e-3 * b


@pytest.mark.parametrize("name", ["llama", "tied"])
def test_one_example_before_several(cuda, name, monkeypatch):
    """The passes of two and three examples are captured without a warm-up of their own."""
    from opake_b200.parallel import engine as E

    cfg, engines = _model(name), []
    for joined in (True, False):
        monkeypatch.setattr(E, "_JOIN_VALUES", (1 << 23) if joined else 0)
        eng = E.ShardedDPEngine(cfg, E.EngineConfig(logical_batch=4, noise_multiplier=0.1, accumulate_group=3, lr=1e-3), cuda)
        gen = torch.Generator().manual_seed(0)
        for B in (1, 2, 1, 8, 3):
            tok = torch.rand(B, cfg.vocab_size, generator=gen).argsort(1)[:, :61].to(torch.int32).contiguous().pin_memory()
            eng.step(tok, torch.roll(tok, -1, 1).clone())
        engines.append(eng)
    a, b = engines
    for x, y in ((a.params, b.params), (a.m, b.m), (a.v, b.v)):
        for p, q in zip(a.layout.views(x).values(), b.layout.views(y).values()):
            assert torch.equal(p, q)


@pytest.mark.parametrize("graph", [True, False])
def test_losses_are_added_in_the_order_of_the_examples(cuda, graph, monkeypatch):
    """The loss of a step has the bits that the examples one by one give."""
    from opake_b200.parallel import engine as E

    cfg, losses = _model("llama"), []
    for values in (1 << 23, 0):
        monkeypatch.setattr(E, "_JOIN_VALUES", values)
        eng = E.ShardedDPEngine(cfg, E.EngineConfig(logical_batch=4, noise_multiplier=0.1, accumulate_group=5, lr=1e-3, use_cuda_graph=graph), cuda)
        gen = torch.Generator().manual_seed(1)
        for B in (1, 5, 9, 13, 13, 13, 2):
            tok = torch.rand(B, cfg.vocab_size, generator=gen).argsort(1)[:, :77].to(torch.int32).contiguous().pin_memory()
            losses.append(eng.step(tok, torch.roll(tok, -1, 1).clone()).clone())
    half = len(losses) // 2
    assert all(torch.equal(a, b) for a, b in zip(losses[:half], losses[half:]))
