"""Buffers of the one-rank engine over steps of different lengths: what graphs read stays, what is optional gives way."""
import gc

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


@pytest.fixture(autouse=True)
def _no_garbage():
    """A patched method makes a cycle of its engine, whose graphs must not go while another test captures."""
    yield
    gc.collect()


def _scarce(monkeypatch, eng, room):
    """``room`` bytes more for this engine's runtime than torch has handed out now: what the device says and what allocations do."""
    from opake_b200.ops import _lib

    cap, inner = torch.cuda.memory_allocated() + room, eng.runtime._alloc

    def alloc(*shape, dtype, name):
        t = inner(*shape, dtype=dtype, name=name)
        if torch.cuda.memory_allocated() > cap:
            raise torch.cuda.OutOfMemoryError("the test's limit")
        return t

    monkeypatch.setattr(eng.runtime, "_alloc", alloc)
    monkeypatch.setattr(_lib, "free_bytes", lambda device, plenty=None: max(0, cap - torch.cuda.memory_allocated()))


@pytest.mark.parametrize("graph", [True, False])
def test_examples_go_one_by_one_where_several_do_not_fit(cuda, graph, monkeypatch):
    """Whole and partial groups, a step of one example first; the bits of an engine that never takes several."""
    from opake_b200.parallel import engine as E

    a, b = _engine(cuda, use_cuda_graph=graph), _engine(cuda, use_cuda_graph=graph)
    inner = a.runtime._alloc

    def alloc(*shape, dtype, name):
        if name.startswith("workspace[T=144]"):          # three examples of 48 tokens
            raise torch.cuda.OutOfMemoryError("the test's limit")
        return inner(*shape, dtype=dtype, name=name)

    monkeypatch.setattr(a.runtime, "_alloc", alloc)
    steps = [_batch(a.model_cfg, B, 48, B) for B in (1, 7, 4, 2)]
    for batch in steps:
        a.step(*batch)
    monkeypatch.setattr(E, "_JOIN_VALUES", 0)
    for batch in steps:
        b.step(*batch)
    assert a._join_limit == {48: 1} and set(a.runtime._ws) == {(48, 1)}
    _same(a, b)


@pytest.mark.parametrize("experts", [False, True])
def test_what_is_optional_gives_way_to_more_lengths(cuda, experts, monkeypatch):
    """Every length fits one by one; with the sets and logits of the earlier ones it does not. Captured steps, a sequence that is only
    evaluated among them, then the earlier lengths again."""
    from opake_b200.models.config import tiny_llama

    cfg = tiny_llama(n_experts=8, top_k=2, expert_ffn=64) if experts else tiny_llama()
    lengths = (64, 60, 56, 52, 48, 44)
    plain, empty = _engine(cuda, cfg), torch.cuda.memory_allocated()
    probe = _engine(cuda, cfg)
    before = torch.cuda.memory_allocated()
    for T in (*lengths, 70):
        probe.runtime.workspace(T)
    room = torch.cuda.memory_allocated() - before + (1 << 20)         # the scratch of a pass is not in it
    del probe
    assert torch.cuda.memory_allocated() <= empty                     # nothing waits for a garbage collection
    steps = [_batch(cfg, B, T, T + B) for B in (4, 7) for T in lengths]
    tok = _batch(cfg, 1, 70, 0)[0][0].to(cuda)
    for batch in steps:
        plain.step(*batch)
    want = plain.runtime.logits(tok)
    eng = _engine(cuda, cfg)
    with monkeypatch.context() as m:
        _scarce(m, eng, room)
        for batch in steps:
            eng.step(*batch)
        got = eng.runtime.logits(tok)
    assert eng.runtime.lean and all(n == 1 for _, n in eng.runtime._ws) and not eng.runtime._logits
    assert torch.equal(got, want) and ("joined", 64) in eng._warm          # a rank must not warm up again by itself
    _same(eng, plain)


@pytest.mark.parametrize("name", ["llama", "tied", "experts", "biases"])
def test_guard_bands_watch_the_passes_that_steps_take(cuda, name):
    """With guard bands, examples go through the model together as they do without: the same bits, every band intact, and a write behind
    a gradient slot is reported."""
    from opake_b200.models.config import tiny_llama
    from opake_b200.utils import DeviceIntegrityError

    cfg = {"llama": tiny_llama(), "tied": tiny_llama(tie_embeddings=True), "biases": tiny_llama(qkv_bias=True),
           "experts": tiny_llama(n_experts=8, top_k=2, expert_ffn=64)}[name]
    for graph in (False, True):
        a, b = _engine(cuda, cfg, use_cuda_graph=graph, debug_canaries=True), _engine(cuda, cfg, use_cuda_graph=graph)
        for B, T in ((7, 45), (4, 45), (1, 33)):
            batch = _batch(cfg, B, T, B)
            a.step(*batch), b.step(*batch)
        assert a._joined(45) == b._joined(45) == 3 and (45, 3) in a.runtime._ws
        if name != "biases":                                   # whose gradients are added by fp32 atomics
            _same(a, b)
        slot = a.runtime.Gs[1]
        slot.as_strided((1,), (1,), slot.storage_offset() + slot.numel()).zero_()
        with pytest.raises(DeviceIntegrityError, match="grad_slot1: after the buffer"):
            a.step(*batch)
