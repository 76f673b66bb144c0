"""The step kernel that adds the last group of per-example gradients itself against the separate accumulation pass."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_group", [0, 1, 2, 3, 8])
@pytest.mark.parametrize("skip", [False, True])
@pytest.mark.parametrize("n,group_len", [(8192, 8192), (4099, 4096), (70_001, 60_000), (6, 4)])
def test_same_bits_as_a_separate_pass(cuda, n_group, skip, n, group_len):
    from opake_b200.ops import kernels as K

    gs = [torch.randn(group_len, device=cuda).to(torch.bfloat16) for _ in range(n_group)]
    scales = [torch.rand(1, device=cuda) for _ in range(n_group)]
    acc = torch.randn(n, device=cuda)
    out = []
    for fused in (False, True):
        a = acc.clone()
        p = torch.linspace(-1, 1, n, device=cuda).to(torch.bfloat16)
        m, v = torch.full((n,), 0.01, device=cuda), torch.full((n,), 0.02, device=cuda)
        extra = {}
        if fused:
            if skip:
                a[:group_len] = float("nan")          # must not be read
            extra = dict(group=gs, group_scales=scales, group_len=group_len, skip_sum=skip)
        else:
            if skip:
                a[:group_len] = 0
            if n_group:
                head = a[:group_len].clone()
                K.clip_accumulate_group(gs, scales, head)
                a[:group_len] = head
        K.dp_step(grad_src=[a.data_ptr()], shard_begin=0, shard_len=n, inv_batch=0.25, sigma=0.01, seed=3, step=1, m=m, v=v, master=None,
                  param_dst=[p.data_ptr()], param_src=p, lr=0.1, beta1=0.9, beta2=0.99, eps=1e-8, weight_decay=0.01, bc1=0.1, bc2=0.01,
                  phi_hat=1e-5, device=cuda, **extra)
        out.append((p, m, v))
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("graph", [False, True])
def test_engine_steps_of_changing_batch_sizes(cuda, graph):
    """Whole, partial and empty last groups in turn (groups of two): equal to an engine that adds every group in its own pass."""
    from opake_b200.models.config import tiny_llama
    from opake_b200.parallel.engine import EngineConfig, ShardedDPEngine

    cfg = tiny_llama()
    engines = []
    for fused in (True, False):
        e = ShardedDPEngine(cfg, EngineConfig(logical_batch=4, noise_multiplier=0.1, accumulate_group=2, use_cuda_graph=graph), cuda)
        e._fuse_last_group = fused
        engines.append(e)
    gen = torch.Generator().manual_seed(0)
    for B in (4, 1, 0, 5, 2, 3):
        tok = torch.randint(0, cfg.vocab_size, (B, 64), dtype=torch.int32, generator=gen).pin_memory()
        lab = torch.roll(tok, -1, 1).clone()
        for e in engines:
            e.step(tok, lab) if B else e.apply_update()
    a, b = engines
    assert torch.equal(a.params, b.params) and torch.equal(a.m, b.m) and torch.equal(a.v, b.v)


@pytest.mark.parametrize("tied", [False, True])
@pytest.mark.parametrize("graph", [False, True])
def test_sums_that_a_caller_fills_are_applied(cuda, graph, tied):
    """`acc` is zero between steps, and what a caller adds to it is part of the next update, with or without a step in between:
    equal to an engine that runs every pass from its first step on."""
    from dataclasses import replace

    from opake_b200.models.config import tiny_llama
    from opake_b200.parallel.engine import EngineConfig, ShardedDPEngine

    cfg = replace(tiny_llama(), tie_embeddings=tied)
    engines = []
    for fused in (True, False):
        e = ShardedDPEngine(cfg, EngineConfig(logical_batch=4, noise_multiplier=0.1, accumulate_group=2, use_cuda_graph=graph), cuda)
        e._fuse_last_group = fused
        engines.append(e)
    gen = torch.Generator().manual_seed(0)
    add = [torch.randn(engines[0].layout.total, generator=torch.Generator().manual_seed(i)).to(cuda) for i in range(2)]

    def step(B):
        tok = torch.randint(0, cfg.vocab_size, (B, 64), dtype=torch.int32, generator=gen).pin_memory()
        for e in engines:
            e.step(tok, torch.roll(tok, -1, 1).clone())

    def same():
        a, b = engines
        assert torch.equal(a.params, b.params) and torch.equal(a.m, b.m) and torch.equal(a.v, b.v)

    step(5)
    same()
    before = engines[0].m.clone()
    for e in engines:
        assert not bool(e.acc.any())
        e.acc.copy_(add[0])
        e.apply_update()
        assert not bool(e.acc.any())
    same()
    assert float((engines[0].m - 0.9 * before).norm()) > 0.02 * float(add[0].norm()) / 4        # the sums were applied, not noise alone
    for e in engines:
        e.acc.add_(add[1])
    step(3)
    same()
    step(2)
    same()


def test_sums_seen_by_an_update_that_looks_at_them(cuda):
    """A subclass that reads the sums before they are applied sees all groups of the step."""
    from opake_b200.models.config import tiny_llama
    from opake_b200.parallel.engine import EngineConfig, ShardedDPEngine

    cfg = tiny_llama()
    seen = {}

    class Looking(ShardedDPEngine):
        def apply_update(self):
            seen.setdefault(self.tag, []).append(self.acc.clone())
            super().apply_update()

    gen = torch.Generator().manual_seed(0)
    batches = [torch.randint(0, cfg.vocab_size, (B, 64), dtype=torch.int32, generator=gen).pin_memory() for B in (3, 1, 4)]
    for tag, fused in (("a", True), ("b", False)):
        e = Looking(cfg, EngineConfig(logical_batch=4, noise_multiplier=0.1, accumulate_group=2), cuda)
        e.tag, e._fuse_last_group = tag, fused
        for tok in batches:
            e.step(tok, torch.roll(tok, -1, 1).clone())
    for x, y in zip(seen["a"], seen["b"]):
        assert bool(x.any()) and torch.equal(x, y)


def test_step_after_an_update_that_failed(cuda):
    """The groups of a step whose update raised stay in the sums, as they do in separate passes."""
    from opake_b200.models.config import tiny_llama
    from opake_b200.parallel.engine import EngineConfig, ShardedDPEngine

    cfg = tiny_llama()
    gen = torch.Generator().manual_seed(0)
    batches = [torch.randint(0, cfg.vocab_size, (B, 64), dtype=torch.int32, generator=gen).pin_memory() for B in (3, 1, 4)]
    engines = []
    for fused in (True, False):
        e = ShardedDPEngine(cfg, EngineConfig(logical_batch=4, noise_multiplier=0.1, accumulate_group=2), cuda)
        e._fuse_last_group = fused
        engines.append(e)
        update = e.apply_update
        for i, tok in enumerate(batches):
            def fail():
                raise OSError("interrupted")

            e.apply_update = fail if i == 0 else update
            try:
                e.step(tok, torch.roll(tok, -1, 1).clone())
            except OSError:
                assert i == 0
    a, b = engines
    assert torch.equal(a.params, b.params) and torch.equal(a.m, b.m)


@pytest.mark.parametrize("n_group,group_len", [(0, 0), (2, 4096), (3, 7000)])
@pytest.mark.parametrize("noise", ["independent", "blt 2", "blt 6", "toeplitz 1", "toeplitz 5"])
@pytest.mark.parametrize("sgd,master", [(False, False), (False, True), (True, False)])
def test_vectors_of_eight_and_of_four_give_the_same_bits(cuda, n_group, group_len, noise, sgd, master):
    """One shard whose arrays start on 32-byte boundaries against shards that start at 4, 12, ... (16 bytes), ragged at the end."""
    from opake_b200.ops import kernels as K

    n = 8008                                      # rows of correlation state are whole vectors
    gs = [torch.randn(n, device=cuda).to(torch.bfloat16) for _ in range(n_group)]
    scales = [torch.rand(1, device=cuda) for _ in range(n_group)]
    acc, start = torch.randn(n, device=cuda), torch.randn(n, device=cuda)
    kind, rows = noise.split()[0], int(noise.split()[-1]) if " " in noise else 0
    state = torch.randn(rows, n, device=cuda)
    coef = torch.rand(rows + 1, device=cuda) + 0.5
    out = []
    for cuts in ([0, n], [0, 4, 12, 4100, n]):
        p = start.to(torch.bfloat16)
        full = dict(m=torch.full((n,), 0.01, device=cuda), v=torch.full((n,), 0.02, device=cuda), master=start.clone(), state=state.clone())
        for a, b in zip(cuts, cuts[1:]):
            part = {k: t[..., a:b].clone() for k, t in full.items()}          # own allocations: the shard's state starts aligned
            if len(cuts) > 2:                                                 # ... and here 16 bytes after such a boundary
                part = {k: torch.empty(t.numel() + 4, device=cuda)[4:].view(t.shape).copy_(t) for k, t in part.items()}
            corr = {}
            if kind == "blt":
                corr = dict(blt_state=part["state"], blt_decay=coef[1:] / 2, blt_scale=coef[1:] / 8)
            elif kind == "toeplitz":
                corr = dict(toep_state=part["state"], toep_coef=coef, toep_pos=rows - 1)
            K.dp_step(grad_src=[acc.data_ptr()], shard_begin=a, shard_len=b - a, inv_batch=0.25, sigma=0.01, seed=3, step=1,
                      m=None if sgd else part["m"], v=None if sgd else part["v"], master=part["master"] if master else None,
                      param_dst=[p.data_ptr()], param_src=p, lr=0.1, beta1=0.9, beta2=0.99, eps=1e-8, weight_decay=0.01, bc1=0.1,
                      bc2=0.01, phi_hat=1e-5, device=cuda, sgd_mode=sgd, group=gs, group_scales=scales, group_len=group_len, **corr)
            for k, t in full.items():
                t[..., a:b] = part[k]
        out.append((p, *full.values()))
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n_group,group_len", [(0, 0), (2, 4096), (3, 7000)])
@pytest.mark.parametrize("noise", ["independent", "blt 4", "toeplitz 3"])
def test_vectors_of_eight_and_of_four_with_master_weights_under_sgd(cuda, n_group, group_len, noise):
    test_vectors_of_eight_and_of_four_give_the_same_bits(cuda, n_group, group_len, noise, True, True)
