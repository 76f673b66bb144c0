"""Several examples of an accumulation group in one pass through the model: every example as in a pass of its own."""
from dataclasses import replace

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,H,KV", [(64, 4, 4), (64, 8, 2), (128, 4, 2)])
@pytest.mark.parametrize("T", [1, 63, 128, 129, 300])
def test_attention_of_several_sequences(cuda, hd, H, KV, T):
    """Bits of one launch per sequence; a neighbour's infinities stay where they are; nothing behind the last row is written."""
    from opake_b200.ops.flash import flash_bwd, flash_fwd
    from opake_b200.ops._lib import raise_if_device_error

    n, cols = 3, (H + 2 * KV) * hd
    torch.manual_seed(T)
    qkv = torch.randn(n * T + 128, cols, device=cuda).to(torch.bfloat16)
    dout = torch.randn(n * T, H * hd, device=cuda).to(torch.bfloat16)
    qkv[2 * T : 3 * T] = float("inf")
    out = torch.full((n * T + 128, H * hd), 3.0, device=cuda, dtype=torch.bfloat16)
    dqkv = torch.full((n * T + 128, cols), 5.0, device=cuda, dtype=torch.bfloat16)
    _, lse = flash_fwd(qkv[: n * T], H, KV, hd, out=out[: n * T], n_seq=n)
    flash_bwd(dout, qkv[: n * T], out[: n * T], lse, H, KV, hd, dqkv[: n * T], n_seq=n)
    raise_if_device_error(cuda)
    assert bool((out[n * T :] == 3.0).all()) and bool((dqkv[n * T :] == 5.0).all())
    for j in range(2):
        r = slice(j * T, (j + 1) * T)
        o, l = flash_fwd(qkv[r], H, KV, hd)
        d = torch.empty_like(qkv[r])
        flash_bwd(dout[r], qkv[r], o, l, H, KV, hd, d)
        assert torch.equal(out[r], o) and torch.equal(lse[j * H : (j + 1) * H], l) and torch.equal(dqkv[r], d)


def _model(name):
    from opake_b200.models.config import gpt2_small, tiny_llama

    return {"llama": tiny_llama(), "tied": tiny_llama(tie_embeddings=True, qk_norm="head"), "wide norm": tiny_llama(qk_norm=True, qkv_bias=True),
            "geglu": tiny_llama(act="geglu"), "experts": tiny_llama(n_experts=8, top_k=2, expert_ffn=64, qk_norm=True),
            "gpt2": replace(gpt2_small(), vocab_size=515, d_model=192, n_layers=2, n_heads=3, n_kv_heads=3, ffn=768, max_seq=320)}[name]


@pytest.mark.parametrize("name", ["llama", "tied", "wide norm", "geglu", "gpt2", "experts"])
@pytest.mark.parametrize("T,graph", [(33, True), (128, False), (300, True)])
def test_steps_equal_those_of_single_examples(cuda, name, T, graph, monkeypatch):
    """Groups of three, joined in twos, whole and partial: losses, norms, gradients and updates. RMSNorm models to the bit;
    LayerNorm and bias gradients are added by fp32 atomics, in an order that changes from run to run: 1e-2 is the bf16 noise that
    a flipped last bit grows to."""
    from opake_b200.parallel import engine as E

    cfg = replace(_model(name), max_seq=max(320, T))
    exact = name != "gpt2" and name != "wide norm"
    runs = []
    for joined in (2, 1):
        monkeypatch.setattr(E, "_JOIN_VALUES", joined * T * cfg.d_model)
        eng = E.ShardedDPEngine(cfg, E.EngineConfig(logical_batch=4, noise_multiplier=0.1, accumulate_group=3, use_cuda_graph=graph, lr=1e-3), cuda)
        assert eng._joined(T) == joined
        gen, out = torch.Generator().manual_seed(0), []
        for B in (7, 1, 4):
            # no token twice in an example: the rows of a repeated one are added by fp32 atomics as well
            tok = torch.rand(B, cfg.vocab_size, generator=gen).argsort(1)[:, :T].to(torch.int32).contiguous().pin_memory()
            lab = torch.roll(tok, -1, 1).clone()
            lab[:, : T // 4] = -100
            loss = eng.step(tok, lab)
            n = B % 3 or 3
            full = [eng.layout.views(t) for t in (eng.params, eng.m, eng.v)]          # without the gaps between the tensors
            out.append([loss.clone(), *[t.clone() for views in (*eng.runtime.gs[:n], *full) for t in views.values()],
                        *[t.clone() for t in eng.runtime.norms[:n]], eng.runtime.clip_count.clone()])
            eng.runtime.logits(tok[0].to(cuda))           # a workspace of its own for one sequence
        runs.append(out)
    for step, (a, b) in enumerate(zip(*runs)):
        assert abs(a[0].item() - b[0].item()) <= 1e-5 * abs(b[0].item()) + (0 if exact else 0.02 * step)
        for x, y in zip(a[1:], b[1:]):
            if exact:
                assert torch.equal(x, y)
            elif step == 0:                                 # later steps start from parameters that differ already
                x, y = x.double(), y.double()
                assert (x - y).norm() <= 1e-2 * y.norm() + 1e-12


@pytest.mark.parametrize("batch,N", [(1, 256), (3, 256), (8, 384), (9, 256)])      # sums kept per warp, and added per tile beyond eight
def test_norms_of_several_gradients_in_one_launch(cuda, batch, N):
    from opake_b200.ops import gemm as G

    T, Kd = 70, 136
    dy = torch.randn(batch, T, N, device=cuda).to(torch.bfloat16)
    x = torch.randn(batch, T, Kd, device=cuda).to(torch.bfloat16)
    dy[batch - 1] = 0
    sums = torch.zeros(batch, dtype=torch.float64, device=cuda)
    out = torch.empty(batch, N * Kd + 64, device=cuda, dtype=torch.bfloat16)[:, : N * Kd].unflatten(1, (N, Kd))
    G.linear_wgrad(dy, x, out=out, sumsq=sums)
    for j in range(batch):
        one = torch.zeros(1, dtype=torch.float64, device=cuda)
        assert torch.equal(G.linear_wgrad(dy[j], x[j], sumsq=one), out[j])
        assert abs(one.item() - sums[j].item()) <= 1e-12 * one.item()


@pytest.mark.parametrize("E,k,examples,T", [(8, 2, 2, 33), (64, 8, 4, 200), (3, 1, 3, 1), (128, 4, 2, 65), (64, 8, 1, 1025),
                                                (4, 2, 3, 3001)])
def test_routing_plan_of_several_examples(cuda, E, k, examples, T):
    """Rows sorted by expert, then example, in order; parts of whole 64-row blocks (empty ones too), segments of whole tiles; a
    plan for the first example alone in the same buffers."""
    from opake_b200.ops import kernels as K

    plan = K.MoePlan(examples * T, E, k, cuda, examples=examples)
    idx = torch.randint(0, max(1, E - 1), (examples * T, k), dtype=torch.int32)          # the last expert gets nothing
    idx[::7, 0] = E                                                                       # dropped
    for n in (examples, 1):
        p = plan.part(n) if n < examples else plan
        p.build(idx[: n * T].to(cuda))
        unit, off, flat = (64 if n > 1 else 128), 0, idx[: n * T].reshape(-1).tolist()
        src, dest = torch.full((p.R,), -1), torch.full((len(flat),), -1)
        gk, tiles = torch.zeros(n, E, 2), torch.full((p.R // 128,), -1)
        for e in range(E):
            start = off
            for j in range(n):
                rows = [i for i in range(j * T * k, (j + 1) * T * k) if flat[i] == e]
                for r, i in enumerate(rows):
                    src[off + r], dest[i] = i, off + r
                padded = max(unit, -(-len(rows) // unit) * unit)
                gk[j, e] = torch.tensor([off, padded // 64])
                off += padded
            off = -(-off // 128) * 128
            tiles[start // 128 : off // 128] = e
        assert torch.equal(p.src_entry.cpu().long(), src) and torch.equal(p.dest.cpu().long().reshape(-1), dest)
        assert torch.equal(p.group_k.cpu().float().reshape(n, E, 2), gk) and torch.equal(p.tile_group.cpu().long(), tiles)
