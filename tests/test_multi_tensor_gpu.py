"""Multi-tensor kernels of the functional API against the leaf-by-leaf formulas that they replace."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tree(cuda, dtypes=(torch.float32, torch.bfloat16)):
    """Leaf sizes around the kernels' chunks (4, 1024, 2048, 4096 elements), a scalar, an empty leaf, a misaligned one; more
    leaves than one launch takes."""
    sizes = [(1,), (3, 5), (8,), (1023,), (1024,), (1025,), (2048, 3), (4097,), (0, 4), ()] + [(7, k) for k in range(1, 45)]
    out = {}
    for i, s in enumerate(sizes):
        t = torch.randn(s, device=cuda, dtype=torch.float32)
        out[f"l{i:03d}"] = t.to(dtypes[i % len(dtypes)])
    out["odd"] = torch.randn(4001, device=cuda)[1:].to(dtypes[0])
    out["shifted"] = torch.randn(2001, device=cuda, dtype=torch.float32)[1:]
    return out


def _off(monkeypatch):
    from opake_b200.ops import multi_tensor as MT

    monkeypatch.setattr(MT, "usable", lambda *a: False)


@pytest.mark.parametrize("correct", [False, True])
def test_optimizer_chain_matches_the_leafwise_formulas(cuda, monkeypatch, correct):
    from opake_b200.engine.types import NoisedPytree
    from opake_b200.ops import _lib
    from opake_b200.optimizers import adamw, apply_updates

    params, grads = _tree(cuda), _tree(cuda, (torch.float32,))
    results = []
    for fused in (True, False):
        if not fused:
            _off(monkeypatch)
        opt = adamw(1e-2, eps=1e-6, weight_decay=0.1, noise_bias_correction=correct)
        p, st, n0 = params, opt.init(params), _lib.LAUNCHES[0]
        for k in range(3):
            g = {q: t * (k + 1) for q, t in grads.items()}
            u, st = opt.update(NoisedPytree(g, 1.0, 0.3), st, params=p)
            p = apply_updates(p, u)
        assert (_lib.LAUNCHES[0] > n0) == fused
        results.append((p, st.moment.mu, st.moment.nu, u))
    for which, (a, b) in enumerate(zip(*results)):
        for q in a:
            assert a[q].dtype == b[q].dtype
            # the same correctly rounded operations in the same order: the same bits. Nothing looser would do for the bias
            # correction, which amplifies an ulp of v_hat by v_hat / (v_hat - phi), without a bound near phi.
            assert torch.equal(a[q], b[q]), (which, q)


def test_noise_is_the_leafwise_noise(cuda, monkeypatch):
    from opake_b200.dpsgd.noise import add_gaussian_noise_tree
    from opake_b200.engine.random import key

    tree = _tree(cuda)
    a = add_gaussian_noise_tree(tree, 0.37, key(5))
    same = add_gaussian_noise_tree(tree, 0.0, key(5))
    assert all(same[q] is tree[q] for q in tree)
    _off(monkeypatch)
    b = add_gaussian_noise_tree(tree, 0.37, key(5))
    for q in tree:
        assert a[q].dtype == b[q].dtype and torch.equal(a[q], b[q]), q


@pytest.mark.parametrize("B", [1, 3, 64])
@pytest.mark.parametrize("clip", [0.0, 0.5, 1e9, float("inf")])
def test_clip_and_sum(cuda, B, clip):
    from opake_b200.engine.clipping.streaming import stream_clip_and_sum
    from opake_b200.engine.clipping import numerics as N
    from opake_b200.ops.clip_sum import fused_clip_sum

    leaves = [torch.randn(B, *t.shape, device=cuda).to(t.dtype) for t in _tree(cuda).values()]
    leaves[0][0] = float("nan")
    leaves[3][B - 1, 5] = float("inf")
    leaves[5][0] = 0
    sums, norms, mask, post = fused_clip_sum(leaves, clip, with_postsq=True)
    ref, _, rn, rm, rp = stream_clip_and_sum([N.sanitize(l) for l in leaves], clip, with_postsq=True)
    assert bool(((norms - rn).abs() <= rn * 1e-12).all()) and torch.equal(mask, rm)
    for s, r, l in zip(sums, ref, leaves):
        # the factors agree up to the order of an fp64 sum: a stored bf16 value may round the other way
        tol = 2.0 ** -8 if l.dtype == torch.bfloat16 else 2.0 ** -22 * B
        assert bool(((s - r).abs() <= tol * N.sanitize(l).float().abs().sum(0) * (min(clip, 1.0)) + 1e-30).all())
    assert bool(((post - rp).abs() <= rp * 1e-3 + 1e-30).all())
    if clip == 0.5:
        assert bool((post <= clip).all())
    # micro-batches: added to the earlier sums, scaled once
    if B > 1:
        first, *_ = fused_clip_sum([l[:1] for l in leaves], clip)
        both, *_ = fused_clip_sum([l[1:] for l in leaves], clip, prev=first, scale=0.25)
        rest, *_ = fused_clip_sum([l[1:] for l in leaves], clip)
        for f, r, b in zip(first, rest, both):
            assert torch.equal((f + r) * 0.25, b)


def test_watched_tensors_keep_the_torch_formulas(cuda):
    from opake_b200.ops import multi_tensor as MT
    from opake_b200.optimizers import apply_updates

    p, u = {"w": torch.randn(8, device=cuda)}, {"w": torch.randn(8, device=cuda)}
    assert MT.usable([p["w"]], [u["w"]])
    assert not MT.usable([p["w"].t().expand(2, 8)]) and not MT.usable([p["w"].double()]) and not MT.usable([p["w"]], [u["w"][:4]])
    w = p["w"].clone().requires_grad_()
    assert not MT.usable([w])
    out = apply_updates({"w": w}, u)["w"]
    assert out.requires_grad                                      # autograd still sees the addition
    batched = torch.func.vmap(lambda a, b: apply_updates({"w": a}, {"w": b})["w"])(p["w"].view(2, 4), u["w"].view(2, 4))
    assert torch.equal(batched.view(8), p["w"] + u["w"])


def test_rope_of_a_batch(cuda):
    from opake_b200.ops.kernels import rope_table
    from opake_b200.patches.kernels import opake_rope_qk

    T, H, hd = 37, 3, 32
    table = rope_table(T, hd, device=cuda)
    x = torch.randn(5, T, H * hd + 16, device=cuda).to(torch.bfloat16)
    one = torch.stack([opake_rope_qk(x[b], table, H, hd) for b in range(5)])
    assert torch.equal(torch.func.vmap(lambda t: opake_rope_qk(t, table, H, hd))(x), one)
    nested = torch.func.vmap(torch.func.vmap(lambda t: opake_rope_qk(t, table, H, hd)))(x[:4].view(2, 2, T, -1))
    assert torch.equal(nested.view(4, T, -1), one[:4])


def test_noise_of_a_huge_standard_deviation(cuda):
    """Beyond the fp32 range the leaf-by-leaf formula gives infinities; so does the kernel."""
    from opake_b200.dpsgd.noise import add_gaussian_noise_tree
    from opake_b200.engine.random import key

    tree = {"a": torch.zeros(1000, device=cuda), "b": torch.ones(33, device=cuda, dtype=torch.bfloat16)}
    got = add_gaussian_noise_tree(tree, 1e39, key(0))
    ref = add_gaussian_noise_tree({**tree, "c": torch.zeros(4, device=cuda, dtype=torch.float64)}, 1e39, key(0))     # leaf by leaf
    for n in tree:
        assert torch.equal(got[n], ref[n]) and bool(got[n].isinf().all())


def test_earlier_sums_of_any_strides(cuda):
    from opake_b200.ops.clip_sum import fused_clip_sum

    leaves = [torch.randn(3, 40, 24, device=cuda), torch.randn(3, 7, device=cuda).to(torch.bfloat16)]
    prev = [torch.randn(24, 40, device=cuda).t(), torch.randn(7, device=cuda)]
    got = fused_clip_sum(leaves, 1.0, prev=prev, scale=0.5)[0]
    want = fused_clip_sum(leaves, 1.0, prev=[p.clone(memory_format=torch.contiguous_format) for p in prev], scale=0.5)[0]
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_micro_batches_on_either_side_of_the_kernel_limit(cuda):
    """65,540 examples go through the portable path, the last 3 through the kernel: equal to one portable pass."""
    from opake_b200 import patches
    from opake_b200.dpsgd.clipping import clipped_grad

    patches.apply_runtime_patches(compat=False)
    p = {"w": torch.randn(3, 5, device=cuda)}
    x = torch.randn(65543, 5, device=cuda)
    loss = lambda q, xe: ((xe @ q["w"].t()) ** 2).sum()
    sums = []
    for micro in (65540, 65543):
        fn, st = clipped_grad(loss, clipping_norm=1.0, normalize_by=65543.0, microbatch_size=micro)
        sums.append(fn(p, x, state=st)[0].pytree["w"])
    # fp32 sums of 65,543 terms of at most 1 in another order
    assert float((sums[0] - sums[1]).abs().max()) <= 65543 ** 0.5 * 2.0 ** -23
