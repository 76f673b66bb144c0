"""Fused linear cross-entropy whose forward pass leaves its logits for the backward pass."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(shape, dev, std=1.0):
    return (torch.randn(shape, device=dev) * std).to(torch.bfloat16)


@pytest.mark.parametrize("rows", [1, 31, 33, 257, 600])        # 32-row blocks, the single-CTA and the two-CTA product
@pytest.mark.parametrize("vocab", [8, 255, 257, 4999])         # 32-column blocks, ragged and odd row pitches, several column tiles
@pytest.mark.parametrize("cap", [0.0, 30.0])
def test_gradient_from_stored_logits_has_the_bits_of_the_second_product(cuda, rows, vocab, cap):
    from opake_b200.ops import gemm as G, kernels as K
    from opake_b200.ops._lib import raise_if_device_error

    torch.manual_seed(rows * 7 + vocab)
    D, alpha = 136, 0.7
    h, w = _rand((rows, D), cuda), _rand((vocab, D), cuda, 0.4)
    labels = torch.randint(0, vocab, (rows,), device=cuda, dtype=torch.int32)
    labels[::5] = -100
    tiles = G.lce_tiles(vocab, parts=2 if cap else 1)
    pmax, psum = (torch.empty(rows, tiles, device=cuda) for _ in range(2))
    tgt, z = torch.zeros(rows, device=cuda), torch.full((G.lce_logits_floats(rows, vocab),), float("nan"), device=cuda)
    G.gemm(h, w, epilogue=G.EPI_LCE_FWD, labels=labels, pmax=pmax, psum=psum, tgt=tgt, alpha=alpha, softcap=cap, z=z)
    lse, _ = K.lce_finalize(pmax, psum, tgt, labels)
    coef = (labels >= 0).float() * torch.rand(rows, device=cuda)
    pitch = (vocab + 7) // 8 * 8 + 8
    out = torch.full((2, rows, pitch), 7.0, device=cuda, dtype=torch.bfloat16)
    want = G.gemm(h, w, out=out[0, :, :vocab], epilogue=G.EPI_LCE_BWD, labels=labels, lse=lse, coef=coef, alpha=alpha, softcap=cap)
    got = G.lce_grad(z, labels, lse, coef, out[1, :, :vocab], cap)
    raise_if_device_error(cuda)
    assert torch.equal(got, want) and bool((out[:, :, vocab:] == 7.0).all())


@pytest.mark.parametrize("cap", [0.0, 30.0])
def test_loss_gradients_do_not_depend_on_kept_logits(cuda, cap, monkeypatch):
    """Autograd, vmap(grad), a vmap over cotangents and saved-tensor hooks: the same bits with and without kept logits."""
    from opake_b200.ops import lce

    torch.manual_seed(0)
    B, T, D, V = 3, 70, 64, 1000
    h, w = _rand((B, T, D), cuda), _rand((V, D), cuda, 0.2)
    lab = torch.randint(0, V, (B, T), device=cuda)
    lab[:, ::4] = -1
    kept = []
    inner = lce._native_fwd
    monkeypatch.setattr(lce, "_native_fwd", lambda *a: (kept.append(r := inner(*a)), r)[1])

    def run():
        nll = lambda hh, ww, ll: lce.linear_cross_entropy(hh, ww, ll, logit_softcapping=cap)
        hr, wr = h[0].clone().requires_grad_(), w.clone().requires_grad_()
        plain = torch.autograd.grad(nll(hr, wr, lab[0]).sum(), (hr, wr))
        per = torch.func.vmap(torch.func.grad(lambda hh, ww, ll: nll(hh, ww, ll).sum(), (0, 1)), (0, None, 0))(h, w, lab)
        _, pull = torch.func.vjp(lambda hh: nll(hh, w, lab[0]), h[0])
        many = torch.func.vmap(pull)(torch.eye(T, device=cuda)[:4])
        with torch.autograd.graph.save_on_cpu():
            hooked = nll(hr, wr, lab[0]).sum()
        return [*plain, *per, many[0], *torch.autograd.grad(hooked, (hr, wr))]

    first = run()
    assert [k[3].numel() > 0 for k in kept] == [True, True, True, False]
    monkeypatch.setattr(lce, "KEEP_BYTES", 0)
    kept.clear()
    second = run()
    assert all(k[3].numel() == 0 for k in kept)
    assert all(torch.equal(a, b) for a, b in zip(first, second))
    with torch.no_grad():
        lce.linear_cross_entropy(h[0], w, lab[0])
    assert kept[-1][3].numel() == 0


def test_losses_that_wait_share_one_limit_and_give_way_to_scarce_memory(cuda, monkeypatch):
    """Several losses before one backward pass (preference pairs, sums of losses) keep no more logits together than one may, none at all
    where memory is short, and the same bits come out; the room is free again when their graphs are gone."""
    from opake_b200.ops import _lib, gemm as G, lce

    torch.manual_seed(1)
    T, D, V = 40, 64, 700
    one = 4 * G.lce_logits_floats(T, V)
    hs, w = [_rand((T, D), cuda) for _ in range(4)], _rand((V, D), cuda, 0.2).requires_grad_()
    lab = torch.randint(0, V, (T,), device=cuda)
    sizes = []
    inner = lce._native_fwd
    monkeypatch.setattr(lce, "_native_fwd", lambda *a: (r := inner(*a), sizes.append(4 * r[3].numel()))[0])

    def run():
        sizes.clear()
        grads = torch.autograd.grad(sum(lce.linear_cross_entropy(h, w, lab).sum() for h in hs), w)
        return grads[0], list(sizes)

    want, all_kept = run()
    assert all_kept == [one] * 4
    monkeypatch.setattr(lce, "KEEP_BYTES", 5 * one // 2)
    for _ in range(2):                                   # the first pass's logits are gone when the second one begins
        got, kept = run()
        assert kept == [one, one, 0, 0] and torch.equal(got, want)
    monkeypatch.setattr(lce, "_UNASKED_BYTES", 0)
    assert run()[1] == [one, one, 0, 0]
    monkeypatch.setattr(_lib, "free_bytes", lambda device, plenty=None: 2 * one)
    got, kept = run()
    assert kept == [0] * 4 and torch.equal(got, want)
