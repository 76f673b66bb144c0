"""Kernels that start under the tail of their predecessor (programmatic dependent launch) on two streams that exchange work."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [40, 300, 1024])
@pytest.mark.parametrize("mode", ["eager", "graph"])
def test_chain_on_two_streams_has_the_bits_of_single_kernels(cuda, T, mode):
    """A layer's forward and backward chain (row kernels, narrow / single / paired products, attention forward and backward) on one
    stream, products over its intermediates on another, which read buffers that the chain overwrites in the next round: every
    result equals that of the same calls with the device idle in between."""
    from opake_b200.ops import gemm as G, kernels as K
    from opake_b200.ops._lib import raise_if_device_error
    from opake_b200.ops.flash import flash_bwd, flash_fwd

    torch.manual_seed(0)
    bf = torch.bfloat16
    D, H, KV, hd, F = 512, 8, 2, 64, 1408
    rnd = lambda *s: (torch.randn(*s, device=cuda) * s[-1] ** -0.5).to(bf)
    wqkv, wo, wgu, wd, nw = rnd((H + 2 * KV) * hd, D), rnd(D, H * hd), rnd(2 * F, D), rnd(D, F), torch.ones(D, device=cuda, dtype=bf)
    table = K.rope_table(T, hd, device=cuda)
    x0 = torch.randn(T, D, device=cuda).to(bf)
    side = torch.cuda.Stream()
    sums = [torch.zeros(1, dtype=torch.float64, device=cuda) for _ in range(3)]
    e = lambda *s: torch.empty(*s, dtype=bf, device=cuda)
    b = dict(x=x0.clone(), xn=e(T, D), qkv=e(T, (H + 2 * KV) * hd), dqkv=e(T, (H + 2 * KV) * hd), mid=e(T, D), gu=e(T, 2 * F), act=e(T, F), dgu=e(T, 2 * F),
             out=e(T, D), dx=e(T, D), gqkv=e((H + 2 * KV) * hd, D), ggu=e(2 * F, D), gd=e(D, F))

    def one_round(wait):
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        main.wait_stream(side)                              # the products of the round before still read these buffers
        xn, _ = K.rmsnorm_fwd(b["x"], nw, out=b["xn"])
        wait()
        G.gemm(xn, wqkv, out=b["qkv"])
        wait()
        K.rope_(b["qkv"], table, H + KV, hd)
        wait()
        att, lse = flash_fwd(b["qkv"], H, KV, hd)
        wait()
        G.gemm(att, wo, out=b["mid"], residual=b["x"])
        wait()
        G.gemm(b["mid"], wgu, out=b["gu"], epilogue=G.EPI_SWIGLU, act=b["act"])
        wait()
        G.gemm(b["act"], wd, out=b["out"], residual=b["mid"])
        wait()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            G.linear_wgrad(b["out"], b["act"], out=b["gd"], sumsq=sums[0])
        wait()
        G.swiglu_dgrad(b["out"], wd, b["gu"], out=b["dgu"])
        wait()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            G.linear_wgrad(b["dgu"], b["mid"], out=b["ggu"], sumsq=sums[1])
        wait()
        G.gemm(b["dgu"], wgu, b_mn=True, out=b["dx"])
        wait()
        datt = G.gemm(b["dx"], wo, b_mn=True)
        wait()
        flash_bwd(datt, b["qkv"], att, lse, H, KV, hd, b["dqkv"])
        wait()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            G.linear_wgrad(b["dqkv"], xn, out=b["gqkv"], sumsq=sums[2])
        wait()
        y, _ = K.rmsnorm_fwd(b["out"], nw)
        wait()
        b["x"].copy_(y)                                     # input of the next round
        main.wait_stream(side)

    def run(rounds, wait):
        b["x"].copy_(x0)
        for s in sums:
            s.zero_()
        torch.cuda.synchronize()
        for _ in range(rounds):
            one_round(wait)
        torch.cuda.synchronize()
        raise_if_device_error(cuda)
        return {k: v.clone() for k, v in b.items()} | {f"s{i}": s.clone() for i, s in enumerate(sums)}

    want = run(6, torch.cuda.synchronize)
    if mode == "graph":
        run(1, lambda: None)
        b["x"].copy_(x0)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(6):
                one_round(lambda: None)
    for _ in range(8):
        if mode == "eager":
            got = run(6, lambda: None)
        else:
            b["x"].copy_(x0)
            for s in sums:
                s.zero_()
            g.replay()
            torch.cuda.synchronize()
            got = {k: v.clone() for k, v in b.items()} | {f"s{i}": s.clone() for i, s in enumerate(sums)}
        for k, v in want.items():
            if k[0] == "s":      # one atomic per CTA in fp64: the order of about 100 additions is free
                assert abs(float(got[k] - v)) <= float(v) * 128 * 2.0 ** -53, k
            else:
                assert torch.equal(got[k], v), k
