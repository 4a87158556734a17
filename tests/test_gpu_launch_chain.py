"""Chains of overlapped launches: a kernel may start while the one before it drains and waits for it before it touches global
memory.  Every chain gives the same bytes with a synchronisation behind each call, one call after the other, on a second
stream, and replayed from a graph -- several times over changing inputs, so that a kernel that read too early would meet the
values of the pass before."""
import pytest
import torch

from util import need_lib

pytestmark = pytest.mark.gpu


def _mx_chain(g, gen, M):
    """quantise, re-tile (which lets its successor start before its own wait), GEMM; twice, as in a feed-forward."""
    K, F = 128, 256
    mx = lambda n, k: (lambda q, s: (q, g.mx_scales_to_tiled(s, k)))(*g.mxfp8_quantize((torch.randn(n, k, generator=gen) * k ** -0.5).half().cuda()))
    (wg, sg), (wu, su), (wd, sd) = mx(F, K), mx(F, K), mx(K, F)
    x = torch.zeros(M, K, dtype=torch.float16, device="cuda")

    def run(sync):
        q, s = g.mxfp8_quantize(x); sync()
        t = g.mx_scales_to_tiled(s, K); sync()
        h = g.dual_gemm_mxfp8_silu(q, t, wg, wu, sg, su); sync()
        q2, s2 = g.mxfp8_quantize(h); sync()
        t2 = g.mx_scales_to_tiled(s2, F); sync()
        y = g.gemm_mxfp8(q2, t2, wd, sd); sync()
        return h, y
    return x, run


def _cell_chain(g, gen, B):
    """The low-rank cell over time: each step (which lets its successor start before its own wait) writes the h that the next
    down-projection reads, and the c that the next step reads and writes."""
    T, H, R = 12, 256, 64
    f8 = lambda *s: ((torch.rand(*s, generator=gen) * 2 - 1) * 100).to(torch.float8_e4m3fn).cuda()
    f16 = lambda *s: (torch.randn(*s, generator=gen) * 0.3).half().cuda()
    dn, up_hh, up_ih = f8(R, H), f16(4 * H, R), f16(4 * H, R)
    b = (torch.randn(4 * H, generator=gen) * 0.1).cuda()
    sdn, sx = torch.full((1,), 1e-2, device="cuda"), torch.full((B,), 1 / 448.0, device="cuda")
    x = torch.zeros(T * B, R, dtype=torch.float16, device="cuda")
    h, c = torch.zeros(T + 1, B, H, dtype=torch.uint8, device="cuda"), torch.zeros(B, H, device="cuda")

    def run(sync):
        h.zero_()
        c.zero_()
        for t in range(T):
            hh = g.fp8_down_proj(h[t].view(torch.float8_e4m3fn), sx, dn, sdn); sync()
            g.factored_lstm_step(h[t + 1], c, hh, up_hh, b, x[t * B:(t + 1) * B], up_ih, None); sync()
        return h.clone(), c.clone()
    return x, run


@pytest.mark.parametrize("chain,size", [(_mx_chain, 77), (_mx_chain, 20001), (_cell_chain, 33), (_cell_chain, 256)])
def test_chain_gives_the_bytes_of_synchronised_calls(chain, size):
    g = need_lib()
    gen = torch.Generator().manual_seed(size)
    x, run = chain(g, gen, size)
    inputs = [torch.randn(x.shape, generator=gen).half().cuda() for _ in range(3)]
    want = []
    for v in inputs:
        x.copy_(v)
        want.append([t.clone() for t in run(torch.cuda.synchronize)])
    same = lambda got, ref: all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(got, ref))
    nothing = lambda: None
    for v, ref in zip(inputs, want):
        x.copy_(v)
        assert same(run(nothing), ref), "one call after the other"
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for v, ref in zip(inputs, want):
            x.copy_(v)
            assert same(run(nothing), ref), "on a second stream"
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run(nothing)
    for _ in range(3):
        for v, ref in zip(inputs, want):
            x.copy_(v)
            graph.replay()
            assert same(out, ref), "replayed"
    assert g.device_status()[0] == 0
