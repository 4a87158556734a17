"""GPU checks of the MXFP8 pieces (parity unpinned: the rule is this library's, see oracle/mx.py).
The activation quantiser is compared bit for bit with the CPU statement of the rule; the fused
SwiGLU->MXFP8 epilogue is held to the error bound of the format against the fp32 reference math."""
import pytest
import torch

import oracle
from util import assert_bitexact, launches, need_lib, rand_scales

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K", [(64, 512), (1000, 2048), (3, 32), (129, 384)])
def test_mx_activation_quantiser_bitexact(M, K):
    g = need_lib()
    gen = torch.Generator().manual_seed(M + K)
    x = (torch.randn(M, K, generator=gen) * torch.logspace(-3, 3, M)[:, None]).half()
    x[0, :32] = 0
    q_ref, s_ref = oracle.mx_block_quantize(x.float())
    q, s = g.mxfp8_quantize(x.cuda())
    assert_bitexact(s, s_ref, "E8M0 scale bytes")
    assert_bitexact(q, q_ref, "E4M3 elements")


@pytest.mark.parametrize("M,N,K", [(256, 2048, 512), (1000, 256, 512), (130, 160, 128)])
def test_dual_silu_mxfp8_output(M, N, K):
    g = need_lib()
    gen = torch.Generator().manual_seed(7 + M + N)
    A, sa = oracle.fp8_quantize_per_token(torch.randn(M, K, generator=gen))
    Wg = ((torch.rand(N, K, generator=gen) * 2 - 1) * 448).to(torch.float8_e4m3fn)
    Wu = ((torch.rand(N, K, generator=gen) * 2 - 1) * 448).to(torch.float8_e4m3fn)
    sbg, sbu = rand_scales(gen, N, 2e-4, 2e-3), rand_scales(gen, N, 2e-4, 2e-3)
    q, s = g.dual_gemm_fp8_silu_mxfp8(A.cuda(), Wg.cuda(), Wu.cuda(), sa.cuda(), sbg.cuda(), sbu.cuda())
    ref = oracle.fp8_dual_silu_ref(A, Wg, Wu, sa, sbg, sbu)
    got = oracle.mx_dequantize(q.cpu(), s.cpu())
    blk_amax = ref.reshape(M, N // 32, 32).abs().amax(-1, keepdim=True).expand(M, N // 32, 32).reshape(M, N)
    err = (got - ref).abs()
    # E4M3 carries 3 mantissa bits; a scaled block maximum in (448, 512) saturates: error <= 12.5 % of the block maximum
    assert bool((err <= 0.13 * blk_amax + 1e-6).all()), float((err / (blk_amax + 1e-12)).max())
    assert float((err / (blk_amax + 1e-12)).mean()) < 0.02
    # scale bytes follow the rule on the reference values except where the block maximum sits at a binade edge
    _, s_ref = oracle.mx_block_quantize(ref)
    assert float((s.cpu() != s_ref).float().mean()) < 0.01
    assert int((s.cpu().int() - s_ref.int()).abs().max()) <= 1
    # fused output == two-step path: the plain SwiGLU kernel's fp16 result dequantises to the same values within fp16 + e4m3 rounding
    h = g.dual_gemm_fp8_silu(A.cuda(), Wg.cuda(), Wu.cuda(), sa.cuda(), sbg.cuda(), sbu.cuda()).cpu().float()
    assert bool(((got - h).abs() <= 0.13 * blk_amax + 1e-3).all())


def tiled_ref(s, K):
    """CPU statement of the 128 x 4 scale tile order."""
    rows = s.shape[0]
    rb, kt = (rows + 127) // 128, K // 128
    out = torch.full((rb * kt * 512,), 127, dtype=torch.uint8)
    r = torch.arange(rows)[:, None]
    b = torch.arange(K // 32)[None, :]
    idx = ((r // 128) * kt + b // 4) * 512 + (r % 32) * 16 + ((r % 128) // 32) * 4 + b % 4
    out[idx.reshape(-1)] = s.reshape(-1)
    return out


def test_scale_retiling():
    g = need_lib()
    gen = torch.Generator().manual_seed(4)
    for rows, K in [(128, 128), (300, 512), (5, 256)]:
        s = torch.randint(0, 255, (rows, K // 32), generator=gen, dtype=torch.uint8)
        got = g.mx_scales_to_tiled(s.cuda(), K)
        assert torch.equal(got.cpu(), tiled_ref(s, K))


def mx_operand(gen, rows, K, spread=True):
    v = torch.randn(rows, K, generator=gen)
    if spread:
        v = v * torch.logspace(-2, 2, K // 32).repeat_interleave(32)[None, :]     # different block magnitudes
    return oracle.mx_block_quantize(v)


# K <= 512 runs the weight-stationary kernel (256-column slices: N % 256 of 0, 128 and other remainders, 3 and 4
# K blocks, ragged M, more row blocks than one group walks), K = 2048 the streaming one
@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (128, 128, 512), (300, 512, 512), (1000, 512, 2048), (64, 96, 256),
                                   (300, 384, 512), (257, 2048, 512), (200, 640, 384), (20000, 256, 512),
                                   (20000, 256, 640), (40000, 128, 1024)])   # streaming form, several tiles per CTA: both pipelines
def test_block_scaled_gemm(M, N, K):
    g = need_lib()
    gen = torch.Generator().manual_seed(M + N + K)
    Aq, As = mx_operand(gen, M, K)
    Wq, Ws = mx_operand(gen, N, K)
    c = g.gemm_mxfp8(Aq.cuda(), g.mx_scales_to_tiled(As.cuda(), K), Wq.cuda(), g.mx_scales_to_tiled(Ws.cuda(), K))
    ref = oracle.mx_gemm_ref(Aq, As, Wq, Ws)
    assert g.device_status()[0] == 0
    from util import assert_close
    assert_close(c, ref.half(), atol=float(ref.abs().max()) * 2 ** -9, rtol=2e-2, what="block-scaled GEMM")


@pytest.mark.parametrize("M,N,K", [(128, 64, 128), (256, 2048, 512), (1000, 192, 512), (300, 320, 512), (129, 2048, 256),
                                   (20000, 128, 384), (700, 256, 1024), (20000, 128, 640)])
def test_block_scaled_dual_silu(M, N, K):
    g = need_lib()
    gen = torch.Generator().manual_seed(3 * M + N + K)
    Aq, As = mx_operand(gen, M, K, spread=False)
    Wg = oracle.mx_block_quantize(torch.randn(N, K, generator=gen) * 0.05)
    Wu = oracle.mx_block_quantize(torch.randn(N, K, generator=gen) * 0.05)
    t = lambda s: g.mx_scales_to_tiled(s.cuda(), K)
    c = g.dual_gemm_mxfp8_silu(Aq.cuda(), t(As), Wg[0].cuda(), Wu[0].cuda(), t(Wg[1]), t(Wu[1]))
    ref = oracle.mx_dual_silu_ref(Aq, As, Wg[0], Wg[1], Wu[0], Wu[1])
    from util import assert_close
    assert_close(c, ref.half(), atol=float(ref.abs().max()) * 2 ** -9, rtol=2e-2, what="block-scaled SwiGLU")


def test_mx_ffn_chain():
    """fp8 SwiGLU emitting MXFP8 -> block-scaled down-projection consuming it (activation scales per 32 K)."""
    g = need_lib()
    gen = torch.Generator().manual_seed(77)
    M, D, F = 512, 512, 1024
    A, sa = oracle.fp8_quantize_per_token(torch.randn(M, D, generator=gen))
    Wg = ((torch.rand(F, D, generator=gen) * 2 - 1) * 448).to(torch.float8_e4m3fn)
    Wu = ((torch.rand(F, D, generator=gen) * 2 - 1) * 448).to(torch.float8_e4m3fn)
    sbg, sbu = rand_scales(gen, F, 2e-4, 2e-3), rand_scales(gen, F, 2e-4, 2e-3)
    Wd = oracle.mx_block_quantize(torch.randn(D, F, generator=gen) * 0.05)
    hq, hs = g.dual_gemm_fp8_silu_mxfp8(A.cuda(), Wg.cuda(), Wu.cuda(), sa.cuda(), sbg.cuda(), sbu.cuda())
    y = g.gemm_mxfp8(hq, g.mx_scales_to_tiled(hs, F), Wd[0].cuda(), g.mx_scales_to_tiled(Wd[1].cuda(), F))
    ref = oracle.mx_gemm_ref(hq.cpu(), hs.cpu(), Wd[0], Wd[1])         # oracle fed with the device's own MXFP8 activations
    from util import assert_close
    assert_close(y, ref.half(), atol=float(ref.abs().max()) * 2 ** -9, rtol=2e-2, what="MX down-projection")


# shapes that take the 256-column tiles (enough tiles, K > 512): column tails with one and with two scale tiles in the last
# tile, ragged rows, K blocks that do not divide the ring, one and several tiles per CTA
@pytest.mark.parametrize("M,N,K", [(9001, 384, 640), (9088, 512, 768), (19000, 480, 640), (37889, 512, 1152), (18945, 512, 2048)])
def test_block_scaled_gemm_256_column_tiles(M, N, K):
    g = need_lib()
    gen = torch.Generator().manual_seed(M + N + K)
    Aq, As = mx_operand(gen, M, K)
    Wq, Ws = mx_operand(gen, N, K)
    c = g.gemm_mxfp8(Aq.cuda(), g.mx_scales_to_tiled(As.cuda(), K), Wq.cuda(), g.mx_scales_to_tiled(Ws.cuda(), K))
    torch.cuda.synchronize()
    assert g.device_status()[0] == 0
    # the same rows in a call small enough for the 128-column tiles: the same sums in the same order, the same bytes
    from util import assert_close
    for lo in (0, 5000, M - 300):
        Ar, Sr = Aq[lo:lo + 300].contiguous(), As[lo:lo + 300].contiguous()
        part = g.gemm_mxfp8(Ar.cuda(), g.mx_scales_to_tiled(Sr.cuda(), K), Wq.cuda(), g.mx_scales_to_tiled(Ws.cuda(), K))
        ref = oracle.mx_gemm_ref(Ar, Sr, Wq, Ws)
        assert_close(c[lo:lo + 300], ref.half(), atol=float(ref.abs().max()) * 2 ** -9, rtol=2e-2, what="256-column tiles")
        assert torch.equal(part, c[lo:lo + 300])


@pytest.mark.parametrize("M,N,K", [(1, 32, 128), (129, 96, 512), (333, 480, 96), (2000, 2048, 512), (700, 160, 384), (20000, 512, 128)])
def test_dual_silu_mxfp8_epilogue_forms_agree(M, N, K):
    """The twelve-warp form (staged boxes, both scales of an item in one store where aligned) against the eight-warp form:
    the same bytes, with N ending inside a 64-column item, odd scale rows and an output that is a slice of a wider buffer."""
    g = need_lib()
    gen = torch.Generator().manual_seed(M + N + K)
    A = (torch.randn(M, K, generator=gen) * 100).clamp(-448, 448).to(torch.float8_e4m3fn).cuda()
    W = [(torch.randn(N, K, generator=gen) * 100).clamp(-448, 448).to(torch.float8_e4m3fn).cuda() for _ in range(2)]
    sa, sg, su = [(1e-4 + 1e-3 * torch.rand(n, generator=gen)).cuda() for n in (M, N, N)]
    res = []
    try:
        for ew in (8, -1):
            assert g.lib().gsb200_set_gemm_variant(ew, -1) == 0
            q = torch.zeros(M, N + 32, dtype=torch.uint8, device="cuda")
            s = torch.zeros(M, N // 32 + 3, dtype=torch.uint8, device="cuda")
            g.dual_gemm_fp8_silu_mxfp8(A, W[0], W[1], sa, sg, su, out=q[:, :N], out_scale=s[:, :N // 32])
            res.append((q, s))
    finally:
        g.lib().gsb200_set_gemm_variant(-1, -1)
    torch.cuda.synchronize()
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    assert int(res[1][0][:, N:].count_nonzero()) == 0 and int(res[1][1][:, N // 32:].count_nonzero()) == 0
    assert g.device_status()[0] == 0


# (which of these the 256-column tiles take on 148 SMs; M = 9001 leaves a row block of 41 rows, M = 3001 one of 57)
FORM_256W = [(True, 9001, 2080, 512, True), (True, 20000, 544, 384, True), (True, 40000, 160, 128, False), (True, 19000, 288, 256, False),
             (False, 9001, 2080, 512, True), (False, 20000, 544, 384, False), (False, 40000, 160, 128, True), (False, 19000, 288, 256, False)]
FORM_256W += [(True, m, n, k, True) for k in (128, 256, 384, 512) for m, n in ((9001, 160), (3001, 544))]
FORM_256W += [(False, m, n, k, True) for k in (128, 256, 384, 512) for m, n in ((9001, 288), (3001, 800))]


@pytest.mark.parametrize("dual,M,N,K,wide", FORM_256W)
def test_block_scaled_weight_stationary_256_column_tiles(dual, M, N, K, wide):
    """Many row blocks run on 256-column weight-stationary tiles where their rounds are cheaper; a slice of two row blocks (one
    round) on 128-column ones.  Rows are independent, so the slices must give the same bytes: ragged last tiles in M and N (half
    of a column tile, one without scale tiles), one to four K blocks through the ring of four."""
    g = need_lib()
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    def mx(n):
        q, s = g.mxfp8_quantize(torch.randn(n, K, generator=gen, device="cuda").half())
        return q, s, g.mx_scales_to_tiled(s, K)
    (a, sa, ta), (w, _, tw), (u, _, tu) = mx(M), mx(N), mx(N)
    run = (lambda x, t: g.dual_gemm_mxfp8_silu(x, t, w, u, tw, tu)) if dual else (lambda x, t: g.gemm_mxfp8(x, t, w, tw))
    got = run(a, ta)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        few, tf = a[:256].contiguous(), g.mx_scales_to_tiled(sa[:256].contiguous(), K)
        assert [("mx_gemm256w" in n) for n, _ in launches(lambda: run(a, ta))] == [wide]
        assert [("mx_gemm256w" in n) for n, _ in launches(lambda: run(few, tf))] == [False]
    for lo in (0, M // 2 // 128 * 128, (M - 1) // 128 * 128 - 128):
        hi = min(M, lo + 256)
        assert_bitexact(got[lo:hi], run(a[lo:hi].contiguous(), g.mx_scales_to_tiled(sa[lo:hi].contiguous(), K)), f"rows {lo}:{hi}")
    assert g.device_status()[0] == 0


@pytest.mark.parametrize("dual,N,M,form", [(False, 18976, 100, "mx_gemm256w"), (False, 18976, 1300, "mx_gemm256_k"), (False, 37888, 1300, "mx_gemm256w"),
                                           (True, 9504, 100, "mx_gemm256w"), (True, 9504, 1300, "mx_gemm_k"), (True, 18944, 1300, "mx_gemm256w")])
def test_block_scaled_gemm_of_many_column_slices(dual, N, M, form):
    """More 128-column slices than SMs: 256-column weight-stationary tiles only where they beat the streaming kernel, which has work
    for every SM.  Either way the bytes are those of the same columns asked for by themselves."""
    g = need_lib()
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are either side of the line for 148 SMs")
    K = 256
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    def mx(n):
        q, s = g.mxfp8_quantize(torch.randn(n, K, generator=gen, device="cuda").half())
        return q, s, g.mx_scales_to_tiled(s, K)
    (a, _, ta), (w, sw, tw), (u, su, tu) = mx(M), mx(N), mx(N)
    out = torch.empty(M, N, dtype=torch.float16, device="cuda")
    run = lambda: g.dual_gemm_mxfp8_silu(a, ta, w, u, tw, tu, out=out) if dual else g.gemm_mxfp8(a, ta, w, tw, out=out)
    run()
    names = [n for n, _ in launches(run)]
    assert len(names) == 1 and form in names[0], names
    for lo in (0, N // 2 // 128 * 128, (N - 1) // 128 * 128):
        hi = min(N, lo + 256)
        part = lambda t: t[lo:hi].contiguous()
        tiled = lambda s: g.mx_scales_to_tiled(part(s), K)
        ref = g.dual_gemm_mxfp8_silu(a, ta, part(w), part(u), tiled(sw), tiled(su)) if dual else g.gemm_mxfp8(a, ta, part(w), tiled(sw))
        assert_bitexact(out[:, lo:hi], ref, f"columns {lo}:{hi}")
    assert g.device_status()[0] == 0


@pytest.mark.parametrize("dual,M,N,K,maps", [(False, 1024, 2048, 512, 3), (True, 1024, 2048, 512, 4), (False, 128, 2048, 512, 3), (True, 128, 2048, 512, 4),
                                             (False, 20000, 512, 1024, 3), (True, 300, 512, 1024, 4)])
def test_a_block_scaled_call_encodes_the_maps_it_uses(dual, M, N, K, maps):
    """On buffers not seen before: one tensor map each for A, a weight and the output, whichever kernel runs."""
    g = need_lib()
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    def mx(n):
        q, s = g.mxfp8_quantize(torch.randn(n, K, generator=gen, device="cuda").half())
        return q, g.mx_scales_to_tiled(s, K)
    (a, ta), (w, tw), (u, tu) = mx(M), mx(N), mx(N)
    out = torch.empty(M, N + 8 * (1 + dual), dtype=torch.float16, device="cuda")[:, :N]       # (a stride of this test's own)
    a, w, u = [torch.empty(t.shape[0], K + 16 * (3 + dual), dtype=t.dtype, device="cuda")[:, :K].copy_(t) for t in (a, w, u)]
    n0 = int(g.lib().gsb200_tensor_map_encodes())
    g.dual_gemm_mxfp8_silu(a, ta, w, u, tw, tu, out=out) if dual else g.gemm_mxfp8(a, ta, w, tw, out=out)
    assert int(g.lib().gsb200_tensor_map_encodes()) - n0 == maps
