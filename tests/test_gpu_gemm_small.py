"""GPU parity of the few-tile GEMM form (tiles of 64 or 128 rows, one per CTA) at the edges of its tiles, its ring and its range.

The persistent kernel, which an override of the variant choice selects, runs the same calls: both must give the same
bytes, and INT8 results must be the exact-accumulator model's.  Outputs lie inside wider buffers, whose other columns
must stay as they were."""
import pytest
import torch

import oracle
from util import assert_bitexact, f16_equal_up_to_signed_zero, launches, need_lib, rand_i8, rand_scales

pytestmark = pytest.mark.gpu

GUARD = 24


def both(call, M, N, dtype=torch.float16):
    """call(out) with the library's choice and with the persistent kernel; returns the two results."""
    g = need_lib()
    outs = []
    for variant in ((-1, -1), (8, 0)):
        buf = torch.full((M + 1, N + GUARD), 0x5A, dtype=torch.uint8).to(torch.uint8).cuda()
        buf = (buf.to(torch.float16) if dtype == torch.float16 else buf.view(dtype))
        before = buf.clone()
        try:
            assert g.lib().gsb200_set_gemm_variant(*variant) == 0
            call(buf[:M, :N])
        finally:
            assert g.lib().gsb200_set_gemm_variant(-1, -1) == 0
        assert_bitexact(buf[:, N:], before[:, N:], "columns past the output")
        assert_bitexact(buf[M:], before[M:], "rows past the output")
        outs.append(buf[:M, :N].clone())
    assert g.device_status()[0] == 0
    assert_bitexact(outs[0], outs[1], "few-tile form against the persistent kernel")
    return outs[0]


def operands(gen, fp8, M, N, K):
    if not fp8:
        return rand_i8(gen, M, K), rand_i8(gen, N, K)
    q = lambda n: ((torch.rand(n, K, generator=gen) * 2 - 1) * 448).to(torch.float8_e4m3fn)
    return q(M), q(N)


# one row; tile edges; a column tile cut after its first part and after 8 columns; a ragged K block; rings that are
# reused (K = 2048 and 3 * 128 with one to three CTAs per SM); the last two take 128-row tiles
SHAPES = [(1, 8, 16), (63, 64, 128), (64, 96, 144), (65, 72, 512), (130, 520, 2048), (777, 1032, 384), (2048, 512, 2048), (3000, 512, 512),
          (1025, 1536, 640), (3601, 520, 384), (4700, 512, 2048)]


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_dequant(fp8, M, N, K):
    g = need_lib()
    gen = torch.Generator().manual_seed(M + 3 * N + 7 * K)
    A, B = operands(gen, fp8, M, N, K)
    sa, sb = rand_scales(gen, M, 5e-3, 5e-2), rand_scales(gen, N)
    Ac, Bc, sac, sbc = A.cuda(), B.cuda(), sa.cuda(), sb.cuda()
    c = both(lambda out: (g.gemm_fp8 if fp8 else g.gemm_i8)(Ac, Bc, sac, sbc, out=out), M, N)
    if not fp8:
        assert f16_equal_up_to_signed_zero(c, oracle.gemm_dequant_exact(A, B, sa, sb)) == 0


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("M,N,K", [(1, 8, 16), (64, 32, 128), (65, 72, 512), (200, 2048, 512), (330, 1000, 2048), (700, 1544, 384), (1001, 2040, 512), (700, 2040, 1024), (570, 2040, 1040)])
def test_swiglu(fp8, M, N, K):
    g = need_lib()
    gen = torch.Generator().manual_seed(M + 5 * N + 7 * K)
    A, G = operands(gen, fp8, M, N, K)
    U = operands(gen, fp8, M, N, K)[1]
    sa, sg, su = rand_scales(gen, M, 5e-3, 5e-2).cuda(), rand_scales(gen, N).cuda() * 1e-2, rand_scales(gen, N).cuda()
    A, G, U = A.cuda(), G.cuda(), U.cuda()
    both(lambda out: (g.dual_gemm_fp8_silu if fp8 else g.dual_gemm_i8_silu)(A, G, U, sa, sg, su, out=out), M, N)


@pytest.mark.parametrize("M,K,kernel", [(700, 1024, "gemm_small"), (700, 1040, "gemm_tcgen05"), (570, 1040, "gemm_small"), (570, 4096, "gemm_small")])
def test_swiglu_few_tile_form_by_k(M, K, kernel):
    """Three 64-row tiles per SM (M = 700) only up to K = 1024, two (M = 570) at any K; the same bytes from either kernel."""
    g = need_lib()
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are either side of the line for 148 SMs")
    gen = torch.Generator().manual_seed(M + K)
    A, G = operands(gen, False, M, 2048, K)
    U = operands(gen, False, M, 2048, K)[1]
    sa, sg, su = rand_scales(gen, M, 5e-3, 5e-2).cuda(), rand_scales(gen, 2048).cuda() * 1e-2, rand_scales(gen, 2048).cuda()
    A, G, U = A.cuda(), G.cuda(), U.cuda()
    both(lambda out: g.dual_gemm_i8_silu(A, G, U, sa, sg, su, out=out), M, 2048)
    out = torch.empty(M, 2048, dtype=torch.float16, device="cuda")
    names = [n for n, _ in launches(lambda: g.dual_gemm_i8_silu(A, G, U, sa, sg, su, out=out))]
    assert len(names) == 1 and kernel in names[0], names


@pytest.mark.parametrize("M,N,K", [(1, 32, 128), (65, 96, 512), (200, 2048, 512), (500, 1056, 2048), (500, 2048, 2048), (590, 1056, 1024)])
def test_swiglu_to_mxfp8(M, N, K):
    g = need_lib()
    gen = torch.Generator().manual_seed(M + 5 * N + 7 * K)
    A, G = operands(gen, True, M, N, K)
    U = operands(gen, True, M, N, K)[1]
    sa, sg, su = rand_scales(gen, M, 5e-3, 5e-2).cuda(), rand_scales(gen, N).cuda() * 1e-2, rand_scales(gen, N).cuda()
    A, G, U = A.cuda(), G.cuda(), U.cuda()
    scales = []

    def call(out):
        s = torch.full((M, N // 32 + 3), 0x5A, dtype=torch.uint8, device="cuda")
        # (an output row stride that is a multiple of 16 bytes is part of the call's contract)
        wide = torch.empty(M, (N + 31) // 16 * 16, dtype=torch.float8_e4m3fn, device="cuda")[:, :N]
        g.dual_gemm_fp8_silu_mxfp8(A, G, U, sa, sg, su, out=wide, out_scale=s[:, :N // 32])
        out.copy_(wide)
        assert bool((s[:, N // 32:] == 0x5A).all())
        scales.append(s)
    both(call, M, N, dtype=torch.float8_e4m3fn)
    assert_bitexact(scales[0], scales[1], "block scales")


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("head_dim,rotary_dim", [(64, 64), (64, 32), (128, 128), (128, 64)])
@pytest.mark.parametrize("M,nhead,K,seqlen,row_offset", [(1, 1, 128, 1, 0), (65, 3, 64, 17, 5), (333, 4, 512, 333, 70000), (600, 4, 2048, 100, 99)])
def test_rotary(fp8, head_dim, rotary_dim, M, nhead, K, seqlen, row_offset):
    g = need_lib()
    N = 3 * nhead * head_dim
    gen = torch.Generator().manual_seed(M + N + K + rotary_dim)
    A, B = operands(gen, fp8, M, N, K)
    sa, sb = rand_scales(gen, M, 5e-3, 5e-2), rand_scales(gen, N)
    sn, cs = oracle.rope_tables(seqlen, rotary_dim // 2, head_dim)
    d = [t.cuda() for t in (A, B, sa, sb, sn, cs)]
    fn = g.gemm_fp8_rotary if fp8 else g.gemm_i8_rotary
    c = both(lambda out: fn(*d, nhead, head_dim, rotary_dim, seqlen, row_offset=row_offset, out=out), M, N)
    if not fp8 and row_offset % seqlen < 2000:
        pad = row_offset % seqlen
        exact = oracle.rotary_exact(torch.cat([torch.zeros(pad, K, dtype=torch.int8), A]), B, torch.cat([torch.ones(pad), sa]), sb, sn, cs,
                                    nhead, head_dim, rotary_dim, seqlen)[pad:]
        assert f16_equal_up_to_signed_zero(c, exact) == 0


def test_scalar_and_absent_scales_and_a_capped_grid():
    """One weight scale for all columns (the down-projections of the low-rank LSTM), and a cap on the SMs that leaves the
    form no room: the persistent kernel answers, with the same bytes."""
    g = need_lib()
    gen = torch.Generator().manual_seed(3)
    M, N, K = 256, 128, 1024
    A, B = operands(gen, True, M, N, K)
    sa, sb = rand_scales(gen, M).cuda(), rand_scales(gen, 1).cuda()
    A, B = A.cuda(), B.cuda()
    c = both(lambda out: out.copy_(g.fp8_down_proj(A, sa, B, sb)), M, N)
    try:
        assert g.lib().gsb200_set_sm_limit(2) == 0
        assert_bitexact(g.fp8_down_proj(A, sa, B, sb), c.contiguous())
    finally:
        assert g.lib().gsb200_set_sm_limit(0) == 0


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("with_a,with_b", [(False, True), (True, False), (False, False)])
@pytest.mark.parametrize("M,N,K", [(65, 72, 144), (3000, 512, 512), (4700, 512, 512)])
def test_null_scales_count_as_one(fp8, with_a, with_b, M, N, K):
    """The C entry points take null for either scale of a plain GEMM: 64-row and 128-row tiles against the persistent kernel, and the
    products against exact sums."""
    g = need_lib()
    gen = torch.Generator().manual_seed(M + N)
    draw = lambda n: torch.randint(-3, 4, (n, K), generator=gen, dtype=torch.int8)
    A, B = draw(M), draw(N)
    sa, sb = rand_scales(gen, M, 0.5, 2.0).cuda(), rand_scales(gen, N, 0.5, 2.0).cuda()
    Ac, Bc = (t.to(torch.float8_e4m3fn).cuda() if fp8 else t.cuda() for t in (A, B))
    entry = g.lib().gsb200_gemm_fp8_f16 if fp8 else g.lib().gsb200_gemm_i8_f16
    stream = torch.cuda.current_stream().cuda_stream

    def call(out):
        assert entry(Ac.data_ptr(), Ac.stride(0), Bc.data_ptr(), Bc.stride(0), out.data_ptr(), out.stride(0), sa.data_ptr() if with_a else None,
                     sb.data_ptr() if with_b else None, M, N, K, 0, stream) == 0
    c = both(call, M, N)
    acc = A.cuda().float() @ B.cuda().float().t()
    assert float(acc.abs().max()) < 2 ** 15                # (whole numbers, exact in fp32)
    ref = acc.double() * (sa.double()[:, None] if with_a else 1) * (sb.double() if with_b else 1)
    # two products in fp32 and one rounding to fp16
    assert bool(((c.double() - ref).abs() <= ref.abs() * (2 ** -11 + 2 ** -22)).all())
