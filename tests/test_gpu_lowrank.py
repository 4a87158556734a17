"""GPU parity of the one-launch low-rank input projection (R = 64 and 128): x_down stays on chip, column tiles of a row block are
shared out among CTAs.  Its two products exist as calls of their own, which must give the same bytes where the bias is zero; a row
of zeros must give the bias; an output inside a wider buffer must leave the other columns alone."""
import pytest
import torch

from util import assert_bitexact, f16_equal_up_to_signed_zero, need_lib

pytestmark = pytest.mark.gpu


def make(M, C, R, N):
    gen = torch.Generator(device="cuda").manual_seed(M + C + R + N)
    rnd = lambda *s: torch.rand(*s, generator=gen, device="cuda") * 2 - 1
    x, dn = (rnd(M, C) * 448).to(torch.float8_e4m3fn), (rnd(R, C) * 448).to(torch.float8_e4m3fn)
    sx, sdn = rnd(M).abs() * 1e-3 + 1e-4, rnd(1).abs() * 1e-3 + 1e-4
    return x, sx, dn, sdn, rnd(N, R).half(), rnd(N)


# one row; ragged rows, K blocks and column tiles; every CTA one share, some two; whole rounds and a shared last one; one column tile
@pytest.mark.parametrize("M,C,R,N", [(1, 16, 64, 64), (127, 256, 128, 1024), (129, 1024, 128, 4096), (9001, 272, 128, 1544), (19589, 512, 64, 1536),
                                     (40001, 1040, 128, 520), (38000, 128, 64, 200)])
def test_is_the_two_products(M, C, R, N):
    g = need_lib()
    x, sx, dn, sdn, up, bias = make(M, C, R, N)
    zero = torch.zeros_like(bias)
    xd = g.fp8_down_proj(x, sx, dn, sdn)
    buf = torch.full((M + 1, N + 24), 90.0, dtype=torch.float16, device="cuda")
    g.fp8_factored_gemm(x, sx, dn, sdn, up, zero, out=buf[:M, :N])
    assert bool((buf[:, N:] == 90).all()) and bool((buf[M:] == 90).all())
    assert f16_equal_up_to_signed_zero(buf[:M, :N].contiguous(), g.gemm_f16(xd, up)) == 0
    # with the bias: f16(acc + b), one rounding.  |acc| is known to fp16, so the sum to half an ulp of either
    out = g.fp8_factored_gemm(x, sx, dn, sdn, up, bias)
    acc = buf[:M, :N].float()
    assert bool(((out.float() - (acc + bias)).abs() <= 2 ** -11 * (acc.abs() + out.float().abs()) + 2 ** -24).all())
    lo = M // 2
    x[lo].zero_()
    out = g.fp8_factored_gemm(x, sx, dn, sdn, up, bias)
    assert_bitexact(out[lo], bias.half())
    assert g.device_status()[0] == 0


def test_same_bytes_on_a_capped_grid():
    """On all SMs the last round's row blocks are shared; on one and on 37 CTAs the rounds and shares are others."""
    g = need_lib()
    a = make(5000, 384, 128, 1032)
    ref = g.fp8_factored_gemm(*a)
    try:
        for cap in (1, 37):
            assert g.lib().gsb200_set_sm_limit(cap) == 0
            assert_bitexact(g.fp8_factored_gemm(*a), ref, f"{cap} CTAs")
    finally:
        assert g.lib().gsb200_set_sm_limit(0) == 0
    assert g.device_status()[0] == 0
