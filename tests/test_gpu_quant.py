"""GPU parity: per-token quantisers through the C ABI vs the CPU oracle (bit-exact)."""
import pytest
import torch

import oracle
from conftest import load_golden
from util import T, assert_bitexact, need_lib

pytestmark = pytest.mark.gpu


def test_int8_quantiser_golden():
    g = need_lib()
    gold = load_golden("quant_i8")
    x = T(gold["x_f16"]).cuda()
    q, s = g.quantize_tensor(x)
    assert_bitexact(q, T(gold["q"]), "int8 values vs reference golden")
    assert_bitexact(s, T(gold["scale"]), "scales vs reference golden")
    q32, s32 = g.quantize_tensor(x.float())
    assert_bitexact(q32, T(gold["q"]), "fp32-input path")
    assert_bitexact(s32, T(gold["scale"]), "fp32-input path scales")


@pytest.mark.parametrize("M,K", [(16384, 512), (1, 512), (129, 2048), (777, 384), (33, 1024), (5, 8), (64, 4096 + 64)])
def test_int8_quantiser_bitexact(M, K):
    g = need_lib()
    gen = torch.Generator().manual_seed(1001)
    x = torch.randn(M, K, generator=gen).half()
    q_ref, s_ref = oracle.quantize_tensor(x.float())
    q, s = g.quantize_tensor(x.cuda())
    assert_bitexact(q, q_ref, f"int8 [{M},{K}]")
    assert_bitexact(s, s_ref, f"scale [{M},{K}]")


def test_int8_quantiser_strided_and_empty():
    g = need_lib()
    gen = torch.Generator().manual_seed(7)
    big = torch.randn(100, 1024, generator=gen).half().cuda()
    view = big[:, :512]                       # row stride 1024
    q, s = g.quantize_tensor(view)
    q_ref, s_ref = oracle.quantize_tensor(view.cpu().float())
    assert_bitexact(q, q_ref)
    assert_bitexact(s, s_ref)
    q0, s0 = g.quantize_tensor(torch.empty(0, 512, dtype=torch.float16, device="cuda"))
    assert q0.shape == (0, 512) and s0.shape == (0,)


def test_int8_requant_of_swiglu_shaped_activations():
    g = need_lib()
    gen = torch.Generator().manual_seed(3003)
    x = (torch.randn(4096, 2048, generator=gen) * 3).half()
    q_ref, s_ref = oracle.quantize_tensor(x.float())
    q, s = g.quantize_tensor(x.cuda())
    assert_bitexact(q, q_ref)
    assert_bitexact(s, s_ref)


@pytest.mark.parametrize("torch_form", [True, False])
@pytest.mark.parametrize("M,K", [(48, 256), (1000, 512), (130, 2048), (9, 384)])
def test_fp8_quantiser_bitexact(M, K, torch_form):
    g = need_lib()
    gen = torch.Generator().manual_seed(1005)
    x = torch.randn(M, K, generator=gen).half()
    x[0] = 0
    if M > 4:
        x[4] *= 300
    fn = oracle.fp8_quantize_per_token if torch_form else oracle.fp8_quantize_per_token_kernel
    q_ref, s_ref = fn(x.float())
    q, s = g.fp8_quantize_per_token(x.cuda(), torch_formulation=torch_form)
    assert_bitexact(s, s_ref, "fp8 scale")
    assert_bitexact(q, q_ref, "fp8 bytes")


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("K", [256, 768, 2048, 2304])
def test_fp8_quantiser_quotients_bitexact(dtype, K):
    """The torch formulation divides every element by the row scale: every finite fp16 value (both zeros and the
    subnormals among them) under row maxima from 2^-24 to 65504, bit for bit."""
    g = need_lib()
    every = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.float16)
    every = every[torch.isfinite(every)]
    every = every[torch.argsort(every.abs().float())]           # rows of like magnitude, so that every E4M3 binade is met
    M = (every.numel() + K - 1) // K
    x = torch.zeros(M * K, dtype=torch.float16)
    x[: every.numel()] = every
    x = x.view(M, K).to(dtype)
    gen = torch.Generator().manual_seed(K)
    mixed = torch.randn(64, K, generator=gen) * torch.logspace(-6, 3, 64)[:, None]
    x = torch.cat([x, mixed.to(dtype)])
    q_ref, s_ref = oracle.fp8_quantize_per_token(x.float())
    q, s = g.fp8_quantize_per_token(x.cuda())
    assert_bitexact(s, s_ref, "fp8 scale")
    assert_bitexact(q, q_ref, "fp8 bytes")


def test_fp8_quantiser_golden():
    g = need_lib()
    gold = load_golden("fp8_quant")
    q, s = g.fp8_quantize_per_token(T(gold["x"]).cuda(), torch_formulation=True)
    assert_bitexact(q.view(torch.uint8), T(gold["xq"]), "fp8 bytes vs reference golden")
    assert_bitexact(s, T(gold["xs"]), "fp8 scales vs reference golden")


def test_bounded_wait_gives_up_and_reports():
    """A wait nothing satisfies must end by itself and leave a code in the status word."""
    g = need_lib()
    L = g.lib()
    assert g.device_status()[0] == 0
    assert L.gsb200_set_spin_budget(200000) == 0          # ~0.1 ms of SM clocks
    try:
        assert L.gsb200_selftest_wait_timeout(None) == 0
        torch.cuda.synchronize()
        st = g.device_status()
        assert st[0] & 4 and st[1] == 0xdead
        assert g.device_status()[0] == 0                    # read clears
    finally:
        assert L.gsb200_set_spin_budget(0) == 0
    x = torch.randn(64, 512).half().cuda()                  # context still healthy
    q, s = g.quantize_tensor(x)
    q_ref, _ = oracle.quantize_tensor(x.cpu().float())
    assert torch.equal(q.cpu(), q_ref)


def _rows_with_nan_and_inf(K, dtype):
    """Rows of N(0, 1) values: finite ones between rows that hold a NaN (of either sign), an infinity, both, or nothing else."""
    gen = torch.Generator().manual_seed(K)
    nan, inf = float("nan"), float("inf")
    x = torch.randn(24, K, generator=gen)
    last = K - 1
    for row, put in enumerate([{}, {0: nan}, {}, {last: -nan}, {K // 2: inf}, {}, {3: -inf}, {1: nan, 2: inf}, {last: inf, 0: -inf, 7: nan}]):
        for i, v in put.items():
            x[row, i] = v
    x[9], x[10], x[11] = nan, inf, 0.0
    x[12, :8], x[12, 8:] = nan, 0.0
    x[13, ::2], x[13, 1::2] = inf, -0.0
    return x.to(dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("K", [8, 512, 1024, 2048, 2304])
def test_fp8_quantiser_rows_with_nan_and_infinity(dtype, K):
    """A NaN does not take part in the row maximum; an infinity does (scale infinity: the row's finite values become zeros).
    What is not a number after the scaling is -448 in the torch formulation (the clamp) and NaN in the kernel formulation."""
    g = need_lib()
    x = _rows_with_nan_and_inf(K, dtype)
    xf = x.float()
    amax = torch.where(xf.isnan(), torch.zeros(()), xf.abs()).amax(dim=1, keepdim=True).clamp(min=1e-12)
    scale = amax / 448.0
    for torch_form in (True, False):
        v = xf / scale if torch_form else xf * (torch.full_like(amax, 448.0) / amax)
        q_ref = v.clamp(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8)
        q_ref[v.isnan()] = 0xFE if torch_form else 0x7F
        q, s = g.fp8_quantize_per_token(x.cuda(), torch_formulation=torch_form)
        assert_bitexact(s, scale.squeeze(1), f"scale, torch_formulation={torch_form}")
        assert_bitexact(q.view(torch.uint8), q_ref, f"bytes, torch_formulation={torch_form}")


@pytest.mark.parametrize("K", [512, 1024, 2048, 2304])
def test_fp8_quantiser_at_the_limits_of_fp32(K):
    """Quotients without a division: row maxima up to the largest fp32 number and down to (and below) the floor of 1e-12, with
    elements far smaller than the maximum, subnormals and both zeros among them."""
    g = need_lib()
    gen = torch.Generator().manual_seed(K + 1)
    rows = []
    for top in (3.4028234e38, 3e38, 2.0 ** 100, 448.0, 1.0, 1e-11, 1e-12, 9e-13, 1e-30, 1.2e-38, 1e-45):
        for binades in (12, 140, 140):
            x = (torch.rand(K, generator=gen) * 2 - 1) * top
            x = x * torch.exp2(-torch.randint(0, binades, (K,), generator=gen).double()).float()
            x[0], x[1], x[2], x[3] = top, 0.0, -0.0, 1e-45
            x[4:12] = -top * torch.tensor([1.0, 0.5, 0.4999, 2 ** -6, 2 ** -9, 2 ** -10, 2 ** -10 * 1.0001, 2 ** -17])
            rows.append(x)
    x = torch.stack(rows)
    q_ref, s_ref = oracle.fp8_quantize_per_token(x)
    q, s = g.fp8_quantize_per_token(x.cuda())
    assert_bitexact(s, s_ref, "fp8 scale")
    assert_bitexact(q, q_ref, "fp8 bytes")


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("K", [32, 512, 2048, 2304])
def test_mx_quantiser_blocks_with_nan_and_infinity(dtype, K):
    """Per block of 32: a NaN does not take part in the maximum and stays a NaN; an infinity gives the scale 2^120 and saturates."""
    g = need_lib()
    x = _rows_with_nan_and_inf(K, dtype)
    blk = x.float().view(len(x), K // 32, 32)
    amax = torch.where(blk.isnan(), torch.zeros(()), blk.abs()).amax(dim=-1)
    byte = (((amax.view(torch.int32) >> 23) & 0xFF) - 8).clamp(0, 254)
    v = blk * torch.ldexp(torch.ones_like(amax), 127 - byte).unsqueeze(-1)
    q_ref = v.clamp(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8)
    q_ref[v.isnan()] = 0x7F
    q, s = g.mxfp8_quantize(x.cuda())
    assert_bitexact(s, byte.to(torch.uint8), "E8M0 scales")
    assert_bitexact(q.view(torch.uint8), q_ref.view(len(x), K), "bytes")


def test_fp8_quotients_of_every_fp16_pair():
    """The torch formulation divides by amax / 448; the kernel gets the quotient of an fp16 row from one refinement of a product.
    Every fp16 significand as the row maximum, with every fp16 value up to it: 16 million pairs, scaled to three places in the fp16
    range (a power of two changes nothing but the exponents)."""
    g = need_lib()
    bits = torch.arange(0x3C00, 0x4000, dtype=torch.int32, device="cuda")          # 1 <= amax < 2
    val = torch.arange(0, 0x4000, dtype=torch.int32, device="cuda")
    per = -(-len(val) // 511)
    body = torch.zeros(per * 511, dtype=torch.int32, device="cuda")
    body[:len(val)] = val
    body = body.view(per, 511).to(torch.int16).view(torch.float16)
    for shift in (-13, 0, 14):
        for chunk in bits.split(128):
            amax = chunk.to(torch.int16).view(torch.float16)
            x = torch.empty(len(chunk), per, 512, dtype=torch.float16, device="cuda")
            x[:, :, 0] = amax[:, None]
            x[:, :, 1:] = torch.minimum(body[None], amax[:, None, None])
            x[:, 1::2] *= -1
            x = (x.view(-1, 512) * 2.0 ** shift)
            q, s = g.fp8_quantize_per_token(x)
            ref_s = x.abs().amax(1).float() / torch.full((len(x),), 448.0, device="cuda")     # (a tensor: torch multiplies by 1 / scalar)
            assert torch.equal(s, ref_s)
            ref = (x.float() / ref_s[:, None]).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
            assert torch.equal(q.view(torch.uint8), ref.view(torch.uint8))
