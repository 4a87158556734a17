"""Workloads of the quantized-GEMM path, as a program that uses the package runs them.

Each case is one call sequence of the public functions on device-resident inputs: what a transformer or LSTM
basecaller built on this library does for one batch of chunks.  Sizes are those of the benchmark configurations
(65536 tokens = 32 chunks x 2048 steps, d_model 512, feed-forward 2048; LSTM stack of 5 x 384 over 512 x 2000) and
of the tests, from a single short read up to the full batch.

    linear        quantise activations per token, GEMM with dequant epilogue          (any projection of a layer)
    qkv           quantise, QKV GEMM with the rotary embedding in its epilogue        (attention input of a layer)
    ffn           quantise, SwiGLU dual GEMM, re-quantise, down-projection            (feed-forward of a layer)
    lowrank       quantise, low-rank input projection of a factored LSTM over all timesteps
    lstm_stack    quantise, LSTM stack: hoisted projections and recurrences of every layer
    lstm_cell     the factored LSTM cell stepped through time, two calls per timestep (a decoder's inner loop)
"""
import math

import torch

import gigaslop_b200 as g
from gigaslop_b200.lstm import lstm_stack_workspace

DEV = "cuda"


def listed():
    return [
        # the attention input of one full batch, INT8: the benchmark's headline step
        dict(name="qkv_i8_batch", op="qkv", dtype="int8", M=65536, nhead=8, head_dim=64, rotary_dim=64, seqlen=2048, row_offset=0),
        # one short read alone: the smallest calls, latency and launches count
        dict(name="qkv_i8_read", op="qkv", dtype="int8", M=333, nhead=8, head_dim=64, rotary_dim=64, seqlen=333, row_offset=0),
        # FP8 and wide heads, a shard of a batch (ragged rows, positions continue from the shard before)
        dict(name="qkv_fp8_h128_shard", op="qkv", dtype="fp8", M=20001, nhead=4, head_dim=128, rotary_dim=128, seqlen=2048, row_offset=20001),
        # a square projection over 8 chunks (attention output), INT8
        dict(name="linear_i8_16k", op="linear", dtype="int8", x="f16", M=16384, N=512, K=512),
        # the feed-forward of a full batch in each of the three precisions
        dict(name="ffn_i8_batch", op="ffn", dtype="int8", M=65536, K=512, F=2048),
        dict(name="ffn_fp8_ragged", op="ffn", dtype="fp8", M=9001, K=512, F=2048),
        dict(name="ffn_mxfp8_batch", op="ffn", dtype="mxfp8", M=65536, K=512, F=2048),
        # the feed-forward of a small batch
        dict(name="ffn_i8_small", op="ffn", dtype="int8", M=256, K=512, F=2048),
        # the deployed low-rank LSTM: input projection over all timesteps, and its recurrence (16 steps of it)
        dict(name="lowrank_batch", op="lowrank", M=131072, C=1024, R=128, N=4096),
        dict(name="lstm_cell_steps", op="lstm_cell", T=16, B=256, H=1024, K_hh=128, R=128),
        # the full-rank LSTM stack: the benchmark's full batch (next layer's projection on a second stream) ...
        dict(name="lstm_stack_batch", op="lstm_stack", T=2000, B=512, C=384, H=384, layers=5, overlap=True),
        # ... and a small model on a few chunks
        dict(name="lstm_stack_small", op="lstm_stack", T=200, B=70, C=96, H=128, layers=3, overlap=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tokens(rng):
    """1 .. 65536 rows: ragged, or a whole number of 128-row tiles."""
    m = _log(rng, 1, 65536)
    return m if rng.random() < 0.7 else max(128, m // 128 * 128)


def draw(rng):
    op = rng.choice(["linear", "qkv", "qkv", "ffn", "ffn", "lowrank", "lstm_stack", "lstm_cell"])
    if op == "linear":
        return dict(op=op, dtype=rng.choice(["int8", "fp8"]), x=rng.choice(["f16", "f16", "f16", "f32"]), M=_tokens(rng),
                    N=8 * _log(rng, 16, 256), K=rng.choice([128, 256, 384, 512, 512, 768, 1024, 2048]))
    if op == "qkv":
        head_dim = rng.choice([64, 64, 128])
        rotary_dim = rng.choice([head_dim, head_dim, head_dim // 2])
        d_model = rng.choice([256, 384, 512, 512, 768, 1024])
        seqlen = _log(rng, 64, 2048)
        return dict(op=op, dtype=rng.choice(["int8", "fp8"]), M=_tokens(rng), nhead=d_model // head_dim, head_dim=head_dim,
                    rotary_dim=rotary_dim, seqlen=seqlen, row_offset=rng.choice([0, rng.randrange(0, 65536)]))
    if op == "ffn":
        k = rng.choice([128, 256, 384, 512, 512])
        return dict(op=op, dtype=rng.choice(["int8", "fp8", "mxfp8", "fp8_mx"]), M=_tokens(rng), K=k, F=4 * k)
    if op == "lowrank":
        return dict(op=op, M=_log(rng, 64, 131072), C=rng.choice([256, 512, 1024]), R=rng.choice([64, 128]), N=rng.choice([1024, 1536, 4096]))
    if op == "lstm_stack":
        t = _log(rng, 25, 2000)
        return dict(op=op, T=t, B=max(1, min(512, rng.randrange(16, 513))), C=rng.choice([64, 128, 256, 384]),
                    H=rng.choice([128, 192, 256, 384, 384, 512]), layers=rng.choice([1, 2, 3, 5]), overlap=rng.random() < 0.5)
    return dict(op=op, T=_log(rng, 1, 64), B=rng.randrange(1, 513), H=rng.choice([512, 1024]), K_hh=rng.choice([64, 128]), R=rng.choice([64, 128]))


# ---- inputs ---------------------------------------------------------------------------------------------------
class _Rand:
    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV).manual_seed(seed)

    def act(self, *shape, dtype=torch.float16):               # activations ~ N(0, 1)
        return torch.randn(*shape, generator=self.gen, device=DEV, dtype=dtype)

    def i8(self, n, k):                                       # INT8 weight, uniform in [-127, 127]
        return torch.randint(-127, 128, (n, k), generator=self.gen, device=DEV, dtype=torch.int8)

    def f8(self, n, k, amp=448.0):                            # E4M3 weight, uniform
        return ((torch.rand(n, k, generator=self.gen, device=DEV) * 2 - 1) * amp).to(torch.float8_e4m3fn)

    def scale(self, n, lo=1e-3, hi=1e-2):                     # per-channel weight scales
        return lo + (hi - lo) * torch.rand(n, generator=self.gen, device=DEV)

    def normal(self, *shape, std=1.0):
        return torch.randn(*shape, generator=self.gen, device=DEV) * std


def _weight(r, dtype, n, k):
    """Quantised weight with per-channel scales such that outputs are O(1) for N(0, 1) activations."""
    unit = 1.73 / (127.0 if dtype == "int8" else 448.0) / math.sqrt(k)
    return (r.i8(n, k) if dtype == "int8" else r.f8(n, k)), r.scale(n, 0.7 * unit, 1.3 * unit)


def _mx_weight(r, n, k):
    """MXFP8 weight: E4M3 elements and E8M0 scales in the tile order of the block-scaled GEMMs."""
    q, s = g.mxfp8_quantize(r.normal(n, k, std=1.0 / math.sqrt(k)).half())
    return q, g.mx_scales_to_tiled(s, k)


def _rope(seqlen, half, head_dim):
    inv = 1.0 / (10000.0 ** (torch.arange(half, device=DEV).float() * 2 / head_dim))
    ang = torch.outer(torch.arange(seqlen, device=DEV).float(), inv)
    return ang.sin().contiguous(), ang.cos().contiguous()


def prepare(case, seed):
    r = _Rand(seed)
    op = case["op"]
    s = dict(case=case)
    if op == "linear":
        s["x"] = r.act(case["M"], case["K"], dtype=torch.float32 if case["x"] == "f32" else torch.float16)
        s["w"], s["sw"] = _weight(r, case["dtype"], case["N"], case["K"])
    elif op == "qkv":
        k = case["nhead"] * case["head_dim"]
        s["x"] = r.act(case["M"], k)
        s["w"], s["sw"] = _weight(r, case["dtype"], 3 * k, k)
        s["sin"], s["cos"] = _rope(case["seqlen"], case["rotary_dim"] // 2, case["head_dim"])
    elif op == "ffn":
        k, f = case["K"], case["F"]
        s["x"] = r.act(case["M"], k)
        if case["dtype"] == "mxfp8":
            s["wg"], s["sg"] = _mx_weight(r, f, k)
            s["wu"], s["su"] = _mx_weight(r, f, k)
        else:
            d = "int8" if case["dtype"] == "int8" else "fp8"
            s["wg"], s["sg"] = _weight(r, d, f, k)
            s["wu"], s["su"] = _weight(r, d, f, k)
        s["wd"], s["sd"] = _mx_weight(r, k, f) if case["dtype"] in ("mxfp8", "fp8_mx") else _weight(r, case["dtype"], k, f)
    elif op == "lowrank":
        c, rk = case["C"], case["R"]
        s["x"] = r.act(case["M"], c)
        s["dn"], s["sdn"] = r.f8(rk, c), torch.full((1,), 1.73 / 448.0 / math.sqrt(c), device=DEV)
        s["up"] = r.normal(case["N"], rk, std=1.0 / math.sqrt(rk)).half()
        s["bias"] = r.normal(case["N"], std=0.1)
    elif op == "lstm_stack":
        t, b, h = case["T"], case["B"], case["H"]
        s["x"] = r.act(t * b, case["C"])
        s["layers"] = []
        for i in range(case["layers"]):
            c = case["C"] if i == 0 else h
            s["layers"].append(dict(W_ih=r.f8(4 * h, c, 44.8), s_ih=r.scale(4 * h, 0.9 / 448, 1.1 / 448), b=r.normal(4 * h, std=0.05),
                                    W_hh=r.f8(4 * h, h, 44.8), s_hh=r.scale(4 * h, 0.9 / 448, 1.1 / 448)))
        s["ws"] = lstm_stack_workspace(t, b, h, torch.device(DEV, torch.cuda.current_device()), case["overlap"])
        s["aux"] = torch.cuda.Stream() if case["overlap"] else None
    elif op == "lstm_cell":
        t, b, h, kh, rk = case["T"], case["B"], case["H"], case["K_hh"], case["R"]
        s["x_down"] = r.normal(t, b, rk, std=0.3).half()              # hoisted low-rank projection of the inputs
        s["dn"], s["sdn"] = r.f8(kh, h), torch.full((1,), 1.73 / 448.0 / math.sqrt(h), device=DEV)
        s["up_hh"] = r.normal(4 * h, kh, std=1.0 / math.sqrt(kh)).half()
        s["up_ih"] = r.normal(4 * h, rk, std=1.0 / math.sqrt(rk)).half()
        s["b_hh"], s["b_ih"] = r.normal(4 * h, std=0.05), r.normal(4 * h, std=0.05)
        s["sx"] = torch.full((b,), 1.0 / 448.0, device=DEV)           # h is E4M3 at the fixed scale 1/448
        s["h"] = torch.empty(t + 1, b, h, dtype=torch.uint8, device=DEV)
        s["c"] = torch.empty(b, h, device=DEV)
    else:
        raise ValueError(op)
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "linear":
        if case["dtype"] == "int8":
            q, sa = g.quantize_tensor(s["x"])
            return g.gemm_i8(q, s["w"], sa, s["sw"])
        q, sa = g.fp8_quantize_per_token(s["x"])
        return g.gemm_fp8(q, s["w"], sa, s["sw"])
    if op == "qkv":
        args = (s["w"], s["sw"], s["sin"], s["cos"], case["nhead"], case["head_dim"], case["rotary_dim"], case["seqlen"])
        if case["dtype"] == "int8":
            q, sa = g.quantize_tensor(s["x"])
            return g.gemm_i8_rotary(q, args[0], sa, *args[1:], row_offset=case["row_offset"])
        q, sa = g.fp8_quantize_per_token(s["x"])
        return g.gemm_fp8_rotary(q, args[0], sa, *args[1:], row_offset=case["row_offset"])
    if op == "ffn":
        if case["dtype"] == "int8":
            q, sa = g.quantize_tensor(s["x"])
            h = g.dual_gemm_i8_silu(q, s["wg"], s["wu"], sa, s["sg"], s["su"])
            q, sa = g.quantize_tensor(h)
            return g.gemm_i8(q, s["wd"], sa, s["sd"])
        if case["dtype"] == "fp8":
            q, sa = g.fp8_quantize_per_token(s["x"])
            h = g.dual_gemm_fp8_silu(q, s["wg"], s["wu"], sa, s["sg"], s["su"])
            q, sa = g.fp8_quantize_per_token(h)
            return g.gemm_fp8(q, s["wd"], sa, s["sd"])
        if case["dtype"] == "mxfp8":                          # block scales on both operands throughout
            q, sa = g.mxfp8_quantize(s["x"])
            h = g.dual_gemm_mxfp8_silu(q, g.mx_scales_to_tiled(sa, case["K"]), s["wg"], s["wu"], s["sg"], s["su"])
            q, sa = g.mxfp8_quantize(h)
            return g.gemm_mxfp8(q, g.mx_scales_to_tiled(sa, case["F"]), s["wd"], s["sd"])
        q, sa = g.fp8_quantize_per_token(s["x"])              # FP8 SwiGLU that emits MXFP8 for the down-projection
        q, sa = g.dual_gemm_fp8_silu_mxfp8(q, s["wg"], s["wu"], sa, s["sg"], s["su"])
        return g.gemm_mxfp8(q, g.mx_scales_to_tiled(sa, case["F"]), s["wd"], s["sd"])
    if op == "lowrank":
        q, sx = g.fp8_quantize_per_token(s["x"])
        return g.fp8_factored_gemm(q, sx, s["dn"], s["sdn"], s["up"], s["bias"])
    if op == "lstm_stack":
        q, sx = g.fp8_quantize_per_token(s["x"])
        return g.lstm_stack(q, sx, s["layers"], case["T"], case["B"], workspace=s["ws"], aux_stream=s["aux"])
    h, c = s["h"], s["c"]                                     # lstm_cell: a new batch starts from zero state
    h[0].zero_()
    c.zero_()
    for t in range(case["T"]):
        hh = g.fp8_down_proj(h[t].view(torch.float8_e4m3fn), s["sx"], s["dn"], s["sdn"])
        g.factored_lstm_step(h[t + 1], c, hh, s["up_hh"], s["b_hh"], s["x_down"][t], s["up_ih"], s["b_ih"])
    return h[1:].view(torch.float8_e4m3fn), c


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def work(case):
    """Inputs (activations, weights, tables) read once, results written once; intermediates are not counted."""
    op = case["op"]
    if op == "linear":
        m, n, k = case["M"], case["N"], case["K"]
        return dict(bytes=m * k * (4 if case["x"] == "f32" else 2) + n * k + 4 * n + 2 * m * n, flops=2 * m * n * k)
    if op == "qkv":
        m, k = case["M"], case["nhead"] * case["head_dim"]
        return dict(bytes=2 * m * k + 3 * k * k + 12 * k + 6 * m * k + 4 * case["seqlen"] * case["rotary_dim"], flops=6 * m * k * k)
    if op == "ffn":
        m, k, f = case["M"], case["K"], case["F"]
        return dict(bytes=4 * m * k + 3 * k * f + 8 * f + 4 * k, flops=6 * m * k * f)
    if op == "lowrank":
        m, c, r, n = case["M"], case["C"], case["R"], case["N"]
        return dict(bytes=2 * m * c + r * c + 2 * n * r + 4 * n + 2 * m * n, flops=2 * m * r * (c + n))
    if op == "lstm_stack":
        rows, c, h, layers = case["T"] * case["B"], case["C"], case["H"], case["layers"]
        w = 4 * h * c + (layers - 1) * 4 * h * h + layers * (4 * h * h + 36 * h)
        return dict(bytes=2 * rows * c + 2 * rows * h + w, flops=2 * rows * 4 * h * (c + h * (2 * layers - 1)))
    t, b, h, kh, r = case["T"], case["B"], case["H"], case["K_hh"], case["R"]
    w = kh * h + 8 * h * (kh + r) + 32 * h
    return dict(bytes=2 * t * b * r + t * b * h + 4 * b * h + w, flops=2 * t * b * (kh * h + 4 * h * (kh + r)))


def tolerance(case):
    """About four times the 2-norm difference measured between a pass and the same path with its sums and functions in
    64 bits, quantised at the same points.  INT8 is exact up to the fp16 result (2.1e-4); an E4M3 activation whose scale
    differs in its last bit may round to the neighbouring value, 2^-3 away (9e-4 after one quantiser, 3.9e-3 after the
    two of a feed-forward); the recurrences feed such flips back (3e-3 in the cell, 5e-3 to 2e-2 in the stack)."""
    op, fp8 = case["op"], case.get("dtype") != "int8"
    if op in ("linear", "qkv", "lowrank"):
        return {"rel": 4e-3 if fp8 else 8e-4}
    if op == "ffn":
        return {"rel": {"int8": 2e-3, "fp8": 1.6e-2, "mxfp8": 3.5e-3, "fp8_mx": 1.6e-2}[case["dtype"]]}
    if op == "lstm_cell":
        return {"rel": 1.2e-2}
    return {"rel": 8e-2 if case["H"] >= 256 else 3e-2}
