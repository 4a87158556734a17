"""The native call path of the operators (csrc/binding.cpp): it takes plain CUDA tensors only and leaves every other
call to the Python function, and what it takes gives the bytes of the ctypes path."""
import pytest
import torch

import oracle
from util import need_lib


def test_native_path_declines_what_is_not_plain():
    from gigaslop_b200 import _lib
    _lib.lib()
    n = _lib.native
    x = torch.zeros(4, 64, dtype=torch.float16)
    w = torch.zeros(8, 64, dtype=torch.int8)
    s = torch.zeros(8)
    assert n.quantize(0, x, None, None) is None                  # CPU tensors
    assert n.quantize(0, "x", None, None) is None and n.quantize(0, x) is None
    assert n.gemm(0, w, w, s, s, None, 0) is None
    assert n.gemm(0, w, w, s, s, None, 1 << 40) is None and n.gemm(0, w, w, s, s, None, 0.0) is None
    assert n.quantize(0, torch.nn.Parameter(x), None, None) is None
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        assert n.quantize(0, torch.empty(4, 64, dtype=torch.float16, device="cuda"), None, None) is None
    with pytest.raises(RuntimeError):
        need_lib().quantize_tensor(x)


def run_python(code):
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    return subprocess.run([sys.executable, "-c", f"import sys; sys.path.insert(0, {root!r})\n" + code], capture_output=True, text=True,
                          timeout=120)


def test_package_works_without_the_native_path():
    """The extension is a shortcut: without it the library loads, with a warning, and every call goes through ctypes."""
    r = run_python("import warnings; sys.modules['gigaslop_b200._native'] = None\n"
                   "import gigaslop_b200 as g; from gigaslop_b200 import _lib\n"
                   "with warnings.catch_warnings(record=True) as w:\n"
                   "    warnings.simplefilter('always'); g.lib(); g.lib()\n"
                   "assert [x.category for x in w] == [RuntimeWarning] and '_native.so' in str(w[0].message), w\n"
                   "assert _lib.native is None and g.mx_scales_to_tiled and g.lib().gsb200_mx_tiled_scale_bytes(128, 128) == 512\n")
    assert r.returncode == 0, r.stdout + r.stderr


def test_native_path_belongs_to_one_torch(monkeypatch):
    """The extension looks into torch's tensors: one built for another torch is rebuilt, and not used."""
    from gigaslop_b200 import build
    build.build_native()
    assert not build.native_is_stale()
    monkeypatch.setattr(torch, "__version__", "99.0")
    assert build.native_is_stale()
    r = run_python("import warnings, torch; torch.__version__ = '99.0'\n"
                   "import gigaslop_b200 as g; from gigaslop_b200 import _lib\n"
                   "with warnings.catch_warnings(record=True) as w:\n"
                   "    warnings.simplefilter('always'); g.lib()\n"
                   "assert len(w) == 1 and 'torch 99.0' in str(w[0].message), w\n"
                   "assert _lib.native is None\n")
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_native_path_gives_the_bytes_of_the_checked_path(monkeypatch):
    g = need_lib()
    from gigaslop_b200 import _lib
    gen = torch.Generator().manual_seed(5)
    M, K, nh = 77, 256, 4
    x = torch.randn(M, K, generator=gen).half().cuda()
    xs = torch.randn(M, 2 * K, generator=gen).half().cuda()[:, :K]             # strided rows
    w = torch.randint(-127, 128, (3 * K, K), generator=gen, dtype=torch.int8).cuda()
    w8 = ((torch.rand(3 * K, K, generator=gen) * 2 - 1) * 400).to(torch.float8_e4m3fn).cuda()
    sw = (1e-3 + 1e-2 * torch.rand(3 * K, generator=gen)).cuda()
    sin, cos = [t.cuda() for t in oracle.rope_tables(M, 32, 64)]
    up = torch.randn(128, 64, generator=gen).half().cuda()
    bias = torch.randn(128, generator=gen).cuda()
    one = torch.full((1,), 2e-3, device="cuda")
    H, R, B = 64, 64, 33
    fac = lambda *shape: (torch.randn(*shape, generator=gen) * 0.2).half().cuda()
    hh, uhh, xd, uih = fac(B, R), fac(4 * H, R), fac(B, R), fac(4 * H, R)
    qi, si = g.quantize_tensor(x)
    q8, s8 = g.fp8_quantize_per_token(x)
    qm, sm = g.mxfp8_quantize(x)
    wm, swm = g.mxfp8_quantize(torch.randn(3 * K, K, generator=gen).half().cuda())
    swm = g.mx_scales_to_tiled(swm, K)
    tm = g.mx_scales_to_tiled(sm, K)

    def step():
        h, c = torch.zeros(B, H, dtype=torch.uint8, device="cuda"), torch.zeros(B, H, device="cuda")
        return g.factored_lstm_step(h, c, hh, uhh, None, xd, uih, bias[:1].expand(4 * H).contiguous())

    buf = lambda *shape, dtype=torch.float16: torch.empty(*shape, dtype=dtype, device="cuda")
    rope = (sin, cos, nh, 64, 64, M, 3)
    calls = {
        "quantize_tensor": lambda: g.quantize_tensor(xs), "quantize_tensor f32": lambda: g.quantize_tensor(x.float(), 1, buf(M, K, dtype=torch.int8)),
        "fp8": lambda: g.fp8_quantize_per_token(xs), "fp8 kernel": lambda: g.fp8_quantize_per_token(x, False, out_scale=buf(M, dtype=torch.float32)),
        "mxfp8": lambda: g.mxfp8_quantize(xs), "tile": lambda: g.mx_scales_to_tiled(sm, K),
        "gemm_i8": lambda: g.gemm_i8(qi, w, si, sw), "gemm_i8 out": lambda: g.gemm_i8(qi, w, si, sw, buf(M, 4 * K)[:, :3 * K]),
        "gemm_fp8": lambda: g.gemm_fp8(q8, w8, s8, sw), "down": lambda: g.fp8_down_proj(q8, s8, w8[:64], one),
        "rotary i8": lambda: g.gemm_i8_rotary(qi, w, si, sw, *rope), "rotary fp8": lambda: g.gemm_fp8_rotary(q8, w8, s8, sw, *rope),
        "silu i8": lambda: g.dual_gemm_i8_silu(qi, w[:K], w[K:2 * K], si, sw[:K], sw[K:2 * K]),
        "silu fp8": lambda: g.dual_gemm_fp8_silu(q8, w8[:K], w8[K:2 * K], s8, sw[:K], sw[K:2 * K]),
        "silu mx": lambda: g.dual_gemm_fp8_silu_mxfp8(q8, w8[:K], w8[K:2 * K], s8, sw[:K], sw[K:2 * K]),
        "gemm mx": lambda: g.gemm_mxfp8(qm, tm, wm, swm), "dual mx": lambda: g.dual_gemm_mxfp8_silu(qm, tm, wm, wm, swm, swm),
        "factored": lambda: g.fp8_factored_gemm(q8, s8, w8[:64], one, up, bias), "step": step,
    }
    flat = lambda r: [t.cpu().contiguous().view(torch.uint8) for t in (r if isinstance(r, tuple) else (r,))]
    taken = []

    class Spy:                                                   # every one of these calls is one the native path takes
        def __getattr__(self, name):
            fn = getattr(_lib_native, name)
            return lambda *a: taken.append((name, r := fn(*a))) or r

    _lib_native = _lib.native
    monkeypatch.setattr(_lib, "native", Spy())
    native = {k: flat(f()) for k, f in calls.items()}
    assert len(taken) == len(calls) and all(r is not None for _, r in taken), [n for n, r in taken if r is None]
    monkeypatch.setattr(_lib, "native", None)
    for k, f in calls.items():
        for a, b in zip(native[k], flat(f())):
            assert torch.equal(a, b), k
    # a view handed in as `out` comes back as the same object, on both paths
    out = buf(M, 3 * K)
    assert g.gemm_i8(qi, w, si, sw, out) is out
    monkeypatch.undo()
    assert g.gemm_i8(qi, w, si, sw, out) is out
    # another stream: the launch goes to the stream that is current at the call
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        r = g.gemm_i8(qi, w, si, sw)
    side.synchronize()
    assert torch.equal(flat(r)[0], native["gemm_i8"][0])
    with pytest.raises(ValueError):
        g.gemm_i8(qi[:, ::2], w, si, sw)
    with pytest.raises(TypeError):
        g.gemm_fp8(qi, w, si, sw)


@pytest.mark.gpu
def test_error_of_a_copy_on_write_tensor_is_raised():
    """Taking the data pointer of a lazily cloned tensor makes its copy, which can fail: the error is an ordinary exception (it
    is thrown while the interpreter lock is held).  In a child process, which is given little memory and leaves without
    freeing the tensor: torch itself aborts there after a copy that failed."""
    r = run_python(
        "import os, torch\n"
        "import gigaslop_b200 as g; from gigaslop_b200 import _lib\n"
        "g.lib(); assert _lib.native is not None\n"
        "x = torch.randn(1 << 16, 512, device='cuda').half(); torch.cuda.synchronize(); torch.cuda.empty_cache()\n"
        "q, s = torch.empty(x.shape, dtype=torch.int8, device='cuda'), torch.empty(len(x), device='cuda')\n"
        "want = g.quantize_tensor(x)[0].cpu()\n"
        "assert torch.equal(g.quantize_tensor(torch._lazy_clone(x), out=q, out_scale=s)[0].cpu(), want)\n"
        "y = torch._lazy_clone(x); torch.cuda.empty_cache()\n"
        "total = torch.cuda.get_device_properties(0).total_memory\n"
        "torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (8 << 20)) / total)\n"
        "try:\n"
        "    g.quantize_tensor(y, out=q, out_scale=s)\n"
        "    print('no error')\n"
        "except torch.OutOfMemoryError:\n"
        "    print('raised')\n"
        "sys.stdout.flush(); os._exit(0)\n")
    assert r.returncode == 0 and r.stdout.split() == ["raised"], r.stdout + r.stderr


@pytest.mark.gpu
def test_call_that_the_library_refuses_is_made_once(monkeypatch):
    """A refusal raises from the native path: the Python function does not allocate, print and launch a second time."""
    g = need_lib()
    from gigaslop_b200 import ops
    entered = []
    for name in dir(ops):
        if name.startswith("_checked_"):
            monkeypatch.setattr(ops, name, lambda *a, _n=name: entered.append(_n))
    z = lambda *shape, dtype=torch.float16: torch.zeros(*shape, dtype=dtype, device="cuda")
    f8 = lambda *shape: z(*shape, dtype=torch.uint8).view(torch.float8_e4m3fn)
    i8, f32 = lambda *shape: z(*shape, dtype=torch.int8), lambda *shape: z(*shape, dtype=torch.float32)
    x, w, s, tab = 24, 64, f32(192), f32(8, 32)                   # K = 24: not a multiple of 16 (nor of 32, 64 or 128)
    calls = {
        "quantize_tensor": lambda: g.quantize_tensor(z(4, 4)), "fp8_quantize_per_token": lambda: g.fp8_quantize_per_token(z(4, 4)),
        "mxfp8_quantize": lambda: g.mxfp8_quantize(z(4, 40)), "gemm_i8": lambda: g.gemm_i8(i8(4, x), i8(w, x), s, s),
        "gemm_fp8": lambda: g.gemm_fp8(f8(4, x), f8(w, x), s, s),
        "gemm_i8_rotary": lambda: g.gemm_i8_rotary(i8(4, x), i8(192, x), s, s, tab, tab, 1, 64, 64, 8),
        "gemm_fp8_rotary": lambda: g.gemm_fp8_rotary(f8(4, x), f8(192, x), s, s, tab, tab, 1, 64, 64, 8),
        "dual_gemm_i8_silu": lambda: g.dual_gemm_i8_silu(i8(4, x), i8(w, x), i8(w, x), s, s, s),
        "dual_gemm_fp8_silu": lambda: g.dual_gemm_fp8_silu(f8(4, x), f8(w, x), f8(w, x), s, s, s),
        "dual_gemm_fp8_silu_mxfp8": lambda: g.dual_gemm_fp8_silu_mxfp8(f8(4, x), f8(w, x), f8(w, x), s, s, s),
        "mx_scales_to_tiled": lambda: g.mx_scales_to_tiled(z(4, 3, dtype=torch.uint8), 96),
        "gemm_mxfp8": lambda: g.gemm_mxfp8(f8(4, x), f8(512), f8(w, x), f8(512)),
        "dual_gemm_mxfp8_silu": lambda: g.dual_gemm_mxfp8_silu(f8(4, x), f8(512), f8(w, x), f8(w, x), f8(512), f8(512)),
        "fp8_factored_gemm": lambda: g.fp8_factored_gemm(f8(4, 64), f32(4), f8(12, 64), f32(1), z(64, 12), f32(64)),
        "factored_lstm_step": lambda: g.factored_lstm_step(f8(4, 64), f32(4, 64), z(4, x), z(256, x), None, z(4, x), z(256, x), None),
    }
    for name, call in calls.items():
        with pytest.raises(RuntimeError, match=rf"gigaslop_b200\.{name}: .* \(status -"):
            call()
        assert not entered, name


@pytest.mark.gpu
@pytest.mark.parametrize("native", [True, False])
def test_gate_and_up_weights_share_shape_and_stride(native, monkeypatch):
    """The library describes both weights with the gate's row count and stride: an up weight with fewer rows would be read past
    its end, one with another stride misread.  All four SwiGLU operators raise for both."""
    g = need_lib()
    from gigaslop_b200 import _lib
    if not native:
        monkeypatch.setattr(_lib, "native", None)
    z = lambda *shape: torch.zeros(*shape, dtype=torch.uint8, device="cuda")
    s, M, N, K = torch.ones(256, device="cuda"), 8, 256, 128
    sf = lambda rows: z(g.lib().gsb200_mx_tiled_scale_bytes(rows, K))
    f8 = torch.float8_e4m3fn
    for up in (z(N // 2, K), z(2 * N, K), z(N, 2 * K)[:, :K]):
        a, gate = z(M, K), z(N, K)
        with pytest.raises(ValueError):
            g.dual_gemm_i8_silu(a.view(torch.int8), gate.view(torch.int8), up.view(torch.int8), s, s, s)
        with pytest.raises(ValueError):
            g.dual_gemm_fp8_silu(a.view(f8), gate.view(f8), up.view(f8), s, s, s)
        with pytest.raises(ValueError):
            g.dual_gemm_fp8_silu_mxfp8(a.view(f8), gate.view(f8), up.view(f8), s, s, s)
        with pytest.raises(ValueError):
            g.dual_gemm_mxfp8_silu(a.view(f8), sf(M), gate.view(f8), up.view(f8), sf(N), sf(N))


@pytest.mark.gpu
def test_native_path_declines_one_argument_that_is_not_plain():
    """CUDA operands throughout, so that nothing but the one argument named is the reason."""
    need_lib()
    from gigaslop_b200 import _lib
    n = _lib.native
    x = torch.randn(4, 64, device="cuda").half()
    a, w = torch.ones(4, 64, dtype=torch.int8, device="cuda"), torch.ones(8, 64, dtype=torch.int8, device="cuda")
    sa, sw = torch.ones(4, device="cuda"), torch.ones(8, device="cuda")
    assert n.gemm(0, a, w, sa, sw, None, 0) is not None and n.quantize(0, x, None, None) is not None

    class Sub(torch.Tensor):
        pass

    declined = {
        "flags beyond 32 bits": (0, a, w, sa, sw, None, 1 << 40), "flags beyond 64 bits": (0, a, w, sa, sw, None, 1 << 80),
        "float flags": (0, a, w, sa, sw, None, 0.0), "K mismatch": (0, a[:, :32], w, sa, sw, None, 0),
        "1-D operand": (0, a[0], w, sa, sw, None, 0), "inner stride": (0, a[:, ::2], w[:, :32], sa, sw, None, 0),
        "wrong type": (0, a.float(), w, sa, sw, None, 0), "INT8 for FP8": (1, a, w, sa, sw, None, 0),
        "subclass": (0, a.as_subclass(Sub), w, sa, sw, None, 0), "CPU scale": (0, a, w, sa.cpu(), sw, None, 0),
        "CPU output": (0, a, w, sa, sw, torch.empty(4, 8, dtype=torch.float16), 0), "not a tensor": (0, a, w, [1.0], sw, None, 0),
        "conjugate view": (0, a, w, torch.ones(4, dtype=torch.complex64, device="cuda").conj(), sw, None, 0),
        "negative view": (0, a, w, torch.ones(4, dtype=torch.complex64, device="cuda").conj().imag, sw, None, 0),
        "an argument too few": (0, a, w, sa, sw, None),
    }
    for what, args in declined.items():
        assert n.gemm(*args) is None, what
    assert n.quantize(0, x.double(), None, None) is None
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode
    for mode in (TorchFunctionMode, TorchDispatchMode):
        with mode():
            assert n.gemm(0, a, w, sa, sw, None, 0) is None, mode.__name__
    seen = []

    def batched(t):
        seen.append(n.quantize(0, t, None, None))
        return t

    torch.vmap(batched)(x[None])
    assert seen == [None]


@pytest.mark.gpu
def test_outputs_are_what_torch_empty_makes():
    """Outputs come from torch's CUDA allocation function without the dispatcher: ordinary tensors, inference tensors under
    inference mode, and the dispatcher's (filled) ones in the deterministic mode -- with the same bytes in each."""
    g = need_lib()
    x = torch.randn(300, 512, generator=torch.Generator().manual_seed(2)).half().cuda()
    q, s = g.quantize_tensor(x)
    for t in (q, s):
        e = torch.empty(t.shape, dtype=t.dtype, device="cuda")
        assert type(t) is torch.Tensor and t.stride() == e.stride() and t.storage_offset() == 0 and t.device == e.device
        assert t.untyped_storage().nbytes() == e.untyped_storage().nbytes() and t._version == 0 and not t.is_inference()
        assert torch._C._dispatch_keys(t) == torch._C._dispatch_keys(e)
    with torch.inference_mode():
        qi, si = g.quantize_tensor(x)
        assert qi.is_inference() and si.is_inference() and torch.equal(qi, q) and torch.equal(si, s)
    try:
        torch.use_deterministic_algorithms(True)
        qd, sd = g.quantize_tensor(x)
        assert torch.equal(qd, q) and torch.equal(sd, s)
    finally:
        torch.use_deterministic_algorithms(False)
    e, se = g.quantize_tensor(x[:0])
    assert e.shape == (0, 512) and se.shape == (0,)


@pytest.mark.gpu
def test_a_profiler_sees_the_outputs_allocated():
    """Under a profiler of operator calls the outputs come through the dispatcher, so a trace shows them as torch.empty's."""
    g = need_lib()
    x = torch.randn(300, 512, generator=torch.Generator().manual_seed(2)).half().cuda()
    want = g.quantize_tensor(x)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        got = g.quantize_tensor(x)
    assert sum(e.count for e in prof.key_averages() if e.key == "aten::empty") == 2
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
