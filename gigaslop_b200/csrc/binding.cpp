// Native call path of the Python operators: argument checks, output allocation and the C-ABI call without the
// interpreter in between.  It takes the plain case only -- ordinary CUDA tensors of one device, that device current, no
// torch-function or dispatch mode active, every shape, stride and type check of the Python function passed -- and
// returns None for everything else, upon which the Python function runs its own checks (and raises what it always
// raised) and calls the library through ctypes.  A status other than 0 raises here, with the exception that the Python
// function makes of it.  Nothing is kept between calls.
//
// Why: through Python and ctypes an operator costs the host 17 to 22 us (device checks 3, torch.empty 2 to 4, stream
// lookup 2, about 15 converted arguments 4, launch 4); small calls never reached the GPU's own time.  Here it is 3 to 4.5: the
// launch is 2.1 of them, a GEMM into a given output 3.0, with its output allocated 4.1, a quantiser with two outputs 4.4 (with
// the outputs allocated through the dispatcher 4.5 and 5.1).
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "gigaslop_b200/gigaslop_b200.h"

namespace {

// Entry points of the loaded library, handed over as addresses (the ctypes handle owns the library).
enum Entry { PTQ_INT8, PTQ_FP8, PTQ_MXFP8, GEMM_I8, GEMM_FP8, ROT_I8, ROT_FP8, DUAL_I8, DUAL_FP8, DUAL_FP8_MX, MX_BYTES, MX_TILE, MX_GEMM,
             MX_DUAL, FAC_GEMM, FAC_STEP, N_ENTRIES };
void* g_entry[N_ENTRIES];
PyObject* g_check;             // check(status, what), raises
template <typename Fn>
Fn entry(Entry e, Fn) { return reinterpret_cast<Fn>(g_entry[e]); }
#define ENTRY(e, name) entry(e, &name)

// One call's view of its tensors: false from any method = not the plain case.
struct Call {
  c10::Device device{c10::kCPU};
  bool have = false;

  bool tensor(PyObject* o, const at::Tensor*& t) {
    if (!THPVariable_CheckExact(o)) return false;
    t = &THPVariable_Unpack(o);
    if (!t->defined()) return false;
    static const uint64_t plain = c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::AutocastCUDA}).raw_repr();
    const c10::DispatchKeySet ks = t->unsafeGetTensorImpl()->key_set();
    if ((ks.raw_repr() & ~plain) != 0 || !t->is_cuda()) return false;
    if (!have) {
      device = t->device();
      have = true;
      return device.index() == c10::cuda::current_device();
    }
    return t->device() == device;
  }
  bool optional(PyObject* o, const at::Tensor*& t) {
    t = nullptr;
    return o == Py_None || tensor(o, t);
  }
  // 2-D with unit inner stride
  bool rows(PyObject* o, const at::Tensor*& t) { return tensor(o, t) && t->dim() == 2 && t->stride(1) == 1; }
  bool out_rows(PyObject* o, const at::Tensor*& t) { return optional(o, t) && (!t || t->dim() >= 1); }
  gsb200_stream_t stream() const { return c10::cuda::getCurrentCUDAStream(device.index()).stream(); }
  // An output.  torch's own CUDA allocation function directly: the way to it through the dispatcher is most of what at::empty
  // costs.  The dispatcher is asked where something may want to see the call: dispatch keys switched on for this
  // thread (functorch, tracing), observers of operator calls (a profiler), or the deterministic mode, in which at::empty
  // fills its result.
  int direct = -1;             // what empty() found for this call
  at::Tensor empty(at::IntArrayRef size, at::ScalarType dt) {
    if (direct < 0) {
      const c10::DispatchKeySet on = c10::impl::tls_local_dispatch_key_set().included_;
      direct = (on - c10::default_included_set).empty() && !at::hasCallbacks() && !at::globalContext().deterministicAlgorithms() ? 1 : 0;
    }
    if (direct) return at::Tensor(at::detail::empty_cuda(size, dt, device, std::nullopt));
    return at::empty(size, at::TensorOptions().device(device).dtype(dt));
  }
};

bool modes_active() { return c10::impl::dispatch_mode_enabled() || at::impl::torch_function_mode_enabled(); }

bool integer(PyObject* o, long long& v) {
  if (!PyLong_Check(o)) return false;
  int overflow = 0;
  v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}
bool int32(PyObject* o, int32_t& v) {
  long long x;
  if (!integer(o, x) || x < INT32_MIN || x > INT32_MAX) return false;
  v = (int32_t)x;
  return true;
}
bool fits(int64_t a) { return a <= INT32_MAX; }
bool is_i8(const at::Tensor* t) { return t->scalar_type() == at::kChar; }
bool is_f8(const at::Tensor* t) { return t->scalar_type() == at::kFloat8_e4m3fn || t->scalar_type() == at::kByte; }
bool operand(bool fp8, const at::Tensor* t) { return fp8 ? is_f8(t) : is_i8(t); }
template <typename T>
T* ptr(const at::Tensor& t) { return static_cast<T*>(t.data_ptr()); }
template <typename T>
T* ptr(const at::Tensor* t) { return t ? static_cast<T*>(t->data_ptr()) : nullptr; }

// The library call without the interpreter lock (as ctypes makes it).  Its arguments are values that the caller made with the
// lock held: taking a tensor's data pointer can allocate and throw (copy-on-write), the entry points do neither.
template <typename Fn, typename... A>
int32_t call(Fn fn, A... a) {
  int32_t rc;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(a...);
  Py_END_ALLOW_THREADS
  return rc;
}
// What the library refuses is refused: the package's own `check` raises.  (Not None: the Python function would allocate, print
// and launch once more.)
PyObject* refused(int32_t rc, const char* what) {
  PyObject* r = PyObject_CallFunction(g_check, "is", (int)rc, what);
  if (r) {
    Py_DECREF(r);
    PyErr_SetString(PyExc_SystemError, "gigaslop_b200: check accepted an error status");
  }
  return nullptr;
}

PyObject* wrap(const at::Tensor& t) { return THPVariable_Wrap(t); }
// The result tensor as Python hands it out: the caller's own object if one was given.
PyObject* result(PyObject* given, const at::Tensor& t) {
  if (given == Py_None) return wrap(t);
  Py_INCREF(given);
  return given;
}
PyObject* pair(PyObject* a, PyObject* b) {
  if (!a || !b) { Py_XDECREF(a); Py_XDECREF(b); return nullptr; }
  PyObject* r = PyTuple_New(2);
  if (!r) { Py_DECREF(a); Py_DECREF(b); return nullptr; }
  PyTuple_SET_ITEM(r, 0, a);
  PyTuple_SET_ITEM(r, 1, b);
  return r;
}

#define SLOW_UNLESS(cond) do { if (!(cond)) Py_RETURN_NONE; } while (0)
#define CHECK(rc, what) do { const int32_t rc_ = (rc); if (rc_ != 0) return refused(rc_, what); } while (0)
#define OPERATOR(name, n)                                                       \
  PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t nargs) {             \
    HANDLE_TH_ERRORS                                                            \
    SLOW_UNLESS(nargs == (n) && !modes_active());                               \
    Call c;
#define OPERATOR_END END_HANDLE_TH_ERRORS }

// (kind, x, out, out_scale): kind 0 = int8, 1 = E4M3 kernel formulation, 2 = E4M3 torch formulation
OPERATOR(quantize, 4)
  long long kind;
  const at::Tensor *x, *q0, *s0;
  SLOW_UNLESS(integer(a[0], kind) && c.rows(a[1], x) && c.out_rows(a[2], q0) && c.optional(a[3], s0));
  const bool f16 = x->scalar_type() == at::kHalf;
  SLOW_UNLESS((f16 || x->scalar_type() == at::kFloat) && fits(x->size(1)));
  const int64_t M = x->size(0), K = x->size(1);
  const at::Tensor q = q0 ? *q0 : c.empty({M, K}, kind == 0 ? at::kChar : at::kFloat8_e4m3fn);
  const at::Tensor s = s0 ? *s0 : c.empty({M}, at::kFloat);
  const int32_t dt = f16 ? GSB200_F16 : GSB200_F32;
  const gsb200_stream_t st = c.stream();
  const int32_t rc = kind == 0
      ? call(ENTRY(PTQ_INT8, gsb200_ptq_int8), x->data_ptr(), dt, x->stride(0), ptr<int8_t>(q), q.stride(0), ptr<float>(s), M, (int32_t)K, st)
      : call(ENTRY(PTQ_FP8, gsb200_ptq_fp8), x->data_ptr(), dt, x->stride(0), ptr<uint8_t>(q), q.stride(0), ptr<float>(s), M, (int32_t)K,
             kind == 2, st);
  CHECK(rc, kind == 0 ? "quantize_tensor" : "fp8_quantize_per_token");
  return pair(result(a[2], q), result(a[3], s));
OPERATOR_END

// (x, out, out_scale)
OPERATOR(quantize_mx, 3)
  const at::Tensor *x, *q0, *s0;
  SLOW_UNLESS(c.rows(a[0], x) && c.out_rows(a[1], q0) && c.out_rows(a[2], s0));
  const bool f16 = x->scalar_type() == at::kHalf;
  SLOW_UNLESS((f16 || x->scalar_type() == at::kFloat) && fits(x->size(1)));
  const int64_t M = x->size(0), K = x->size(1);
  const at::Tensor q = q0 ? *q0 : c.empty({M, K}, at::kFloat8_e4m3fn);
  const at::Tensor s = s0 ? *s0 : c.empty({M, K / 32}, at::kByte);
  const gsb200_stream_t st = c.stream();
  CHECK(call(ENTRY(PTQ_MXFP8, gsb200_ptq_mxfp8), x->data_ptr(), f16 ? GSB200_F16 : GSB200_F32, x->stride(0), ptr<uint8_t>(q),
             q.stride(0), ptr<uint8_t>(s), s.stride(0), M, (int32_t)K, st), "mxfp8_quantize");
  return pair(result(a[1], q), result(a[2], s));
OPERATOR_END

// (fp8, A, B, scale_a, scale_b, out, flags)
OPERATOR(gemm, 7)
  long long fp8;
  const at::Tensor *A, *B, *sa, *sb, *C0;
  int32_t flags;
  SLOW_UNLESS(integer(a[0], fp8) && c.rows(a[1], A) && c.rows(a[2], B) && c.tensor(a[3], sa) && c.tensor(a[4], sb) && c.out_rows(a[5], C0) && int32(a[6], flags));
  SLOW_UNLESS(operand(fp8, A) && operand(fp8, B) && A->size(1) == B->size(1) && fits(B->size(0)) && fits(A->size(1)));
  const int64_t M = A->size(0), N = B->size(0), K = A->size(1);
  const at::Tensor C = C0 ? *C0 : c.empty({M, N}, at::kHalf);
  const gsb200_stream_t st = c.stream();
  const int32_t rc = fp8
      ? call(ENTRY(GEMM_FP8, gsb200_gemm_fp8_f16), ptr<uint8_t>(A), A->stride(0), ptr<uint8_t>(B), B->stride(0), C.data_ptr(), C.stride(0),
             ptr<float>(sa), ptr<float>(sb), M, (int32_t)N, (int32_t)K, flags, st)
      : call(ENTRY(GEMM_I8, gsb200_gemm_i8_f16), ptr<int8_t>(A), A->stride(0), ptr<int8_t>(B), B->stride(0), C.data_ptr(), C.stride(0),
             ptr<float>(sa), ptr<float>(sb), M, (int32_t)N, (int32_t)K, flags, st);
  CHECK(rc, fp8 ? "gemm_fp8" : "gemm_i8");
  return result(a[5], C);
OPERATOR_END

// (fp8, A, B, scale_a, scale_b, sin, cos, nhead, head_dim, rotary_dim, seqlen, row_offset, out, flags)
OPERATOR(rotary, 14)
  long long fp8, row_offset;
  const at::Tensor *A, *B, *sa, *sb, *sn, *cs, *C0;
  int32_t nhead, head_dim, rotary_dim, seqlen, flags;
  SLOW_UNLESS(integer(a[0], fp8) && c.rows(a[1], A) && c.rows(a[2], B) && c.tensor(a[3], sa) && c.tensor(a[4], sb) && c.tensor(a[5], sn) && c.tensor(a[6], cs));
  SLOW_UNLESS(int32(a[7], nhead) && int32(a[8], head_dim) && int32(a[9], rotary_dim) && int32(a[10], seqlen) && integer(a[11], row_offset) &&
              c.out_rows(a[12], C0) && int32(a[13], flags));
  SLOW_UNLESS(operand(fp8, A) && operand(fp8, B) && A->size(1) == B->size(1) && fits(B->size(0)) && fits(A->size(1)));
  SLOW_UNLESS(sn->scalar_type() == at::kFloat && sn->is_contiguous() && cs->is_contiguous() && sn->dim() >= 2 && rotary_dim >= 0 &&
              sn->size(0) >= seqlen && sn->size(1) == rotary_dim / 2);
  const int64_t M = A->size(0), N = B->size(0), K = A->size(1);
  const at::Tensor C = C0 ? *C0 : c.empty({M, N}, at::kHalf);
  const gsb200_stream_t st = c.stream();
  const int32_t rc = fp8
      ? call(ENTRY(ROT_FP8, gsb200_gemm_fp8_rotary_f16), ptr<uint8_t>(A), A->stride(0), ptr<uint8_t>(B), B->stride(0), C.data_ptr(), C.stride(0),
             ptr<float>(sa), ptr<float>(sb), ptr<float>(sn), ptr<float>(cs), M, (int32_t)N, (int32_t)K, nhead, head_dim, rotary_dim, seqlen,
             row_offset, flags, st)
      : call(ENTRY(ROT_I8, gsb200_gemm_i8_rotary_f16), ptr<int8_t>(A), A->stride(0), ptr<int8_t>(B), B->stride(0), C.data_ptr(), C.stride(0),
             ptr<float>(sa), ptr<float>(sb), ptr<float>(sn), ptr<float>(cs), M, (int32_t)N, (int32_t)K, nhead, head_dim, rotary_dim, seqlen,
             row_offset, flags, st);
  CHECK(rc, fp8 ? "gemm_fp8_rotary" : "gemm_i8_rotary");
  return result(a[12], C);
OPERATOR_END

// (fp8, A, B_gate, B_up, scale_a, scale_b_gate, scale_b_up, out, flags)
OPERATOR(dual, 9)
  long long fp8;
  const at::Tensor *A, *G, *U, *sa, *sg, *su, *C0;
  int32_t flags;
  SLOW_UNLESS(integer(a[0], fp8) && c.rows(a[1], A) && c.rows(a[2], G) && c.rows(a[3], U) && c.tensor(a[4], sa) && c.tensor(a[5], sg) &&
              c.tensor(a[6], su) && c.out_rows(a[7], C0) && int32(a[8], flags));
  SLOW_UNLESS(operand(fp8, A) && operand(fp8, G) && operand(fp8, U) && A->size(1) == G->size(1) && G->sizes() == U->sizes() &&
              G->stride(0) == U->stride(0) && fits(G->size(0)) && fits(A->size(1)));
  const int64_t M = A->size(0), N = G->size(0), K = A->size(1);
  const at::Tensor C = C0 ? *C0 : c.empty({M, N}, at::kHalf);
  const gsb200_stream_t st = c.stream();
  const int32_t rc = fp8
      ? call(ENTRY(DUAL_FP8, gsb200_dual_gemm_fp8_silu_f16), ptr<uint8_t>(A), A->stride(0), ptr<uint8_t>(G), ptr<uint8_t>(U), G->stride(0),
             C.data_ptr(), C.stride(0), ptr<float>(sa), ptr<float>(sg), ptr<float>(su), M, (int32_t)N, (int32_t)K, flags, st)
      : call(ENTRY(DUAL_I8, gsb200_dual_gemm_i8_silu_f16), ptr<int8_t>(A), A->stride(0), ptr<int8_t>(G), ptr<int8_t>(U), G->stride(0),
             C.data_ptr(), C.stride(0), ptr<float>(sa), ptr<float>(sg), ptr<float>(su), M, (int32_t)N, (int32_t)K, flags, st);
  CHECK(rc, fp8 ? "dual_gemm_fp8_silu" : "dual_gemm_i8_silu");
  return result(a[7], C);
OPERATOR_END

// (A, B_gate, B_up, scale_a, scale_b_gate, scale_b_up, out, out_scale, flags)
OPERATOR(dual_mx, 9)
  const at::Tensor *A, *G, *U, *sa, *sg, *su, *q0, *s0;
  int32_t flags;
  SLOW_UNLESS(c.rows(a[0], A) && c.rows(a[1], G) && c.rows(a[2], U) && c.tensor(a[3], sa) && c.tensor(a[4], sg) && c.tensor(a[5], su) &&
              c.out_rows(a[6], q0) && c.out_rows(a[7], s0) && int32(a[8], flags));
  SLOW_UNLESS(is_f8(A) && is_f8(G) && is_f8(U) && A->size(1) == G->size(1) && G->sizes() == U->sizes() && G->stride(0) == U->stride(0) &&
              fits(G->size(0)) && fits(A->size(1)));
  const int64_t M = A->size(0), N = G->size(0), K = A->size(1);
  const at::Tensor q = q0 ? *q0 : c.empty({M, N}, at::kFloat8_e4m3fn);
  const at::Tensor s = s0 ? *s0 : c.empty({M, N / 32}, at::kByte);
  const gsb200_stream_t st = c.stream();
  CHECK(call(ENTRY(DUAL_FP8_MX, gsb200_dual_gemm_fp8_silu_mxfp8), ptr<uint8_t>(A), A->stride(0), ptr<uint8_t>(G), ptr<uint8_t>(U),
             G->stride(0), ptr<uint8_t>(q), q.stride(0), ptr<uint8_t>(s), s.stride(0), ptr<float>(sa), ptr<float>(sg),
             ptr<float>(su), M, (int32_t)N, (int32_t)K, flags, st), "dual_gemm_fp8_silu_mxfp8");
  return pair(result(a[6], q), result(a[7], s));
OPERATOR_END

// (scales, K)
OPERATOR(mx_tile, 2)
  const at::Tensor* s;
  int32_t K;
  SLOW_UNLESS(c.tensor(a[0], s) && s->dim() >= 1 && int32(a[1], K));
  const int64_t bytes = ENTRY(MX_BYTES, gsb200_mx_tiled_scale_bytes)(s->size(0), K);
  SLOW_UNLESS(bytes >= 0);
  const at::Tensor out = c.empty({bytes}, at::kByte);
  const gsb200_stream_t st = c.stream();
  CHECK(call(ENTRY(MX_TILE, gsb200_mx_scales_to_tiled), ptr<uint8_t>(s), s->stride(0), s->size(0), K, ptr<uint8_t>(out), st), "mx_scales_to_tiled");
  return wrap(out);
OPERATOR_END

// (A, sfa_tiled, B, sfb_tiled, out)
OPERATOR(mx_gemm, 5)
  const at::Tensor *A, *sfa, *B, *sfb, *C0;
  SLOW_UNLESS(c.rows(a[0], A) && c.tensor(a[1], sfa) && c.rows(a[2], B) && c.tensor(a[3], sfb) && c.out_rows(a[4], C0));
  SLOW_UNLESS(is_f8(A) && is_f8(B) && A->size(1) == B->size(1) && fits(B->size(0)) && fits(A->size(1)));
  const int64_t M = A->size(0), N = B->size(0), K = A->size(1);
  const at::Tensor C = C0 ? *C0 : c.empty({M, N}, at::kHalf);
  const gsb200_stream_t st = c.stream();
  CHECK(call(ENTRY(MX_GEMM, gsb200_gemm_mxfp8_f16), ptr<uint8_t>(A), A->stride(0), ptr<uint8_t>(sfa), ptr<uint8_t>(B), B->stride(0),
             ptr<uint8_t>(sfb), C.data_ptr(), C.stride(0), M, (int32_t)N, (int32_t)K, st), "gemm_mxfp8");
  return result(a[4], C);
OPERATOR_END

// (A, sfa_tiled, B_gate, B_up, sfb_gate_tiled, sfb_up_tiled, out)
OPERATOR(mx_dual, 7)
  const at::Tensor *A, *sfa, *G, *U, *sg, *su, *C0;
  SLOW_UNLESS(c.rows(a[0], A) && c.tensor(a[1], sfa) && c.rows(a[2], G) && c.rows(a[3], U) && c.tensor(a[4], sg) && c.tensor(a[5], su) && c.out_rows(a[6], C0));
  SLOW_UNLESS(is_f8(A) && is_f8(G) && is_f8(U) && A->size(1) == G->size(1) && G->sizes() == U->sizes() && G->stride(0) == U->stride(0) &&
              fits(G->size(0)) && fits(A->size(1)));
  const int64_t M = A->size(0), N = G->size(0), K = A->size(1);
  const at::Tensor C = C0 ? *C0 : c.empty({M, N}, at::kHalf);
  const gsb200_stream_t st = c.stream();
  CHECK(call(ENTRY(MX_DUAL, gsb200_dual_gemm_mxfp8_silu_f16), ptr<uint8_t>(A), A->stride(0), ptr<uint8_t>(sfa), ptr<uint8_t>(G),
             ptr<uint8_t>(U), G->stride(0), ptr<uint8_t>(sg), ptr<uint8_t>(su), C.data_ptr(), C.stride(0), M, (int32_t)N, (int32_t)K,
             st), "dual_gemm_mxfp8_silu");
  return result(a[6], C);
OPERATOR_END

// (x, scale_x, dn, scale_dn, up, bias, out)
OPERATOR(fac_gemm, 7)
  const at::Tensor *x, *sx, *dn, *sdn, *up, *bias, *C0;
  SLOW_UNLESS(c.rows(a[0], x) && c.tensor(a[1], sx) && c.rows(a[2], dn) && c.tensor(a[3], sdn) && c.rows(a[4], up) && c.tensor(a[5], bias) && c.out_rows(a[6], C0));
  SLOW_UNLESS(x->scalar_type() == at::kFloat8_e4m3fn && dn->scalar_type() == at::kFloat8_e4m3fn && up->scalar_type() == at::kHalf);
  const int64_t M = x->size(0), Cc = x->size(1), R = dn->size(0), N = up->size(0);
  SLOW_UNLESS(dn->size(1) == Cc && up->size(1) == R && bias->numel() == N && sx->numel() == M && fits(Cc) && fits(R) && fits(N));
  const at::Tensor C = C0 ? *C0 : c.empty({M, N}, at::kHalf);
  const gsb200_stream_t st = c.stream();
  CHECK(call(ENTRY(FAC_GEMM, gsb200_fac_gemm_fp8_f16), ptr<uint8_t>(x), x->stride(0), ptr<float>(sx), ptr<uint8_t>(dn),
             dn->stride(0), ptr<float>(sdn), up->data_ptr(), up->stride(0), ptr<float>(bias), C.data_ptr(), C.stride(0), M,
             (int32_t)Cc, (int32_t)R, (int32_t)N, st), "fp8_factored_gemm");
  return result(a[6], C);
OPERATOR_END

// (h_fp8_out, c_inout, hh_down, up_hh, bias_hh, x_down, up_ih, bias_ih) -> True
OPERATOR(fac_step, 8)
  const at::Tensor *h, *cc, *hh, *uhh, *bhh, *xd, *uih, *bih;
  SLOW_UNLESS(c.tensor(a[0], h) && c.tensor(a[1], cc) && c.tensor(a[2], hh) && c.tensor(a[3], uhh) && c.optional(a[4], bhh) && c.tensor(a[5], xd) &&
              c.tensor(a[6], uih) && c.optional(a[7], bih));
  SLOW_UNLESS(hh->dim() == 2 && uhh->dim() >= 1 && xd->dim() >= 2 && h->is_contiguous() && cc->is_contiguous() && hh->is_contiguous() &&
              uhh->is_contiguous() && xd->is_contiguous() && uih->is_contiguous());
  const int64_t B = hh->size(0), K = hh->size(1), H = uhh->size(0) / 4, R = xd->size(1);
  SLOW_UNLESS(fits(K) && fits(H) && fits(R));
  const gsb200_stream_t st = c.stream();
  CHECK(call(ENTRY(FAC_STEP, gsb200_factored_lstm_step), ptr<uint8_t>(h), ptr<float>(cc), hh->data_ptr(), uhh->data_ptr(),
             ptr<float>(bhh), xd->data_ptr(), uih->data_ptr(), ptr<float>(bih), B, (int32_t)H, (int32_t)K, (int32_t)R, st), "factored_lstm_step");
  Py_RETURN_TRUE;
OPERATOR_END

// bind(addresses, check): the entry points' addresses in the order of `Entry`, and what turns a status into an exception
PyObject* bind(PyObject*, PyObject* args) {
  PyObject *seq, *check;
  if (!PyArg_ParseTuple(args, "OO:bind", &seq, &check)) return nullptr;
  PyObject* f = PySequence_Fast(seq, "bind takes a sequence of addresses");
  if (!f) return nullptr;
  if (PySequence_Fast_GET_SIZE(f) != N_ENTRIES) {
    Py_DECREF(f);
    PyErr_SetString(PyExc_ValueError, "bind: wrong number of entry points");
    return nullptr;
  }
  for (int i = 0; i < N_ENTRIES; ++i) {
    g_entry[i] = PyLong_AsVoidPtr(PySequence_Fast_GET_ITEM(f, i));
    if (PyErr_Occurred()) { Py_DECREF(f); return nullptr; }
  }
  Py_DECREF(f);
  Py_INCREF(check);
  Py_XDECREF(g_check);
  g_check = check;
  Py_RETURN_NONE;
}

#define METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, nullptr}, METHOD(quantize), METHOD(quantize_mx), METHOD(gemm), METHOD(rotary), METHOD(dual),
                         METHOD(dual_mx), METHOD(mx_tile), METHOD(mx_gemm), METHOD(mx_dual), METHOD(fac_gemm), METHOD(fac_step),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
  PyObject* m = PyModule_Create(&module);
  // (the loader compares it before the first call)
  if (m && PyModule_AddStringConstant(m, "TARGET", GSB200_NATIVE_TARGET) != 0) { Py_DECREF(m); return nullptr; }
  return m;
}
