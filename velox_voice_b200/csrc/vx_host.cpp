// Native host path of the Python operators: argument checks, output allocation and the C-ABI calls of one
// operator in one C++ function, called from Python through the vectorcall protocol.
//
// Why it exists: the kernels of a short call (a streaming chunk, an utterance) run for 3-10 us, while the same
// call through ctypes spent 15-25 us per launch in Python (descriptor fields, torch.empty, data_ptr, stream
// look-up).  Here an operator costs its allocations (about 0.5 us each) and its launches (about 2 us each).
//
// Every function covers the ordinary call (CUDA tensors, unit column stride, matching shapes) and returns None for
// anything else; the Python operator then takes its general route, which copies where a copy is needed and words the
// errors.  So no check is weaker than before, and results do not depend on the route.
//
// The C-ABI entry points are taken from the library that ctypes loaded (init(path)); nothing is linked against it.

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <atomic>
#include <string>
#include <vector>

#include "../../include/velox_b200.h"

namespace {

#define VX_FUNCS(X)                                                                                                 \
  X(vx_last_error) X(vx_quantize_pack) X(vx_ln_quantize_pack) X(vx_ln2_quantize_pack) X(vx_amax) X(vx_bsgemm)        \
  X(vx_bsgemm_natural_sf_supported) X(vx_bsgemm_residual_ln_supported) X(vx_bsgemm_residual_ln) X(vx_bsgemm_residual_ln2) X(vx_argmax_ids) X(vx_relpos_attention)   \
  X(vx_power_mel_log) X(vx_power_mel_log_supported) X(vx_sf_from_natural_pair) X(vx_rowscale_linear) X(vx_rowscale_linear_scratch) X(vx_ctc_topk_rows) X(vx_ctc_topk)        \
  X(vx_conformer_pass_supported) X(vx_conformer_pass_scratch) X(vx_conformer_pass)
struct Api {
#define X(f) decltype(&::f) f = nullptr;
  VX_FUNCS(X)
#undef X
} g;

PyObject* g_error = nullptr;      // VeloxError
PyObject* g_quantized = nullptr;  // class Quantized
PyObject *s_fmt, *s_rows, *s_k, *s_codes, *s_scales, *s_sf, *s_amax, *s_q, *s_bias;
std::atomic<int64_t> g_launches{0};

void count(int64_t n = 1) { g_launches.fetch_add(n, std::memory_order_relaxed); }

struct PyFail {};                           // a Python error is set
struct CallFail { int rc; const char* what; };  // a C-ABI call failed on this thread

void check(int rc, const char* what) {
  if (rc != 0) throw CallFail{rc, what};
}
void set_error(const CallFail& f) {
  if (f.rc < 0) PyErr_Format(g_error, "%s: argument error: %s", f.what, g.vx_last_error());
  else PyErr_Format(g_error, "%s: CUDA error %d: %s", f.what, f.rc, g.vx_last_error());
}

// Allocations and launches run without the interpreter lock: a launch blocks while the stream's queue is full, and an
// allocation may wait for the device.  No Python object is touched in its scope; tensors that come out of Python objects
// other threads may change (the fields of a Quantized, a plan's layers) are held by value.
struct NoGil {
  PyThreadState* const state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

// ---------------------------------------------------------------- small helpers
at::Tensor empty(at::IntArrayRef size, at::ScalarType dt, const at::Device& dev) {
  return at::Tensor(at::detail::empty_cuda(size, dt, dev, std::nullopt));
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

bool is_cuda_tensor(PyObject* o) { return THPVariable_Check(o) && THPVariable_Unpack(o).is_cuda(); }
int dtype_code(const at::Tensor& t) {
  if (t.scalar_type() == at::kFloat) return VX_F32;
  if (t.scalar_type() == at::kBFloat16) return VX_BF16;
  return -1;
}
bool rows2d(const at::Tensor& t) { return t.dim() == 2 && t.stride(1) == 1; }
bool has_sf(int fmt) { return fmt >= VX_FMT_BLK16_A && fmt <= VX_FMT_NV16; }
int fmt_block(int fmt) { return fmt == VX_FMT_MX32 ? 32 : (fmt == VX_FMT_FP8_1X128 ? 128 : 16); }
int64_t kgroups(int fmt, int64_t K) { return (K + 255) / 256 * (fmt == VX_FMT_MX32 ? 2 : 4); }
int64_t sf_bytes(int fmt, int64_t M, int64_t K) { return (M + 127) / 128 * kgroups(fmt, K) * 512; }

// fp32 vector of at least n contiguous entries on `dev`
bool vector_ok(const at::Tensor& t, int64_t n, const at::Device& dev) {
  return t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel() >= n && t.device() == dev;
}
// optional fp32 vector argument: its pointer, or sets `ok` to false when the general route has to look at it
const float* f32_ptr(const at::Tensor& t) { return t.defined() ? static_cast<const float*>(t.data_ptr()) : nullptr; }
const float* vector_arg(PyObject* o, int64_t n, const at::Device& dev, bool& ok) {
  if (o == Py_None) return nullptr;
  if (!is_cuda_tensor(o)) { ok = false; return nullptr; }
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!vector_ok(t, n, dev)) { ok = false; return nullptr; }
  return static_cast<const float*>(t.data_ptr());
}

PyObject* wrap(const at::Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}

struct Outputs {
  at::Tensor codes, scales, sf;
};
Outputs alloc_outputs(int fmt, int64_t M, int64_t K, const at::Device& dev, bool natural, bool sf) {
  Outputs o;
  const bool fp8 = fmt == VX_FMT_FP8_1X128;
  o.codes = empty({M, fp8 ? K : K / 2}, at::kByte, dev);
  if (natural) {
    if (fmt == VX_FMT_ROWSCALE) o.scales = empty({M}, at::kByte, dev);
    else if (fmt == VX_FMT_BLK16_A) o.scales = empty({K / 16, M / 2}, at::kByte, dev);
    else if (fmt == VX_FMT_BLK16_B) o.scales = empty({K / 16, M}, at::kByte, dev);
    else if (fp8) o.scales = empty({M, K / 128}, at::kFloat, dev);
    else o.scales = empty({M, K / fmt_block(fmt)}, at::kByte, dev);
  }
  if (sf && has_sf(fmt)) o.sf = empty({(M + 127) / 128, kgroups(fmt, K), 512}, at::kByte, dev);
  return o;
}
void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

PyObject* make_quantized(int fmt, int64_t M, int64_t K, const Outputs& o, PyObject* amax) {
  PyObject* a[7] = {PyLong_FromLong(fmt), PyLong_FromLongLong(M), PyLong_FromLongLong(K), wrap(o.codes), wrap(o.scales), wrap(o.sf),
                    Py_NewRef(amax)};
  PyObject* r = PyObject_Vectorcall(g_quantized, a, 7, nullptr);
  for (PyObject* p : a) Py_XDECREF(p);
  return r;
}

// One GEMM operand out of a Python `Quantized`
struct Operand {
  int fmt = -1;
  int64_t rows = 0, k = 0;
  at::Tensor codes, scales, amax;
};
// false: not an ordinary operand (the general route decides what it is)
bool read_operand(PyObject* o, Operand& r) {
  if (reinterpret_cast<PyObject*>(Py_TYPE(o)) != g_quantized) return false;
  auto get = [&](PyObject* name) {
    PyObject* v = PyObject_GetAttr(o, name);
    if (!v) throw PyFail{};
    Py_DECREF(v);  // (the instance keeps it alive until the tensor in it has been taken)
    return v;
  };
  r.fmt = static_cast<int>(PyLong_AsLong(get(s_fmt)));
  r.rows = PyLong_AsLongLong(get(s_rows));
  r.k = PyLong_AsLongLong(get(s_k));
  if (PyErr_Occurred()) throw PyFail{};
  PyObject* c = get(s_codes);
  PyObject* s = get(has_sf(r.fmt) ? s_sf : s_scales);
  if (!is_cuda_tensor(c) || !is_cuda_tensor(s)) return false;
  r.codes = THPVariable_Unpack(c);
  r.scales = THPVariable_Unpack(s);
  if (r.codes.dim() != 2) return false;
  if (r.fmt == VX_FMT_NV16) {
    PyObject* a = get(s_amax);
    if (!is_cuda_tensor(a)) return false;
    r.amax = THPVariable_Unpack(a);
  }
  return true;
}
bool operands(PyObject* pa, PyObject* pb, Operand& a, Operand& b, vx_gemm_desc& d) {
  if (!read_operand(pa, a) || !read_operand(pb, b)) return false;
  if (a.fmt == VX_FMT_BLK16_A ? b.fmt != VX_FMT_BLK16_B : a.fmt != b.fmt) return false;
  if (a.k != b.k || a.codes.device() != b.codes.device()) return false;
  d = vx_gemm_desc{};
  d.struct_size = sizeof(vx_gemm_desc);
  d.fmt = a.fmt;
  d.M = a.rows; d.N = b.rows; d.K = a.k;
  d.a_codes = a.codes.data_ptr(); d.lda = a.codes.stride(0);
  d.b_codes = b.codes.data_ptr(); d.ldb = b.codes.stride(0);
  d.a_scales = a.scales.data_ptr(); d.b_scales = b.scales.data_ptr();
  d.a_amax = f32_ptr(a.amax); d.b_amax = f32_ptr(b.amax);
  return true;
}

long as_long(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyFail{};
  return v;
}
bool as_bool(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PyFail{};
  return v != 0;
}
double as_double(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyFail{};
  return v;
}

#define VX_BEGIN                                                    \
  HANDLE_TH_ERRORS                                                  \
  try {
#define VX_END                                                      \
  } catch (const PyFail&) {                                         \
    return nullptr;                                                 \
  } catch (const CallFail& f) {                                     \
    set_error(f);                                                   \
    return nullptr;                                                 \
  }                                                                 \
  END_HANDLE_TH_ERRORS
#define VX_ARGS(n)                                                                   \
  if (nargs != (n)) {                                                                \
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", (n), nargs);     \
    return nullptr;                                                                  \
  }

// ---------------------------------------------------------------- quantizers
at::Tensor tensor_amax(const at::Tensor& x, int dt) {
  at::Tensor am = empty({1}, at::kFloat, x.device());
  check(g.vx_amax(x.data_ptr(), dt, x.size(0), x.size(1), x.stride(0), static_cast<float*>(am.data_ptr()), stream()), "vx_amax");
  count();
  return am;
}

// quantize(x, fmt, natural, sf, amax | None) -> Quantized | None
PyObject* py_quantize(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(5)
  if (!is_cuda_tensor(a[0])) Py_RETURN_NONE;
  const at::Tensor& x = THPVariable_Unpack(a[0]);
  const int dt = dtype_code(x), fmt = static_cast<int>(as_long(a[1]));
  if (dt < 0 || !rows2d(x)) Py_RETURN_NONE;
  const bool natural = as_bool(a[2]) || fmt == VX_FMT_ROWSCALE || fmt == VX_FMT_FP8_1X128;
  const int64_t M = x.size(0), K = x.size(1);
  const bool sf = as_bool(a[3]), measure = fmt == VX_FMT_NV16 && a[4] == Py_None;
  at::Tensor amax;
  if (fmt == VX_FMT_NV16 ? !measure && !is_cuda_tensor(a[4]) : a[4] != Py_None) Py_RETURN_NONE;
  if (fmt == VX_FMT_NV16 && !measure) amax = THPVariable_Unpack(a[4]);
  Outputs o;
  {
    NoGil nogil;
    if (measure) amax = tensor_amax(x, dt);
    o = alloc_outputs(fmt, M, K, x.device(), natural, sf);
    check(g.vx_quantize_pack(x.data_ptr(), dt, M, K, x.stride(0), fmt, ptr(o.codes), o.codes.stride(0), ptr(o.scales), ptr(o.sf),
                             f32_ptr(amax), stream()),
          "vx_quantize_pack");
    count();
  }
  if (!measure) return make_quantized(fmt, M, K, o, a[4]);
  PyObject* made = wrap(amax);
  PyObject* r = make_quantized(fmt, M, K, o, made);
  Py_XDECREF(made);
  return r;
  VX_END
}

// ln_quantize(x, gamma, beta, eps, fmt, natural, sf, amax | None) -> Quantized | None
PyObject* py_ln_quantize(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(8)
  if (!is_cuda_tensor(a[0])) Py_RETURN_NONE;
  const at::Tensor& x = THPVariable_Unpack(a[0]);
  const int dt = dtype_code(x), fmt = static_cast<int>(as_long(a[4]));
  if (dt < 0 || !rows2d(x)) Py_RETURN_NONE;
  const int64_t M = x.size(0), K = x.size(1);
  bool ok = true;
  const float* gamma = vector_arg(a[1], K, x.device(), ok);
  const float* beta = vector_arg(a[2], K, x.device(), ok);
  if (!ok || !gamma || !beta) Py_RETURN_NONE;
  const float* am = nullptr;
  if (fmt == VX_FMT_NV16) {
    am = vector_arg(a[7], 1, x.device(), ok);
    if (!ok || !am) Py_RETURN_NONE;
  } else if (a[7] != Py_None) {
    Py_RETURN_NONE;
  }
  const bool natural = as_bool(a[5]) || fmt == VX_FMT_ROWSCALE || fmt == VX_FMT_FP8_1X128;
  const bool sf = as_bool(a[6]);
  const float eps = static_cast<float>(as_double(a[3]));
  Outputs o;
  {
    NoGil nogil;
    o = alloc_outputs(fmt, M, K, x.device(), natural, sf);
    check(g.vx_ln_quantize_pack(x.data_ptr(), dt, M, K, x.stride(0), gamma, beta, eps, fmt, ptr(o.codes), o.codes.stride(0), ptr(o.scales),
                                ptr(o.sf), am, nullptr, 0, K, stream()),
          "vx_ln_quantize_pack");
    count();
  }
  return make_quantized(fmt, M, K, o, a[7]);
  VX_END
}

// ---------------------------------------------------------------- GEMMs
// A [M, n] output; 16-bit rows are padded to a pitch of 16 bytes so that the TMA store path applies.
at::Tensor new_out(int64_t M, int64_t n, at::ScalarType dt, const at::Device& dev) {
  if (dt == at::kBFloat16 && n % 8 != 0)
    return at::Tensor(at::detail::empty_strided_cuda({M, n}, {(n + 7) / 8 * 8, 1}, dt, dev));
  return empty({M, n}, dt, dev);
}

void launch(const vx_gemm_desc& d) {
  check(g.vx_bsgemm(&d, stream()), "vx_bsgemm");
  count();
}

// bsgemm(a, b, epilogue, bias, residual, alpha, out_dtype, out, out_fmt, out_amax, out_natural, flags)
//   -> Tensor | Quantized | None
PyObject* py_bsgemm(PyObject*, PyObject* const* p, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(12)
  Operand a, b;
  vx_gemm_desc d;
  if (!operands(p[0], p[1], a, b, d)) Py_RETURN_NONE;
  const at::Device dev = a.codes.device();
  bool ok = true;
  d.bias = vector_arg(p[3], d.N, dev, ok);
  if (!ok) Py_RETURN_NONE;
  d.epilogue = static_cast<int>(as_long(p[2]));
  const int64_t n_out = d.epilogue == VX_EPI_BIAS_GLU ? d.N / 2 : d.N;
  if (d.epilogue == VX_EPI_BIAS_RESIDUAL) {
    if (!is_cuda_tensor(p[4])) Py_RETURN_NONE;
    const at::Tensor& r = THPVariable_Unpack(p[4]);
    if (!rows2d(r) || r.size(0) != d.M || r.size(1) != d.N || r.device() != dev || dtype_code(r) < 0) Py_RETURN_NONE;
    d.residual = r.data_ptr(); d.residual_dtype = dtype_code(r); d.ldr = r.stride(0);
    d.alpha = static_cast<float>(as_double(p[5]));
  }
  d.flags = static_cast<int>(as_long(p[11]));
  if (p[8] != Py_None) {  // re-quantized output
    const int ofmt = static_cast<int>(as_long(p[8]));
    if (ofmt == VX_FMT_NV16) {
      d.out_amax = vector_arg(p[9], 1, dev, ok);
      if (!ok || !d.out_amax) Py_RETURN_NONE;
    } else if (ofmt != VX_FMT_MX32 || p[9] != Py_None) {
      Py_RETURN_NONE;
    }
    const bool natural = as_bool(p[10]);
    Outputs o;
    {
      NoGil nogil;
      o = alloc_outputs(ofmt, d.M, n_out, dev, natural, true);
      d.out_dtype = VX_FP4; d.out = ptr(o.codes); d.ldo = o.codes.stride(0);
      d.out_fmt = ofmt; d.out_scales_sf = ptr(o.sf); d.out_scales = ptr(o.scales);
      launch(d);
    }
    return make_quantized(ofmt, d.M, n_out, o, p[9]);
  }
  if (p[7] != Py_None) {
    if (!is_cuda_tensor(p[7])) Py_RETURN_NONE;
    const at::Tensor& o = THPVariable_Unpack(p[7]);
    if (!rows2d(o) || o.size(0) != d.M || o.size(1) != n_out || o.device() != dev || dtype_code(o) < 0) Py_RETURN_NONE;
    d.out_dtype = dtype_code(o); d.out = o.data_ptr(); d.ldo = o.stride(0);
    {
      NoGil nogil;
      launch(d);
    }
    return Py_NewRef(p[7]);
  }
  if (!THPDtype_Check(p[6])) Py_RETURN_NONE;
  const at::ScalarType odt = reinterpret_cast<THPDtype*>(p[6])->scalar_type;
  if (odt != at::kFloat && odt != at::kBFloat16) Py_RETURN_NONE;
  at::Tensor o;
  {
    NoGil nogil;
    o = new_out(d.M, n_out, odt, dev);
    d.out_dtype = odt == at::kFloat ? VX_F32 : VX_BF16; d.out = o.data_ptr(); d.ldo = o.stride(0);
    launch(d);
  }
  return wrap(o);
  VX_END
}

// residual_ln(a, b, bias, residual, gamma, beta, eps, alpha, out, gamma2, beta2, flags) -> (out, Quantized) | None
PyObject* py_residual_ln(PyObject*, PyObject* const* p, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(12)
  Operand a, b;
  vx_gemm_desc d;
  if (!operands(p[0], p[1], a, b, d)) Py_RETURN_NONE;
  const at::Device dev = a.codes.device();
  bool ok = true;
  d.bias = vector_arg(p[2], d.N, dev, ok);
  const float* gamma = vector_arg(p[4], d.N, dev, ok);
  const float* beta = vector_arg(p[5], d.N, dev, ok);
  const float* gamma2 = vector_arg(p[9], d.N, dev, ok);
  const float* beta2 = vector_arg(p[10], d.N, dev, ok);
  if (!ok || !gamma || !beta || (gamma2 == nullptr) != (beta2 == nullptr) || !is_cuda_tensor(p[3])) Py_RETURN_NONE;
  const at::Tensor& r = THPVariable_Unpack(p[3]);
  if (!rows2d(r) || r.size(0) != d.M || r.size(1) != d.N || r.device() != dev || dtype_code(r) < 0) Py_RETURN_NONE;
  at::Tensor out;
  if (p[8] == Py_None) {
    NoGil nogil;
    out = empty({d.M, d.N}, at::kBFloat16, dev);
  }
  else if (is_cuda_tensor(p[8])) out = THPVariable_Unpack(p[8]);
  else Py_RETURN_NONE;
  if (!rows2d(out) || out.size(0) != d.M || out.size(1) != d.N || out.device() != dev || dtype_code(out) < 0) Py_RETURN_NONE;
  d.epilogue = VX_EPI_BIAS_RESIDUAL;
  d.residual = r.data_ptr(); d.residual_dtype = dtype_code(r); d.ldr = r.stride(0);
  d.alpha = static_cast<float>(as_double(p[7]));
  d.out_dtype = dtype_code(out); d.out = out.data_ptr(); d.ldo = out.stride(0);
  d.flags = static_cast<int>(as_long(p[11]));
  const float eps = static_cast<float>(as_double(p[6]));
  Outputs o;
  {
    NoGil nogil;
    o = alloc_outputs(VX_FMT_MX32, d.M, d.N, dev, false, true);
    if (!gamma2)
      check(g.vx_bsgemm_residual_ln(&d, gamma, beta, eps, ptr(o.codes), o.codes.stride(0), ptr(o.sf), stream()), "vx_bsgemm_residual_ln");
    else
      check(g.vx_bsgemm_residual_ln2(&d, gamma, beta, gamma2, beta2, eps, ptr(o.codes), o.codes.stride(0), ptr(o.sf), stream()),
            "vx_bsgemm_residual_ln2");
    count();
  }
  PyObject* q = make_quantized(VX_FMT_MX32, d.M, d.N, o, Py_None);
  if (!q) return nullptr;
  PyObject* pair = PyTuple_New(2);
  if (!pair) { Py_DECREF(q); return nullptr; }
  PyTuple_SET_ITEM(pair, 0, p[8] == Py_None ? wrap(out) : Py_NewRef(p[8]));
  PyTuple_SET_ITEM(pair, 1, q);
  return pair;
  VX_END
}

// rowscale_linear(x [..., K], wq [N, K/2], ws [N], bias | None) -> f32 [..., N] | None: the reference's per-row lane, one
// or two launches.
PyObject* py_rowscale_linear(PyObject*, PyObject* const* p, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(4)
  if (!is_cuda_tensor(p[0]) || !is_cuda_tensor(p[1]) || !is_cuda_tensor(p[2])) Py_RETURN_NONE;
  const at::Tensor &x = THPVariable_Unpack(p[0]), &wq = THPVariable_Unpack(p[1]), &ws = THPVariable_Unpack(p[2]);
  const at::Device dev = x.device();
  const int dt = dtype_code(x);
  if (dt < 0 || x.dim() < 1 || !x.is_contiguous() || !rows2d(wq) || wq.scalar_type() != at::kByte || ws.scalar_type() != at::kByte ||
      !ws.is_contiguous() || wq.device() != dev || ws.device() != dev)
    Py_RETURN_NONE;
  const int64_t K = x.size(-1), N = wq.size(0);
  if (K == 0 || x.numel() == 0 || wq.size(1) * 2 != K || ws.numel() < N) Py_RETURN_NONE;
  const int64_t M = x.numel() / K;
  bool ok = true;
  const float* bias = vector_arg(p[3], N, dev, ok);
  if (!ok) Py_RETURN_NONE;
  at::Tensor out;
  {
    NoGil nogil;
    const int64_t need = g.vx_rowscale_linear_scratch(M, N, K);
    at::Tensor scratch;
    if (need) scratch = empty({need}, at::kByte, dev);
    c10::SmallVector<int64_t, 8> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = N;
    out = empty(shape, at::kFloat, dev);
    check(g.vx_rowscale_linear(x.data_ptr(), dt, M, K, K, wq.data_ptr(), wq.stride(0), ws.data_ptr(), N, bias, ptr(scratch),
                               static_cast<float*>(out.data_ptr()), N, stream()),
          "vx_rowscale_linear");
    count(need ? 2 : 1);
  }
  return wrap(out);
  VX_END
}

// blkscale_gemm(pack_a, pack_b, scale_a, scale_b) -> f32 [M, N] | None: the reference's per-16 block-scaled product.  Up to one
// tile per SM the GEMM takes the scales as they are; beyond, the tensor-core copies of both operands' scales live in one
// scratch block, made by one launch.
PyObject* py_blkscale_gemm(PyObject*, PyObject* const* p, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(4)
  for (int i = 0; i < 4; ++i)
    if (!is_cuda_tensor(p[i])) Py_RETURN_NONE;
  const at::Tensor &pa = THPVariable_Unpack(p[0]), &pb = THPVariable_Unpack(p[1]);
  const at::Tensor &sa = THPVariable_Unpack(p[2]), &sb = THPVariable_Unpack(p[3]);
  const at::Device dev = pa.device();
  if (!rows2d(pa) || !rows2d(pb) || pa.size(1) != pb.size(1) || pb.device() != dev) Py_RETURN_NONE;
  const int64_t M = pa.size(0), N = pb.size(0), K = pa.size(1) * 2;
  if (M == 0 || N == 0 || K == 0 || M % 2 || K % 16) Py_RETURN_NONE;
  for (const at::Tensor* s : {&sa, &sb})
    if (s->scalar_type() != at::kByte || !s->is_contiguous() || s->device() != dev) Py_RETURN_NONE;
  if (sa.numel() < K / 16 * (M / 2) || sb.numel() < K / 16 * N) Py_RETURN_NONE;
  at::Tensor out;
  {
    NoGil nogil;
    vx_gemm_desc d{};
    at::Tensor scratch;
    if (g.vx_bsgemm_natural_sf_supported(M, N, K)) {
      d.flags = VX_GEMM_NATURAL_SF;
      d.a_scales = sa.data_ptr(); d.b_scales = sb.data_ptr();
    } else {
      const int64_t na = sf_bytes(VX_FMT_BLK16_A, M, K), nb = sf_bytes(VX_FMT_BLK16_B, N, K);
      scratch = empty({na + nb}, at::kByte, dev);
      uint8_t* const sf = static_cast<uint8_t*>(scratch.data_ptr());
      check(g.vx_sf_from_natural_pair(VX_FMT_BLK16_A, sa.data_ptr(), M, sf, VX_FMT_BLK16_B, sb.data_ptr(), N, sf + na, K, stream()),
            "vx_sf_from_natural_pair");
      count();
      d.a_scales = sf; d.b_scales = sf + na;
    }
    out = empty({M, N}, at::kFloat, dev);
    d.struct_size = sizeof(d);
    d.fmt = VX_FMT_BLK16_A;
    d.M = M; d.N = N; d.K = K;
    d.a_codes = pa.data_ptr(); d.lda = pa.stride(0);
    d.b_codes = pb.data_ptr(); d.ldb = pb.stride(0);
    d.epilogue = VX_EPI_NONE;
    d.out_dtype = VX_F32; d.out = out.data_ptr(); d.ldo = N;
    launch(d);
  }
  return wrap(out);
  VX_END
}

// ---------------------------------------------------------------- CTC head
// topk(a, b, bias | None, k) -> (logp f32 [M, k], ids i64 [M, k]) | None.  The bf16 logits exist for a block of rows at a
// time, in one scratch block small enough to stay in L2 between the GEMM that writes it and the kernel that reads it.
PyObject* py_topk(PyObject*, PyObject* const* p, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(4)
  Operand a, b;
  vx_gemm_desc d;
  if (!operands(p[0], p[1], a, b, d) || a.fmt == VX_FMT_FP8_1X128) Py_RETURN_NONE;
  const at::Device dev = a.codes.device();
  bool ok = true;
  d.bias = vector_arg(p[2], d.N, dev, ok);
  const long k = as_long(p[3]);
  if (!ok || k < 1 || k > 16 || (d.N + 255) / 256 * 4 < k || d.M == 0) Py_RETURN_NONE;
  at::Tensor logp, ids;
  {
    NoGil nogil;
    logp = empty({d.M, k}, at::kFloat, dev);
    ids = empty({d.M, k}, at::kLong, dev);
    const int64_t rows = g.vx_ctc_topk_rows(d.N), block = rows < d.M ? rows : d.M;
    const at::Tensor scratch = empty({block, (d.N + 7) / 8 * 8}, at::kBFloat16, dev);
    check(g.vx_ctc_topk(&d, static_cast<int>(k), scratch.data_ptr(), block, static_cast<float*>(logp.data_ptr()),
                        static_cast<int64_t*>(ids.data_ptr()), stream()),
          "vx_ctc_topk");
    count(2 * ((d.M + block - 1) / block));
  }
  PyObject* pair = PyTuple_New(2);
  if (!pair) return nullptr;
  PyTuple_SET_ITEM(pair, 0, wrap(logp));
  PyTuple_SET_ITEM(pair, 1, wrap(ids));
  return pair;
  VX_END
}

// ---------------------------------------------------------------- attention
bool bf16_cube(PyObject* o, const at::Tensor** t) {
  if (!is_cuda_tensor(o)) return false;
  *t = &THPVariable_Unpack(o);
  return (*t)->scalar_type() == at::kBFloat16 && (*t)->dim() == 3 && (*t)->is_contiguous();
}

// relpos_attention(q2, k2, v2, kv_len) -> bf16 [T, h dk] | None
PyObject* py_relpos_attention(PyObject*, PyObject* const* p, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(4)
  const at::Tensor *q, *k, *v;
  if (!bf16_cube(p[0], &q) || !bf16_cube(p[1], &k) || !bf16_cube(p[2], &v)) Py_RETURN_NONE;
  if (k->sizes() != q->sizes() || v->sizes() != q->sizes() || q->size(2) != 128 || k->device() != q->device() || v->device() != q->device())
    Py_RETURN_NONE;
  const int64_t h = q->size(0), T = q->size(1);
  const int64_t kv_len = p[3] == Py_None ? 0 : as_long(p[3]);
  at::Tensor out;
  {
    NoGil nogil;
    out = empty({T, h * 64}, at::kBFloat16, q->device());
    check(g.vx_relpos_attention(q->data_ptr(), k->data_ptr(), v->data_ptr(), T, static_cast<int>(h), 64, kv_len, out.data_ptr(), h * 64,
                                stream()),
          "vx_relpos_attention");
    count();
  }
  return wrap(out);
  VX_END
}

// qkv_pack_gemm(a, w, bias | None, pos_u, pos_v, scale, packed | None) -> bf16 [3, h, M, 2 dk] | None
PyObject* py_qkv_pack_gemm(PyObject*, PyObject* const* p, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(7)
  Operand a, b;
  vx_gemm_desc d;
  if (!operands(p[0], p[1], a, b, d) || a.fmt == VX_FMT_ROWSCALE || !is_cuda_tensor(p[3]) || !is_cuda_tensor(p[4])) Py_RETURN_NONE;
  const at::Device dev = a.codes.device();
  bool ok = true;
  d.bias = vector_arg(p[2], d.N, dev, ok);
  const at::Tensor &u = THPVariable_Unpack(p[3]), &v = THPVariable_Unpack(p[4]);
  const at::ScalarType pt = u.scalar_type();
  if (!ok || u.dim() != 2 || u.sizes() != v.sizes() || v.scalar_type() != pt || (pt != at::kFloat && pt != at::kBFloat16) ||
      !u.is_contiguous() || !v.is_contiguous() || u.device() != dev || v.device() != dev)
    Py_RETURN_NONE;
  // (the kernel reads 16 bytes at a time; the general route's cast to bf16 copies fp32 biases of any address)
  if (((reinterpret_cast<uintptr_t>(u.data_ptr()) | reinterpret_cast<uintptr_t>(v.data_ptr())) & 15) != 0) Py_RETURN_NONE;
  const int64_t h = u.size(0), dk = u.size(1);
  if (d.N != 3 * h * dk) Py_RETURN_NONE;
  at::Tensor packed;
  if (p[6] == Py_None) {
    NoGil nogil;
    packed = empty({3, h, d.M, 2 * dk}, at::kBFloat16, dev);
  }
  else if (is_cuda_tensor(p[6])) packed = THPVariable_Unpack(p[6]);
  else Py_RETURN_NONE;
  if (packed.scalar_type() != at::kBFloat16 || !packed.is_contiguous() || packed.device() != dev ||
      packed.sizes() != at::IntArrayRef({3, h, d.M, 2 * dk}))
    Py_RETURN_NONE;
  d.epilogue = VX_EPI_BIAS_QKVPACK;
  d.out_dtype = VX_BF16; d.out = packed.data_ptr(); d.ldo = 2 * dk;
  d.heads = static_cast<int>(h); d.head_dim = static_cast<int>(dk);
  d.pos_u = u.data_ptr(); d.pos_v = v.data_ptr(); d.qk_scale = static_cast<float>(as_double(p[5]));
  d.flags = pt == at::kFloat ? VX_GEMM_POS_F32 : 0;
  {
    NoGil nogil;
    launch(d);
  }
  return p[6] == Py_None ? wrap(packed) : Py_NewRef(p[6]);
  VX_END
}

// heads_gemm(a, w, bias | None, out [h, M, width], col_off) -> out | None
PyObject* py_heads_gemm(PyObject*, PyObject* const* p, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(5)
  Operand a, b;
  vx_gemm_desc d;
  const at::Tensor* out;
  if (!operands(p[0], p[1], a, b, d) || !bf16_cube(p[3], &out)) Py_RETURN_NONE;
  const at::Device dev = a.codes.device();
  bool ok = true;
  d.bias = vector_arg(p[2], d.N, dev, ok);
  const int64_t h = out->size(0);
  if (!ok || h == 0 || out->size(1) != d.M || d.N % h || out->device() != dev) Py_RETURN_NONE;
  d.epilogue = d.bias ? VX_EPI_BIAS : VX_EPI_NONE;
  d.out_dtype = VX_BF16; d.out = out->data_ptr(); d.ldo = out->size(2);
  d.heads = static_cast<int>(h); d.head_dim = static_cast<int>(d.N / h); d.head_col_off = static_cast<int>(as_long(p[4]));
  d.flags = VX_GEMM_OUT_HEADS;
  {
    NoGil nogil;
    launch(d);
  }
  return Py_NewRef(p[3]);
  VX_END
}

// ---------------------------------------------------------------- front-end
// power_mel_log(spec c64 [T, F], mel f32 [M, F], mean | None, istd | None) -> f32 [T, M] | None
PyObject* py_power_mel_log(PyObject*, PyObject* const* p, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(4)
  if (!is_cuda_tensor(p[0]) || !is_cuda_tensor(p[1])) Py_RETURN_NONE;
  const at::Tensor &spec = THPVariable_Unpack(p[0]), &mel = THPVariable_Unpack(p[1]);
  const at::Device dev = spec.device();
  if (spec.scalar_type() != at::kComplexFloat || spec.dim() != 2 || !spec.is_contiguous() || spec.is_conj() || !rows2d(mel) ||
      mel.scalar_type() != at::kFloat || mel.device() != dev || mel.size(1) != spec.size(1))
    Py_RETURN_NONE;
  const int64_t T = spec.size(0), F = spec.size(1), M = mel.size(0);
  bool ok = true;
  const float* mean = vector_arg(p[2], M, dev, ok);
  const float* istd = vector_arg(p[3], M, dev, ok);
  if (!ok || (mean == nullptr) != (istd == nullptr) || !g.vx_power_mel_log_supported(F, M)) Py_RETURN_NONE;
  at::Tensor out;
  {
    NoGil nogil;
    out = empty({T, M}, at::kFloat, dev);
    check(g.vx_power_mel_log(spec.data_ptr(), T, F, F, static_cast<const float*>(mel.data_ptr()), M, mel.stride(0), mean, istd,
                             static_cast<float*>(out.data_ptr()), M, stream()),
          "vx_power_mel_log");
    count();
  }
  return wrap(out);
  VX_END
}

// ---------------------------------------------------------------- the encoder's linear stack
// A plan holds what one forward pass needs besides its frames: the packed weights, LayerNorm parameters and calibrated
// maxima as plain pointers, and the tensors they point into.  forward() walks the layer sequence that stack.py documents and
// issues every launch of the pass; its intermediate tensors live in one workspace block.
struct Lin {
  const void* codes; int64_t ld; const void* scales; const float* amax; const float* bias; int64_t N, K;
  int flags;  // VX_GEMM_CONST_B for what PackedLinear packs: see PackedLinear._const
};
struct Norm { const float *g, *b; };
enum { L_FFM1, L_FFM2, L_QKV, L_LO, L_LP, L_PW1, L_PW2, L_FF1, L_FF2, L_COUNT };
enum { N_FFM, N_MHA, N_CONV, N_FF, N_FINAL, N_COUNT };
enum { A_FFM, A_FFM_H, A_MHA, A_CTX, A_CONV, A_GLU, A_FF, A_FF_H, A_COUNT };

struct Plan {
  int fmt;
  int64_t d, ffn = 0, glu = 0, vocab = 0;  // the widest FFN intermediate and GLU output of the blocks
  float eps;
  bool fuse_ffn;
  int blocks;
  std::vector<Lin> lin;          // [block][L_COUNT], then the CTC head
  Lin lp_all{};                  // the positional projections of all blocks as one weight (codes nullptr: none)
  std::vector<Norm> norm;        // [block][N_COUNT], then after_norm
  std::vector<const float*> am;  // [block][A_COUNT], then after_norm, then the positions (NV16)
  // everything the pointers above point into, as it was when they were taken
  struct Kept { at::Tensor t; const void* ptr; int64_t numel, ld; };
  std::vector<Kept> kept;
  bool converted = false;        // a LayerNorm parameter was converted for this pass: the plan serves no other
  // the Python objects the plan was made of, see py_stack_plan_current
  struct Layer { PyObject *name, *layer, *q, *bias, *codes, *scales, *amax; };
  struct Named { PyObject *name, *object; };
  std::vector<Layer> layers;
  std::vector<Named> norms, maxima;
  std::vector<PyObject*> refs;
  PyObject* own(PyObject* o) {  // (takes over a reference)
    if (!o) throw PyFail{};
    refs.push_back(o);
    return o;
  }
  ~Plan() {
    for (PyObject* o : refs) Py_DECREF(o);
  }
  static int64_t row_stride(const at::Tensor& t) { return t.dim() > 0 ? t.stride(0) : 0; }
  void keep(const at::Tensor& t) {
    if (t.defined()) kept.push_back({t, t.data_ptr(), t.numel(), row_stride(t)});
  }
  // a tensor may have been given other storage (`t.data = ...`), and its former one freed
  bool in_place() const {
    for (const Kept& k : kept)
      if (k.t.data_ptr() != k.ptr || k.t.numel() != k.numel || row_stride(k.t) != k.ld) return false;
    return true;
  }
  Lin layer(const Operand& w, const float* bias, int flags) {
    for (const at::Tensor& t : {w.codes, w.scales, w.amax}) keep(t);
    return {w.codes.data_ptr(), w.codes.stride(0), w.scales.data_ptr(), f32_ptr(w.amax), bias, w.rows, w.k, flags};
  }
  const float* amax(size_t i) const { return am.empty() ? nullptr : am[i]; }
};

// quantized activation inside the workspace
struct Act { uint8_t* codes; uint8_t* scales; int64_t K; const float* amax; };

struct Pass {
  const Plan& p;
  int64_t M;
  void* st;
  int64_t launches = 0;

  int64_t code_ld(int64_t K) const { return p.fmt == VX_FMT_FP8_1X128 ? K : K / 2; }
  int64_t code_bytes(int64_t K) const { return (M * code_ld(K) + 255) / 256 * 256; }
  int64_t act_bytes(int64_t K) const {
    const int64_t s = p.fmt == VX_FMT_FP8_1X128 ? M * (K / 128) * 4 : sf_bytes(p.fmt, M, K);
    return code_bytes(K) + (s + 255) / 256 * 256;
  }
  Act act(uint8_t* base, int64_t K, const float* amax) const { return {base, base + code_bytes(K), K, amax}; }
  bool natural() const { return p.fmt == VX_FMT_FP8_1X128; }

  void quantize(const void* x, int dt, int64_t ld, const Act& q) {
    check(g.vx_quantize_pack(x, dt, M, q.K, ld, p.fmt, q.codes, code_ld(q.K), natural() ? q.scales : nullptr,
                             natural() ? nullptr : q.scales, q.amax, st), "vx_quantize_pack");
    ++launches;
  }
  void ln_quantize(const void* x, int64_t ld, const Norm& n, const Act& q) {
    check(g.vx_ln_quantize_pack(x, VX_BF16, M, q.K, ld, n.g, n.b, p.eps, p.fmt, q.codes, code_ld(q.K), natural() ? q.scales : nullptr,
                                natural() ? nullptr : q.scales, q.amax, nullptr, 0, q.K, st), "vx_ln_quantize_pack");
    ++launches;
  }
  void ln2_quantize(void* x, int64_t ld, const Norm& n1, const Norm& n2, const Act& q) {
    check(g.vx_ln2_quantize_pack(x, VX_BF16, M, q.K, ld, n1.g, n1.b, n2.g, n2.b, p.eps, p.fmt, q.codes, code_ld(q.K),
                                 natural() ? q.scales : nullptr, natural() ? nullptr : q.scales, q.amax, x, VX_BF16, ld, st),
          "vx_ln2_quantize_pack");
    ++launches;
  }
  vx_gemm_desc desc(const Act& a, const Lin& w, int epi) const {
    vx_gemm_desc d{};
    d.struct_size = sizeof(d);
    d.fmt = p.fmt;
    d.M = M; d.N = w.N; d.K = w.K;
    d.a_codes = a.codes; d.lda = code_ld(a.K);
    d.b_codes = w.codes; d.ldb = w.ld;
    d.a_scales = a.scales; d.b_scales = w.scales;
    d.a_amax = a.amax; d.b_amax = w.amax;
    d.epilogue = epi == VX_EPI_BIAS && !w.bias ? VX_EPI_NONE : epi;
    d.flags = w.flags;
    d.bias = w.bias;
    return d;
  }
  void run(const vx_gemm_desc& d) {
    check(g.vx_bsgemm(&d, st), "vx_bsgemm");
    ++launches;
  }
  void gemm(const Act& a, const Lin& w, int epi, void* out, int64_t ldo) {
    vx_gemm_desc d = desc(a, w, epi);
    d.out_dtype = VX_BF16; d.out = out; d.ldo = ldo;
    run(d);
  }
  // Swish or GLU with the result quantized in the epilogue
  void gemm_quant(const Act& a, const Lin& w, int epi, const Act& h) {
    vx_gemm_desc d = desc(a, w, epi);
    d.out_dtype = VX_FP4; d.out = h.codes; d.ldo = code_ld(h.K);
    d.out_fmt = p.fmt; d.out_scales_sf = h.scales; d.out_amax = h.amax;
    run(d);
  }
  // bf16 result whose columns from `col0` on are also quantized in the epilogue
  void gemm_tail_quant(const Act& a, const Lin& w, void* out, int64_t ldo, int64_t col0, const Act& t) {
    vx_gemm_desc d = desc(a, w, VX_EPI_BIAS);
    d.out_dtype = VX_BF16; d.out = out; d.ldo = ldo;
    d.flags |= VX_GEMM_QUANT_TAIL;
    d.out_fmt = p.fmt; d.out_scales = t.codes; d.out_scales_sf = t.scales; d.out_amax = t.amax; d.quant_col0 = static_cast<int>(col0);
    run(d);
  }
  // x <- alpha w(a) + x, then the LayerNorm(s) that read x next and the quantizer: `n2` set = x <- LN_n(x) is stored and
  // LN_n2 of it quantized (the end of a block)
  // (`from`: the residual is read there, x otherwise)
  void residual(const Act& a, const Lin& w, void* x, int64_t ldx, float alpha, const Norm& n, const Norm* n2, const Act& q, bool fused,
                const void* from = nullptr, int64_t ldf = 0) {
    vx_gemm_desc d = desc(a, w, VX_EPI_BIAS_RESIDUAL);
    d.residual = from ? from : x; d.residual_dtype = VX_BF16; d.ldr = from ? ldf : ldx; d.alpha = alpha;
    d.out_dtype = VX_BF16; d.out = x; d.ldo = ldx;
    if (fused && g.vx_bsgemm_residual_ln_supported(p.fmt, w.N, w.K)) {
      if (n2)
        check(g.vx_bsgemm_residual_ln2(&d, n.g, n.b, n2->g, n2->b, p.eps, q.codes, code_ld(q.K), q.scales, st), "vx_bsgemm_residual_ln2");
      else
        check(g.vx_bsgemm_residual_ln(&d, n.g, n.b, p.eps, q.codes, code_ld(q.K), q.scales, st), "vx_bsgemm_residual_ln");
      ++launches;
      return;
    }
    run(d);
    if (n2) ln2_quantize(x, ldx, n, *n2, q);
    else ln_quantize(x, ldx, n, q);
  }
};

// How a pass runs its residual GEMMs and LayerNorms: separate launches, with the LayerNorm + quantizer in the GEMM, or all
// blocks in one launch where the shapes and addresses allow it (separate launches where not).
enum { ROUTE_SEPARATE, ROUTE_FUSED, ROUTE_WHOLE };

void plan_free(PyObject* cap) {
  delete static_cast<Plan*>(PyCapsule_GetPointer(cap, "velox_stack_plan"));
}

// Frames up to which the positional projections of all blocks run as one launch: they depend on the positions only, and
// a pass this short is bound by its launches (twelve of 5 us against one of 10 us at 375 frames).  Beyond it their
// outputs would take blocks * d_model columns of workspace for nothing.
constexpr int64_t LP_BATCH_MAX = 4096;

// stack_plan(fmt, d, eps, fuse_ffn, blocks, layers, norms, maxima, positions | None) -> capsule
//   layers: ((name, PackedLinear)...); norms: ((name, (gamma, beta))...); maxima: ((name, tensor | None)...), or empty;
//   positions: the Quantized whose parts the positional projections of the blocks are
PyObject* py_stack_plan(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(9)
  auto plan = std::make_unique<Plan>();
  plan->fmt = static_cast<int>(as_long(a[0]));
  plan->d = as_long(a[1]);
  plan->eps = static_cast<float>(as_double(a[2]));
  plan->fuse_ffn = as_bool(a[3]);
  plan->blocks = static_cast<int>(as_long(a[4]));
  auto bad = [](const char* what) { PyErr_SetString(PyExc_ValueError, what); throw PyFail{}; };
  const char* const vectors = "the stack's biases, LayerNorm parameters and maxima have to be CUDA vectors of the layers' widths";
  for (int i = 5; i < 8; ++i) {
    if (!PyTuple_Check(a[i])) bad("stack_plan: tuples expected");
    for (Py_ssize_t j = 0; j < PyTuple_GET_SIZE(a[i]); ++j)
      if (!PyTuple_Check(PyTuple_GET_ITEM(a[i], j)) || PyTuple_GET_SIZE(PyTuple_GET_ITEM(a[i], j)) != 2) bad("stack_plan: pairs expected");
  }
  if (PyTuple_GET_SIZE(a[5]) != plan->blocks * L_COUNT + 1 || PyTuple_GET_SIZE(a[6]) != plan->blocks * N_COUNT + 1 ||
      (PyTuple_GET_SIZE(a[7]) != 0 && PyTuple_GET_SIZE(a[7]) != plan->blocks * A_COUNT + 2))
    bad("stack_plan: wrong number of layers, norms or maxima");
  auto f32 = [&](PyObject* o, int64_t n) -> const float* {
    if (!is_cuda_tensor(o)) bad(vectors);
    const at::Tensor& t = THPVariable_Unpack(o);
    if (t.scalar_type() != at::kFloat || !t.is_contiguous() || t.numel() < n) bad(vectors);
    plan->keep(t);
    return static_cast<const float*>(t.data_ptr());
  };
  // a LayerNorm's parameters may be of another type or strided; their copies are not kept, they would not follow the originals
  auto norm_vector = [&](PyObject* o) -> const float* {
    if (!is_cuda_tensor(o)) bad(vectors);
    const at::Tensor& t = THPVariable_Unpack(o);
    if (t.scalar_type() == at::kFloat && t.is_contiguous()) return f32(o, plan->d);
    if (t.numel() < plan->d) bad(vectors);
    plan->converted = true;
    at::Tensor c;
    {
      NoGil nogil;
      c = t.detach().to(at::kFloat).contiguous();
    }
    plan->keep(c);
    return static_cast<const float*>(c.data_ptr());
  };
  const bool sf = has_sf(plan->fmt);
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(a[5]); ++i) {
    Plan::Layer y;
    y.name = plan->own(Py_NewRef(PyTuple_GET_ITEM(PyTuple_GET_ITEM(a[5], i), 0)));
    y.layer = plan->own(Py_NewRef(PyTuple_GET_ITEM(PyTuple_GET_ITEM(a[5], i), 1)));
    y.q = plan->own(PyObject_GetAttr(y.layer, s_q));
    y.bias = plan->own(PyObject_GetAttr(y.layer, s_bias));
    if (reinterpret_cast<PyObject*>(Py_TYPE(y.q)) != g_quantized) bad("stack_plan: bad layer");
    y.codes = plan->own(PyObject_GetAttr(y.q, s_codes));
    y.scales = plan->own(PyObject_GetAttr(y.q, sf ? s_sf : s_scales));
    if (sf && y.scales == Py_None) {  // made from the natural layout, and kept by the Quantized
      plan->own(PyObject_CallMethod(y.q, "gemm_scales", nullptr));
      y.scales = plan->own(PyObject_GetAttr(y.q, s_sf));
    }
    y.amax = plan->own(PyObject_GetAttr(y.q, s_amax));
    Operand w;
    if (!read_operand(y.q, w)) bad("stack_plan: bad layer");
    // the widths come from the layers; what follows one another has to fit
    const int64_t d = plan->d;
    const bool head = i == plan->blocks * L_COUNT;
    const int l = head ? L_COUNT : static_cast<int>(i % L_COUNT);
    const bool wide = l == L_FFM1 || l == L_FF1 || l == L_PW1 || head;  // its number of outputs is free
    const int64_t before = l == L_FFM2 || l == L_FF2 ? plan->lin.back().N : (l == L_PW2 ? plan->lin.back().N / 2 : d);
    if (w.fmt != plan->fmt || w.k != before || (!wide && w.rows != (l == L_QKV ? 3 * d : d)))
      bad("a layer of the stack does not fit the format, d_model or the layer before it");
    if (l == L_FFM1 || l == L_FF1) plan->ffn = std::max(plan->ffn, w.rows);
    if (l == L_PW1) plan->glu = std::max(plan->glu, w.rows / 2);
    if (head) plan->vocab = w.rows;
    const bool packed = plan->own(PyObject_GetAttr(y.q, s_scales)) != Py_None;
    plan->lin.push_back(plan->layer(w, y.bias == Py_None ? nullptr : f32(y.bias, w.rows), packed ? VX_GEMM_CONST_B : 0));
    plan->layers.push_back(y);
  }
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(a[6]); ++i) {
    PyObject* const e = PyTuple_GET_ITEM(a[6], i);
    PyObject* const pr = PyTuple_GET_ITEM(e, 1);
    if (!PyTuple_Check(pr) || PyTuple_GET_SIZE(pr) != 2) bad("stack_plan: a LayerNorm is a pair (gamma, beta)");
    plan->norms.push_back({plan->own(Py_NewRef(PyTuple_GET_ITEM(e, 0))), plan->own(Py_NewRef(pr))});
    const float* const gamma = norm_vector(PyTuple_GET_ITEM(pr, 0));
    plan->norm.push_back({gamma, norm_vector(PyTuple_GET_ITEM(pr, 1))});
  }
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(a[7]); ++i) {
    PyObject* const e = PyTuple_GET_ITEM(a[7], i);
    PyObject* const o = PyTuple_GET_ITEM(e, 1);
    plan->maxima.push_back({plan->own(Py_NewRef(PyTuple_GET_ITEM(e, 0))), plan->own(Py_NewRef(o))});
    plan->am.push_back(o == Py_None ? nullptr : f32(o, 1));
  }
  if (a[8] != Py_None) {  // used as long as every block's projection is its part of it
    Operand w;
    bool parts = read_operand(a[8], w) && w.fmt == plan->fmt && w.k == plan->d && plan->blocks > 0 && w.rows == plan->blocks * plan->d;
    for (int i = 0; parts && i < plan->blocks; ++i) {
      const Lin& L = plan->lin[i * L_COUNT + L_LP];
      const int64_t scale_bytes = static_cast<int64_t>(w.scales.nbytes()) / plan->blocks;
      parts = !L.bias && L.ld == w.codes.stride(0) && L.codes == static_cast<uint8_t*>(w.codes.data_ptr()) + i * plan->d * L.ld &&
              L.scales == static_cast<uint8_t*>(w.scales.data_ptr()) + i * scale_bytes;
    }
    if (parts) plan->lp_all = plan->layer(w, nullptr, VX_GEMM_CONST_B);
  }
  PyObject* cap = PyCapsule_New(plan.get(), "velox_stack_plan", plan_free);
  if (!cap) return nullptr;
  plan.release();
  return cap;
  VX_END
}

// stack_plan_current(plan, layers by name, norms by name, maxima by name, eps, fuse_ffn, blocks) -> bool: whether the stack still holds the
// objects the plan was made of, with the storage they had.  A program may replace a layer, its weight or bias, a LayerNorm's parameters or a
// maximum between passes; about 10 us of a host call that is ahead of the GPU by more.
PyObject* py_stack_plan_current(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(7)
  const Plan* plan = static_cast<const Plan*>(PyCapsule_GetPointer(a[0], "velox_stack_plan"));
  if (!plan) return nullptr;
  if (static_cast<float>(as_double(a[4])) != plan->eps || as_bool(a[5]) != plan->fuse_ffn || as_long(a[6]) != plan->blocks ||
      plan->converted || !plan->in_place())
    Py_RETURN_FALSE;
  auto held = [](PyObject* dict, PyObject* name) {
    PyObject* now = PyDict_GetItemWithError(dict, name);
    if (!now && PyErr_Occurred()) throw PyFail{};
    return now ? now : Py_None;
  };
  auto same = [](PyObject* o, PyObject* name, PyObject* was) {
    PyObject* v = PyObject_GetAttr(o, name);
    if (!v) throw PyFail{};
    Py_DECREF(v);
    return v == was;
  };
  PyObject* const s_gemm_scales = has_sf(plan->fmt) ? s_sf : s_scales;
  for (const Plan::Layer& y : plan->layers)
    if (held(a[1], y.name) != y.layer || !same(y.layer, s_q, y.q) || !same(y.layer, s_bias, y.bias) || !same(y.q, s_codes, y.codes) ||
        !same(y.q, s_gemm_scales, y.scales) || !same(y.q, s_amax, y.amax))
      Py_RETURN_FALSE;
  for (const Plan::Named& n : plan->norms)
    if (held(a[2], n.name) != n.object) Py_RETURN_FALSE;
  for (const Plan::Named& n : plan->maxima)
    if (held(a[3], n.name) != n.object) Py_RETURN_FALSE;
  Py_RETURN_TRUE;
  VX_END
}

// Whether the blocks of a pass can run as one launch (vx_conformer_pass): the model's own widths, unit pieces of 16 bytes.
bool one_launch(const Plan& p, const void* x, int64_t ldx, const void* src, int64_t ld_src) {
  if (p.blocks == 0 || !p.fuse_ffn || !g.vx_conformer_pass_supported(p.fmt, p.d, p.lin[L_FFM1].N, p.lin[L_PW1].N, p.blocks)) return false;
  for (int i = 0; i < p.blocks; ++i) {
    const Lin* L = &p.lin[i * L_COUNT];
    if (L[L_FFM1].N != p.lin[L_FFM1].N || L[L_FF1].N != p.lin[L_FFM1].N || L[L_PW1].N != p.lin[L_PW1].N) return false;
    for (int l = 0; l < L_COUNT; ++l)
      if ((l != L_LP && (!L[l].bias || (reinterpret_cast<uintptr_t>(L[l].bias) & 15))) || ((reinterpret_cast<uintptr_t>(L[l].codes) | reinterpret_cast<uintptr_t>(L[l].scales) | L[l].ld) & 15) != 0) return false;
  }
  for (const Norm& n : p.norm)
    if (((reinterpret_cast<uintptr_t>(n.g) | reinterpret_cast<uintptr_t>(n.b)) & 15) != 0) return false;
  // (rows that overlap are for the separate launches to refuse)
  return ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(src)) & 15) == 0 && ((ldx | ld_src) & 7) == 0 && ldx >= p.d && ld_src >= p.d;
}

// Every launch of one pass.  `src` (row stride ld_src): the features, where they are not in x; `pt`: the positions, or not
// defined; of the outputs those that the caller did not bring are made.
void stack_pass(const Plan& p, const at::Tensor& xt, const void* src, int64_t ld_src, const at::Tensor& pt, int route, bool greedy,
                at::Tensor& keys, at::Tensor& ids, at::Tensor& logits) {
  const at::Device dev = xt.device();
  const int64_t M = xt.size(0), ldx = xt.stride(0), d = p.d;
  void* const x = xt.data_ptr();
  const bool with_pos = pt.defined(), fused = route == ROUTE_FUSED;
  const bool whole = route == ROUTE_WHOLE && M > 0 && one_launch(p, x, ldx, src ? src : x, src ? ld_src : ldx);
  Pass s{p, M, stream()};
  Pass sp{p, with_pos ? pt.size(0) : 0, s.st};  // the positions' own rows

  // workspace: [activations | positions | context / GLU activations | FFN intermediate or q|k|v or GLU output | lp output]
  const int64_t ba = s.act_bytes(d), bc = s.act_bytes(d > p.glu ? d : p.glu);
  const int64_t bh = p.fuse_ffn ? s.act_bytes(p.ffn) : s.act_bytes(p.ffn) + (M * p.ffn * 2 + 255) / 256 * 256;
  int64_t big = bh > M * 3 * d * 2 ? bh : M * 3 * d * 2;
  if (big < M * p.glu * 2) big = M * p.glu * 2;
  if (whole) big = M * 3 * d * 2 + 256 + g.vx_conformer_pass_scratch(M, p.ffn);  // q|k|v, then the kernel's scratch
  big = (big + 255) / 256 * 256;
  const int64_t bp = sp.act_bytes(d);
  const bool lp_batched = with_pos && p.lp_all.codes && sp.M <= LP_BATCH_MAX;
  const int64_t total = ba + bc + big + bp + sp.M * d * 2 * (lp_batched ? p.blocks : 1);
  const at::Tensor ws = empty({total}, at::kByte, dev);
  uint8_t* const base = static_cast<uint8_t*>(ws.data_ptr());
  uint8_t* const w_act = base;
  uint8_t* const w_ctx = w_act + ba;
  uint8_t* const w_big = w_ctx + bc;
  uint8_t* const w_pos = w_big + big;
  uint8_t* const w_lp = w_pos + bp;

  Act pos_q{};
  if (with_pos) {
    pos_q = sp.act(w_pos, d, p.amax(p.blocks * A_COUNT + 1));
    sp.quantize(pt.data_ptr(), dtype_code(pt), pt.stride(0), pos_q);
  }
  if (lp_batched) sp.gemm(pos_q, p.lp_all, VX_EPI_NONE, w_lp, p.blocks * d);
  // the quantizers of the value third and of the GLU output run in the epilogues that produce them
  const bool fp4 = p.fmt != VX_FMT_FP8_1X128;
  auto ffn = [&](const Act& q, const Lin& w1, const Lin& w2, const float* am_h, const Norm& n, const Norm* n2, const Act& q_next,
                 const void* from = nullptr) {
    const Act h = s.act(w_big, w1.N, am_h);
    if (p.fuse_ffn) {
      s.gemm_quant(q, w1, VX_EPI_BIAS_SWISH, h);
    } else {
      void* const hb = w_big + s.act_bytes(w1.N);
      s.gemm(q, w1, VX_EPI_BIAS_SWISH, hb, w1.N);
      s.quantize(hb, VX_BF16, w1.N, h);
    }
    s.residual(h, w2, x, ldx, 0.5f, n, n2, q_next, fused, from, ld_src);
  };
  Act q = s.act(w_act, d, p.amax(p.blocks > 0 ? A_FFM : 0));
  if (whole) {
    std::vector<vx_pass_block> blocks(p.blocks);
    vx_pass_desc c{};
    c.struct_size = sizeof(c);
    c.const_weights = 1;
    for (int i = 0; i < p.blocks; ++i) {
      constexpr int order[VX_PASS_LINEARS] = {L_FFM1, L_FFM2, L_QKV, L_LO, L_PW1, L_PW2, L_FF1, L_FF2};
      for (int l = 0; l < VX_PASS_LINEARS; ++l) {
        const Lin& w = p.lin[i * L_COUNT + order[l]];
        blocks[i].lin[l] = {w.codes, w.ld, w.scales, w.bias};
        if (!(w.flags & VX_GEMM_CONST_B)) c.const_weights = 0;
      }
      for (int n = 0; n < N_COUNT; ++n) {
        blocks[i].gamma[n] = p.norm[i * N_COUNT + n].g;
        blocks[i].beta[n] = p.norm[i * N_COUNT + n].b;
      }
    }
    c.blocks = p.blocks; c.M = M; c.ffn = p.ffn; c.eps = p.eps;
    c.block = blocks.data();
    c.after_gamma = p.norm[p.blocks * N_COUNT].g; c.after_beta = p.norm[p.blocks * N_COUNT].b;
    c.src = src ? src : x; c.ld_src = src ? ld_src : ldx;
    c.x = x; c.ldx = ldx;
    c.qkv = w_big;
    c.scratch = w_big + (M * 3 * d * 2 + 255) / 256 * 256;
    c.codes = q.codes; c.scales_sf = q.scales;
    check(g.vx_conformer_pass(&c, s.st), "vx_conformer_pass");
    ++s.launches;
    for (int i = 0; i < p.blocks && with_pos && !lp_batched; ++i) sp.gemm(pos_q, p.lin[i * L_COUNT + L_LP], VX_EPI_BIAS, w_lp, d);
  } else
    s.ln_quantize(src ? src : x, src ? ld_src : ldx, p.norm[p.blocks > 0 ? N_FFM : 0], q);
  for (int i = 0; i < p.blocks && !whole; ++i) {
    const Lin* L = &p.lin[i * L_COUNT];
    const Norm* n = &p.norm[i * N_COUNT];
    const float* const* am = p.am.empty() ? nullptr : &p.am[i * A_COUNT];
    auto mx = [&](int k) { return am ? am[k] : nullptr; };
    Act q_mha = s.act(w_act, d, mx(A_MHA)), q_conv = s.act(w_act, d, mx(A_CONV)), q_ff = s.act(w_act, d, mx(A_FF));
    ffn(q, L[L_FFM1], L[L_FFM2], mx(A_FFM_H), n[N_MHA], nullptr, q_mha, i == 0 ? src : nullptr);
    const Act ctx = s.act(w_ctx, d, mx(A_CTX));
    if (fp4 && d % 256 == 0) {
      s.gemm_tail_quant(q_mha, L[L_QKV], w_big, 3 * d, 2 * d, ctx);
    } else {
      s.gemm(q_mha, L[L_QKV], VX_EPI_BIAS, w_big, 3 * d);
      s.quantize(w_big + 2 * d * 2, VX_BF16, 3 * d, ctx);
    }
    if (with_pos && !lp_batched) sp.gemm(pos_q, L[L_LP], VX_EPI_BIAS, w_lp, d);  // feeds the attention scores only
    s.residual(ctx, L[L_LO], x, ldx, 1.0f, n[N_CONV], nullptr, q_conv, fused);
    const int64_t glu = L[L_PW1].N / 2;
    const Act gl = s.act(w_ctx, glu, mx(A_GLU));
    if (fp4 && glu % 256 == 0) {
      s.gemm_quant(q_conv, L[L_PW1], VX_EPI_BIAS_GLU, gl);
    } else {
      s.gemm(q_conv, L[L_PW1], VX_EPI_BIAS_GLU, w_big, glu);
      s.quantize(w_big, VX_BF16, glu, gl);
    }
    s.residual(gl, L[L_PW2], x, ldx, 1.0f, n[N_FF], nullptr, q_ff, fused);
    // norm_final of this block and the LayerNorm that reads it next: the first of the next block, or after_norm
    const bool last = i + 1 == p.blocks;
    q = s.act(w_act, d, p.amax(last ? p.blocks * A_COUNT : (i + 1) * A_COUNT + A_FFM));
    ffn(q_ff, L[L_FF1], L[L_FF2], mx(A_FF_H), n[N_FINAL], last ? &p.norm[p.blocks * N_COUNT] : n + N_COUNT + N_FFM, q);
  }
  const Lin& head = p.lin[p.blocks * L_COUNT];
  vx_gemm_desc e = s.desc(q, head, greedy ? VX_EPI_BIAS_ARGMAX : VX_EPI_BIAS);
  if (greedy) {
    if (!keys.defined()) keys = empty({M}, at::kLong, dev);
    if (!ids.defined()) ids = empty({M}, at::kInt, dev);
    e.out_dtype = VX_F32; e.out = keys.data_ptr(); e.ldo = 1;
    s.run(e);
    check(g.vx_argmax_ids(keys.data_ptr(), M, static_cast<int32_t*>(ids.data_ptr()), nullptr, s.st), "vx_argmax_ids");
    ++s.launches;
  } else {
    if (!logits.defined()) logits = new_out(M, p.vocab, at::kBFloat16, dev);
    e.out_dtype = dtype_code(logits); e.out = logits.data_ptr(); e.ldo = logits.stride(0);
    s.run(e);
  }
  count(s.launches + sp.launches);
}

// stack_forward(plan, x, pos | None, route, head, keys | None, ids | None, logits | None, source | None) -> logits / ids
//   x bf16 [T, d] (overwritten; with `source`, bf16 [T, d], the features are read there and x only receives the residual
//   stream); head 0: bf16 logits [T, vocab], 1: greedy ids i32 [T]
PyObject* py_stack_forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  VX_BEGIN
  VX_ARGS(9)
  const Plan* plan = static_cast<const Plan*>(PyCapsule_GetPointer(a[0], "velox_stack_plan"));
  if (!plan) return nullptr;
  const Plan& p = *plan;
  auto bad = [](const char* what) { PyErr_SetString(PyExc_ValueError, what); throw PyFail{}; };
  if (!is_cuda_tensor(a[1])) {
    PyErr_SetString(PyExc_RuntimeError, "x must be a CUDA tensor: this library has no CPU path");
    return nullptr;
  }
  const at::Tensor& xt = THPVariable_Unpack(a[1]);
  if (xt.scalar_type() != at::kBFloat16 || !rows2d(xt) || xt.size(1) != p.d) bad("x must be bf16 [T, d_model] with unit column stride");
  const at::Device dev = xt.device();
  const int64_t M = xt.size(0), d = p.d;
  const void* src = nullptr;
  int64_t ld_src = 0;
  if (a[8] != Py_None) {
    if (!is_cuda_tensor(a[8])) bad("source must be a CUDA tensor");
    const at::Tensor& t = THPVariable_Unpack(a[8]);
    if (t.scalar_type() != at::kBFloat16 || !rows2d(t) || t.sizes() != xt.sizes() || t.device() != xt.device())
      bad("source must be bf16 of x's shape on x's device with unit column stride");
    src = t.data_ptr();
    ld_src = t.stride(0);
  }
  const bool with_pos = a[2] != Py_None;
  if (with_pos && !is_cuda_tensor(a[2])) bad("pos must be a CUDA tensor");
  at::Tensor pt, keys, ids, logits;
  if (with_pos) {
    pt = THPVariable_Unpack(a[2]);
    if (!rows2d(pt) || pt.size(1) != d || pt.device() != dev || dtype_code(pt) < 0)
      bad("pos must be a float32 or bf16 [frames, d_model] tensor on x's device with unit column stride");
  }
  const int route = static_cast<int>(as_long(a[3]));
  const bool greedy = as_long(a[4]) != 0;
  auto out_vec = [&](PyObject* o, at::ScalarType dt, const char* what, at::Tensor& t) {
    if (o == Py_None) return;
    if (!is_cuda_tensor(o)) bad(what);
    t = THPVariable_Unpack(o);
    if (t.scalar_type() != dt || !t.is_contiguous() || t.numel() < M || t.device() != dev) bad(what);
  };
  if (greedy) {
    out_vec(a[5], at::kLong, "keys must be a contiguous int64 tensor with at least T entries", keys);
    out_vec(a[6], at::kInt, "ids must be a contiguous int32 tensor with at least T entries", ids);
  } else if (a[7] != Py_None) {
    if (is_cuda_tensor(a[7])) logits = THPVariable_Unpack(a[7]);
    if (!logits.defined() || !rows2d(logits) || logits.size(0) != M || logits.size(1) != p.vocab || logits.device() != dev || dtype_code(logits) < 0)
      bad("out_logits must be a [T, vocab] CUDA tensor with unit column stride");
  }
  {
    NoGil nogil;
    stack_pass(p, xt, src, ld_src, pt, route, greedy, keys, ids, logits);
  }
  PyObject* given = a[greedy ? 6 : 7];
  return given == Py_None ? wrap(greedy ? ids : logits) : Py_NewRef(given);
  VX_END
}

// ---------------------------------------------------------------- module
PyObject* py_launches(PyObject*, PyObject*) { return PyLong_FromLongLong(g_launches.load()); }
PyObject* py_reset(PyObject*, PyObject*) {
  g_launches.store(0);
  Py_RETURN_NONE;
}

// init(library path, VeloxError, Quantized)
PyObject* py_init(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  VX_ARGS(3)
  const char* path = PyUnicode_AsUTF8(a[0]);
  if (!path) return nullptr;
  void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (!h) {
    PyErr_Format(PyExc_RuntimeError, "cannot load %s: %s", path, dlerror());
    return nullptr;
  }
#define X(f)                                                                              \
  g.f = reinterpret_cast<decltype(g.f)>(dlsym(h, #f));                                    \
  if (!g.f) {                                                                             \
    PyErr_Format(PyExc_RuntimeError, "%s: missing export %s", path, #f);                  \
    return nullptr;                                                                       \
  }
  VX_FUNCS(X)
#undef X
  Py_XSETREF(g_error, Py_NewRef(a[1]));
  Py_XSETREF(g_quantized, Py_NewRef(a[2]));
  Py_RETURN_NONE;
}

#define VX_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    VX_METHOD("init", py_init),
    VX_METHOD("quantize", py_quantize),
    VX_METHOD("ln_quantize", py_ln_quantize),
    VX_METHOD("bsgemm", py_bsgemm),
    VX_METHOD("residual_ln", py_residual_ln),
    VX_METHOD("rowscale_linear", py_rowscale_linear),
    VX_METHOD("blkscale_gemm", py_blkscale_gemm),
    VX_METHOD("topk", py_topk),
    VX_METHOD("relpos_attention", py_relpos_attention),
    VX_METHOD("qkv_pack_gemm", py_qkv_pack_gemm),
    VX_METHOD("heads_gemm", py_heads_gemm),
    VX_METHOD("power_mel_log", py_power_mel_log),
    VX_METHOD("stack_plan", py_stack_plan),
    VX_METHOD("stack_plan_current", py_stack_plan_current),
    VX_METHOD("stack_forward", py_stack_forward),
    {"launches", py_launches, METH_NOARGS, nullptr},
    {"reset_launches", py_reset, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_vx_host", "native host path of velox_voice_b200", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__vx_host() {
  s_fmt = PyUnicode_InternFromString("fmt");
  s_rows = PyUnicode_InternFromString("rows");
  s_k = PyUnicode_InternFromString("k");
  s_codes = PyUnicode_InternFromString("codes");
  s_scales = PyUnicode_InternFromString("scales");
  s_sf = PyUnicode_InternFromString("sf");
  s_amax = PyUnicode_InternFromString("amax");
  s_q = PyUnicode_InternFromString("q");
  s_bias = PyUnicode_InternFromString("bias");
  return PyModule_Create(&kModule);
}
