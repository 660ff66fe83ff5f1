// Python binding of the operators (module _native): argument checks, output allocation and the call into libintfa.so in
// native code, because in Python they cost more than the kernels of a small call (75 us of host time against 20 us of
// device time for one attention call of batch 1, heads 4, 512 tokens; 23 us in all now).
// Semantics and error types are those of the reference's Python operators and of ops.py, which calls this.
#include <torch/csrc/python_headers.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <initializer_list>
#include <mutex>
#include <string>

#include "../../include/intfa.h"

namespace {

PyObject* g_error_class = nullptr;      // IntfaError(code, message)

// thrown where a Python exception has been set already
struct PySet {};
[[noreturn]] void raise(PyObject* type, const std::string& msg) {
  PyErr_SetString(type, msg.c_str());
  throw PySet();
}
void check(int rc) {
  if (rc == INTFA_OK) return;
  char buf[512];
  intfa_last_error(buf, sizeof(buf));
  if (!g_error_class) raise(PyExc_RuntimeError, buf);
  PyObject* e = PyObject_CallFunction(g_error_class, "is", rc, buf);
  if (e) {
    PyErr_SetObject(g_error_class, e);
    Py_DECREF(e);
  }
  throw PySet();
}

const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) raise(PyExc_TypeError, std::string(what) + " must be a torch.Tensor");
  return THPVariable_Unpack(o);
}
void need_cuda(const at::Tensor& t) {
  if (!t.is_cuda()) raise(PyExc_RuntimeError, "int-flashattention_b200 runs on CUDA tensors only (there is no CPU path)");
}
at::Tensor empty(at::IntArrayRef size, at::ScalarType type, c10::Device dev) {
  return at::detail::empty_cuda(size, type, dev, c10::nullopt);
}
bool is(const at::Tensor& t, at::ScalarType s) { return t.scalar_type() == s; }
void* stream_of(c10::Device dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

// one status word per device, which the kernels report bounded-wait expiry into
at::Tensor status_word(c10::Device dev) {
  static std::mutex mu;
  static std::array<at::Tensor, 64> words;
  const int i = dev.index();
  if (i < 0 || i >= 64) raise(PyExc_RuntimeError, "bad device index");
  std::lock_guard<std::mutex> lock(mu);
  if (!words[i].defined()) words[i] = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(dev));
  return words[i];
}

// TMA wants a contiguous last dim and 16-byte multiples for every other stride
at::Tensor tma_ready(const at::Tensor& t) {
  const int64_t es = t.element_size();
  bool ok = t.stride(-1) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  for (int64_t i = 0; ok && i + 1 < t.dim(); ++i) ok = t.stride(i) > 0 && (t.stride(i) * es) % 16 == 0;
  return ok ? t : t.contiguous();
}
// scales as the kernel reads them: fp32 or fp16 (what benchmark.py makes), contiguous
at::Tensor scales(const at::Tensor& s) {
  return is(s, at::kFloat) || is(s, at::kHalf) ? s.contiguous() : s.to(at::kFloat).contiguous();
}

// ---------------------------------------------------------------------------------------------------------------
// keyword arguments of the attention operators
// ---------------------------------------------------------------------------------------------------------------
constexpr int kAutoG = -0x7fffffff;     // no G given
struct Options {
  int G = kAutoG, p_round = 0, kv_order = 0;
  bool have_state = false, return_state = false, return_lse = false, write_o = true, tap = false;
  at::Tensor m, l, acc;
  int64_t q_offset = 0, kv_offset = 0;
  int tap_tile = 0, tap_step = 0, wait_kcycles = 0, skip_k = 0;
  at::ScalarType out = at::kHalf;
};
enum Name { N_G, N_P_ROUND, N_KV_ORDER, N_STATE, N_Q_OFFSET, N_KV_OFFSET, N_RETURN_STATE, N_RETURN_LSE, N_WRITE_O, N_TAP, N_OUT, N_WAIT,
            N_COUNT };
const char* const kNames[N_COUNT] = {"G", "p_round", "kv_order", "state", "q_offset", "kv_offset", "return_state", "return_lse",
                                     "write_o", "debug_tap", "out_dtype", "debug_wait"};
PyObject* g_names[N_COUNT];             // interned

// int(o) and float(o): any number, a tensor of one element, a string
int64_t as_long(PyObject* o) {
  PyObject* i = PyNumber_Long(o);
  if (!i) throw PySet();
  const long long v = PyLong_AsLongLong(i);
  Py_DECREF(i);
  if (v == -1 && PyErr_Occurred()) throw PySet();
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PySet();
  return v != 0;
}
double as_double(PyObject* o) {
  PyObject* f = PyNumber_Float(o);
  if (!f) throw PySet();
  const double v = PyFloat_AS_DOUBLE(f);
  Py_DECREF(f);
  return v;
}
bool equals(PyObject* s, const char* w) { return PyUnicode_Check(s) && PyUnicode_CompareWithASCIIString(s, w) == 0; }
// index of a word in a list of two, KeyError otherwise
int word(PyObject* o, const char* a, const char* b) {
  if (equals(o, a)) return 0;
  if (equals(o, b)) return 1;
  PyErr_SetObject(PyExc_KeyError, o);
  throw PySet();
}
int name_index(PyObject* name) {
  for (int i = 0; i < N_COUNT; ++i)
    if (name == g_names[i]) return i;
  for (int i = 0; i < N_COUNT; ++i)
    if (PyUnicode_CompareWithASCIIString(name, kNames[i]) == 0) return i;
  return -1;
}
void pair_of_ints(PyObject* v, int* a, int* b) {
  PyObject* t = PySequence_Tuple(v);
  if (!t) throw PySet();
  PyObject* i[2] = {nullptr, nullptr};
  const bool ok = PyTuple_GET_SIZE(t) == 2;
  for (int n = 0; ok && n < 2 && (n == 0 || i[0]); ++n) i[n] = PyNumber_Long(PyTuple_GET_ITEM(t, n));
  const long x = i[0] ? PyLong_AsLong(i[0]) : 0, y = i[1] ? PyLong_AsLong(i[1]) : 0;
  Py_XDECREF(i[0]);
  Py_XDECREF(i[1]);
  Py_DECREF(t);
  if (PyErr_Occurred()) throw PySet();
  if (!ok) raise(PyExc_ValueError, "expected a pair");
  *a = static_cast<int>(x);
  *b = static_cast<int>(y);
}
// takes one keyword argument; false: not one of the attention options
bool take_option(Options& o, int name, PyObject* v) {
  switch (name) {
    case N_G: if (v != Py_None) o.G = static_cast<int>(as_long(v)); return true;
    case N_P_ROUND: o.p_round = word(v, "triton", "rne"); return true;
    case N_KV_ORDER: o.kv_order = word(v, "ascending", "descending"); return true;
    case N_STATE: {
      if (v == Py_None) return true;
      PyObject* t = PySequence_Tuple(v);
      if (!t) throw PySet();
      if (PyTuple_GET_SIZE(t) != 3) {
        Py_DECREF(t);
        raise(PyExc_ValueError, "state is (m, l, acc)");
      }
      at::Tensor* dst[3] = {&o.m, &o.l, &o.acc};
      bool ok = true;
      for (int i = 0; i < 3; ++i) {
        PyObject* x = PyTuple_GET_ITEM(t, i);
        ok = ok && THPVariable_Check(x);
        if (ok) *dst[i] = THPVariable_Unpack(x);
      }
      Py_DECREF(t);
      if (!ok) raise(PyExc_TypeError, "state holds tensors");
      for (at::Tensor* x : dst)
        if (!x->is_contiguous() || !is(*x, at::kFloat)) raise(PyExc_AssertionError, "state tensors are contiguous float32");
      o.have_state = true;
      return true;
    }
    case N_Q_OFFSET: o.q_offset = as_long(v); return true;
    case N_KV_OFFSET: o.kv_offset = as_long(v); return true;
    case N_RETURN_STATE: o.return_state = truth(v); return true;
    case N_RETURN_LSE: o.return_lse = truth(v); return true;
    case N_WRITE_O: o.write_o = truth(v); return true;
    case N_TAP: if (v != Py_None) { o.tap = true; pair_of_ints(v, &o.tap_tile, &o.tap_step); } return true;
    case N_OUT: {
      if (!THPDtype_Check(v)) raise(PyExc_TypeError, "out_dtype must be torch.float16 or torch.bfloat16");
      o.out = reinterpret_cast<THPDtype*>(v)->scalar_type;
      if (o.out != at::kHalf && o.out != at::kBFloat16) raise(PyExc_TypeError, "out_dtype must be torch.float16 or torch.bfloat16");
      return true;
    }
    case N_WAIT: if (v != Py_None) pair_of_ints(v, &o.wait_kcycles, &o.skip_k); return true;
    default: return false;
  }
}
void take_options(Options& o, PyObject* const* values, PyObject* kwnames) {
  const Py_ssize_t n = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
  for (Py_ssize_t i = 0; i < n; ++i)
    if (!take_option(o, name_index(PyTuple_GET_ITEM(kwnames, i)), values[i]))
      raise(PyExc_TypeError, std::string("unexpected keyword argument '") + PyUnicode_AsUTF8(PyTuple_GET_ITEM(kwnames, i)) + "'");
}

int default_G(int64_t D, bool full) {
  if (!full) return D == 256 ? 64 : 128;
  return D >= 128 ? 128 : D >= 64 ? 64 : 32;
}

void set_sizes(IntfaFwdParams& P, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, bool full, int G) {
  P.B = q.size(0);
  P.H = q.size(1);
  P.Nq = q.size(2);
  P.D = q.size(3);
  P.Nk = k.size(2);
  P.H_kv = k.size(1);                       // grouped-query attention: fewer K/V heads than query heads
  if (P.H_kv <= 0 || v.size(1) != P.H_kv || P.H % P.H_kv != 0)
    raise(PyExc_ValueError, "k and v must have the same number of heads, dividing the " + std::to_string(P.H) + " query heads");
  // (longer ones are read in part)
  if (k.size(0) < P.B || v.size(0) < P.B) raise(PyExc_ValueError, "k and v must have the batch size of q, " + std::to_string(P.B));
  if (v.size(2) < P.Nk) raise(PyExc_ValueError, "v must have the " + std::to_string(P.Nk) + " keys of k, got " + std::to_string(v.size(2)));
  P.variant = full ? INTFA_VARIANT_FULL : is(v, at::kFloat8_e5m2) ? INTFA_VARIANT_HALF_FP8 : INTFA_VARIANT_HALF;
  P.G = G != kAutoG ? G : default_G(P.D, full);
}
void need_4d(const at::Tensor& t, const char* what) {
  if (t.dim() != 4) raise(PyExc_ValueError, std::string(what) + " must have four dimensions [B,H,N,D]");
}
void check_v_type(const at::Tensor& v, bool full) {
  if (full && !is(v, at::kChar)) raise(PyExc_TypeError, "full-int8: v must be int8");
  // V (and with it P) in fp8: flash_atten_int8.py:55-56
  if (!full && !is(v, at::kHalf) && !is(v, at::kFloat8_e5m2)) raise(PyExc_TypeError, "half-int8: v must be float16 or float8_e5m2");
}
// The kernels read a scale tensor by its strides: `last` is the index of the last element they touch.
void need_scales(const at::Tensor& s, const char* what, int64_t last) {
  if (last >= s.numel())
    raise(PyExc_ValueError, std::string(what) + " is too short: element " + std::to_string(last) + " is read, it holds " + std::to_string(s.numel()));
}
void check_head_dims(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v) {
  // shape constraints, as flash_atten_full_int8.py:189-193
  const int64_t d = q.size(-1);
  if (k.size(-1) != d || v.size(-1) != d || (d != 16 && d != 32 && d != 64 && d != 128 && d != 256))
    raise(PyExc_AssertionError, "head dims of q, k and v must be equal and one of 16, 32, 64, 128, 256");
}

PyObject* tuple_of(std::initializer_list<at::Tensor> ts) {
  PyObject* t = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
  Py_ssize_t n = 0;
  for (const at::Tensor& x : ts) PyTuple_SET_ITEM(t, n++, THPVariable_Wrap(x));
  return t;
}

// the forward on prepared tensors: P holds the tensors, strides, sizes and variant
PyObject* forward(IntfaFwdParams& P, Options& o, c10::Device dev, bool causal, double sm_scale) {
  const int64_t B = P.B, H = P.H, Nq = P.Nq, D = P.D;
  at::Tensor out = o.write_o ? empty({B, H, Nq, D}, o.out, dev) : empty({1, 1, 1, 8}, o.out, dev);
  P.o = out.data_ptr();
  for (int i = 0; i < 3; ++i) P.o_stride[i] = out.stride(i);
  P.o_dtype = o.out == at::kBFloat16 ? INTFA_OUT_BF16 : INTFA_OUT_FP16;
  P.causal = causal ? 1 : 0;
  P.sm_scale = static_cast<float>(sm_scale);
  P.p_round = o.p_round;
  P.kv_order = o.kv_order;
  P.q_offset = o.q_offset;
  P.kv_offset = o.kv_offset;
  at::Tensor lse, tap_s, tap_p;
  if (o.return_lse) {
    lse = empty({B, H, Nq}, at::kFloat, dev);
    P.lse_out = lse.data_ptr<float>();
  }
  if (o.have_state || o.return_state) {
    if (o.have_state) {
      const int64_t rows = B * H * Nq;
      for (const at::Tensor* x : {&o.m, &o.l, &o.acc})
        if (x->device() != dev || x->numel() < (x == &o.acc ? rows * D : rows))
          raise(PyExc_ValueError, "state is (m, l [B,H,Nq], acc [B,H,Nq,D]) on the device of q");
    } else {
      o.m = empty({B, H, Nq}, at::kFloat, dev);
      o.l = empty({B, H, Nq}, at::kFloat, dev);
      o.acc = empty({B, H, Nq, D}, at::kFloat, dev);
    }
    P.state_in = o.have_state;
    P.state_out = o.return_state;
    P.state_m = o.m.data_ptr<float>();
    P.state_l = o.l.data_ptr<float>();
    P.state_acc = o.acc.data_ptr<float>();
  }
  P.write_o = o.write_o;
  if (o.tap) {
    const auto opt = at::TensorOptions().device(dev);
    tap_s = at::zeros({128, P.G}, opt.dtype(at::kInt));
    tap_p = at::zeros({128, P.G}, opt.dtype(P.variant == INTFA_VARIANT_FULL ? at::kChar : P.variant == INTFA_VARIANT_HALF_FP8 ? at::kByte : at::kHalf));
    P.dbg_s = tap_s.data_ptr<int>();
    P.dbg_p = tap_p.data_ptr();
    P.dbg_tile = o.tap_tile;
    P.dbg_step = o.tap_step;
  }
  P.debug_wait_limit_kcycles = o.wait_kcycles;
  P.debug_skip_k_load = o.skip_k;
  at::Tensor ws;
  if (const size_t bytes = intfa_fwd_workspace_bytes(&P)) {
    ws = empty({static_cast<int64_t>(bytes)}, at::kByte, dev);
    P.workspace = ws.data_ptr();
    P.workspace_bytes = bytes;
  }
  const at::Tensor st = status_word(dev);
  P.status = st.data_ptr<int>();
  void* stream = stream_of(dev);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = intfa_fwd(&P, stream);
  Py_END_ALLOW_THREADS
  check(rc);
  PyObject* po = o.write_o ? THPVariable_Wrap(out) : Py_NewRef(Py_None);
  const int extra = (o.return_state ? 1 : 0) + (o.return_lse ? 1 : 0) + (o.tap ? 1 : 0);
  if (extra == 0) return po;
  PyObject* t = PyTuple_New(1 + extra);
  Py_ssize_t n = 0;
  PyTuple_SET_ITEM(t, n++, po);
  if (o.return_state) PyTuple_SET_ITEM(t, n++, tuple_of({o.m, o.l, o.acc}));
  if (o.return_lse) PyTuple_SET_ITEM(t, n++, THPVariable_Wrap(lse));
  if (o.tap) PyTuple_SET_ITEM(t, n++, tuple_of({tap_s, tap_p}));
  return t;
}

// fwd(full, q, k, v, q_scale, k_scale, v_scale | None, causal, sm_scale, **options)
PyObject* fwd(PyObject*, PyObject* const* a, Py_ssize_t n, PyObject* kwnames) {
  HANDLE_TH_ERRORS
  try {
    if (n != 9) raise(PyExc_TypeError, "fwd takes 9 positional arguments");
    const bool full = truth(a[0]);
    const at::Tensor &q0 = tensor(a[1], "q"), &k0 = tensor(a[2], "k"), &v0 = tensor(a[3], "v");
    check_head_dims(q0, k0, v0);
    const at::Tensor &qs0 = tensor(a[4], "q_scale"), &ks0 = tensor(a[5], "k_scale");
    for (const at::Tensor* t : {&q0, &k0, &v0, &qs0, &ks0}) need_cuda(*t);
    if (a[6] != Py_None) need_cuda(tensor(a[6], "v_scale"));
    for (const at::Tensor* t : {&k0, &v0, &qs0, &ks0})
      if (t->device() != q0.device()) raise(PyExc_ValueError, "all tensors must be on the device of q");
    if (!is(q0, at::kChar) || !is(k0, at::kChar)) raise(PyExc_TypeError, "q and k must be int8");
    check_v_type(v0, full);
    need_4d(q0, "q");
    need_4d(k0, "k");
    need_4d(v0, "v");
    if (qs0.dim() < 2 || ks0.dim() < 2) raise(PyExc_ValueError, "q_scale and k_scale must have shape (B,H,N)");
    Options o;
    take_options(o, a + n, kwnames);
    IntfaFwdParams P{};
    set_sizes(P, q0, k0, v0, full, o.G);
    const c10::Device dev = q0.device();
    c10::cuda::CUDAGuard guard(dev);
    const at::Tensor q = tma_ready(q0), k = tma_ready(k0), v = tma_ready(v0), qs = scales(qs0);
    at::Tensor ks = scales(ks0);
    // (where the last KV step is partial, one scale per (batch, head) has always stood for all its keys)
    const bool ragged = P.G > 0 && P.Nk % P.G != 0;
    if (ragged && ks.dim() == 3 && ks.size(2) == 1) ks = ks.expand({ks.size(0), ks.size(1), P.Nk}).contiguous();
    at::Tensor vs;
    P.q = q.data_ptr();
    P.k = k.data_ptr();
    P.v = v.data_ptr();
    P.q_scale = qs.data_ptr();
    P.k_scale = ks.data_ptr();
    for (int i = 0; i < 3; ++i) {
      P.q_stride[i] = q.stride(i);
      P.k_stride[i] = k.stride(i);
      P.v_stride[i] = v.stride(i);
    }
    for (int i = 0; i < 2; ++i) {
      P.qs_stride[i] = qs.stride(i);
      P.ks_stride[i] = ks.stride(i);
    }
    need_scales(qs, "q_scale", (P.B - 1) * P.qs_stride[0] + (P.H - 1) * P.qs_stride[1] + P.Nq - 1);
    need_scales(ks, "k_scale", (P.B - 1) * P.ks_stride[0] + (P.H_kv - 1) * P.ks_stride[1] + P.Nk - 1);
    // (... and rows of another length an error)
    if (ragged && (ks.dim() != 3 || ks.size(2) != P.Nk))
      raise(PyExc_ValueError, "k_scale must have shape (B,H," + std::to_string(P.Nk) + ")");
    P.scale_f16 = (is(qs, at::kHalf) ? INTFA_SCALE_F16_Q : 0) | (is(ks, at::kHalf) ? INTFA_SCALE_F16_K : 0);
    if (full) {
      vs = scales(tensor(a[6], "v_scale"));
      P.scale_f16 |= is(vs, at::kHalf) ? INTFA_SCALE_F16_V : 0;
      P.v_scale = vs.data_ptr();
      const int64_t d = vs.dim();
      if (d < 2 || d > 4) raise(PyExc_ValueError, "v_scale must have shape (B,H), (B,H,D) or (B,H,ceil(Nk/G),D)");
      P.vs_stride[0] = vs.stride(0);
      P.vs_stride[1] = vs.stride(1);
      // (B,H): one scale per (batch, head), benchmark.py:102-107; (B,H,D): per channel; (B,H,ceil(Nk/G),D): one row per KV tile,
      // the CUDA path's layout
      P.vs_stride[2] = d == 2 ? 0 : vs.stride(d - 1);
      if (d == 4) {
        const int64_t want = P.G > 0 ? (P.Nk + P.G - 1) / P.G : 0;
        if (vs.size(2) != want)
          raise(PyExc_ValueError, "per-tile v_scale needs ceil(Nk/G) = " + std::to_string(want) + " rows, got " + std::to_string(vs.size(2)));
        P.vs_stride_blk = vs.stride(2);
      }
      if (vs.device() != dev) raise(PyExc_ValueError, "all tensors must be on the device of q");
      need_scales(vs, "v_scale", (P.B - 1) * P.vs_stride[0] + (P.H_kv - 1) * P.vs_stride[1] + (P.D - 1) * P.vs_stride[2] +
                                     (d == 4 ? (vs.size(2) - 1) * P.vs_stride_blk : 0));
    }
    return forward(P, o, dev, truth(a[7]), as_double(a[8]));
  } catch (const PySet&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------------------------
// quantisers
// ---------------------------------------------------------------------------------------------------------------
at::Tensor quant_in(const at::Tensor& x) {
  need_cuda(x);
  if (!is(x, at::kHalf) || x.dim() != 4) raise(PyExc_TypeError, "quantisers take a float16 [B,H,N,D] tensor");
  const bool ok = x.stride(3) == 1 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0 && x.stride(0) % 8 == 0 && x.stride(1) % 8 == 0 &&
                  x.stride(2) % 8 == 0;
  return ok ? x : x.contiguous();
}

PyObject* quant_pertoken(PyObject*, PyObject* arg) {
  HANDLE_TH_ERRORS
  try {
    const at::Tensor& x0 = tensor(arg, "X");
    need_cuda(x0);
    c10::cuda::CUDAGuard guard(x0.device());
    const at::Tensor x = quant_in(x0);
    at::Tensor x8 = empty(x.sizes(), at::kChar, x.device());
    at::Tensor s = empty(x.sizes().slice(0, 3), at::kFloat, x.device());
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = intfa_quant_pertoken(x.data_ptr(), x.strides().data(), x8.data_ptr(), s.data_ptr<float>(), x.size(0), x.size(1), x.size(2), x.size(3),
                              stream_of(x.device()));
    Py_END_ALLOW_THREADS
    check(rc);
    return tuple_of({x8, s});
  } catch (const PySet&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// quant_v(X, mode)
PyObject* quant_v(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    if (n != 2) raise(PyExc_TypeError, "quant_v takes 2 arguments");
    const at::Tensor& x0 = tensor(a[0], "X");
    need_cuda(x0);
    const int mode = static_cast<int>(as_long(a[1]));
    c10::cuda::CUDAGuard guard(x0.device());
    const at::Tensor x = quant_in(x0);
    const int64_t B = x.size(0), H = x.size(1), N = x.size(2), D = x.size(3);
    at::Tensor x8 = empty({B, H, N, D}, at::kChar, x.device());
    at::Tensor s = mode == INTFA_VSCALE_PER_CHANNEL ? empty({B, H, D}, at::kFloat, x.device()) : empty({B, H}, at::kFloat, x.device());
    const size_t bytes = intfa_quant_v_partial_workspace_bytes(B, H, N, D);
    at::Tensor ws = empty({static_cast<int64_t>(bytes)}, at::kByte, x.device());
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = intfa_quant_v_partial(x.data_ptr(), x.strides().data(), x8.data_ptr(), s.data_ptr<float>(), mode, B, H, N, D, ws.data_ptr(), bytes,
                               stream_of(x.device()));
    Py_END_ALLOW_THREADS
    check(rc);
    return tuple_of({x8, s});
  } catch (const PySet&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// the three tensors of one call, checked and with the strides the prologue takes
struct Qkv {
  at::Tensor q, k, v;
  int64_t B, H, Hkv, Nq, Nk, D;
};
Qkv qkv_in(const at::Tensor& q0, const at::Tensor& k0, const at::Tensor* v0) {
  Qkv x;
  if (k0.device() != q0.device() || (v0 && v0->device() != q0.device())) raise(PyExc_ValueError, "q, k and v must be on the same device");
  x.q = quant_in(q0).contiguous();
  x.k = quant_in(k0).contiguous();
  if (v0) {
    x.v = quant_in(*v0);
    if (x.v.sizes() != x.k.sizes()) raise(PyExc_ValueError, "k and v must have the same shape");
  }
  x.B = x.q.size(0);
  x.H = x.q.size(1);
  x.Nq = x.q.size(2);
  x.D = x.q.size(3);
  x.Hkv = x.k.size(1);
  x.Nk = x.k.size(2);
  if (x.k.size(0) < x.B) raise(PyExc_ValueError, "k must have the batch size of q, " + std::to_string(x.B));
  return x;
}
void run_quant_qkv(const Qkv& x, void* q8, void* k8, void* v8, float* qs, float* ks, float* vs, int mode, void* ws, size_t ws_bytes) {
  int rc;
  const bool v = x.v.defined();
  const int64_t none[4] = {0, 0, 0, 0};
  Py_BEGIN_ALLOW_THREADS
  rc = intfa_quant_qkv(x.q.data_ptr(), x.k.data_ptr(), v ? x.v.data_ptr() : nullptr, v ? x.v.strides().data() : none, q8, k8, v8, qs, ks, vs, mode,
                       x.B, x.H, x.Hkv, x.Nq, x.Nk, x.D, ws, ws_bytes, stream_of(x.q.device()));
  Py_END_ALLOW_THREADS
  check(rc);
}

// quant_qkv(q, k, v | None, mode)
PyObject* quant_qkv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    if (n != 4) raise(PyExc_TypeError, "quant_qkv takes 4 arguments");
    const at::Tensor& q0 = tensor(a[0], "q");
    const at::Tensor& k0 = tensor(a[1], "k");
    const bool have_v = a[2] != Py_None;
    need_cuda(q0);
    const int mode = static_cast<int>(as_long(a[3]));
    const c10::Device dev = q0.device();
    c10::cuda::CUDAGuard guard(dev);
    const Qkv x = qkv_in(q0, k0, have_v ? &tensor(a[2], "v") : nullptr);
    if (x.k.size(3) != x.D) raise(PyExc_ValueError, "q and k must have the same head dim");
    at::Tensor q8 = empty({x.B, x.H, x.Nq, x.D}, at::kChar, dev), k8 = empty({x.B, x.Hkv, x.Nk, x.D}, at::kChar, dev);
    at::Tensor qs = empty({x.B, x.H, x.Nq}, at::kFloat, dev), ks = empty({x.B, x.Hkv, x.Nk}, at::kFloat, dev);
    if (!have_v) {
      run_quant_qkv(x, q8.data_ptr(), k8.data_ptr(), nullptr, qs.data_ptr<float>(), ks.data_ptr<float>(), nullptr, mode, nullptr, 0);
      return tuple_of({q8, qs, k8, ks});
    }
    at::Tensor v8 = empty({x.B, x.Hkv, x.Nk, x.D}, at::kChar, dev);
    at::Tensor vs = mode == INTFA_VSCALE_PER_CHANNEL ? empty({x.B, x.Hkv, x.D}, at::kFloat, dev) : empty({x.B, x.Hkv}, at::kFloat, dev);
    const size_t bytes = intfa_quant_qkv_workspace_bytes(x.B, x.Hkv, x.Nk, x.D);
    at::Tensor ws = empty({static_cast<int64_t>(bytes)}, at::kByte, dev);
    run_quant_qkv(x, q8.data_ptr(), k8.data_ptr(), v8.data_ptr(), qs.data_ptr<float>(), ks.data_ptr<float>(), vs.data_ptr<float>(), mode,
                  ws.data_ptr(), bytes);
    return tuple_of({q8, qs, k8, ks, v8, vs});
  } catch (const PySet&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// flash(q, k, v, causal, sm_scale, variant, v_mode, **options): prologue and forward, with the quantised tensors, their scales
// and the scratch in ONE buffer
PyObject* flash(PyObject*, PyObject* const* a, Py_ssize_t n, PyObject* kwnames) {
  HANDLE_TH_ERRORS
  try {
    if (n != 7) raise(PyExc_TypeError, "flash takes 7 positional arguments");
    Options o;
    take_options(o, a + n, kwnames);
    const bool full = equals(a[5], "full");
    const int mode = equals(a[6], "per_channel") ? INTFA_VSCALE_PER_CHANNEL : INTFA_VSCALE_PER_TENSOR;
    const at::Tensor &q0 = tensor(a[0], "q"), &k0 = tensor(a[1], "k"), &v0 = tensor(a[2], "v");
    need_cuda(q0);
    const c10::Device dev = q0.device();
    c10::cuda::CUDAGuard guard(dev);
    const Qkv x = qkv_in(q0, k0, full ? &v0 : nullptr);
    at::Tensor v = x.v;
    if (!full) {
      need_cuda(v0);
      if (v0.device() != dev) raise(PyExc_ValueError, "q, k and v must be on the same device");
      check_v_type(v0, false);
      need_4d(v0, "v");
      v = tma_ready(v0);
    }
    check_head_dims(x.q, x.k, v);
    IntfaFwdParams P{};
    set_sizes(P, x.q, x.k, v, full, o.G);
    size_t used = 0;
    const auto take = [&](size_t bytes) {
      const size_t r = used;
      used += (bytes + 255) / 256 * 256;
      return r;
    };
    const bool pc = mode == INTFA_VSCALE_PER_CHANNEL;
    const size_t rq = static_cast<size_t>(x.B) * x.H * x.Nq, rk = static_cast<size_t>(x.B) * x.Hkv * x.Nk, sv = static_cast<size_t>(x.B) * x.Hkv * (pc ? x.D : 1);
    const size_t o_q = take(rq * x.D), o_k = take(rk * x.D), o_qs = take(rq * 4), o_ks = take(rk * 4);
    const size_t ws_bytes = full ? intfa_quant_qkv_workspace_bytes(x.B, x.Hkv, x.Nk, x.D) : 0;
    const size_t o_v = take(full ? rk * x.D : 0), o_vs = take(full ? sv * 4 : 0), o_ws = take(ws_bytes);
    at::Tensor buf = empty({static_cast<int64_t>(used)}, at::kByte, dev);
    char* b = static_cast<char*>(buf.data_ptr());
    run_quant_qkv(x, b + o_q, b + o_k, b + o_v, reinterpret_cast<float*>(b + o_qs), reinterpret_cast<float*>(b + o_ks),
                  reinterpret_cast<float*>(b + o_vs), mode, b + o_ws, ws_bytes);
    P.q = b + o_q;
    P.k = b + o_k;
    P.v = full ? b + o_v : v.data_ptr();
    P.q_scale = b + o_qs;
    P.k_scale = b + o_ks;
    P.v_scale = full ? b + o_vs : nullptr;
    const int64_t sq[3] = {x.H * x.Nq * x.D, x.Nq * x.D, x.D}, sk[3] = {x.Hkv * x.Nk * x.D, x.Nk * x.D, x.D};
    for (int i = 0; i < 3; ++i) {
      P.q_stride[i] = sq[i];
      P.k_stride[i] = sk[i];
      P.v_stride[i] = full ? sk[i] : v.stride(i);
    }
    P.qs_stride[0] = x.H * x.Nq;
    P.qs_stride[1] = x.Nq;
    P.ks_stride[0] = x.Hkv * x.Nk;
    P.ks_stride[1] = x.Nk;
    if (full) {
      P.vs_stride[0] = pc ? x.Hkv * x.D : x.Hkv;
      P.vs_stride[1] = pc ? x.D : 1;
      P.vs_stride[2] = pc ? 1 : 0;
    }
    return forward(P, o, dev, truth(a[3]), as_double(a[4]));
  } catch (const PySet&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// the status word (int32[1] tensor) of a CUDA device
PyObject* status(PyObject*, PyObject* arg) {
  HANDLE_TH_ERRORS
  try {
    return THPVariable_Wrap(status_word(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(as_long(arg)))));
  } catch (const PySet&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

PyObject* set_error_class(PyObject*, PyObject* cls) {
  Py_INCREF(cls);
  Py_XSETREF(g_error_class, cls);
  Py_RETURN_NONE;
}

template <typename F>
PyCFunction method(F f) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}
PyMethodDef kMethods[] = {{"fwd", method(fwd), METH_FASTCALL | METH_KEYWORDS, nullptr},
                          {"flash", method(flash), METH_FASTCALL | METH_KEYWORDS, nullptr},
                          {"quant_pertoken", quant_pertoken, METH_O, nullptr},
                          {"quant_v", method(quant_v), METH_FASTCALL, nullptr},
                          {"quant_qkv", method(quant_qkv), METH_FASTCALL, nullptr},
                          {"status", status, METH_O, nullptr},
                          {"set_error_class", set_error_class, METH_O, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};
}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  for (int i = 0; i < N_COUNT; ++i)
    if (!(g_names[i] = PyUnicode_InternFromString(kNames[i]))) return nullptr;
  return PyModule_Create(&kModule);
}
