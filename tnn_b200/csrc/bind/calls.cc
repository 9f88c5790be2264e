// Calls from Python into the kernel library without ctypes.
//
// What bounds small models launched one by one is the host's time per launch, and a third of that was ctypes: 22 arguments
// converted one after the other through generic code, and a Python-level data_ptr() for every tensor among them. `Call`
// converts the arguments of an entry point itself and takes tensors as they are, `empty` allocates an output like torch.empty,
// `gemm` is the front of ops/gemm.py's gemm for its usual calls. Us of host time per call, the launch itself being 2.3: gemm
// 10.8 and 5.0, into a given output 7.7 and 3.6, layernorm_fwd 12.3 and 8.0, act_fwd 5.8 and 4.7. A step of a small GPT, 106
// launches, 1254 -> 770 us, with the shorter kernels of its products.
//
// An entry point is named by its address and a signature with one letter per argument (all return int):
//   p pointer (None, int or torch.Tensor)   i int   l long long   u unsigned long long   U unsigned   f float
// Signatures are compiled in (SIGNATURES below). Arguments that are none of these objects (ctypes values, arrays) send the
// whole call to `slow`, a Python callable with the same arguments.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ops/empty.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <utility>

namespace {

union Slot {
  void* p;
  unsigned long long n;  // every integer, two's complement: narrower parameters take the low bits, like ctypes
  float f;
};

template <size_t N>
struct Text {
  char s[N];
  constexpr Text(const char (&t)[N]) {
    for (size_t i = 0; i < N; ++i) s[i] = t[i];
  }
  static constexpr size_t size = N - 1;
};

template <char C> struct Param;
template <> struct Param<'p'> { using T = void*; static T get(const Slot& s) { return s.p; } };
template <> struct Param<'i'> { using T = int; static T get(const Slot& s) { return (int)s.n; } };
template <> struct Param<'l'> { using T = long long; static T get(const Slot& s) { return (long long)s.n; } };
template <> struct Param<'u'> { using T = unsigned long long; static T get(const Slot& s) { return s.n; } };
template <> struct Param<'U'> { using T = unsigned; static T get(const Slot& s) { return (unsigned)s.n; } };
template <> struct Param<'f'> { using T = float; static T get(const Slot& s) { return s.f; } };

using Invoke = int (*)(void* fn, const Slot* a);

template <Text S, size_t... I>
int invoke_as(void* fn, const Slot* a, std::index_sequence<I...>) {
  return reinterpret_cast<int (*)(typename Param<S.s[I]>::T...)>(fn)(Param<S.s[I]>::get(a[I])...);
}
template <Text S>
int invoke(void* fn, const Slot* a) {
  return invoke_as<S>(fn, a, std::make_index_sequence<S.size>());
}

struct Entry {
  const char* sig;
  Invoke invoke;
};
#define SIG(S) {S, &invoke<S>}
const Entry SIGNATURES[] = {
    SIG("pppiiiiilllppplpliiipp"),                      // gemm_bf16
    SIG("pppiiiiillli" "pp" "ipp"),                     // gemm_bf16_heads
    SIG("pppiii" "lllpppppfpliipp"),                    // gemm_bf16_norm
    SIG("pppppppp" "fpiiiiiiiiiiiiiipp"),               // conv2d_fwd_norm
    SIG("pplifp"), SIG("ppplifp"), SIG("pppliip"),      // act_fwd, act_bwd, binary
    SIG("pplfupp"),                                     // dropout
    SIG("ppppliillfupp"),                               // embedding_fwd, embedding_bwd
    SIG("plplip"), SIG("pplp"), SIG("plpplip"),         // colsum_accum, cast_f32_bf16, scale_by
    SIG("pppppppp" "liffupp"),                          // layernorm_fwd
    SIG("pppppppppp" "lifupp"), SIG("ppppppppppp" "lifupp"),  // layernorm_bwd, layernorm_bwd_db
    SIG("plpplppplif" "fp"),                            // softmax_ce
    SIG("ppppplffffffffpp"), SIG("pppplfffpp"),         // adam_step, sgd_step
    SIG("pppiiiiifpp"), SIG("pppppppiiiiifpp"),         // attn_fwd, attn_bwd
    SIG("pppliilfip"), SIG("ppppppliilfip"), SIG("pppiiiip"),  // attn_softmax_fwd, attn_softmax_bwd, attn_delta
    SIG("ppppppppp" "liffiip"), SIG("pppppppppp" "liffiip"), SIG("ppppppppppp" "liip"),  // batchnorm_fwd, _fwd_res, _bwd
    SIG("ppiiiiiiiiiiip"), SIG("pppiiiiiiiiiiip"),      // im2col, col2im; pool_fwd, pool_bwd
    SIG("ppiiiiiiiiiip"),                               // conv_weight_t
    SIG("ppppiiiiiiiiiiiipp"),                          // conv2d_fwd_implicit
    SIG("pppiiiiiiiiiiiiiiiiipp"),                      // conv2d_fwd_implicit_strided
    SIG("ppppiiiiiiiiiipp"), SIG("pppiiiiiiiiipp"), SIG("pppiiiiiiiiiiipp"),  // conv2d_fwd_halo, wgrad_halo, wgrad_implicit
};
constexpr int MAX_ARGS = 32;
constexpr const char* GEMM_SIG = "pppiiiiilllppplpliiipp";

struct Call {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  PyObject* slow;
  void* fn;
  Invoke invoke;
  int n;
  char sig[MAX_ARGS + 1];
};

PyObject* call_slow(Call* c, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  return PyObject_Vectorcall(c->slow, args, nargsf, kwnames);
}

// 1: converted, 0: not an object this code knows, -1: Python error set
int convert(char kind, PyObject* o, Slot& s) {
  if (kind == 'p') {
    if (o == Py_None) {
      s.p = nullptr;
      return 1;
    }
    if (THPVariable_CheckExact(o)) {
      s.p = THPVariable_Unpack(o).data_ptr();  // throws for tensors without memory of their own
      return 1;
    }
  }
  if (kind == 'f') {
    const double v = PyFloat_Check(o) ? PyFloat_AS_DOUBLE(o) : PyLong_Check(o) ? PyLong_AsDouble(o) : 0.0;
    if (!PyFloat_Check(o) && !PyLong_Check(o)) return 0;
    if (v == -1.0 && PyErr_Occurred()) return -1;
    s.f = (float)v;
    return 1;
  }
  if (!PyLong_Check(o)) return 0;
  s.n = PyLong_AsUnsignedLongLongMask(o);
  return s.n == (unsigned long long)-1 && PyErr_Occurred() ? -1 : 1;
}

PyObject* call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  HANDLE_TH_ERRORS
  Call* c = reinterpret_cast<Call*>(self);
  if (kwnames || PyVectorcall_NARGS(nargsf) != c->n) return call_slow(c, args, nargsf, kwnames);
  Slot a[MAX_ARGS];
  for (int i = 0; i < c->n; ++i) {
    const int ok = convert(c->sig[i], args[i], a[i]);
    if (ok < 0) return nullptr;
    if (ok == 0) return call_slow(c, args, nargsf, kwnames);
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS  // a launch waits when the driver's queue is full
  rc = c->invoke(c->fn, a);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

void call_dealloc(PyObject* self) {
  Py_XDECREF(reinterpret_cast<Call*>(self)->slow);
  Py_TYPE(self)->tp_free(self);
}

PyTypeObject CallType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// bind(address, signature, slow) -> callable, or None for a signature that is not compiled in
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3 || !PyLong_Check(args[0]) || !PyUnicode_Check(args[1]) || !PyCallable_Check(args[2])) {
    PyErr_SetString(PyExc_TypeError, "bind(address, signature, slow)");
    return nullptr;
  }
  const char* sig = PyUnicode_AsUTF8(args[1]);
  if (!sig) return nullptr;
  void* fn = PyLong_AsVoidPtr(args[0]);
  if (!fn && PyErr_Occurred()) return nullptr;
  for (const Entry& e : SIGNATURES) {
    if (fn && std::strcmp(e.sig, sig) == 0) {
      Call* c = PyObject_New(Call, &CallType);
      if (!c) return nullptr;
      c->vectorcall = call;
      c->slow = Py_NewRef(args[2]);
      c->fn = fn;
      c->invoke = e.invoke;
      c->n = (int)std::strlen(sig);
      std::strcpy(c->sig, sig);
      return reinterpret_cast<PyObject*>(c);
    }
  }
  Py_RETURN_NONE;
}

// at::empty without the interpreter lock, like torch.empty: an allocation may wait for the device, and the other threads should not.
at::Tensor empty_unlocked(at::IntArrayRef sizes, const at::TensorOptions& opt) {
  struct Unlocked {
    PyThreadState* state = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(state); }
  } unlocked;
  return at::empty(sizes, opt);
}

// empty(like, *sizes): an uninitialised contiguous tensor of like's dtype on its device; empty(like, dtype, *sizes): of dtype
PyObject* empty(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 1 || !THPVariable_Check(args[0])) {
    PyErr_SetString(PyExc_TypeError, "empty(like, [dtype,] *sizes)");
    return nullptr;
  }
  const at::Tensor& like = THPVariable_Unpack(args[0]);
  at::TensorOptions opt = at::TensorOptions().device(like.device()).dtype(like.dtype());
  Py_ssize_t first = 1;
  if (n > 1 && THPDtype_Check(args[1])) {
    opt = opt.dtype(reinterpret_cast<THPDtype*>(args[1])->scalar_type);
    first = 2;
  }
  int64_t sizes[8];
  if (n - first > 8) {
    PyErr_SetString(PyExc_TypeError, "empty: at most 8 dimensions");
    return nullptr;
  }
  for (Py_ssize_t i = first; i < n; ++i) {
    sizes[i - first] = PyLong_AsLongLong(args[i]);
    if (sizes[i - first] == -1 && PyErr_Occurred()) return nullptr;
  }
  return THPVariable_Wrap(empty_unlocked(at::IntArrayRef(sizes, (size_t)(n - first)), opt));
  END_HANDLE_TH_ERRORS
}

// A matrix as the products take it: 2-D bf16 with a unit inner stride, row pitch and address multiples of 16 bytes.
bool operand(const at::Tensor& t, int64_t& ld) {
  if (t.dim() != 2 || t.scalar_type() != at::kBFloat16 || t.stride(1) != 1) return false;
  ld = t.size(0) > 1 ? t.stride(0) : std::max(t.stride(0), t.size(1));
  return ld % 8 == 0 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}

// gemm(entry, a, b, a_t, b_t, bias, z, dgelu_of, residual, out, dtype, flags, split_k, force_bn, status, stream) -> out
// The usual calls of ops/gemm.py's gemm on a GPU, checked and launched without Python in between: `entry` is the bound
// tnnb_gemm_bf16, flags the epilogue bits that are not implied by a tensor. None for anything unusual (operands that must be
// copied first, wrong shapes or types), which ops/gemm.py then handles or refuses itself.
enum { F_BIAS = 1, F_GELU = 2, F_DGELU = 4, F_RESID = 8, F_RELU = 16, F_ATOMIC = 32, F_OUT_F32 = 64, F_ACCUM = 128 };
PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 16 || Py_TYPE(args[0]) != &CallType || !THPVariable_CheckExact(args[1]) || !THPVariable_CheckExact(args[2])) Py_RETURN_NONE;
  const Call* c = reinterpret_cast<const Call*>(args[0]);
  if (std::strcmp(c->sig, GEMM_SIG) != 0) Py_RETURN_NONE;
  const at::Tensor &a = THPVariable_Unpack(args[1]), &b = THPVariable_Unpack(args[2]);
  const int a_t = PyObject_IsTrue(args[3]), b_t = PyObject_IsTrue(args[4]);
  if (a_t < 0 || b_t < 0) return nullptr;
  int64_t lda, ldb;
  if (!a.is_cuda() || a.device() != b.device() || !operand(a, lda) || !operand(b, ldb)) Py_RETURN_NONE;
  const int64_t M = a.size(a_t ? 1 : 0), K = a.size(a_t ? 0 : 1), N = b.size(b_t ? 1 : 0);
  if (b.size(b_t ? 0 : 1) != K || M > INT_MAX || N > INT_MAX || K > INT_MAX) Py_RETURN_NONE;
  // bias, z, dgelu_of, residual: absent, or plain tensors of the right type and extent
  const at::Tensor* t[4] = {nullptr, nullptr, nullptr, nullptr};
  for (int i = 0; i < 4; ++i) {
    if (args[5 + i] == Py_None) continue;
    if (!THPVariable_CheckExact(args[5 + i])) Py_RETURN_NONE;
    t[i] = &THPVariable_Unpack(args[5 + i]);
    if (t[i]->scalar_type() != at::kBFloat16 || t[i]->device() != a.device()) Py_RETURN_NONE;
    const bool fits = i == 0 ? t[i]->numel() == N && t[i]->is_contiguous()
                             : t[i]->dim() == 2 && t[i]->size(0) == M && t[i]->size(1) == N && t[i]->stride(1) == 1;
    if (!fits) Py_RETURN_NONE;
  }
  long flags = PyLong_AsLong(args[11]);
  const long split_k = PyLong_AsLong(args[12]), force_bn = PyLong_AsLong(args[13]);
  if (PyErr_Occurred()) return nullptr;
  flags |= (t[0] ? F_BIAS : 0) | (t[2] ? F_DGELU : 0) | (t[3] ? F_RESID : 0);
  if (t[1] && !(flags & F_GELU)) Py_RETURN_NONE;
  if (t[1] && t[2]) Py_RETURN_NONE;
  at::Tensor out;
  if (args[9] != Py_None) {
    if (!THPVariable_CheckExact(args[9])) Py_RETURN_NONE;
    out = THPVariable_Unpack(args[9]);
    if (out.dim() != 2 || out.size(0) != M || out.size(1) != N || out.stride(1) != 1 || out.device() != a.device()) Py_RETURN_NONE;
  } else {
    if (args[10] != Py_None && !THPDtype_Check(args[10])) Py_RETURN_NONE;
    const auto type = args[10] == Py_None ? a.scalar_type() : reinterpret_cast<THPDtype*>(args[10])->scalar_type;
    if (type != at::kBFloat16 && type != at::kFloat) Py_RETURN_NONE;
    out = empty_unlocked({M, N}, at::TensorOptions().device(a.device()).dtype(type));
  }
  const bool f32 = out.scalar_type() == at::kFloat;
  if ((!f32 && out.scalar_type() != at::kBFloat16) || ((flags & F_ATOMIC) && !f32)) Py_RETURN_NONE;
  if (flags & F_ATOMIC) flags &= ~F_ACCUM;
  else if (f32) flags |= F_OUT_F32;
  const auto pitch = [](const at::Tensor& x) { return x.size(0) > 1 ? x.stride(0) : std::max(x.stride(0), x.size(1)); };
  const auto ptr = [](const at::Tensor* x) { return x ? x->data_ptr() : nullptr; };
  const at::Tensor* aux = t[1] ? t[1] : t[2];
  Slot s[22];
  s[0].p = a.data_ptr(), s[1].p = b.data_ptr(), s[2].p = out.data_ptr();
  s[3].n = M, s[4].n = N, s[5].n = K, s[6].n = a_t, s[7].n = b_t;
  s[8].n = lda, s[9].n = ldb, s[10].n = pitch(out);
  s[11].p = ptr(t[0]), s[12].p = ptr(t[2]), s[13].p = ptr(t[1]);
  s[14].n = aux ? pitch(*aux) : 0;
  s[15].p = ptr(t[3]), s[16].n = t[3] ? pitch(*t[3]) : 0;
  s[17].n = flags, s[18].n = split_k, s[19].n = force_bn;
  s[20].p = PyLong_AsVoidPtr(args[14]), s[21].p = PyLong_AsVoidPtr(args[15]);
  if (PyErr_Occurred()) return nullptr;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = c->invoke(c->fn, s);
  Py_END_ALLOW_THREADS
  if (rc != 0) {
    PyErr_Format(PyExc_RuntimeError, "tnnb_gemm_bf16 rejected the call (code %d)", rc);
    return nullptr;
  }
  if (args[9] != Py_None) return Py_NewRef(args[9]);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyMethodDef METHODS[] = {
    {"gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(gemm)), METH_FASTCALL, "a product, or None"},
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, "bind(address, signature, slow)"},
    {"empty", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(empty)), METH_FASTCALL, "empty(like, [dtype,] *sizes)"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef MODULE = {PyModuleDef_HEAD_INIT, "_calls", "Calls into the kernel library.", -1, METHODS};

}  // namespace

PyMODINIT_FUNC PyInit__calls() {
  CallType.tp_name = "tnn_b200.Call";
  CallType.tp_basicsize = sizeof(Call);
  CallType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  CallType.tp_vectorcall_offset = offsetof(Call, vectorcall);
  CallType.tp_call = PyVectorcall_Call;
  CallType.tp_dealloc = call_dealloc;
  if (PyType_Ready(&CallType) < 0) return nullptr;
  return PyModule_Create(&MODULE);
}
