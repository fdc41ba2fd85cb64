// The host's side of a launch, as a CPython module: functions of the kernel libraries as callables that take tensors, and the
// checks that the wrappers make on their tensors.  (What torch throws, for a tensor without memory for one, becomes a Python error.)
//
// A small step is bound by the host: per launch, some 3 us in the driver and, with ctypes and the tensors' Python attributes, 9 to
// 12 us around it.  A callable made here turns its arguments (a tensor stands for its address) in some 0.3 us for twenty of them
// where ctypes takes 3, and a check of type, sizes and strides is one call instead of six attributes.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>
#include <unordered_map>
#include <utility>
#include <vector>

namespace {

constexpr int MAX_ARGS = 48;
union Slot {
  void* p;
  int64_t l;
  int i;
  float f;
  size_t z;
};
using P = void*;
using L = int64_t;
using I = int;
using F = float;
using Z = size_t;

template <class T>
T get(const Slot& s);
template <> inline P get<P>(const Slot& s) { return s.p; }
template <> inline L get<L>(const Slot& s) { return s.l; }
template <> inline I get<I>(const Slot& s) { return s.i; }
template <> inline F get<F>(const Slot& s) { return s.f; }
template <> inline Z get<Z>(const Slot& s) { return s.z; }

template <class R, class... A, size_t... K>
int64_t apply(void* fn, const Slot* s, std::index_sequence<K...>) {
  (void)s;
  return (int64_t) reinterpret_cast<R (*)(A...)>(fn)(get<A>(s[K])...);
}
template <class R, class... A>
int64_t thunk(void* fn, const Slot* s) {
  return apply<R, A...>(fn, s, std::index_sequence_for<A...>{});
}
using Thunk = int64_t (*)(void*, const Slot*);

// The signatures that the package's functions have: result, then arguments (written by build.py).
const std::unordered_map<std::string, Thunk>& thunks() {
  static const std::unordered_map<std::string, Thunk> table = {
#include "launch_signatures.inc"
  };
  return table;
}

PyObject* native_error = nullptr;      // raised for tensors that are not on a device

struct Fn {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  void* addr;
  Thunk thunk;
  int n;
  char kind[MAX_ARGS];
  PyObject* name;
};

PyObject* fn_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  HANDLE_TH_ERRORS
  Fn* f = reinterpret_cast<Fn*>(self);
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != f->n || (kwnames && PyTuple_GET_SIZE(kwnames))) return PyErr_Format(PyExc_TypeError, "%U takes %d arguments", f->name, f->n);
  Slot s[MAX_ARGS];
  for (int i = 0; i < f->n; ++i) {
    PyObject* a = args[i];
    switch (f->kind[i]) {
      case 'P':
        if (THPVariable_Check(a)) s[i].p = THPVariable_Unpack(a).data_ptr();
        else if (PyLong_Check(a)) s[i].p = PyLong_AsVoidPtr(a);
        else return PyErr_Format(PyExc_TypeError, "%U: argument %d is a tensor or an address, not %s", f->name, i, Py_TYPE(a)->tp_name);
        break;
      case 'F': s[i].f = (float)PyFloat_AsDouble(a); break;
      case 'I': s[i].i = (int)PyLong_AsLongLong(a); break;
      default: s[i].l = PyLong_AsLongLong(a);
    }
  }
  if (PyErr_Occurred()) return nullptr;
  int64_t r;
  Py_BEGIN_ALLOW_THREADS
  r = f->thunk(f->addr, s);
  Py_END_ALLOW_THREADS
  return PyLong_FromLongLong(r);
  END_HANDLE_TH_ERRORS
}

void fn_dealloc(PyObject* self) {
  Py_XDECREF(reinterpret_cast<Fn*>(self)->name);
  Py_TYPE(self)->tp_free(self);
}

PyTypeObject fn_type = [] {
  PyTypeObject t = {PyVarObject_HEAD_INIT(nullptr, 0)};
  t.tp_name = "atom_launch.Fn";
  t.tp_basicsize = sizeof(Fn);
  t.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  t.tp_vectorcall_offset = offsetof(Fn, vectorcall);
  t.tp_call = PyVectorcall_Call;
  t.tp_dealloc = fn_dealloc;
  return t;
}();

// bind(address, signature, name): the function as a callable, or None for a signature without a thunk.
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) return PyErr_Format(PyExc_TypeError, "bind(address, signature, name)");
  void* addr = PyLong_AsVoidPtr(args[0]);
  Py_ssize_t len = 0;
  const char* sig = PyUnicode_AsUTF8AndSize(args[1], &len);
  if (PyErr_Occurred()) return nullptr;
  const auto it = thunks().find(std::string(sig, len));
  if (it == thunks().end() || len < 1 || len - 1 > MAX_ARGS) Py_RETURN_NONE;
  Fn* f = PyObject_New(Fn, &fn_type);
  if (!f) return nullptr;
  f->vectorcall = fn_call;
  f->addr = addr;
  f->thunk = it->second;
  f->n = (int)len - 1;
  for (int i = 0; i < f->n; ++i) f->kind[i] = sig[i + 1];
  Py_INCREF(args[2]);
  f->name = args[2];
  return reinterpret_cast<PyObject*>(f);
}

// cuda(*tensors): raises NativeError unless each of them is None or a tensor on a device.
PyObject* cuda(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (args[i] == Py_None) continue;
    if (!THPVariable_Check(args[i])) return PyErr_Format(PyExc_TypeError, "a tensor is wanted, not %s", Py_TYPE(args[i])->tp_name);
    if (!THPVariable_Unpack(args[i]).is_cuda()) {
      PyErr_SetString(native_error, "kernels take CUDA tensors only (there is no CPU path)");
      return nullptr;
    }
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

int code_of(at::ScalarType t) { return t == at::kFloat ? 0 : t == at::kBFloat16 ? 1 : t == at::kInt ? 2 : 3; }

// (t, type, *sizes): t has the type (F32 0, BF16 1, I32 2; a tensor: that tensor's; None: any) and, where sizes are given, exactly
// these (None: any).
const at::Tensor* matches(PyObject* const* args, Py_ssize_t n, bool* ok) {
  *ok = false;
  if (n < 2 || !THPVariable_Check(args[0])) {
    PyErr_SetString(PyExc_TypeError, "(tensor, type, sizes ...)");
    return nullptr;
  }
  const at::Tensor& t = THPVariable_Unpack(args[0]);
  if (THPVariable_Check(args[1])) {
    if (t.scalar_type() != THPVariable_Unpack(args[1]).scalar_type()) return &t;
  } else if (args[1] != Py_None) {
    const long code = PyLong_AsLong(args[1]);
    if (code == -1 && PyErr_Occurred()) return nullptr;
    if (code != code_of(t.scalar_type())) return &t;
  }
  if (n > 2) {
    if (t.dim() != n - 2) return &t;
    for (Py_ssize_t i = 2; i < n; ++i) {
      if (args[i] == Py_None) continue;
      const long long want = PyLong_AsLongLong(args[i]);
      if (want == -1 && PyErr_Occurred()) return nullptr;
      if (t.size(i - 2) != want) return &t;
    }
  }
  *ok = true;
  return &t;
}
// dense(t, type, *sizes): ... and t is contiguous.
PyObject* dense(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  bool ok;
  const at::Tensor* t = matches(args, n, &ok);
  return t ? PyBool_FromLong(ok && t->is_contiguous()) : nullptr;
  END_HANDLE_TH_ERRORS
}
// rows(t, type, *sizes): ... and the numbers of its last axis lie one after another.
PyObject* rows(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  bool ok;
  const at::Tensor* t = matches(args, n, &ok);
  return t ? PyBool_FromLong(ok && t->dim() > 0 && t->stride(-1) == 1) : nullptr;
  END_HANDLE_TH_ERRORS
}
// stream(): the current stream's handle.
PyObject* stream(PyObject*, PyObject*) {
  HANDLE_TH_ERRORS
  return PyLong_FromVoidPtr((void*)c10::cuda::getCurrentCUDAStream().stream());
  END_HANDLE_TH_ERRORS
}
// on16(*tensors): every row of these begins on a 16-byte boundary.
PyObject* on16(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (!THPVariable_Check(args[i])) return PyErr_Format(PyExc_TypeError, "a tensor is wanted");
    const at::Tensor& t = THPVariable_Unpack(args[i]);
    if ((uintptr_t)t.data_ptr() % 16 || (t.stride(0) * (int64_t)t.element_size()) % 16) Py_RETURN_FALSE;
  }
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// The GEMM library's scratch memory, one per device and stream (products on two streams may run at once): what `make(out, stream)`
// gives, kept for good.
struct Scratch {
  int device;
  cudaStream_t stream;
  PyObject* tensor;
};
std::vector<Scratch> scratches;
const at::Tensor* scratch_of(PyObject* make, PyObject* out, const at::Tensor& t, cudaStream_t stream) {
  for (const Scratch& s : scratches)
    if (s.device == t.get_device() && s.stream == stream) return &THPVariable_Unpack(s.tensor);
  PyObject* got = PyObject_CallFunction(make, "OK", out, (unsigned long long)(uintptr_t)stream);
  if (!got) return nullptr;
  if (!THPVariable_Check(got)) {
    Py_DECREF(got);
    PyErr_SetString(PyExc_TypeError, "scratch memory is a tensor");
    return nullptr;
  }
  scratches.push_back({(int)t.get_device(), stream, got});
  return &THPVariable_Unpack(got);
}

using Gemm = int (*)(void*, int, const void*, const void*, int, int, int, int64_t, void*, size_t, cudaStream_t);
using GemmBatched = int (*)(void*, int, const void*, const void*, int, int, int, int, int64_t, int64_t, int64_t, int64_t, int64_t, void*, size_t,
                            cudaStream_t);

// gemm_bf16(atom_gemm_bf16, make, out, a, w): out[M, N] (bfloat16 or float32, dense) = a[M, K] w[N, K]^T, a's rows any distance apart.
// gemm_bf16_batched(atom_gemm_bf16_batched, make, out, a, w): the same for a [M, B, K], w [B, N, K] dense, out [M, B, N].
PyObject* product(PyObject* const* args, Py_ssize_t n, bool batched) {
  HANDLE_TH_ERRORS
  if (n != 5 || Py_TYPE(args[0]) != &fn_type || !THPVariable_Check(args[2]) || !THPVariable_Check(args[3]) || !THPVariable_Check(args[4]))
    return PyErr_Format(PyExc_TypeError, "(function, make, out, a, w)");
  const at::Tensor &out = THPVariable_Unpack(args[2]), &a = THPVariable_Unpack(args[3]), &w = THPVariable_Unpack(args[4]);
  if (!out.is_cuda() || !a.is_cuda() || !w.is_cuda()) {
    PyErr_SetString(native_error, "kernels take CUDA tensors only (there is no CPU path)");
    return nullptr;
  }
  const int d = batched ? 3 : 2, code = code_of(out.scalar_type());
  bool ok = a.dim() == d && w.dim() == d && out.dim() == d && a.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 && w.is_contiguous();
  if (ok) {
    const int64_t M = a.size(0), K = a.size(d - 1), N = w.size(d - 2);
    ok = w.size(d - 1) == K && out.size(0) == M && out.size(d - 1) == N && a.stride(d - 1) == 1 &&
         (batched ? w.size(0) == a.size(1) && out.size(1) == a.size(1) && out.stride(2) == 1 : out.is_contiguous());
  }
  if (!ok) {
    PyErr_SetString(PyExc_AssertionError, "a product's types, sizes or strides");
    return nullptr;
  }
  if (code > 1) {
    PyErr_SetString(native_error, "kernels take float32 or bfloat16");
    return nullptr;
  }
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const at::Tensor* ws = scratch_of(args[1], args[2], out, stream);
  if (!ws) return nullptr;
  const int M = (int)a.size(0), K = (int)a.size(d - 1), N = (int)w.size(d - 2);
  void* const fn = reinterpret_cast<Fn*>(args[0])->addr;
  void *po = out.data_ptr(), *pw = ws->data_ptr();
  const void *pa = a.data_ptr(), *pb = w.data_ptr();
  const size_t bytes = ws->nbytes();
  int r;
  Py_BEGIN_ALLOW_THREADS
  if (batched)
    r = reinterpret_cast<GemmBatched>(fn)(po, code, pa, pb, (int)a.size(1), M, N, K, a.stride(0), out.stride(0), a.stride(1), (int64_t)N * K,
                                          out.stride(1), pw, bytes, stream);
  else
    r = reinterpret_cast<Gemm>(fn)(po, code, pa, pb, M, N, K, a.stride(0), pw, bytes, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(r);
  END_HANDLE_TH_ERRORS
}
PyObject* gemm_bf16(PyObject*, PyObject* const* args, Py_ssize_t n) { return product(args, n, false); }
PyObject* gemm_bf16_batched(PyObject*, PyObject* const* args, Py_ssize_t n) { return product(args, n, true); }

PyMethodDef methods[] = {
    {"gemm_bf16", (PyCFunction)(void (*)(void))gemm_bf16, METH_FASTCALL, nullptr},
    {"gemm_bf16_batched", (PyCFunction)(void (*)(void))gemm_bf16_batched, METH_FASTCALL, nullptr},
    {"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, nullptr},
    {"cuda", (PyCFunction)(void (*)(void))cuda, METH_FASTCALL, nullptr},
    {"dense", (PyCFunction)(void (*)(void))dense, METH_FASTCALL, nullptr},
    {"rows", (PyCFunction)(void (*)(void))rows, METH_FASTCALL, nullptr},
    {"on16", (PyCFunction)(void (*)(void))on16, METH_FASTCALL, nullptr},
    {"stream", stream, METH_NOARGS, nullptr},
    {"set_error", [](PyObject*, PyObject* e) -> PyObject* {
       Py_INCREF(e);
       Py_XSETREF(native_error, e);
       Py_RETURN_NONE;
     }, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "atom_launch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_atom_launch(void) {
  if (PyType_Ready(&fn_type) < 0) return nullptr;
  return PyModule_Create(&module);
}
