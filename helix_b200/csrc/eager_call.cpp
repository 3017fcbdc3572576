// Eager operators from Python in one native call.
//
// A call through ctypes reads some twenty tensor attributes and fills a structure field by field: 8 us of Python around a
// launch of 2 us, more than the kernels of small problems take (4096 x 4096 GEMV: 8.0 us).  Here a call whose
// arguments are plain CUDA tensors of the expected types and shapes fills the same helix_launch_t from their C++ side.
// Everything else -- other types, subclasses, modes, wrong shapes, a configuration -- returns None, and the Python
// implementation of the operator runs (and raises what it always raised).  Nothing is kept between calls.
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <climits>
#include <cstring>

#include "../../include/helix_b200.h"

namespace {

int (*g_launch)(const helix_launch_t*, void*, void*) = nullptr;
size_t (*g_workspace_bytes)(const helix_launch_t*) = nullptr;
PyObject* g_status_words = nullptr;   // dict: device -> status word, filled by g_status_word
PyObject* g_status_word = nullptr;    // ops.status_word(device)
PyObject* g_workspace = nullptr;      // ops.workspace(nbytes)
PyObject* g_check = nullptr;          // _lib.check(status, what)

struct Ref {
  PyObject* p = nullptr;
  ~Ref() { Py_XDECREF(p); }
};

bool modes_active() {
  return at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set();
}

// The tensor behind `o` if it is a plain one on a CUDA device, of this type and rank, with memory of its own and no expanded
// dimension (a stride of 0 stands for "contiguous" in helix_launch_t).
const at::Tensor* plain(PyObject* o, at::ScalarType type, int64_t dim) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.scalar_type() != type || t.dim() != dim || t.layout() != at::kStrided || !t.has_storage())
    return nullptr;
  const at::IntArrayRef sizes = t.sizes(), strides = t.strides();
  for (int64_t i = 0; i < dim; ++i)
    if (sizes[i] > INT_MAX || (sizes[i] > 1 && strides[i] == 0)) return nullptr;
  return &t;
}

// Queues `l` on the current stream of `dev`, the current device; false with a Python exception set.
bool queue(helix_launch_t& l, bool own_workspace, int dev) {
  Ref key, made, ws;
  if (own_workspace) {
    const size_t need = g_workspace_bytes(&l);
    if (need) {
      key.p = PyLong_FromSize_t(need);
      ws.p = key.p ? PyObject_CallOneArg(g_workspace, key.p) : nullptr;
      if (!ws.p) return false;
      const at::Tensor& buf = THPVariable_Unpack(ws.p);
      l.ws = buf.data_ptr();
      l.ws_bytes = buf.nbytes();
      Py_CLEAR(key.p);
    }
  }
  key.p = PyLong_FromLong(dev);
  if (!key.p) return false;
  PyObject* word = PyDict_GetItemWithError(g_status_words, key.p);
  if (!word) {
    if (PyErr_Occurred()) return false;
    word = made.p = PyObject_CallOneArg(g_status_word, key.p);
    if (!word) return false;
  }
  void* const status = THPVariable_Unpack(word).data_ptr();
  void* const stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_launch(&l, status, stream);
  Py_END_ALLOW_THREADS
  if (rc != HELIX_OK) {
    Ref r;
    r.p = PyObject_CallFunction(g_check, "is", rc, "helix_launch");
    return false;
  }
  return true;
}

PyObject* none() { Py_RETURN_NONE; }

// `made` is the output when the caller brought none; a, b and c are all on the current device or the call is not covered.
PyObject* finish(helix_launch_t& l, PyObject* out, at::Tensor&& made, const at::Tensor* a, const at::Tensor* b, const at::Tensor* c) {
  const int dev = c10::cuda::current_device();
  if (a->get_device() != dev || b->get_device() != dev || c->get_device() != dev) return none();
  if (!queue(l, true, dev)) return nullptr;
  if (out != Py_None) {
    Py_INCREF(out);
    return out;
  }
  return THPVariable_Wrap(std::move(made));
}

PyObject* gemv(PyObject* const* args, Py_ssize_t nargs, int op, at::ScalarType type) {
  HANDLE_TH_ERRORS
  if (nargs != 3 || modes_active()) return none();
  const at::Tensor *w = plain(args[0], type, 2), *x = plain(args[1], type, 2);
  if (!w || !x || w->stride(1) != 1 || x->stride(1) != 1 || x->size(1) != w->size(1)) return none();
  const int64_t rows = w->size(0), m = x->size(0);
  at::Tensor made;
  const at::Tensor* y;
  if (args[2] == Py_None) {
    made = w->new_empty({m, rows});
    y = &made;
  } else {
    y = plain(args[2], type, 2);
    if (!y || y->size(0) != m || y->size(1) != rows) return none();
  }
  helix_launch_t l;
  std::memset(&l, 0, sizeof(l));
  l.op = op;
  l.a = w->data_ptr(); l.b = x->data_ptr(); l.c = y->data_ptr();
  l.M = static_cast<int>(m); l.N = static_cast<int>(rows); l.K = static_cast<int>(w->size(1));
  l.lda = w->stride(0); l.ldb = x->stride(0);
  l.ldc = y->stride(0); l.ldc_inner = y->stride(1);
  return finish(l, args[2], std::move(made), w, x, y);
  END_HANDLE_TH_ERRORS
}
PyObject* gemv_f16(PyObject*, PyObject* const* args, Py_ssize_t nargs) { return gemv(args, nargs, HELIX_OP_GEMV_F16, at::kHalf); }
PyObject* gemv_f32(PyObject*, PyObject* const* args, Py_ssize_t nargs) { return gemv(args, nargs, HELIX_OP_GEMV_F32, at::kFloat); }

// (a, b_nk, out): 2-D, or 3-D with equal batch counts
PyObject* gemm_f16(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 3 || modes_active() || !THPVariable_CheckExact(args[0])) return none();
  const int64_t dim = THPVariable_Unpack(args[0]).dim();
  if (dim != 2 && dim != 3) return none();
  const at::Tensor *a = plain(args[0], at::kHalf, dim), *b = plain(args[1], at::kHalf, dim);
  if (!a || !b || a->stride(dim - 1) != 1 || b->stride(dim - 1) != 1 || a->size(dim - 1) != b->size(dim - 1) ||
      (dim == 3 && a->size(0) != b->size(0)))
    return none();
  const int64_t M = a->size(dim - 2), N = b->size(dim - 2), batch = dim == 3 ? a->size(0) : 1;
  at::Tensor made;
  const at::Tensor* c;
  if (args[2] == Py_None) {
    made = dim == 3 ? a->new_empty({batch, M, N}) : a->new_empty({M, N});
    c = &made;
  } else {
    c = plain(args[2], at::kHalf, dim);
    if (!c || c->size(dim - 2) != M || c->size(dim - 1) != N || (dim == 3 && c->size(0) != batch)) return none();
  }
  if (c->stride(dim - 1) != 1) return none();
  helix_launch_t l;
  std::memset(&l, 0, sizeof(l));
  l.op = HELIX_OP_GEMM_F16;
  l.a = a->data_ptr(); l.b = b->data_ptr(); l.c = c->data_ptr();
  l.batch = static_cast<int>(batch);
  l.M = static_cast<int>(M); l.N = static_cast<int>(N); l.K = static_cast<int>(a->size(dim - 1));
  l.lda = a->stride(dim - 2); l.ldb = b->stride(dim - 2); l.ldc = c->stride(dim - 2);
  if (dim == 3) { l.stride_a = a->stride(0); l.stride_b = b->stride(0); l.stride_c = c->stride(0); }
  return finish(l, args[2], std::move(made), a, b, c);
  END_HANDLE_TH_ERRORS
}

// (a, b, trans_a, out)
PyObject* gemm_f32(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 4 || modes_active() || !PyBool_Check(args[2])) return none();
  const bool ta = args[2] == Py_True;
  const at::Tensor *a = plain(args[0], at::kFloat, 2), *b = plain(args[1], at::kFloat, 2);
  if (!a || !b || a->stride(1) != 1 || b->stride(1) != 1) return none();
  const int64_t M = a->size(ta ? 1 : 0), K = a->size(ta ? 0 : 1), N = b->size(1);
  if (b->size(0) != K) return none();
  at::Tensor made;
  const at::Tensor* c;
  if (args[3] == Py_None) {
    made = a->new_empty({M, N});
    c = &made;
  } else {
    c = plain(args[3], at::kFloat, 2);
    if (!c || c->size(0) != M || c->size(1) != N) return none();
  }
  if (c->stride(1) != 1) return none();
  helix_launch_t l;
  std::memset(&l, 0, sizeof(l));
  l.op = HELIX_OP_GEMM_F32;
  l.a = a->data_ptr(); l.b = b->data_ptr(); l.c = c->data_ptr();
  l.M = static_cast<int>(M); l.N = static_cast<int>(N); l.K = static_cast<int>(K);
  l.lda = a->stride(0); l.ldb = b->stride(0); l.ldc = c->stride(0);
  l.trans_a = ta ? 1 : 0;
  return finish(l, args[3], std::move(made), a, b, c);
  END_HANDLE_TH_ERRORS
}

// (x, w, stride, pad, out), NHWC
PyObject* conv2d(PyObject* const* args, Py_ssize_t nargs, int op, at::ScalarType type) {
  HANDLE_TH_ERRORS
  if (nargs != 5 || modes_active() || !PyLong_CheckExact(args[2]) || !PyLong_CheckExact(args[3])) return none();
  const long stride = PyLong_AsLong(args[2]), pad = PyLong_AsLong(args[3]);
  if (PyErr_Occurred()) { PyErr_Clear(); return none(); }
  if (stride < 1 || stride > INT_MAX || pad < 0 || pad > INT_MAX / 4) return none();
  const at::Tensor *x = plain(args[0], type, 4), *w = plain(args[1], type, 4);
  if (!x || !w || !x->is_contiguous() || !w->is_contiguous() || x->size(3) != w->size(3)) return none();
  const int64_t H = x->size(1), W = x->size(2), R = w->size(1), S = w->size(2);
  if (H + 2 * pad < R || W + 2 * pad < S) return none();
  const int64_t Ho = (H + 2 * pad - R) / stride + 1, Wo = (W + 2 * pad - S) / stride + 1;
  at::Tensor made;
  const at::Tensor* y;
  if (args[4] == Py_None) {
    made = x->new_empty({x->size(0), Ho, Wo, w->size(0)});
    y = &made;
  } else {
    y = plain(args[4], type, 4);
    if (!y || !y->is_contiguous() || y->size(0) != x->size(0) || y->size(1) != Ho || y->size(2) != Wo || y->size(3) != w->size(0))
      return none();
  }
  helix_launch_t l;
  std::memset(&l, 0, sizeof(l));
  l.op = op;
  l.a = x->data_ptr(); l.b = w->data_ptr(); l.c = y->data_ptr();
  const int64_t geom[9] = {x->size(0), H, W, x->size(3), w->size(0), R, S, stride, pad};
  for (int i = 0; i < 9; ++i) l.conv[i] = static_cast<int>(geom[i]);
  return finish(l, args[4], std::move(made), x, w, y);
  END_HANDLE_TH_ERRORS
}
PyObject* conv2d_f16(PyObject*, PyObject* const* args, Py_ssize_t nargs) { return conv2d(args, nargs, HELIX_OP_CONV_F16, at::kHalf); }
PyObject* conv2d_f32(PyObject*, PyObject* const* args, Py_ssize_t nargs) { return conv2d(args, nargs, HELIX_OP_CONV_F32, at::kFloat); }

// run(launch): a prepared helix_launch_t (a ctypes structure, read through the buffer protocol)
PyObject* run(PyObject*, PyObject* launch) {
  HANDLE_TH_ERRORS
  Py_buffer view;
  if (PyObject_GetBuffer(launch, &view, PyBUF_SIMPLE) != 0) return nullptr;
  if (view.len != static_cast<Py_ssize_t>(sizeof(helix_launch_t))) {
    PyBuffer_Release(&view);
    PyErr_SetString(PyExc_TypeError, "run() takes a prepared Launch");
    return nullptr;
  }
  helix_launch_t l;
  std::memcpy(&l, view.buf, sizeof(l));
  PyBuffer_Release(&view);
  if (!queue(l, false, c10::cuda::current_device())) return nullptr;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// connect(helix_launch, helix_workspace_bytes, status_words, status_word, workspace, check)
PyObject* connect(PyObject*, PyObject* args) {
  unsigned long long launch, bytes;
  PyObject *words, *word, *ws, *check;
  if (!PyArg_ParseTuple(args, "KKO!OOO", &launch, &bytes, &PyDict_Type, &words, &word, &ws, &check)) return nullptr;
  g_launch = reinterpret_cast<decltype(g_launch)>(launch);
  g_workspace_bytes = reinterpret_cast<decltype(g_workspace_bytes)>(bytes);
  Py_INCREF(words); Py_INCREF(word); Py_INCREF(ws); Py_INCREF(check);
  g_status_words = words; g_status_word = word; g_workspace = ws; g_check = check;
  Py_RETURN_NONE;
}

#define HELIX_FASTCALL(fn) {#fn, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    HELIX_FASTCALL(gemv_f16), HELIX_FASTCALL(gemv_f32), HELIX_FASTCALL(gemm_f16), HELIX_FASTCALL(gemm_f32),
    HELIX_FASTCALL(conv2d_f16), HELIX_FASTCALL(conv2d_f32),
    {"run", run, METH_O, nullptr},
    {"connect", connect, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_eager_call", nullptr, -1, methods};

}  // namespace

// Tensors are read through the C++ headers of one torch: under another version the module refuses to be imported.
PyMODINIT_FUNC PyInit__eager_call(void) {
  Ref torch, version;
  torch.p = PyImport_ImportModule("torch");
  version.p = torch.p ? PyObject_GetAttrString(torch.p, "__version__") : nullptr;
  const char* now = version.p && PyUnicode_Check(version.p) ? PyUnicode_AsUTF8(version.p) : nullptr;
  if (!now) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ImportError, "torch has no version");
    return nullptr;
  }
  if (std::strcmp(now, HELIX_TORCH_VERSION) != 0)
    return PyErr_Format(PyExc_ImportError, "built for torch %s, not %s", HELIX_TORCH_VERSION, now);
  return PyModule_Create(&module);
}
