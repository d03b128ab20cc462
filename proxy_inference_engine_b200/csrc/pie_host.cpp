// The host side of nn.fused_rows in one native call: looks the layers and the activations over and makes the launch.  A call from Python spends 13
// of its 19 us on attributes, checks, argument tables and conversions, and a decode layer of few rows makes four of them (one row of a 1B feed-forward,
// whose kernels take 9 us: 39 us).  What it does not take in full it leaves to the Python form, which also reports what is wrong: None.
//
// Nothing is kept between calls but the addresses of the library's functions.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include "../../include/pie_b200.h"

namespace {

decltype(&pie_qmv_fused) qmv_fused = nullptr;
decltype(&pie_qmv_workspace_bytes) qmv_workspace = nullptr;
decltype(&pie_qmt) qmt = nullptr;
decltype(&pie_qmt_scratch_bytes) qmt_scratch = nullptr;

PyObject *s_weight, *s_scales, *s_biases, *s_bias, *s_bits, *s_group_size, *s_eps, *s_device;

// a plain tensor on a GPU: nothing that traces, batches or wraps
bool plain(const at::Tensor& t) {
  return t.is_cuda() && t.layout() == at::kStrided && !t.requires_grad() && !t.is_conj() && !t.is_neg() &&
         !t.key_set().has(c10::DispatchKey::Python) && !t.key_set().has(c10::DispatchKey::FuncTorchBatched) &&
         !t.key_set().has(c10::DispatchKey::FuncTorchGradWrapper) && !t.key_set().has(c10::DispatchKey::Functionalize);
}
bool aligned(const void* p, uintptr_t to) { return reinterpret_cast<uintptr_t>(p) % to == 0; }

// the instance dictionary's entry, borrowed; nullptr (no error set) where there is none
PyObject* entry(PyObject* obj, PyObject* name) {
  PyObject** dict = _PyObject_GetDictPtr(obj);
  PyObject* v = dict && *dict ? PyDict_GetItemWithError(*dict, name) : nullptr;
  if (!v) PyErr_Clear();
  return v;
}
const at::Tensor* tensor_of(PyObject* v) { return v && THPVariable_CheckExact(v) ? &THPVariable_Unpack(v) : nullptr; }
bool int_of(PyObject* v, long& out) {
  if (!v || !PyLong_CheckExact(v)) return false;
  out = PyLong_AsLong(v);
  if (out == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}

// The layers' tensors, held until the launch is queued: while the workspace is asked for, and while the launch waits without the lock, another thread
// may put others in their place, and their memory would be some other tensor's.  (The arguments themselves are the caller's for as long as it calls.)
using Held = c10::SmallVector<at::Tensor, 10>;

// nn._plain, and the pointers
bool segment(PyObject* lin, PyObject* type, long& bits, int64_t K, pie_qmv_seg& seg, Held& held) {
  if ((PyObject*)Py_TYPE(lin) != type || entry(lin, s_bias)) return false;
  long b = 0, gs = 0;
  if (!int_of(entry(lin, s_bits), b) || !int_of(entry(lin, s_group_size), gs) || gs != 64 || (b != 4 && b != 8) || (bits && b != bits)) return false;
  bits = b;
  const at::Tensor *w = tensor_of(entry(lin, s_weight)), *s = tensor_of(entry(lin, s_scales)), *z = tensor_of(entry(lin, s_biases));
  if (!w || !s || !z || !plain(*w) || !plain(*s) || !plain(*z)) return false;
  if (w->scalar_type() != at::kInt || w->dim() != 2 || w->size(1) * 32 != K * b || s->scalar_type() != at::kBFloat16 ||
      z->scalar_type() != at::kBFloat16 || s->sizes() != z->sizes() || s->dim() != 2 || s->size(0) != w->size(0) || s->size(1) != K / 64 ||
      !w->is_contiguous() || !s->is_contiguous() || !z->is_contiguous() || w->size(0) > INT32_MAX)
    return false;
  seg = {(const uint32_t*)w->const_data_ptr(), s->const_data_ptr(), z->const_data_ptr(), (int)w->size(0)};
  held.append({*w, *s, *z});
  return aligned(seg.wq, 16) && aligned(seg.scales, 8) && aligned(seg.biases, 8);
}

// fused_rows(x, linears, norm, residual, swiglu, QuantizedLinear, RMSNorm, workspace): workspace(bytes, device) is asked for the zeroed buffer of
// calls that need one
PyObject* fused_rows(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8 || !qmv_fused || !PyTuple_CheckExact(args[1])) Py_RETURN_NONE;
  const at::Tensor* x = tensor_of(args[0]);
  const Py_ssize_t nseg = PyTuple_GET_SIZE(args[1]);
  if (!x || !plain(*x) || x->scalar_type() != at::kBFloat16 || x->dim() < 1 || !x->is_contiguous() || nseg < 1 || nseg > 3) Py_RETURN_NONE;
  const int64_t K = x->size(-1), M = K > 0 ? x->numel() / K : 0;
  if (M < 1 || M > 128 || K > INT32_MAX || !aligned(x->const_data_ptr(), 16)) Py_RETURN_NONE;
  const bool swiglu = args[4] == Py_True;
  pie_qmv_seg segs[3];
  Held held;
  long bits = 0;
  int64_t N = 0;
  for (Py_ssize_t i = 0; i < nseg; ++i) {
    if (!segment(PyTuple_GET_ITEM(args[1], i), args[5], bits, K, segs[i], held)) Py_RETURN_NONE;
    N += segs[i].N;
  }
  if (K % (1024 / bits)) Py_RETURN_NONE;
  if (swiglu) {
    if (nseg != 2 || segs[0].N != segs[1].N) Py_RETURN_NONE;
    N /= 2;
  }
  if (N > INT32_MAX) Py_RETURN_NONE;
  const void *norm_w = nullptr, *res = nullptr;
  double eps = 0;
  if (args[2] != Py_None) {
    PyObject* e = entry(args[2], s_eps);
    const at::Tensor* w = tensor_of(entry(args[2], s_weight));
    if ((PyObject*)Py_TYPE(args[2]) != args[6] || !e || !PyFloat_CheckExact(e) || !w || !plain(*w) || w->scalar_type() != at::kBFloat16 ||
        w->dim() != 1 || w->size(0) != K || !w->is_contiguous() || !aligned(w->const_data_ptr(), 16))
      Py_RETURN_NONE;
    norm_w = w->const_data_ptr();
    held.push_back(*w);
    eps = PyFloat_AS_DOUBLE(e);
  }
  c10::SmallVector<int64_t, 6> shape(x->sizes().begin(), x->sizes().end());
  shape.back() = N;
  if (args[3] != Py_None) {
    const at::Tensor* r = tensor_of(args[3]);
    if (!r || !plain(*r) || r->scalar_type() != at::kBFloat16 || r->sizes() != at::IntArrayRef(shape) || !r->is_contiguous()) Py_RETURN_NONE;
    res = r->const_data_ptr();
  }
  const int epi = swiglu ? PIE_EPI_SILUMUL : res ? PIE_EPI_RESADD : PIE_EPI_STORE;
  const size_t scratch_bytes = qmt_scratch((int)M, N, (int)K, 64, (int)bits, swiglu);
  if (!scratch_bytes && M > 32) Py_RETURN_NONE;
  at::Tensor ws;
  if (const size_t need = scratch_bytes ? 0 : qmv_workspace((int)M, N, (int)K, (int)bits, swiglu, 0)) {
    THPObjectPtr dev(PyObject_GetAttr(args[0], s_device)), got(dev ? PyObject_CallFunction(args[7], "nO", (Py_ssize_t)need, dev.get()) : nullptr);
    if (!got) return nullptr;
    const at::Tensor* t = tensor_of(got);
    if (!t || !plain(*t)) Py_RETURN_NONE;
    ws = *t;
  }
  at::Tensor out = at::empty(shape, x->options());
  if (!plain(out)) Py_RETURN_NONE;
  void* const stream = c10::cuda::getCurrentCUDAStream().stream();
  int status;
  at::Tensor scratch;
  if (scratch_bytes) scratch = at::empty({(int64_t)scratch_bytes}, x->options().dtype(at::kByte));
  Py_BEGIN_ALLOW_THREADS   // (a launch waits where the queue is full)
  if (scratch_bytes) {
    status = qmt(out.mutable_data_ptr(), (int)N, x->const_data_ptr(), (int)K, (int)M, (int)K, segs, (int)nseg, 64, (int)bits, norm_w, (float)eps, epi,
                 res, scratch.mutable_data_ptr(), scratch_bytes, stream);
  } else {
    status = qmv_fused(out.mutable_data_ptr(), (int)N, x->const_data_ptr(), (int)K, (int)M, (int)K, segs, (int)nseg, 64, (int)bits, norm_w,
                       (float)eps, epi, res, 0, ws.defined() ? ws.mutable_data_ptr() : nullptr, ws.defined() ? (size_t)ws.numel() : 0, 0, stream);
  }
  Py_END_ALLOW_THREADS
  if (status != PIE_OK) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// bind(pie_qmv_fused, pie_qmv_workspace_bytes, pie_qmt, pie_qmt_scratch_bytes): addresses in the loaded library
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long a, b, c, d;
  if (!PyArg_ParseTuple(args, "KKKK", &a, &b, &c, &d)) return nullptr;
  qmv_fused = reinterpret_cast<decltype(qmv_fused)>(a);
  qmv_workspace = reinterpret_cast<decltype(qmv_workspace)>(b);
  qmt = reinterpret_cast<decltype(qmt)>(c);
  qmt_scratch = reinterpret_cast<decltype(qmt_scratch)>(d);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"fused_rows", (PyCFunction)(void (*)(void))fused_rows, METH_FASTCALL, "nn.fused_rows, or None"},
                         {"bind", bind, METH_VARARGS, "addresses of the library's functions"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pie_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__pie_host(void) {
  s_weight = PyUnicode_InternFromString("weight");
  s_scales = PyUnicode_InternFromString("scales");
  s_biases = PyUnicode_InternFromString("biases");
  s_bias = PyUnicode_InternFromString("bias");
  s_bits = PyUnicode_InternFromString("bits");
  s_group_size = PyUnicode_InternFromString("group_size");
  s_eps = PyUnicode_InternFromString("eps");
  s_device = PyUnicode_InternFromString("device");
  return PyModule_Create(&module);
}
