// The host side of calls of few rows, natively: nn.fused_rows (a norm, matrices of one input, and what follows them), the two launches of a
// feed-forward, and a decode step's attention (rotation and cache write, attention).  Each looks the layers and the activations over and makes the
// launches.  From Python a launch spends 13 of its 19 us on attributes, checks, argument tables and conversions, and a decode layer makes
// eight.  Launches are programmatic dependents of whatever is before them on the stream and only ask L2 for weights ahead of their wait; the
// second of a native call reads them ahead of it: the first does not write them, and starts its dependents behind its own wait for all before it.  One row of a 1B feed-forward, whose kernels take 9 us: 39 us
// from Python, 18.5 as two native calls, 14.9 as one; a 1B layer's step of 4 to 8 sequences, attention from Python / natively: 137 -> 57 to 62 (8-bit
// cache 165 -> 68), of an 8B model with five over 7000 tokens of 8-bit cache 166 -> 128.  What they do not take in full they leave to the Python
// form, which also reports what is wrong: None.
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

#define PIE_FUNCTIONS(X)                                                                                                                \
  X(pie_qmv_fused) X(pie_qmv_workspace_bytes) X(pie_qmt) X(pie_qmt_scratch_bytes) X(pie_rope_kv_rows) X(pie_rope_kvq_rows)                \
  X(pie_decode_attn) X(pie_decode_attn_pick_splits_for) X(pie_decode_attn_q8) X(pie_decode_attn_q8_pick_splits) X(pie_decode_attn_workspace_bytes)
struct Library {
#define X(name) decltype(&::name) name = nullptr;
  PIE_FUNCTIONS(X)
#undef X
} lib;
bool bound = false;

#define PIE_NAMES(X)                                                                                                                    \
  X(weight) X(scales) X(biases) X(bias) X(bits) X(group_size) X(eps) X(device) X(num_heads) X(n_kv_heads) X(head_dim) X(scale) X(rope)       \
  X(_freqs) X(traditional) X(dimensions) X(keys) X(values) X(offset)
#define X(name) PyObject* s_##name;
PIE_NAMES(X)
#undef X

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

// What the Python side hands over at every call: its types and where zeroed buffers are had
struct Kit {
  PyObject *linear, *norm, *workspace;   // workspace(bytes, device)
};
// Answers of a step: the result, "not mine" (nothing was launched), or a Python error
enum Answer { DONE, NOT_MINE, FAILED };

// workspace(arguments): a zeroed buffer; `held` keeps it until the launches are queued
Answer buffer(PyObject* args, PyObject* workspace, at::Tensor& out) {
  THPObjectPtr a(args), got(a ? PyObject_Call(workspace, a.get(), nullptr) : nullptr);
  if (!got) return FAILED;
  const at::Tensor* t = tensor_of(got);
  if (!t || !plain(*t)) return NOT_MINE;
  out = *t;
  return DONE;
}

// One launch (two with its preparing kernel) over the rows of x.  `chained`: the launch before it on this stream was made by the same native call.
Answer rows_call(const at::Tensor& x, PyObject* device, PyObject* const* linears, int nseg, PyObject* norm, const at::Tensor* residual, bool swiglu,
                 const Kit& kit, bool chained, Held& held, at::Tensor& out) {
  if (!plain(x) || x.scalar_type() != at::kBFloat16 || x.dim() < 1 || !x.is_contiguous() || nseg < 1 || nseg > 3) return NOT_MINE;
  const int64_t K = x.size(-1), M = K > 0 ? x.numel() / K : 0;
  if (M < 1 || M > 128 || K > INT32_MAX || !aligned(x.const_data_ptr(), 16)) return NOT_MINE;
  pie_qmv_seg segs[3];
  long bits = 0;
  int64_t N = 0;
  for (int i = 0; i < nseg; ++i) {
    if (!segment(linears[i], kit.linear, bits, K, segs[i], held)) return NOT_MINE;
    N += segs[i].N;
  }
  if (K % (1024 / bits)) return NOT_MINE;
  if (swiglu) {
    if (nseg != 2 || segs[0].N != segs[1].N) return NOT_MINE;
    N /= 2;
  }
  if (N > INT32_MAX) return NOT_MINE;
  const void *norm_w = nullptr, *res = nullptr;
  double eps = 0;
  if (norm && norm != Py_None) {
    PyObject* e = entry(norm, s_eps);
    const at::Tensor* w = tensor_of(entry(norm, s_weight));
    if ((PyObject*)Py_TYPE(norm) != kit.norm || !e || !PyFloat_CheckExact(e) || !w || !plain(*w) || w->scalar_type() != at::kBFloat16 ||
        w->dim() != 1 || w->size(0) != K || !w->is_contiguous() || !aligned(w->const_data_ptr(), 16))
      return NOT_MINE;
    norm_w = w->const_data_ptr();
    held.push_back(*w);
    eps = PyFloat_AS_DOUBLE(e);
  }
  c10::SmallVector<int64_t, 6> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = N;
  if (residual) {
    const at::Tensor& r = *residual;
    if (!plain(r) || r.scalar_type() != at::kBFloat16 || r.sizes() != at::IntArrayRef(shape) || !r.is_contiguous()) return NOT_MINE;
    res = r.const_data_ptr();
  }
  const int epi = swiglu ? PIE_EPI_SILUMUL : res ? PIE_EPI_RESADD : PIE_EPI_STORE;
  const size_t scratch_bytes = lib.pie_qmt_scratch_bytes((int)M, N, (int)K, 64, (int)bits, swiglu);
  if (!scratch_bytes && M > 32) return NOT_MINE;
  at::Tensor ws;
  if (const size_t need = scratch_bytes ? 0 : lib.pie_qmv_workspace_bytes((int)M, N, (int)K, (int)bits, swiglu, 0))
    if (const Answer a = buffer(Py_BuildValue("(nO)", (Py_ssize_t)need, device), kit.workspace, ws)) return a;
  out = at::empty(shape, x.options());
  if (!plain(out)) return NOT_MINE;
  void* const stream = c10::cuda::getCurrentCUDAStream().stream();
  int status;
  at::Tensor scratch;
  if (scratch_bytes) scratch = at::empty({(int64_t)scratch_bytes}, x.options().dtype(at::kByte));
  Py_BEGIN_ALLOW_THREADS   // (a launch waits where the queue is full)
  if (scratch_bytes) {
    status = lib.pie_qmt(out.mutable_data_ptr(), (int)N, x.const_data_ptr(), (int)K, (int)M, (int)K, segs, nseg, 64, (int)bits, norm_w, (float)eps,
                         epi, res, scratch.mutable_data_ptr(), scratch_bytes, stream);
  } else {
    status = lib.pie_qmv_fused(out.mutable_data_ptr(), (int)N, x.const_data_ptr(), (int)K, (int)M, (int)K, segs, nseg, 64, (int)bits, norm_w,
                               (float)eps, epi, res, 0, ws.defined() ? ws.mutable_data_ptr() : nullptr, ws.defined() ? (size_t)ws.numel() : 0,
                               chained ? 1 : 2, stream);
  }
  Py_END_ALLOW_THREADS
  return status == PIE_OK ? DONE : NOT_MINE;
}

// fused_rows(x, linears, norm, residual, swiglu, QuantizedLinear, RMSNorm, workspace): workspace(bytes, device) is asked for the zeroed buffer of
// calls that need one
PyObject* fused_rows(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8 || !bound || !PyTuple_CheckExact(args[1])) Py_RETURN_NONE;
  const at::Tensor* x = tensor_of(args[0]);
  const at::Tensor* r = args[3] == Py_None ? nullptr : tensor_of(args[3]);
  const Py_ssize_t nseg = PyTuple_GET_SIZE(args[1]);
  if (!x || (!r && args[3] != Py_None) || nseg < 1 || nseg > 3 || !x->is_cuda()) Py_RETURN_NONE;
  PyObject* linears[3] = {};
  for (Py_ssize_t i = 0; i < nseg; ++i) linears[i] = PyTuple_GET_ITEM(args[1], i);
  THPObjectPtr device(PyObject_GetAttr(args[0], s_device));
  if (!device) return nullptr;
  Held held;
  at::Tensor out;
  switch (rows_call(*x, device, linears, (int)nseg, args[2], r, args[4] == Py_True, {args[5], args[6], args[7]}, false, held, out)) {
    case DONE: return THPVariable_Wrap(std::move(out));
    case FAILED: return nullptr;
    default: Py_RETURN_NONE;
  }
  END_HANDLE_TH_ERRORS
}

// mlp_rows(x, gate, up, down, QuantizedLinear, RMSNorm, workspace) -> down(silu(gate(x)) * up(x)), or the activations alone in a tuple, or None
PyObject* mlp_rows(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const at::Tensor* x = n == 7 && bound ? tensor_of(args[0]) : nullptr;
  if (!x || !x->is_cuda()) Py_RETURN_NONE;
  const Kit kit = {args[4], args[5], args[6]};
  THPObjectPtr device(PyObject_GetAttr(args[0], s_device));
  if (!device) return nullptr;
  // the layers are looked up by the caller, whose references last for the call
  Held held, held2;
  at::Tensor act, out;
  Answer a = rows_call(*x, device, args + 1, 2, nullptr, nullptr, true, kit, false, held, act);
  if (a == FAILED) return nullptr;
  if (a == NOT_MINE) Py_RETURN_NONE;
  a = rows_call(act, device, args + 3, 1, nullptr, nullptr, false, kit, true, held2, out);
  if (a == FAILED) return nullptr;
  if (a == DONE) return THPVariable_Wrap(std::move(out));
  THPObjectPtr v(THPVariable_Wrap(std::move(act)));
  return v ? PyTuple_Pack(1, v.get()) : nullptr;
  END_HANDLE_TH_ERRORS
}

bool heads_cache(const at::Tensor* t, int64_t B, int64_t H, int64_t D, at::ScalarType type) {
  return t && plain(*t) && t->scalar_type() == type && t->dim() == 4 && t->size(0) == B && t->size(1) == H && t->size(3) == D;
}
// a (quants, scales, biases) triple of a quantised cache
bool triple(PyObject* v, int64_t B, int64_t H, int64_t D, const at::Tensor* (&t)[3]) {
  if (!v || !PyTuple_CheckExact(v) || PyTuple_GET_SIZE(v) != 3) return false;
  for (int i = 0; i < 3; ++i) {
    t[i] = tensor_of(PyTuple_GET_ITEM(v, i));
    if (!heads_cache(t[i], B, H, i ? D / 64 : D / 4, i ? at::kBFloat16 : at::kInt) || !t[i]->is_contiguous() || t[i]->size(2) != t[0]->size(2))
      return false;
  }
  return true;
}

// Rotation, cache write and attention of one new token a sequence: Attention.attend for projected rows [B, 1, heads * D].  The cache's offset moves on
// once both launches are queued.
Answer attend_call(const at::Tensor& qkv, PyObject* device, PyObject* at_, PyObject* cache, PyObject* cache_type, PyObject* quantized_type,
                   PyObject* rope_type, PyObject* attention_workspace, Held& held, at::Tensor& out) {
  long Hq = 0, Hkv = 0, D = 0, dims = 0, offset = 0;
  PyObject *sc = entry(at_, s_scale), *rope = entry(at_, s_rope);
  if (!int_of(entry(at_, s_num_heads), Hq) || !int_of(entry(at_, s_n_kv_heads), Hkv) || !int_of(entry(at_, s_head_dim), D) || !sc ||
      !PyFloat_CheckExact(sc) || !rope || (PyObject*)Py_TYPE(rope) != rope_type || entry(rope, s_traditional) != Py_False ||
      !int_of(entry(rope, s_dimensions), dims) || dims != D || (D != 64 && D != 128) || Hq <= 0 || Hkv <= 0 || Hq % Hkv)
    return NOT_MINE;
  const at::Tensor* freqs = tensor_of(entry(rope, s__freqs));
  if (!freqs || !plain(*freqs) || freqs->scalar_type() != at::kFloat || freqs->dim() != 1 || freqs->size(0) != D / 2 || !freqs->is_contiguous())
    return NOT_MINE;
  if (qkv.dim() != 3 || qkv.size(1) != 1 || qkv.size(2) != (Hq + 2 * Hkv) * D || qkv.size(0) > 65535 || Hq + 2 * Hkv > 65535) return NOT_MINE;
  const int B = (int)qkv.size(0);
  const bool quantized = (PyObject*)Py_TYPE(cache) == quantized_type;
  if ((!quantized && (PyObject*)Py_TYPE(cache) != cache_type) || !int_of(entry(cache, s_offset), offset) || offset < 0 || offset >= INT32_MAX - 1)
    return NOT_MINE;
  pie_kv_layout lay = {};
  pie_kvq_cache kvq = {};
  void *kc = nullptr, *vc = nullptr;
  if (quantized) {
    long gs = 0, bits = 0;
    const at::Tensor *k[3], *v[3];
    if (!int_of(entry(cache, s_group_size), gs) || !int_of(entry(cache, s_bits), bits) || gs != 64 || bits != 8 ||
        !triple(entry(cache, s_keys), B, Hkv, D, k) || !triple(entry(cache, s_values), B, Hkv, D, v) || k[0]->size(2) != v[0]->size(2) ||
        offset + 1 > k[0]->size(2))
      return NOT_MINE;
    kvq = {(uint32_t*)k[0]->data_ptr(), k[1]->data_ptr(), k[2]->data_ptr(), (uint32_t*)v[0]->data_ptr(), v[1]->data_ptr(), v[2]->data_ptr(),
           (long long)k[0]->size(2), nullptr, 0, 0, 64, 8};
    for (int i = 0; i < 3; ++i) held.append({*k[i], *v[i]});
  } else {
    const at::Tensor *k = tensor_of(entry(cache, s_keys)), *v = tensor_of(entry(cache, s_values));
    if (!heads_cache(k, B, Hkv, D, at::kBFloat16) || !heads_cache(v, B, Hkv, D, at::kBFloat16) || k->strides() != v->strides() ||
        k->size(2) != v->size(2) || k->stride(3) != 1 || offset + 1 > k->size(2))
      return NOT_MINE;
    lay = {k->stride(0), k->stride(1), k->stride(2), nullptr, 0, 0};
    kc = k->data_ptr();
    vc = v->data_ptr();
    held.append({*k, *v});
  }
  held.push_back(*freqs);
  const int splits = quantized ? lib.pie_decode_attn_q8_pick_splits(B, (int)Hq, (int)Hkv, (int)offset + 1)
                               : lib.pie_decode_attn_pick_splits_for(B, (int)Hq, (int)Hkv, (int)D, (int)offset + 1);
  at::Tensor ws;
  if (const Answer a = buffer(Py_BuildValue("(lnO)", (long)B * Hq, (Py_ssize_t)lib.pie_decode_attn_workspace_bytes(B, (int)Hq, (int)D, splits), device),
                              attention_workspace, ws))
    return a;
  const at::Tensor q = at::empty({B, Hq, D}, qkv.options()), pos = at::empty({B}, qkv.options().dtype(at::kInt));
  out = at::empty({B, 1, Hq * D}, qkv.options());
  if (!plain(out)) return NOT_MINE;
  const uint16_t* const rows = (const uint16_t*)qkv.const_data_ptr();
  const long long row = qkv.size(2);
  const pie_head_rows src[3] = {{rows, row, D, row}, {rows + Hq * D, row, D, row}, {rows + (Hq + Hkv) * D, row, D, row}};
  const float scale = (float)PyFloat_AS_DOUBLE(sc);
  void* const stream = c10::cuda::getCurrentCUDAStream().stream();
  int32_t* const p = (int32_t*)pos.data_ptr();
  const float* const f = (const float*)freqs->const_data_ptr();
  int status;
  Py_BEGIN_ALLOW_THREADS
  if (quantized) {
    status = lib.pie_rope_kvq_rows(q.data_ptr(), &kvq, &src[0], &src[1], &src[2], p, f, B, (int)Hq, (int)Hkv, 1, (int)D, (int)offset, stream);
    if (status == PIE_OK)
      status = lib.pie_decode_attn_q8(out.data_ptr(), q.data_ptr(), &kvq, p, B, (int)Hq, (int)Hkv, (int)D, scale, splits, ws.data_ptr(),
                                      (size_t)ws.numel(), stream);
  } else {
    status = lib.pie_rope_kv_rows(q.data_ptr(), kc, vc, &lay, &src[0], &src[1], &src[2], p, f, B, (int)Hq, (int)Hkv, 1, (int)D, (int)offset, stream);
    if (status == PIE_OK)
      status = lib.pie_decode_attn(out.data_ptr(), q.data_ptr(), kc, vc, &lay, p, B, (int)Hq, (int)Hkv, (int)D, scale, splits, ws.data_ptr(),
                                   (size_t)ws.numel(), stream);
  }
  Py_END_ALLOW_THREADS
  if (status != PIE_OK) return NOT_MINE;   // (the Python form writes the same rows again, and reports it)
  THPObjectPtr next(PyLong_FromLong(offset + 1));
  return next && PyObject_SetAttr(cache, s_offset, next) == 0 ? DONE : FAILED;
}

// attend_rows(attention, qkv, cache, KVCache, QuantizedKVCache, Llama3RoPE, attention_workspace) -> [B, 1, Hq * D], or None (and the cache's offset is
// as it was)
PyObject* attend_rows(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const at::Tensor* qkv = n == 7 && bound ? tensor_of(args[1]) : nullptr;
  if (!qkv || !plain(*qkv) || qkv->scalar_type() != at::kBFloat16 || !qkv->is_contiguous()) Py_RETURN_NONE;
  THPObjectPtr device(PyObject_GetAttr(args[1], s_device));
  if (!device) return nullptr;
  Held held;
  at::Tensor out;
  switch (attend_call(*qkv, device, args[0], args[2], args[3], args[4], args[5], args[6], held, out)) {
    case DONE: return THPVariable_Wrap(std::move(out));
    case FAILED: return nullptr;
    default: Py_RETURN_NONE;
  }
  END_HANDLE_TH_ERRORS
}

// bind({name: address in the loaded library})
PyObject* bind(PyObject*, PyObject* args) {
  PyObject* table;
  if (!PyArg_ParseTuple(args, "O!", &PyDict_Type, &table)) return nullptr;
#define X(name)                                                                                         \
  {                                                                                                     \
    PyObject* v = PyDict_GetItemString(table, #name);                                                   \
    void* const at = v ? PyLong_AsVoidPtr(v) : nullptr;                                                 \
    if (!at) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_KeyError, "bind: no " #name);       \
    lib.name = reinterpret_cast<decltype(lib.name)>(at);                                                \
  }
  PIE_FUNCTIONS(X)
#undef X
  bound = true;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"fused_rows", (PyCFunction)(void (*)(void))fused_rows, METH_FASTCALL, "nn.fused_rows, or None"},
                         {"mlp_rows", (PyCFunction)(void (*)(void))mlp_rows, METH_FASTCALL, "a feed-forward of few rows, or None"},
                         {"attend_rows", (PyCFunction)(void (*)(void))attend_rows, METH_FASTCALL, "a decode step's attention, or None"},
                         {"bind", bind, METH_VARARGS, "addresses of the library's functions"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pie_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__pie_host(void) {
#define X(name) s_##name = PyUnicode_InternFromString(#name);
  PIE_NAMES(X)
#undef X
  PyObject* m = PyModule_Create(&module);
#define X(name) #name,
  const char* const names[] = {PIE_FUNCTIONS(X)};
#undef X
  THPObjectPtr list(m ? PyList_New(0) : nullptr);
  if (!list) return nullptr;
  for (const char* name : names) {
    THPObjectPtr v(PyUnicode_FromString(name));
    if (!v || PyList_Append(list, v) < 0) return nullptr;
  }
  return PyObject_SetAttrString(m, "functions", list) < 0 ? nullptr : m;
}
