// Host side of the calls a decode loop makes once per layer and token: the checks, the launch structure and the
// launch in native code.  A Python caller spends 8 to 25 us per call on attribute look-ups, shape and stride objects
// and ctypes fields; these functions read the same numbers off the tensors directly.
//
// Every function serves the ordinary case and returns None (or False), with nothing launched and nothing changed,
// for anything else -- other dtypes, tensor subclasses, unaligned rows, wrong shapes: the Python code behind it then
// makes contiguous copies or raises the errors of the interface.  Nothing is kept between calls.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <algorithm>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/inquant_b200.h"

namespace {

int (*g_decode)(const inq_decode_args_t*, inq_stream_t) = nullptr;
int (*g_append)(const inq_append_args_t*, inq_stream_t) = nullptr;
PyTypeObject* g_tensor_type = nullptr;

// A plain strided CUDA tensor of exactly torch.Tensor (no subclass, no wrapper of a transform), or nullptr.
const at::Tensor* plain(PyObject* o) {
  if (Py_TYPE(o) != g_tensor_type) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || t.is_conj() || t.is_neg()) return nullptr;
  return &t;
}
bool aligned(const at::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
// [1, heads, tokens, 128] of 16-bit values whose rows are 16-byte vectors
bool dense_rows(const at::Tensor& t, int64_t heads, const at::Tensor& like) {
  return t.dim() == 4 && t.size(0) == 1 && t.size(1) == heads && t.size(3) == 128 && t.scalar_type() == like.scalar_type() &&
         t.device() == like.device() && t.stride(3) == 1 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0 && aligned(t);
}
bool integers(PyObject* const* args, const int* at, int n, long long* out) {
  for (int i = 0; i < n; ++i) {
    out[i] = PyLong_AsLongLong(args[at[i]]);
    if (out[i] == -1 && PyErr_Occurred()) return false;
  }
  return true;
}
PyObject* none() { Py_RETURN_NONE; }
// Exceptions of tensor accessors (a wrapper without storage, ...) never cross into Python: the call is not served.
template <typename F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (...) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
}
// The launch itself does not hold the interpreter: it may wait for room in the launch queue.
template <typename F>
int without_gil(F&& f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  return rc;
}

// bind(address of inq_decode_attention, address of inq_append_token, torch.Tensor)
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) return PyErr_Format(PyExc_TypeError, "bind takes 3 arguments");
  const int at[] = {0, 1};
  long long v[2];
  if (!integers(args, at, 2, v)) return nullptr;
  g_decode = reinterpret_cast<decltype(g_decode)>(v[0]);
  g_append = reinterpret_cast<decltype(g_append)>(v[1]);
  g_tensor_type = reinterpret_cast<PyTypeObject*>(args[2]);
  Py_INCREF(args[2]);
  Py_RETURN_NONE;
}

// append_token(key, value, tail_key, tail_value, sink_key | None, sink_value | None, tail_count, sink_position, status address)
// -> True when the token was written, a negative return code, or None
PyObject* append_token(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 9) return PyErr_Format(PyExc_TypeError, "append_token takes 9 arguments");
  const int at[] = {6, 7, 8};
  long long v[3];
  if (!integers(args, at, 3, v)) return nullptr;
  return guarded([&]() -> PyObject* {
    const at::Tensor *key = plain(args[0]), *value = plain(args[1]), *tk = plain(args[2]), *tv = plain(args[3]);
    if (!key || !value || !tk || !tv || tk->dim() != 4) return none();
    const int64_t heads = tk->size(1), channels = tk->size(3), es = tk->element_size(), row = channels * es;
    if (row % 16 || (tk->stride(1) * es) % 16 || (tk->stride(2) * es) % 16 || tk->stride(3) != 1 || !aligned(*tk)) return none();
    if (tv->sizes() != tk->sizes() || tv->strides() != tk->strides() || !aligned(*tv)) return none();
    for (const at::Tensor* t : {key, value})
      if (t->dim() != 4 || t->size(0) != 1 || t->size(1) != heads || t->size(2) != 1 || t->size(3) != channels || t->scalar_type() != tk->scalar_type() ||
          t->device() != tk->device() || t->stride(3) != 1 || (t->stride(1) * es) % 16 || !aligned(*t))
        return none();
    if (key->stride(1) != value->stride(1)) return none();
    inq_append_args_t a = {};
    a.key = key->data_ptr();
    a.value = value->data_ptr();
    a.src_stride_h = key->stride(1) * es;
    a.tail_key = tk->data_ptr();
    a.tail_value = tv->data_ptr();
    a.tail_stride_h = tk->stride(1) * es;
    a.tail_stride_t = tk->stride(2) * es;
    a.tail_position = (int32_t)v[0];
    a.tail_capacity = (int32_t)tk->size(2);
    a.sink_position = (int32_t)v[1];
    if (v[1] >= 0) {
      const at::Tensor *sk = plain(args[4]), *sv = plain(args[5]);
      if (!sk || !sv || sk->dim() != 4 || sv->sizes() != sk->sizes() || sv->strides() != sk->strides() || v[1] >= sk->size(2)) return none();
      a.sink_key = sk->data_ptr();
      a.sink_value = sv->data_ptr();
      a.sink_stride_h = sk->stride(1) * es;
      a.sink_stride_t = sk->stride(2) * es;
    }
    a.heads = (int32_t)heads;
    a.row_bytes = (int32_t)row;
    a.status = reinterpret_cast<int32_t*>(v[2]);
    const auto stream = c10::cuda::getCurrentCUDAStream(tk->device().index()).stream();
    const int rc = without_gil([&] { return g_append(&a, stream); });
    if (rc != INQ_OK) return PyLong_FromLong(rc);
    Py_RETURN_TRUE;
  });
}

bool query_ok(const at::Tensor& q) {
  const auto type = q.scalar_type();
  return (type == at::kHalf || type == at::kBFloat16) && aligned(q);
}
void scratch(inq_decode_args_t& a, const long long* v) {   // workspace, floats, counters, status
  a.partials = reinterpret_cast<float*>(v[0]);
  a.partials_floats = v[1];
  a.counters = reinterpret_cast<int32_t*>(v[2]);
  a.status = reinterpret_cast<int32_t*>(v[3]);
}

// decode(query, sink_key, sink_value, residual_key, residual_value, scale, kv_heads, n_blocks, block_tokens, n_pad, value_kind,
//        value_groups, table, roles, value_roles, workspace, floats, counters, status) -> output, a return code, or None
PyObject* decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 19) return PyErr_Format(PyExc_TypeError, "decode takes 19 arguments");
  const double scale = PyFloat_AsDouble(args[5]);
  if (scale == -1.0 && PyErr_Occurred()) return nullptr;
  const int at[] = {6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18};
  long long v[13];
  if (!integers(args, at, 13, v)) return nullptr;
  return guarded([&]() -> PyObject* {
    const at::Tensor* q = plain(args[0]);
    const long long kv_heads = v[0], n_blocks = v[1];
    if (!q || q->dim() != 4 || q->size(0) != 1 || q->size(2) != 1 || q->size(3) != 128 || !query_ok(*q)) return none();
    if (q->stride(3) != 1 || q->stride(1) % 8 || q->size(1) < 1 || q->size(1) % kv_heads) return none();
    inq_decode_seq_t s = {};
    int64_t tokens[2] = {0, 0};
    for (int side = 0; side < 2; ++side) {
      PyObject *ko = args[1 + 2 * side], *vo = args[2 + 2 * side];
      if (ko == Py_None && vo == Py_None) continue;
      const at::Tensor *k = plain(ko), *val = plain(vo);
      if (!k || !val || !dense_rows(*k, kv_heads, *q) || !dense_rows(*val, kv_heads, *q) || k->size(2) != val->size(2)) return none();
      tokens[side] = k->size(2);
      if (!tokens[side]) continue;
      (side ? s.tail_key : s.sink_key) = k->data_ptr();
      (side ? s.tail_value : s.sink_value) = val->data_ptr();
      (side ? s.tail_key_stride_h : s.sink_key_stride_h) = k->stride(1);
      (side ? s.tail_key_stride_t : s.sink_key_stride_t) = k->stride(2);
      (side ? s.tail_value_stride_h : s.sink_value_stride_h) = val->stride(1);
      (side ? s.tail_value_stride_t : s.sink_value_stride_t) = val->stride(2);
    }
    if (n_blocks + tokens[0] + tokens[1] == 0) return none();
    at::Tensor out = at::empty(q->sizes(), q->options().memory_format(at::MemoryFormat::Contiguous));
    s.query = q->data_ptr();
    s.output = out.data_ptr();
    s.query_head_stride = q->stride(1);
    s.table = reinterpret_cast<const int64_t*>(v[6]);
    s.roles = reinterpret_cast<const int8_t*>(v[7]);
    s.value_roles = reinterpret_cast<const int8_t*>(v[8]);
    s.n_blocks = (int32_t)n_blocks;
    s.sink_tokens = (int32_t)tokens[0];
    s.tail_tokens = (int32_t)tokens[1];
    inq_decode_args_t a = {};
    a.n_seq = 1;
    a.seq_host = &s;
    a.kv_heads = (int32_t)kv_heads;
    a.q_per_kv = (int32_t)(q->size(1) / kv_heads);
    a.block_tokens = (int32_t)v[2];
    a.n_pad = (int32_t)v[3];
    a.dtype = q->scalar_type() == at::kHalf ? INQ_F16 : INQ_BF16;
    a.scale = (float)scale;
    a.value_kind = (int32_t)v[4];
    a.value_groups = (int32_t)v[5];
    scratch(a, v + 9);
    const auto stream = c10::cuda::getCurrentCUDAStream(q->device().index()).stream();
    const int rc = without_gil([&] { return g_decode(&a, stream); });
    if (rc != INQ_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(out));
  });
}

// paged_decode(query, cache, blocks, dense, output | None, num_pages, tail_tokens, sink_tokens, heads, block_size, page_bytes,
//              offsets, scale, workspace, floats, counters, status) -> output, a return code, or None
PyObject* paged_decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 17) return PyErr_Format(PyExc_TypeError, "paged_decode takes 17 arguments");
  const double scale = PyFloat_AsDouble(args[12]);
  if (scale == -1.0 && PyErr_Occurred()) return nullptr;
  const int at[] = {5, 6, 7, 8, 9, 10, 13, 14, 15, 16};
  long long v[10];
  if (!integers(args, at, 10, v)) return nullptr;
  if (!PyTuple_Check(args[11]) || PyTuple_GET_SIZE(args[11]) != 6) return PyErr_Format(PyExc_TypeError, "six page offsets");
  inq_decode_args_t a = {};
  for (int i = 0; i < 6; ++i) {
    a.page_offsets[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(args[11], i));
    if (a.page_offsets[i] == -1 && PyErr_Occurred()) return nullptr;
  }
  return guarded([&]() -> PyObject* {
    const at::Tensor *q = plain(args[0]), *cache = plain(args[1]), *blocks = plain(args[2]), *dense = plain(args[3]);
    const long long pages = v[0], tail = v[1], sink = v[2], heads = v[3], block = v[4];
    if (!q || !cache || !blocks || !dense) return none();
    if (cache->device() != q->device() || blocks->device() != q->device() || dense->device() != q->device()) return none();
    if (q->dim() != 3 || q->size(0) != 1 || q->size(2) != 128 || q->scalar_type() != at::kBFloat16 || !q->is_contiguous() || !aligned(*q)) return none();
    if (q->size(1) % heads || q->size(1) / heads < 1 || q->size(1) / heads > 16) return none();
    if (blocks->scalar_type() != at::kInt || dense->scalar_type() != q->scalar_type() || !dense->is_contiguous()) return none();
    if (!aligned(*dense) || !aligned(*cache)) return none();
    if (dense->dim() != 4 || dense->size(0) != 2 || dense->size(1) != heads || dense->size(2) != block + 4 || dense->size(3) != 128) return none();
    if (pages * block + tail == 0 && !sink) return none();
    at::Tensor out;
    if (args[4] == Py_None) {
      out = at::empty(q->sizes(), q->options());
    } else {
      const at::Tensor* given = plain(args[4]);
      if (!given || !given->is_contiguous() || given->device() != q->device()) return none();
      out = *given;
    }
    inq_decode_seq_t s = {};
    const int64_t stride_h = dense->stride(1), stride_t = dense->stride(2), plane = dense->stride(0) * 2;
    char* const base = static_cast<char*>(dense->data_ptr());
    s.query = q->data_ptr();
    s.output = out.data_ptr();
    s.query_head_stride = 128;
    s.pool = static_cast<const uint8_t*>(cache->data_ptr());
    s.page_table = static_cast<const int32_t*>(blocks->data_ptr());
    s.n_blocks = (int32_t)pages;
    s.pool_pages = (int32_t)cache->size(0);
    s.sink_key = base;
    s.sink_value = base + plane;
    s.tail_key = base + 4 * stride_t * 2;
    s.tail_value = base + 4 * stride_t * 2 + plane;
    s.sink_key_stride_h = s.sink_value_stride_h = s.tail_key_stride_h = s.tail_value_stride_h = stride_h;
    s.sink_key_stride_t = s.sink_value_stride_t = s.tail_key_stride_t = s.tail_value_stride_t = stride_t;
    s.sink_tokens = (int32_t)sink;
    s.tail_tokens = (int32_t)tail;
    // packed tokens covered by the exact sink are masked; so are tail tokens that the sink holds
    s.first_visible = (int32_t)sink;
    s.tail_skip = (int32_t)std::max<long long>(0, sink - pages * block);
    a.n_seq = 1;
    a.seq_host = &s;
    a.kv_heads = (int32_t)heads;
    a.q_per_kv = (int32_t)(q->size(1) / heads);
    a.block_tokens = (int32_t)block;
    a.n_pad = 16;
    a.layout = 1;
    a.dtype = INQ_BF16;
    a.scale = (float)scale;
    a.page_bytes = v[5];
    scratch(a, v + 6);
    const auto stream = c10::cuda::getCurrentCUDAStream(q->device().index()).stream();
    const int rc = without_gil([&] { return g_decode(&a, stream); });
    if (rc != INQ_OK) return PyLong_FromLong(rc);
    if (args[4] != Py_None) {
      Py_INCREF(args[4]);
      return args[4];
    }
    return THPVariable_Wrap(std::move(out));
  });
}

// same_objects(list, list) -> whether both hold the same objects in the same order
PyObject* same_objects(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) return PyErr_Format(PyExc_TypeError, "same_objects takes 2 arguments");
  if (!PyList_Check(args[0]) || !PyList_Check(args[1])) Py_RETURN_FALSE;
  const Py_ssize_t count = PyList_GET_SIZE(args[0]);
  if (count != PyList_GET_SIZE(args[1])) Py_RETURN_FALSE;
  for (Py_ssize_t i = 0; i < count; ++i)
    if (PyList_GET_ITEM(args[0], i) != PyList_GET_ITEM(args[1], i)) Py_RETURN_FALSE;
  Py_RETURN_TRUE;
}

PyMethodDef methods[] = {{"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(bind)), METH_FASTCALL, nullptr},
                         {"append_token", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(append_token)), METH_FASTCALL, nullptr},
                         {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(decode)), METH_FASTCALL, nullptr},
                         {"paged_decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(paged_decode)), METH_FASTCALL, nullptr},
                         {"same_objects", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(same_objects)), METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  PyObject* const created = PyModule_Create(&module);
  // the PyTorch and the Python this was compiled against, compared before the first use
  if (created && PyModule_AddStringConstant(created, "built_for", INQ_BUILT_FOR) < 0) {
    Py_DECREF(created);
    return nullptr;
  }
  return created;
}
