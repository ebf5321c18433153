// The host half of a decode step, natively: what `CacheLayer.update` and `decode_layer` do per layer for
// one new token, without the interpreter.
//
// A step over a short context is bound by the host (the Python form of these two calls took 20 us per
// layer, the kernels 12): attribute look-ups, tensor methods, filling ctypes records and the ctypes
// call.  Here they are direct accesses to the tensors and the same ShardSeq / ShardDecodeShape records,
// and the library's entry point is called through its address.  Anything out of the ordinary (another
// dtype, layout or device, buffers to grow, a pending token that does not fit) returns None and the Python
// path does it, with its checks and messages.  What torch throws (an allocation that fails) becomes the Python
// exception it would be there.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/shard_b200.h"

namespace {

using DecodeFn = int (*)(const ShardSeq*, int32_t, const ShardDecodeShape*, const float*, const float*, void*, size_t, void*);
using PhaseFn = int (*)(int32_t, int32_t, int32_t, const float*, void*, void*);
DecodeFn g_decode = nullptr;
PhaseFn g_phase = nullptr;
using AppendFn = int (*)(const void*, const void*, int64_t, int64_t, int64_t, int64_t, int32_t, int32_t, void*, void*, int64_t, int64_t, void*);
AppendFn g_append = nullptr;

PyObject *s_pending, *s_stream_n, *s_k_idx, *s_v_idx, *s_k_norm, *s_v_norm, *s_signs, *s_decode_k, *s_decode_v,
    *s_buf_k, *s_buf_v, *s_fresh;

// What does not change from step to step of one layer (the records belong to the Python launch state,
// which keeps this alive).
struct Step {
  ShardSeq* seq;
  ShardDecodeShape* shape;
  const float* inv_freq;
  const float* codebook;
  size_t need;              // workspace bytes
  int device;
};
void step_free(PyObject* cap) { delete static_cast<Step*>(PyCapsule_GetPointer(cap, "shard_b200.step")); }

bool fp16_cuda(const at::Tensor& t, int device) {
  return t.scalar_type() == at::kHalf && t.is_cuda() && t.get_device() == device;
}
const at::Tensor* tensor_at(PyObject* dict, PyObject* key) {
  PyObject* o = PyDict_GetItemWithError(dict, key);
  return o && THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr;
}
void* data_at(PyObject* dict, PyObject* key) {
  const at::Tensor* t = tensor_at(dict, key);
  return t ? t->data_ptr() : nullptr;
}
// (1, heads, 1, hd) whose heads lie hd elements apart
bool one_token(const at::Tensor& t, int64_t heads, int64_t hd) {
  return t.dim() == 4 && t.size(0) == 1 && t.size(1) == heads && t.size(2) == 1 && t.size(3) == hd && t.stride(3) == 1 &&
         (heads == 1 || t.stride(1) == hd) && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 7) == 0;
}

// bind(addresses of shard_b200_decode_attn, shard_b200_phase_table, shard_b200_append_rows)
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 3) return PyErr_Format(PyExc_TypeError, "bind takes 3 arguments");
  g_decode = reinterpret_cast<DecodeFn>(PyLong_AsVoidPtr(a[0]));
  g_phase = reinterpret_cast<PhaseFn>(PyLong_AsVoidPtr(a[1]));
  g_append = reinterpret_cast<AppendFn>(PyLong_AsVoidPtr(a[2]));
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

// phase_table(step, start, pos, n, table): the table of a step's layers, for another query position; returns
// the library's status, or None: not done
PyObject* py_phase_table(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5) return PyErr_Format(PyExc_TypeError, "phase_table takes 5 arguments");
  Step* st = static_cast<Step*>(PyCapsule_GetPointer(a[0], "shard_b200.step"));
  if (!st) return nullptr;
  if (!THPVariable_Check(a[4]) || c10::cuda::current_device() != st->device) Py_RETURN_NONE;
  const int32_t start = (int32_t)PyLong_AsLong(a[1]), pos = (int32_t)PyLong_AsLong(a[2]), tokens = (int32_t)PyLong_AsLong(a[3]);
  if (PyErr_Occurred()) return nullptr;
  return PyLong_FromLong(g_phase(start, pos, tokens, st->inv_freq, THPVariable_Unpack(a[4]).data_ptr(),
                                 c10::cuda::getCurrentCUDAStream(st->device).stream()));
  END_HANDLE_TH_ERRORS
}

// make_step(seq address, shape address, inv_freq pointer, codebook pointer, workspace bytes, device index)
PyObject* py_make_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 6) return PyErr_Format(PyExc_TypeError, "make_step takes 6 arguments");
  Step* s = new Step{static_cast<ShardSeq*>(PyLong_AsVoidPtr(a[0])), static_cast<ShardDecodeShape*>(PyLong_AsVoidPtr(a[1])),
                     static_cast<const float*>(PyLong_AsVoidPtr(a[2])), static_cast<const float*>(PyLong_AsVoidPtr(a[3])),
                     PyLong_AsSize_t(a[4]), (int)PyLong_AsLong(a[5])};
  if (PyErr_Occurred()) { delete s; return nullptr; }
  return PyCapsule_New(s, "shard_b200.step", step_free);
}

// append(gc, k, v, streaming, now) -> True: the token has its row; None: not done.  A token of the stream is left to
// the launch that reads it next.  An fp16 row is written now, on the current stream; without `now` the caller's
// next call is the read-back that writes it.
PyObject* py_append(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5) return PyErr_Format(PyExc_TypeError, "append takes 5 arguments");
  PyObject* gc = a[0];
  if (!PyDict_Check(gc) || !THPVariable_Check(a[1]) || !THPVariable_Check(a[2])) Py_RETURN_NONE;
  const at::Tensor &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]);
  if (k.dim() != 4 || k.scalar_type() != at::kHalf || v.scalar_type() != at::kHalf || !k.is_cuda() || v.device() != k.device()) Py_RETURN_NONE;
  const int64_t heads = k.size(1);
  if (!one_token(k, heads, SHARD_HEAD_DIM) || !one_token(v, heads, SHARD_HEAD_DIM)) Py_RETURN_NONE;
  if (PyDict_GetItemWithError(gc, s_pending)) Py_RETURN_NONE;
  if (a[3] == Py_True) {
    const at::Tensor* buf = tensor_at(gc, s_k_idx);
    if (!buf || !PyDict_GetItemWithError(gc, s_signs)) Py_RETURN_NONE;
    PyObject* so = PyDict_GetItemWithError(gc, s_stream_n);
    const long s = so ? PyLong_AsLong(so) : 0;
    if (s < 0 || s >= buf->size(0)) { PyErr_Clear(); Py_RETURN_NONE; }
    if (buf->dim() != 4 || buf->size(2) != heads) Py_RETURN_NONE;
    PyObject* row = PyLong_FromLong(s);
    PyObject* next = PyLong_FromLong(s + 1);
    PyObject* pend = PyTuple_Pack(3, a[1], a[2], row);
    const bool ok = row && next && pend && !PyDict_SetItem(gc, s_pending, pend) && !PyDict_SetItem(gc, s_stream_n, next);
    Py_XDECREF(row);
    Py_XDECREF(next);
    Py_XDECREF(pend);
    if (!ok) return nullptr;
    Py_RETURN_TRUE;
  }
  // fp16 rows: the views of the rows in use grow by one
  const at::Tensor *bk = tensor_at(gc, s_buf_k), *bv = tensor_at(gc, s_buf_v), *dk = tensor_at(gc, s_decode_k);
  if (!bk || !bv || !dk || bk->scalar_type() != at::kHalf) Py_RETURN_NONE;
  PyObject* so = PyDict_GetItemWithError(gc, s_stream_n);
  if (so && PyLong_AsLong(so) != 0) { PyErr_Clear(); Py_RETURN_NONE; }
  const int64_t rows = dk->size(2), cap = bk->size(2);
  if (rows >= cap || bk->size(1) != heads || dk->data_ptr() != bk->data_ptr()) Py_RETURN_NONE;
  if (a[4] == Py_True) {
    const int device = k.get_device();
    if (c10::cuda::current_device() != device || bk->get_device() != device) Py_RETURN_NONE;
    const int rc = g_append(k.data_ptr(), v.data_ptr(), SHARD_HEAD_DIM, 0, SHARD_HEAD_DIM, 0, 1, (int32_t)heads, bk->data_ptr(),
                            bv->data_ptr(), cap, rows, c10::cuda::getCurrentCUDAStream(device).stream());
    if (rc != 0) Py_RETURN_NONE;                                 // (the general path says why)
  }
  PyObject* nk = THPVariable_Wrap(bk->narrow(2, 0, rows + 1));
  PyObject* nv = THPVariable_Wrap(bv->narrow(2, 0, rows + 1));
  const bool ok = nk && nv && !PyDict_SetItem(gc, s_decode_k, nk) && !PyDict_SetItem(gc, s_decode_v, nv);
  Py_XDECREF(nk);
  Py_XDECREF(nv);
  if (!ok) return nullptr;
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// attend(step, gc, workspace, phase pointer, q, pos, out or None) -> (1, n_q, 1, hd) fp16; None: not done;
// an int: the library's status
PyObject* py_attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 7) return PyErr_Format(PyExc_TypeError, "attend takes 7 arguments");
  Step* st = static_cast<Step*>(PyCapsule_GetPointer(a[0], "shard_b200.step"));
  PyObject* gc = a[1];
  if (!st) return nullptr;
  if (!g_decode || !PyDict_Check(gc) || !THPVariable_Check(a[2]) || !THPVariable_Check(a[4])) Py_RETURN_NONE;
  const at::Tensor &ws = THPVariable_Unpack(a[2]), &q = THPVariable_Unpack(a[4]);
  ShardSeq& seq = *st->seq;
  ShardDecodeShape& sh = *st->shape;
  if (!fp16_cuda(q, st->device) || !one_token(q, sh.n_q, SHARD_HEAD_DIM) || ws.get_device() != st->device ||
      (size_t)ws.numel() < st->need || c10::cuda::current_device() != st->device || PyDict_GetItemWithError(gc, s_fresh))
    Py_RETURN_NONE;
  PyObject* so = PyDict_GetItemWithError(gc, s_stream_n);
  const int n_stream = so ? (int)PyLong_AsLong(so) : 0;
  PyObject* pend = PyDict_GetItemWithError(gc, s_pending);
  const at::Tensor *new_k = nullptr, *new_v = nullptr;
  int append = 0;
  if (pend) {
    if (PyLong_AsLong(PyTuple_GET_ITEM(pend, 2)) != n_stream - 1) Py_RETURN_NONE;
    new_k = &THPVariable_Unpack(PyTuple_GET_ITEM(pend, 0));
    new_v = &THPVariable_Unpack(PyTuple_GET_ITEM(pend, 1));
    append = 1;
  }
  int n_dec = 0, dec_cap = 0;
  if (const at::Tensor* dk = tensor_at(gc, s_decode_k)) {
    const at::Tensor* dv = tensor_at(gc, s_decode_v);
    if (!dv || !fp16_cuda(*dk, st->device) || dk->stride(3) != 1 || dk->stride(2) != SHARD_HEAD_DIM || dv->stride(3) != 1 ||
        dv->stride(2) != SHARD_HEAD_DIM || dv->stride(1) != dk->stride(1))
      Py_RETURN_NONE;
    n_dec = (int)dk->size(2);
    dec_cap = sh.nkv > 1 ? (int)(dk->stride(1) / SHARD_HEAD_DIM) : n_dec;
    seq.dec_k = dk->data_ptr();
    seq.dec_v = dv->data_ptr();
  }
  if (append) {
    if (!fp16_cuda(*new_k, st->device) || !fp16_cuda(*new_v, st->device)) Py_RETURN_NONE;
    seq.new_k = new_k->data_ptr();
    seq.new_v = new_v->data_ptr();
  }
  if (n_stream > 0) {                                            // (asked for at every step: the buffers move when they grow)
    seq.st_k_idx = static_cast<uint8_t*>(data_at(gc, s_k_idx));
    seq.st_v_idx = static_cast<uint8_t*>(data_at(gc, s_v_idx));
    seq.st_k_norm = data_at(gc, s_k_norm);
    seq.st_v_norm = data_at(gc, s_v_norm);
    seq.signs = static_cast<const float*>(data_at(gc, s_signs));
  }
  seq.q = q.data_ptr();
  seq.phase = PyLong_AsVoidPtr(a[3]);
  sh.n_stream = n_stream;
  sh.pos_q = (int32_t)PyLong_AsLong(a[5]);
  sh.append = append;
  sh.n_dec = n_dec;
  sh.dec_cap = dec_cap;
  sh.no_overlap = 0;
  if (PyErr_Occurred()) return nullptr;
  at::Tensor out;
  if (a[6] == Py_None) {
    out = at::empty({1, sh.n_q, 1, SHARD_HEAD_DIM}, q.options());
  } else {
    if (!THPVariable_Check(a[6])) Py_RETURN_NONE;
    const at::Tensor& given = THPVariable_Unpack(a[6]);
    if (!fp16_cuda(given, st->device) || !given.is_contiguous() || given.numel() != (int64_t)sh.n_q * SHARD_HEAD_DIM) Py_RETURN_NONE;
    out = given.view({1, sh.n_q, 1, SHARD_HEAD_DIM});
  }
  seq.out = out.data_ptr();
  const int rc = g_decode(&seq, 1, &sh, st->inv_freq, n_stream > 0 ? st->codebook : nullptr, ws.data_ptr(), (size_t)ws.numel(),
                          c10::cuda::getCurrentCUDAStream(st->device).stream());
  if (rc != 0) return PyLong_FromLong(rc);
  if (append && PyDict_DelItem(gc, s_pending)) return nullptr;
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_bind)), METH_FASTCALL, nullptr},
    {"phase_table", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_phase_table)), METH_FASTCALL, nullptr},
    {"make_step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_make_step)), METH_FASTCALL, nullptr},
    {"append", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_append)), METH_FASTCALL, nullptr},
    {"attend", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attend)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native host half of a decode step.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  const struct { PyObject** s; const char* name; } names[] = {
      {&s_pending, "_pending"}, {&s_stream_n, "stream_n"}, {&s_k_idx, "k_idx_buf"},
      {&s_v_idx, "v_idx_buf"}, {&s_k_norm, "k_norm_buf"}, {&s_v_norm, "v_norm_buf"}, {&s_signs, "signs"},
      {&s_decode_k, "decode_k"}, {&s_decode_v, "decode_v"}, {&s_buf_k, "_dec_buf_k"}, {&s_buf_v, "_dec_buf_v"}, {&s_fresh, "_fresh"}};
  for (const auto& x : names)
    if (!(*x.s = PyUnicode_InternFromString(x.name))) return nullptr;
  return PyModule_Create(&module);
}
