// Native host path of the package: argument checks, pointer extraction and the C-ABI call of the operators that run once
// or more per layer, in one Python -> C++ transition.
//
// What bounds a small call is the host: the Python form of these checks plus ctypes marshalling of 27 arguments took
// 24 us per multi-LoRA call, against 3 - 5 us for the kernel (an eager decode step of one row: 193 us for eight calls).
// Each function here accepts the argument combinations that the serving path uses (tensors on the current device, one
// dtype, dense slabs of one shape) and returns None for anything else; the caller then runs the Python form, which has
// the full set of checks and raises the documented exceptions. A C-ABI status comes back as an int.
//
// The C-ABI library itself links nothing from torch; its entry points reach this module as addresses (`bind`).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <optional>
#include <vector>

#include "../../include/b200_lora.h"

namespace {

decltype(&lora_b200_add) p_add = nullptr;
decltype(&lora_b200_delta) p_delta = nullptr;
decltype(&lora_b200_workspace_bytes) p_workspace_bytes = nullptr;
decltype(&lora_b200_linear_lora) p_linear = nullptr;
decltype(&lora_b200_linear_lora_silu) p_linear_silu = nullptr;
decltype(&lora_b200_glue_add_rmsnorm) p_rmsnorm = nullptr;
decltype(&lora_b200_glue_silu_mul) p_silu = nullptr;
decltype(&lora_b200_glue_rope_kv_store) p_rope = nullptr;
decltype(&lora_b200_shrink_buckets) p_shrink = nullptr;
decltype(&lora_b200_expand_buckets) p_expand = nullptr;
decltype(&lora_b200_prefill_attention) p_attention = nullptr;
PyObject* scratch_for = nullptr;  // lora.scratch_for(device, bytes)
PyObject *s_weight, *s_lora_a, *s_tts, *s_sorted, *s_ids, *s_counts, *s_offsets, *s_num_active;

inline const at::Tensor* tensor_of(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

inline int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kBFloat16: return B200_LORA_BF16;
    case at::kHalf: return B200_LORA_F16;
    case at::kFloat: return B200_LORA_F32;
    default: return -1;
  }
}

// CUDA tensor on `dev` (the current device)
inline bool on(const at::Tensor& t, int dev) { return t.is_cuda() && t.get_device() == dev; }

inline PyObject* not_handled() { Py_RETURN_NONE; }

// Items of a list or tuple; borrowed references, -1 if it is neither.
inline Py_ssize_t items(PyObject* seq, PyObject*** out) {
  if (PyList_CheckExact(seq)) {
    *out = reinterpret_cast<PyListObject*>(seq)->ob_item;
    return PyList_GET_SIZE(seq);
  }
  if (PyTuple_CheckExact(seq)) {
    *out = reinterpret_cast<PyTupleObject*>(seq)->ob_item;
    return PyTuple_GET_SIZE(seq);
  }
  return -1;
}

// Slabs, widths and columns of the slices that have rows, as the C ABI takes them.
struct Slices {
  const void* a[B200_LORA_MAX_SLICES];
  const void* b[B200_LORA_MAX_SLICES];
  int32_t out[B200_LORA_MAX_SLICES], col[B200_LORA_MAX_SLICES];
  int n = 0;
  int64_t S = 0, r = 0, in = 0;

  // false: a combination that the Python form handles
  bool add(PyObject* ao, PyObject* bo, int64_t width, int64_t column, at::ScalarType dt, int dev) {
    const at::Tensor *at_ = tensor_of(ao), *bt = tensor_of(bo);
    if (at_ == nullptr || bt == nullptr || at_->dim() != 3 || bt->dim() != 3) return false;
    if (width == 0) return true;
    if (n == B200_LORA_MAX_SLICES) return false;
    if (!on(*at_, dev) || !on(*bt, dev) || at_->scalar_type() != dt || bt->scalar_type() != dt) return false;
    if (!at_->is_contiguous() || !bt->is_contiguous()) return false;
    const auto as = at_->sizes(), bs = bt->sizes();
    if (n == 0) { S = as[0]; r = as[1]; in = as[2]; }
    if (as[0] != S || as[1] != r || as[2] != in || bs[0] != S || bs[1] != width || bs[2] != r) return false;
    if (S > INT32_MAX || width > INT32_MAX || column > INT32_MAX) return false;
    a[n] = at_->data_ptr(); b[n] = bt->data_ptr(); out[n] = (int32_t)width; col[n] = (int32_t)column;
    ++n;
    return true;
  }
};

// One attribute of the metadata object as an int32 device pointer: 1 = set, 0 = None, -1 = not handled.
inline int meta_ptr(PyObject* meta, PyObject* name, int dev, const int32_t** ptr, int64_t* numel) {
  PyObject* o = PyObject_GetAttr(meta, name);
  if (o == nullptr) { PyErr_Clear(); return -1; }
  int rc = -1;
  if (o == Py_None) {
    *ptr = nullptr; *numel = 0; rc = 0;
  } else if (const at::Tensor* t = tensor_of(o)) {
    if (t->scalar_type() == at::kInt && t->dim() == 1 && t->is_contiguous() && on(*t, dev)) {
      *ptr = static_cast<const int32_t*>(t->data_ptr()); *numel = t->numel(); rc = 1;
    }
  }
  Py_DECREF(o);  // the metadata object keeps the tensor alive over the call
  return rc;
}

struct Buckets {
  const int32_t *tts, *sorted, *ids, *counts, *offsets;
  int n;
};

bool read_metadata(PyObject* meta, int64_t T, int dev, Buckets* k) {
  int64_t n_tts, n_sorted, n_ids, n_counts, n_offsets;
  if (meta_ptr(meta, s_tts, dev, &k->tts, &n_tts) != 1 || n_tts < T) return false;
  const int a = meta_ptr(meta, s_sorted, dev, &k->sorted, &n_sorted), b = meta_ptr(meta, s_ids, dev, &k->ids, &n_ids),
            c = meta_ptr(meta, s_counts, dev, &k->counts, &n_counts), d = meta_ptr(meta, s_offsets, dev, &k->offsets, &n_offsets);
  if (a < 0 || b < 0 || c < 0 || d < 0) return false;
  k->n = 0;
  if (a && b && c && d) {
    int64_t nb = std::min(n_ids, std::min(n_counts, n_offsets - 1));
    PyObject* o = PyObject_GetAttr(meta, s_num_active);
    if (o == nullptr) { PyErr_Clear(); return false; }
    const long active = PyLong_AsLong(o);
    Py_DECREF(o);
    if (active == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    if (active > 0) nb = std::min<int64_t>(nb, active);
    k->n = (int)std::max<int64_t>(nb, 0);
  }
  if (k->n == 0) k->sorted = k->ids = k->counts = k->offsets = nullptr;
  return true;
}

// device pointer of an optional per-slot vector of type `dt`; false = not handled
inline bool optional_vector(PyObject* o, at::ScalarType dt, int64_t S, int dev, const void** ptr) {
  *ptr = nullptr;
  if (o == Py_None) return true;
  const at::Tensor* t = tensor_of(o);
  if (t == nullptr || t->scalar_type() != dt || !t->is_contiguous() || t->numel() < S || !on(*t, dev)) return false;
  *ptr = t->data_ptr();
  return true;
}

// Scratch of the tensor-core kernels: the caller's tensor, or the package's buffer of the current stream. That buffer only grows
// and an outgrown one stays allocated, so the last one seen per device is asked again only when the stream is another one or it
// is too small (asking costs 1 us). Calls that use it keep the GIL over their launches: another thread's on the same stream
// must not come between them.
// Returns a new reference in *keep (may be null); false with a Python error set.
constexpr int kMaxDevices = 64;
struct ScratchSeen {
  PyObject* buffer = nullptr;
  void* stream = nullptr;
} scratch_seen[kMaxDevices];
bool workspace(PyObject* given, const at::Tensor& x, size_t need, PyObject** keep, void** ptr, size_t* bytes) {
  *keep = nullptr; *ptr = nullptr; *bytes = 0;
  PyObject* o = given;
  if (o == Py_None) {
    if (need == 0) return true;
    const int dev = x.get_device();
    void* stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    ScratchSeen none, &seen = dev < kMaxDevices ? scratch_seen[dev] : none;
    if (seen.buffer != nullptr && seen.stream == stream && (size_t)THPVariable_Unpack(seen.buffer).nbytes() >= need) {
      Py_INCREF(seen.buffer);
      *keep = seen.buffer;
    } else {
      PyObject* device = THPDevice_New(x.device());
      if (device == nullptr) return false;
      *keep = PyObject_CallFunction(scratch_for, "On", device, (Py_ssize_t)need);
      Py_DECREF(device);
      if (*keep == nullptr) return false;
      if (dev < kMaxDevices && THPVariable_Check(*keep)) {
        Py_INCREF(*keep);
        seen.stream = stream;
        Py_XSETREF(seen.buffer, *keep);
      }
    }
    o = *keep;
  }
  const at::Tensor* t = tensor_of(o);
  if (t == nullptr) return true;
  *ptr = t->data_ptr();
  *bytes = (size_t)t->numel() * t->element_size();
  return true;
}

// add(y, x, a_slabs, b_slabs, widths, columns, metadata, scaling, rank_per_slot, scale_per_slot, impl, workspace, overwrite)
// columns None: `widths` holds the slices of y themselves, side by side from column 0. Returns the status, or None.
PyObject* add(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 13) { PyErr_SetString(PyExc_TypeError, "add takes 13 arguments"); return nullptr; }
  const at::Tensor *y = tensor_of(args[0]), *x = tensor_of(args[1]);
  if (y == nullptr || x == nullptr || !x->is_cuda() || x->dim() != 2 || y->dim() != 2) return not_handled();
  const int dev = x->get_device();
  const at::ScalarType dt = x->scalar_type();
  const int code = dtype_code(dt);
  if (code < 0 || y->scalar_type() != dt || !on(*y, dev) || dev != c10::cuda::current_device()) return not_handled();
  if (x->stride(1) != 1 || y->stride(1) != 1) return not_handled();
  const int64_t T = x->size(0);
  if (T > INT32_MAX) return not_handled();
  PyObject **ai, **bi, **wi, **ci = nullptr;
  const Py_ssize_t na = items(args[2], &ai), nb = items(args[3], &bi), nw = items(args[4], &wi);
  const bool by_slice = args[5] == Py_None;
  const Py_ssize_t nc = by_slice ? na : items(args[5], &ci);
  if (na < 1 || nb != na || nw != na || nc != na) return not_handled();
  Slices sl;
  int64_t column = 0;
  for (Py_ssize_t i = 0; i < na; ++i) {
    int64_t width;
    if (by_slice) {
      const at::Tensor* t = tensor_of(wi[i]);
      if (t == nullptr || t->dim() < 1) return not_handled();
      width = t->size(-1);
    } else {
      width = PyLong_AsLongLong(wi[i]);
      column = PyLong_AsLongLong(ci[i]);
      if (PyErr_Occurred()) { PyErr_Clear(); return not_handled(); }
    }
    if (!sl.add(ai[i], bi[i], width, column, dt, dev)) return not_handled();
    column += width;
  }
  if (sl.n == 0 || sl.in != x->size(1)) return not_handled();
  const double scaling = PyFloat_AsDouble(args[7]);
  const long impl = PyLong_AsLong(args[10]);
  if (PyErr_Occurred()) { PyErr_Clear(); return not_handled(); }
  Buckets k;
  if (!read_metadata(args[6], T, dev, &k)) return not_handled();
  const void *rank, *scale;
  if (!optional_vector(args[8], at::kInt, sl.S, dev, &rank) || !optional_vector(args[9], at::kFloat, sl.S, dev, &scale))
    return not_handled();
  // (the tensor-core kernels keep the rank-r intermediate in scratch)
  const bool scratch = code != B200_LORA_F32 &&
                       (impl == B200_LORA_IMPL_AUTO || impl == B200_LORA_IMPL_SGMV || impl == B200_LORA_IMPL_GROUPED);
  PyObject* keep;
  void* ws;
  size_t ws_bytes;
  if (!workspace(args[11], *x, scratch ? p_workspace_bytes((int)T, sl.n, (int)sl.r) : 0, &keep, &ws, &ws_bytes)) return nullptr;
  void* stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  const auto fn = args[12] == Py_True ? p_delta : p_add;
  const int rc = fn(y->data_ptr(), y->stride(0), x->data_ptr(), x->stride(0), (int)T, (int)sl.in, sl.n, sl.a, sl.b, sl.out, sl.col,
                    (int)sl.S, (int)sl.r, static_cast<const int32_t*>(rank), static_cast<const float*>(scale), k.tts, k.sorted, k.ids,
                    k.counts, k.offsets, k.n, (float)scaling, code, (int)impl, ws, ws_bytes, stream);
  Py_XDECREF(keep);
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

// Bucket arrays given one by one (mapping, sorted, counts, offsets, ids: five tensors, n_active as an int)
bool read_arrays(PyObject* const* args, int64_t T, int dev, Buckets* k) {
  const at::Tensor* t[5];
  for (int i = 0; i < 5; ++i) {
    t[i] = tensor_of(args[i]);
    if (t[i] == nullptr) {
      if (i == 0 || args[i] != Py_None) return false;
      continue;
    }
    if (t[i]->scalar_type() != at::kInt || t[i]->dim() != 1 || !t[i]->is_contiguous() || !on(*t[i], dev)) return false;
  }
  if (t[0]->numel() < T) return false;
  const long active = PyLong_AsLong(args[5]);
  if (active == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  k->tts = static_cast<const int32_t*>(t[0]->data_ptr());
  k->n = 0;
  k->sorted = k->ids = k->counts = k->offsets = nullptr;
  if (t[1] && t[2] && t[3] && t[4]) {
    int64_t nb = std::min(t[4]->numel(), std::min(t[2]->numel(), t[3]->numel() - 1));
    if (active > 0) nb = std::min<int64_t>(nb, active);
    if (nb > 0) {
      k->n = (int)nb;
      k->sorted = static_cast<const int32_t*>(t[1]->data_ptr()); k->counts = static_cast<const int32_t*>(t[2]->data_ptr());
      k->offsets = static_cast<const int32_t*>(t[3]->data_ptr()); k->ids = static_cast<const int32_t*>(t[4]->data_ptr());
    }
  }
  return true;
}

// Slabs [S, a, b] of one list (lora_A: one shape; lora_B: widths may differ); false = not handled
bool read_slabs(PyObject* list, bool lora_a, at::ScalarType dt, int dev, const void** ptr, int32_t* widths, int* n, int64_t (&shape)[3]) {
  PyObject** it;
  const Py_ssize_t m = items(list, &it);
  if (m < 1 || m > B200_LORA_MAX_SLICES) return false;
  for (Py_ssize_t i = 0; i < m; ++i) {
    const at::Tensor* t = tensor_of(it[i]);
    if (t == nullptr || t->dim() != 3 || !t->is_contiguous() || t->scalar_type() != dt || !on(*t, dev)) return false;
    const auto z = t->sizes();
    if (i == 0) { shape[0] = z[0]; shape[1] = z[1]; shape[2] = z[2]; }
    if (z[0] != shape[0] || z[2] != shape[2] || (lora_a && z[1] != shape[1]) || z[1] > INT32_MAX) return false;
    ptr[i] = t->data_ptr();
    widths[i] = (int32_t)z[1];
  }
  *n = (int)m;
  return shape[0] <= INT32_MAX && shape[2] <= INT32_MAX;
}

// shrink(x, a_slabs, out, mapping, sorted, counts, offsets, ids, n_active, scaling) -> status, or None
PyObject* shrink(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 10) { PyErr_SetString(PyExc_TypeError, "shrink takes 10 arguments"); return nullptr; }
  const at::Tensor *x = tensor_of(args[0]), *out = tensor_of(args[2]);
  if (x == nullptr || out == nullptr || !x->is_cuda() || x->dim() != 2 || x->stride(1) != 1 || out->dim() != 3) return not_handled();
  const int dev = x->get_device();
  const int code = dtype_code(x->scalar_type()), out_code = dtype_code(out->scalar_type());
  const int64_t T = x->size(0);
  if (code < 0 || out_code < 0 || dev != c10::cuda::current_device() || !on(*out, dev) || !out->is_contiguous() || T > INT32_MAX) return not_handled();
  const void* a[B200_LORA_MAX_SLICES];
  int32_t widths[B200_LORA_MAX_SLICES];
  int n;
  int64_t shape[3];
  Buckets k;
  if (!read_slabs(args[1], true, x->scalar_type(), dev, a, widths, &n, shape) || shape[2] != x->size(1) || out->size(0) != n ||
      out->size(1) != T || out->size(2) != shape[1] || !read_arrays(args + 3, T, dev, &k))
    return not_handled();
  const double scaling = PyFloat_AsDouble(args[9]);
  if (PyErr_Occurred()) { PyErr_Clear(); return not_handled(); }
  void* stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = p_shrink(out->data_ptr(), out_code, x->data_ptr(), x->stride(0), (int)T, (int)shape[2], n, a, (int)shape[0], (int)shape[1], k.tts,
                k.sorted, k.ids, k.counts, k.offsets, k.n, (float)scaling, code, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

// expand(tmp, b_slabs, y, mapping, sorted, counts, offsets, ids, n_active, offset_start, add_inputs) -> status, or None
PyObject* expand(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 11) { PyErr_SetString(PyExc_TypeError, "expand takes 11 arguments"); return nullptr; }
  const at::Tensor *tmp = tensor_of(args[0]), *y = tensor_of(args[2]);
  if (tmp == nullptr || y == nullptr || !y->is_cuda() || y->dim() != 2 || y->stride(1) != 1 || tmp->dim() != 3 || !tmp->is_contiguous())
    return not_handled();
  const int dev = y->get_device();
  const int code = dtype_code(y->scalar_type()), tmp_code = dtype_code(tmp->scalar_type());
  const int64_t T = y->size(0);
  if (code < 0 || tmp_code < 0 || dev != c10::cuda::current_device() || !on(*tmp, dev) || T > INT32_MAX) return not_handled();
  const void* b[B200_LORA_MAX_SLICES];
  int32_t widths[B200_LORA_MAX_SLICES], cols[B200_LORA_MAX_SLICES];
  int n;
  int64_t shape[3];
  Buckets k;
  if (!read_slabs(args[1], false, y->scalar_type(), dev, b, widths, &n, shape) || tmp->size(0) != n || tmp->size(1) != T ||
      tmp->size(2) != shape[2] || !read_arrays(args + 3, T, dev, &k))
    return not_handled();
  int64_t col = PyLong_AsLongLong(args[9]);
  if (PyErr_Occurred()) { PyErr_Clear(); return not_handled(); }
  for (int i = 0; i < n; ++i) {
    if (col < 0 || col + widths[i] > y->size(1)) return not_handled();
    cols[i] = (int32_t)col;
    col += widths[i];
  }
  void* stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  const int add_inputs = args[10] == Py_True;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = p_expand(y->data_ptr(), y->stride(0), tmp->data_ptr(), tmp_code, (int)T, n, b, widths, cols, (int)shape[0], (int)shape[2], k.tts,
                k.sorted, k.ids, k.counts, k.offsets, k.n, add_inputs, code, stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

// linear(x, weight, bias, a_slabs, b_slabs, widths, columns, token_to_slot, scaling, scale_per_slot, out)
// Returns (status, out), or None. At least one slice and a slot map; the plain linear stays in Python.
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 11) { PyErr_SetString(PyExc_TypeError, "linear takes 11 arguments"); return nullptr; }
  const at::Tensor *x = tensor_of(args[0]), *w = tensor_of(args[1]), *tts = tensor_of(args[7]);
  if (x == nullptr || w == nullptr || tts == nullptr || !x->is_cuda() || x->dim() != 2 || w->dim() != 2) return not_handled();
  const int dev = x->get_device();
  const at::ScalarType dt = x->scalar_type();
  const int64_t T = x->size(0), in = x->size(1), out_total = w->size(0);
  if (dt != at::kBFloat16 || w->scalar_type() != dt || !on(*w, dev) || dev != c10::cuda::current_device() || w->size(1) != in ||
      x->stride(1) != 1 || w->stride(1) != 1 || T > INT32_MAX)
    return not_handled();
  if (!on(*tts, dev) || tts->scalar_type() != at::kInt || !tts->is_contiguous() || tts->numel() != T) return not_handled();
  const void* bias;
  if (!optional_vector(args[2], dt, out_total, dev, &bias)) return not_handled();
  PyObject **ai, **bi, **wi, **ci;
  const Py_ssize_t na = items(args[3], &ai);
  if (na < 1 || items(args[4], &bi) != na || items(args[5], &wi) != na || items(args[6], &ci) != na) return not_handled();
  Slices sl;
  for (Py_ssize_t i = 0; i < na; ++i) {
    const int64_t width = PyLong_AsLongLong(wi[i]), column = PyLong_AsLongLong(ci[i]);
    if (PyErr_Occurred()) { PyErr_Clear(); return not_handled(); }
    if (width == 0 || !sl.add(ai[i], bi[i], width, column, dt, dev)) return not_handled();
  }
  if (sl.in != in) return not_handled();
  const double scaling = PyFloat_AsDouble(args[8]);
  if (PyErr_Occurred()) { PyErr_Clear(); return not_handled(); }
  const void* scale;
  if (!optional_vector(args[9], at::kFloat, sl.S, dev, &scale)) return not_handled();
  at::Tensor fresh;
  const at::Tensor* out = nullptr;
  if (args[10] == Py_None) {
    fresh = at::empty({T, out_total}, x->options());
    out = &fresh;
  } else {
    out = tensor_of(args[10]);
    if (out == nullptr || !on(*out, dev) || out->scalar_type() != dt || out->dim() != 2 || out->stride(1) != 1 ||
        out->size(0) != T || out->size(1) < out_total)
      return not_handled();
  }
  PyObject* keep;
  void* ws;
  size_t ws_bytes;
  if (!workspace(Py_None, *x, p_workspace_bytes((int)T, sl.n, (int)sl.r), &keep, &ws, &ws_bytes)) return nullptr;
  void* stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  const int rc = p_linear(out->data_ptr(), out->stride(0), x->data_ptr(), x->stride(0), (int)T, (int)in, w->data_ptr(), w->stride(0),
                          (int)out_total, bias, sl.n, sl.a, sl.b, sl.out, sl.col, (int)sl.S, (int)sl.r, static_cast<const float*>(scale),
                          static_cast<const int32_t*>(tts->data_ptr()), (float)scaling, ws, ws_bytes, stream);
  Py_XDECREF(keep);
  if (args[10] != Py_None) return Py_BuildValue("(iO)", rc, args[10]);
  return Py_BuildValue("(iN)", rc, THPVariable_Wrap(fresh));
  END_HANDLE_TH_ERRORS
}

// 2-D row view of a tensor whose rows are the last dim: dense, or 2-D with unit column stride; false otherwise
inline bool rows_of(const at::Tensor& t, int64_t width, int64_t* rows, int64_t* ld) {
  if (t.dim() < 1 || t.size(-1) != width || width == 0) return false;
  if (t.dim() == 2 && t.stride(1) == 1) { *rows = t.size(0); *ld = t.stride(0); return true; }
  if (!t.is_contiguous()) return false;
  *rows = t.numel() / width; *ld = width;
  return true;
}

// add_rms_norm(x, residual, weight, eps, norm_of_rounded_sum) -> (status, normed, hidden | None), or None; fresh outputs
PyObject* add_rms_norm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 5) { PyErr_SetString(PyExc_TypeError, "add_rms_norm takes 5 arguments"); return nullptr; }
  const at::Tensor *x = tensor_of(args[0]), *w = tensor_of(args[2]), *res = nullptr;
  if (x == nullptr || w == nullptr || !x->is_cuda() || x->dim() < 1) return not_handled();
  const int dev = x->get_device();
  const at::ScalarType dt = x->scalar_type();
  const int code = dtype_code(dt);
  const int64_t H = x->size(-1);
  int64_t T, x_ld, res_ld = 0, res_rows = 0;
  if (code < 0 || dev != c10::cuda::current_device() || !rows_of(*x, H, &T, &x_ld) || T > INT32_MAX || H > INT32_MAX) return not_handled();
  if (!on(*w, dev) || w->scalar_type() != dt || w->numel() != H || !w->is_contiguous()) return not_handled();
  if (args[1] != Py_None) {
    res = tensor_of(args[1]);
    if (res == nullptr || !on(*res, dev) || res->scalar_type() != dt || res->sizes() != x->sizes() || !rows_of(*res, H, &res_rows, &res_ld))
      return not_handled();
  }
  const double eps = PyFloat_AsDouble(args[3]);
  if (PyErr_Occurred()) { PyErr_Clear(); return not_handled(); }
  const at::Tensor normed = at::empty(x->sizes(), x->options());
  at::Tensor hidden;
  if (res != nullptr) hidden = at::empty(x->sizes(), x->options());
  const int rc = p_rmsnorm(normed.data_ptr(), H, res ? hidden.data_ptr() : nullptr, H, x->data_ptr(), x_ld,
                           res ? res->data_ptr() : nullptr, res_ld, w->data_ptr(), (int)T, (int)H, (float)eps,
                           args[4] == Py_True ? 1 : 0, code, c10::cuda::getCurrentCUDAStream(dev).stream());
  if (res == nullptr) return Py_BuildValue("(iNO)", rc, THPVariable_Wrap(normed), Py_None);
  return Py_BuildValue("(iNN)", rc, THPVariable_Wrap(normed), THPVariable_Wrap(hidden));
  END_HANDLE_TH_ERRORS
}

// silu_mul(x) -> (status, out), or None; fresh output
PyObject* silu_mul(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 1) { PyErr_SetString(PyExc_TypeError, "silu_mul takes 1 argument"); return nullptr; }
  const at::Tensor* x = tensor_of(args[0]);
  if (x == nullptr || !x->is_cuda() || x->dim() < 1 || x->size(-1) % 2) return not_handled();
  const int dev = x->get_device();
  const int code = dtype_code(x->scalar_type());
  int64_t T, ld;
  if (code < 0 || dev != c10::cuda::current_device() || !rows_of(*x, x->size(-1), &T, &ld) || T > INT32_MAX || x->size(-1) > INT32_MAX)
    return not_handled();
  const int64_t inter = x->size(-1) / 2;
  auto shape = x->sizes().vec();
  shape.back() = inter;
  const at::Tensor out = at::empty(shape, x->options());
  const int rc = p_silu(out.data_ptr(), inter, x->data_ptr(), ld, (int)T, (int)inter, code, c10::cuda::getCurrentCUDAStream(dev).stream());
  return Py_BuildValue("(iN)", rc, THPVariable_Wrap(out));
  END_HANDLE_TH_ERRORS
}

// rope_kv_store(qkv, heads, kv_heads, head_dim, positions, cos, sin, k_cache, v_cache, slot_mapping) -> (status, q, k, v), or
// None; the form with rotation and caches, int64 positions and int32 slots
PyObject* rope_kv_store(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 10) { PyErr_SetString(PyExc_TypeError, "rope_kv_store takes 10 arguments"); return nullptr; }
  const at::Tensor* t[7];
  const at::Tensor* qkv = tensor_of(args[0]);
  if (qkv == nullptr || !qkv->is_cuda() || qkv->dim() != 2 || qkv->stride(1) != 1) return not_handled();
  const int dev = qkv->get_device();
  for (int i = 0; i < 6; ++i) {
    t[i] = tensor_of(args[4 + i]);
    if (t[i] == nullptr || !on(*t[i], dev) || !t[i]->is_contiguous()) return not_handled();
  }
  const at::Tensor &pos = *t[0], &cos = *t[1], &sin = *t[2], &kc = *t[3], &vc = *t[4], &slots = *t[5];
  const int64_t hq = PyLong_AsLongLong(args[1]), hk = PyLong_AsLongLong(args[2]), d = PyLong_AsLongLong(args[3]);
  if (PyErr_Occurred()) { PyErr_Clear(); return not_handled(); }
  const int64_t T = qkv->size(0), q_size = hq * d, kv = hk * d;
  const int code = dtype_code(qkv->scalar_type()), table = dtype_code(cos.scalar_type());
  if (dev != c10::cuda::current_device() || code < 0 || table < 0 || T > INT32_MAX || hq < 0 || hk < 1 || d < 1 ||
      qkv->size(1) != q_size + 2 * kv || pos.scalar_type() != at::kLong || pos.numel() != T || cos.dim() != 2 ||
      cos.sizes() != sin.sizes() || sin.scalar_type() != cos.scalar_type() || slots.scalar_type() != at::kInt || slots.numel() != T ||
      kc.scalar_type() != qkv->scalar_type() || vc.scalar_type() != qkv->scalar_type() || kc.numel() % kv || vc.numel() % kv)
    return not_handled();
  const int64_t ld = qkv->stride(0);
  const int rc = p_rope(qkv->data_ptr(), ld, (int)T, (int)hq, (int)hk, (int)d, static_cast<const int64_t*>(pos.data_ptr()),
                        cos.data_ptr(), sin.data_ptr(), (int)cos.size(1), table, (int)cos.size(0), kc.data_ptr(), vc.data_ptr(),
                        static_cast<const int32_t*>(slots.data_ptr()), code, c10::cuda::getCurrentCUDAStream(dev).stream());
  const int64_t off = qkv->storage_offset();
  auto view = [&](int64_t heads, int64_t first) {
    return THPVariable_Wrap(qkv->as_strided({T, heads, d}, {ld, d, 1}, off + first));
  };
  return Py_BuildValue("(iNNN)", rc, view(hq, 0), view(hk, q_size), view(hk, q_size + kv));
  END_HANDLE_TH_ERRORS
}

// One projection of a decoder layer: (parameters dict of the module, lora_B names | None, widths, columns, rank buffer).
// lora_A is one parameter, stacked [slices, S, r, in] or a single [S, r, in].
struct Projection {
  const at::Tensor* w = nullptr;
  Slices sl;
  const void* rank = nullptr;
  at::Tensor held[2 + B200_LORA_MAX_SLICES];  // (attention may be a Python call, during which another thread may replace a parameter)

  bool read(PyObject* o, int64_t in, int64_t out, int dev) {
    if (!PyTuple_CheckExact(o) || PyTuple_GET_SIZE(o) != 5 || !PyDict_Check(PyTuple_GET_ITEM(o, 0))) return false;
    PyObject* params = PyTuple_GET_ITEM(o, 0);
    auto parameter = [&](PyObject* name) {
      PyObject* v = PyDict_GetItemWithError(params, name);
      return v == nullptr ? nullptr : tensor_of(v);
    };
    w = parameter(s_weight);
    if (w == nullptr || w->dim() != 2 || w->scalar_type() != at::kBFloat16 || !on(*w, dev) || !w->is_contiguous() || w->size(0) != out ||
        w->size(1) != in)
      return false;
    held[0] = *w;
    w = &held[0];
    if (PyTuple_GET_ITEM(o, 1) == Py_None) return true;
    PyObject **names, **wi, **ci;
    const Py_ssize_t n = items(PyTuple_GET_ITEM(o, 1), &names);
    if (n < 1 || n > B200_LORA_MAX_SLICES || items(PyTuple_GET_ITEM(o, 2), &wi) != n || items(PyTuple_GET_ITEM(o, 3), &ci) != n) return false;
    const at::Tensor* a = parameter(s_lora_a);
    if (a == nullptr || a->scalar_type() != at::kBFloat16 || !on(*a, dev) || !a->is_contiguous() || a->dim() < 3 || a->dim() > 4 ||
        (a->dim() == 4 ? a->size(0) : 1) != n || a->size(-1) != in || a->size(-3) > INT32_MAX)
      return false;
    held[1] = *a;
    sl.S = a->size(-3); sl.r = a->size(-2); sl.in = in;
    for (Py_ssize_t i = 0; i < n; ++i) {
      const int64_t width = PyLong_AsLongLong(wi[i]), column = PyLong_AsLongLong(ci[i]);
      if (PyErr_Occurred()) { PyErr_Clear(); return false; }
      if (width == 0) continue;
      const at::Tensor* b = parameter(names[i]);
      if (b == nullptr || b->scalar_type() != at::kBFloat16 || !on(*b, dev) || !b->is_contiguous() || b->dim() != 3 || b->size(0) != sl.S ||
          b->size(1) != width || b->size(2) != sl.r || column < 0 || column + width > out)
        return false;
      sl.a[sl.n] = static_cast<const char*>(a->data_ptr()) + i * sl.S * sl.r * in * 2;
      held[2 + sl.n] = *b;
      sl.b[sl.n] = b->data_ptr();
      sl.out[sl.n] = (int32_t)width;
      sl.col[sl.n++] = (int32_t)column;
    }
    return sl.n == 0 || optional_vector(PyTuple_GET_ITEM(o, 4), at::kInt, sl.S, dev, &rank);
  }
};

// Whether base product and delta of a prefill projection go in one kernel (csrc/linear_pair.cuh) instead of cuBLAS and the add
// behind it. It saves the pass over y and a launch (with `silu`, the activation behind gate_up, a second pass and launch) and
// needs tiles for the SMs: with fewer than 100, cuBLAS's smaller ones win. Whole steps, us, fused / separate: 4001 rows of 1024, 4 layers 888 /
// 1120; 2000 rows of 2048, 3 layers 831 / 957; 1000 rows of 2048 (gate_up 384 tiles, the others 64 to 80) 582 / 609; 1000 rows
// of 1024 (256, the others 32 to 40) 416 / 367.
// Narrow outputs, from 45 tiles on (prefill_cluster_kernel: one launch): us per layer, rank 32, 1024-wide: 1500 rows 135 / 149, 2000
// rows 168 / 172, 3000 rows 190 / 198; 1000 rows (32 and 40 tiles) 121 / 120; 2048-wide 500 rows (32, 40) 167 / 155, 1000 rows 189 / 188.
// Long products are bound by the power cap, and there it takes more energy per operation than cuBLAS, which outweighs the pass
// from 4096 input columns on. us per layer of whole steps, everything separate / only this projection fused, 4096-wide: 4000
// rows gate_up with the activation (940 GFLOP) 2131 / 2318, down (470) 2131 / 2244, o (134) 2131 / 2186; 2000 rows 1020 / 1093,
// 1020 / 1063, 1029 / 1048; 1000 rows 540 / 516 (235), 540 / 547 (118), 540 / 541 (34). 2048-wide down (6144 columns): 4000 rows
// (101) 692 / 705, 2000 rows (50) 355 / 348; its gate_up (2048 columns, 201 and 101) 692 / 651 and 355 / 323.
// Around 1024 input columns one launch (prefill_cluster_kernel with groups of columns) wins: us, cuBLAS + add / fused, rank 32: 1024 ->
// 1280 of 128, 300, 1100, 2700 rows 9.3 / 9.1, 11.0 / 9.4, 14.5 / 11.9, 22.9 / 15.9; 1024 -> 1024 8.4 / 7.6, 8.9 / 7.9, 10.7 / 10.1, 17.1 / 12.8; 1024 ->
// 8192 13.0 / 11.4, 16.4 / 13.6, 34.2 / 23.1; steps of 3 layers of 1024, one prompt of 128, 256, 1000 rows 248 / 225, 265 / 240, 393 / 364. (2048 -> 2048
// 12.1 / 12.5, 13.1 / 14.7, 17.3 / 19.1; 4096 -> 1024 14.9 / 19.5, 15.5 / 21.3, 20.1 / 24.) Narrower models and fewer rows would gain too (one prompt,
// a step of 3 layers of 512, 128 rows 241 / 157, of 1024, 32 rows 245 / 205); they keep cuBLAS and the add, and with it the two roundings that
// the step has layer by layer: a comparison of the two forms of a 256-wide step, not a time, set these two lines.
// Not batches of short prompts: a block of rows reads x again for every one to four runs of it, while the add of so small a batch
// goes by bucket. Steps as above, every prompt an adapter of its own, separate / fused, 128 to 1024 rows: prompts of 4 rows, rank 32, 265 / 469 (128
// rows), 359 / 610 (256); rank 64 306 / 666 and 336 / 638; by rows a prompt, ratio of the two at rank 32 and 64: 24 rows 0.94, 0.92; 32 0.97, 0.98; 40
// 1.01, 1.01; 48 1.02, 1.03; 64 1.03, 1.04; 96 1.06, 1.10.
// Not rank 16, whose intermediate the add of a small batch keeps as two numbers.
inline bool fused_linear_wins(int64_t T, int64_t K, int64_t N, int64_t r, int64_t prompts, bool silu) {
  if (!silu && K >= 768 && K <= 1024 && T >= 128 && T >= 48 * prompts && r > 16) return true;
  return (T + 127) / 128 * ((N + 255) / 256) >= (N <= 1536 ? 45 : 100) && (K < 4096 || 2.0 * (double)T * (double)K * (double)N < (silu ? 300e9 : 60e9));
}

// prefill_layers(embeds, positions, cu_seqlens, max_seqlen, slot_mapping, cos, sin, layers, final_norm, metadata | None, heads,
//                kv_heads, head_dim, intermediate, eps, attend | None) -> (status, normed), or None
// All layers of an eager bf16 prefill step. attend: what to call for attention, attend(qkv) -> [T, heads * head_dim], or None for
// lora_b200_prefill_attention. `layers`: (norm weight, norm weight, k_cache, v_cache, qkv, o, gate_up, down) with
// projections as above. (Layer by layer from Python a step of 400 rows took 270 us of host time per layer, for 86 us of kernels.)
PyObject* prefill_layers(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 16) { PyErr_SetString(PyExc_TypeError, "prefill_layers takes 16 arguments"); return nullptr; }
  const at::Tensor* x = tensor_of(args[0]);
  if (x == nullptr || !x->is_cuda() || x->dim() != 2 || !x->is_contiguous() || x->scalar_type() != at::kBFloat16) return not_handled();
  const int dev = x->get_device();
  const at::Tensor* t[6];
  const int where[6] = {1, 2, 4, 5, 6, 8};
  for (int i = 0; i < 6; ++i) {
    t[i] = tensor_of(args[where[i]]);
    if (t[i] == nullptr || !on(*t[i], dev) || !t[i]->is_contiguous()) return not_handled();
  }
  const at::Tensor slots = t[2]->scalar_type() == at::kLong ? t[2]->to(at::kInt) : *t[2];  // (the store kernel takes int32)
  const at::Tensor &pos = *t[0], &cu = *t[1], &cos = *t[3], &sin = *t[4], &last = *t[5];
  const int64_t max_len = PyLong_AsLongLong(args[3]), hq = PyLong_AsLongLong(args[10]), hk = PyLong_AsLongLong(args[11]),
                d = PyLong_AsLongLong(args[12]), inter = PyLong_AsLongLong(args[13]);
  const double eps = PyFloat_AsDouble(args[14]);
  if (PyErr_Occurred()) { PyErr_Clear(); return not_handled(); }
  const int64_t T = x->size(0), H = x->size(1), q_size = hq * d, kv = hk * d, qkv_width = q_size + 2 * kv;
  const int64_t prompts = cu.numel() - 1;
  const int table = dtype_code(cos.scalar_type());
  if (dev != c10::cuda::current_device() || T < 1 || T > INT32_MAX || hq < 1 || hk < 1 || (d != 64 && d != 128) || hq % hk || inter < 8 || inter % 8 ||
      H % 8 || H > 4096 || max_len < 1 || max_len > T || table < 0)
    return not_handled();
  if (pos.scalar_type() != at::kLong || pos.numel() != T || cu.scalar_type() != at::kInt || cu.numel() < 2 || cu.numel() > 65536 ||
      slots.scalar_type() != at::kInt || slots.numel() != T || cos.dim() != 2 || cos.sizes() != sin.sizes() ||
      sin.scalar_type() != cos.scalar_type() || (cos.size(1) != d && cos.size(1) != d / 2) || last.scalar_type() != at::kBFloat16 || last.numel() != H)
    return not_handled();
  PyObject** it;
  const Py_ssize_t n_layers = items(args[7], &it);
  if (n_layers < 1) return not_handled();
  struct Layer {
    const at::Tensor *ln1, *ln2, *k, *v;
    Projection p[4];
  };
  std::vector<Layer> layers((size_t)n_layers);
  const int64_t in[4] = {H, q_size, H, inter}, out[4] = {qkv_width, H, 2 * inter, H};
  size_t need = 0;
  for (Py_ssize_t i = 0; i < n_layers; ++i) {
    if (!PyTuple_CheckExact(it[i]) || PyTuple_GET_SIZE(it[i]) != 8) return not_handled();
    Layer& l = layers[(size_t)i];
    const at::Tensor** part[4] = {&l.ln1, &l.ln2, &l.k, &l.v};
    for (int j = 0; j < 4; ++j) {
      *part[j] = tensor_of(PyTuple_GET_ITEM(it[i], j));
      if (*part[j] == nullptr || !on(**part[j], dev) || !(*part[j])->is_contiguous() || (*part[j])->scalar_type() != at::kBFloat16) return not_handled();
    }
    if (l.ln1->numel() != H || l.ln2->numel() != H || l.k->numel() % kv || l.v->numel() % kv) return not_handled();
    for (int j = 0; j < 4; ++j) {
      if (!l.p[j].read(PyTuple_GET_ITEM(it[i], 4 + j), in[j], out[j], dev)) return not_handled();
      const Slices& sl = l.p[j].sl;
      if (sl.n > 0) need = std::max(need, p_workspace_bytes((int)T, sl.n, (int)sl.r));
    }
  }
  Buckets b = {};
  if (args[9] != Py_None && !read_metadata(args[9], T, dev, &b)) return not_handled();
  PyObject* keep;
  void* ws;
  size_t ws_bytes;
  if (!workspace(Py_None, *x, need, &keep, &ws, &ws_bytes)) return nullptr;

  std::optional<at::AutoDispatchBelowADInplaceOrView> no_autograd(std::in_place);
  void* stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  const auto opt = x->options();
  at::Tensor normed = at::empty({T, H}, opt), hidden = at::empty({T, H}, opt), qkv = at::empty({T, qkv_width}, opt), attn = at::empty({T, q_size}, opt),
             y = at::empty({T, H}, opt), gate_up = at::empty({T, 2 * inter}, opt), act = at::empty({T, inter}, opt);
  int rc = p_rmsnorm(normed.data_ptr(), H, nullptr, H, x->data_ptr(), H, nullptr, 0, layers[0].ln1->data_ptr(), (int)T, (int)H, (float)eps, 1,
                     B200_LORA_BF16, stream);
  const void* residual = x->data_ptr();
  auto project = [&](const Projection& p, at::Tensor& dst, const at::Tensor& src) {
    if (rc != B200_LORA_OK) return;
    const Slices& sl = p.sl;
    const bool lora = sl.n > 0 && b.tts != nullptr;
    const int K = (int)src.size(1), N = (int)dst.size(1);
    if (lora && fused_linear_wins(T, K, N, sl.r, prompts, false) && K % 64 == 0 && (sl.r == 16 || sl.r == 32 || sl.r == 64)) {
      rc = p_linear(dst.data_ptr(), N, src.data_ptr(), K, (int)T, K, p.w->data_ptr(), K, N, nullptr, sl.n, sl.a, sl.b, sl.out, sl.col, (int)sl.S,
                    (int)sl.r, nullptr, b.tts, 1.0f, ws, ws_bytes, stream);
      return;
    }
    at::mm_out(dst, src, p.w->t());
    if (lora)
      rc = p_add(dst.data_ptr(), N, src.data_ptr(), K, (int)T, K, sl.n, sl.a, sl.b, sl.out, sl.col, (int)sl.S, (int)sl.r,
                 static_cast<const int32_t*>(p.rank), nullptr, b.tts, b.sorted, b.ids, b.counts, b.offsets, b.n, 1.0f, B200_LORA_BF16,
                 B200_LORA_IMPL_AUTO, ws, ws_bytes, stream);
  };
  // gate_up with the activation in its epilogue, by the same line (128 + 128 columns make a tile)
  auto silu_in_linear = [&](const Slices& sl) {
    if (!fused_linear_wins(T, H, 2 * inter, sl.r, prompts, true) || H % 64 || inter % 32) return false;
    if (sl.n > 0 && b.tts != nullptr && sl.r != 16 && sl.r != 32 && sl.r != 64) return false;
    for (int q = 0; q < sl.n; ++q)
      if (sl.out[q] % 32 || sl.col[q] % 32) return false;
    return true;
  };
  auto add_norm = [&](const at::Tensor& weight) {
    if (rc != B200_LORA_OK) return;
    rc = p_rmsnorm(normed.data_ptr(), H, hidden.data_ptr(), H, y.data_ptr(), H, residual, H, weight.data_ptr(), (int)T, (int)H, (float)eps, 1,
                   B200_LORA_BF16, stream);
    residual = hidden.data_ptr();
  };
  for (size_t i = 0; i < layers.size(); ++i) {
    const Layer& l = layers[i];
    project(l.p[0], qkv, normed);
    if (rc == B200_LORA_OK)
      rc = p_rope(qkv.data_ptr(), qkv_width, (int)T, (int)hq, (int)hk, (int)d, pos.data_ptr<int64_t>(), cos.data_ptr(), sin.data_ptr(),
                  (int)cos.size(1), table, (int)cos.size(0), l.k->data_ptr(), l.v->data_ptr(), slots.data_ptr<int32_t>(), B200_LORA_BF16, stream);
    if (rc == B200_LORA_OK && args[15] != Py_None) {
      no_autograd.reset();  // (the callee dispatches as from Python)
      PyObject* rows = THPVariable_Wrap(qkv);
      PyObject* got = rows == nullptr ? nullptr : PyObject_CallOneArg(args[15], rows);
      Py_XDECREF(rows);
      const at::Tensor* t = got == nullptr ? nullptr : tensor_of(got);
      if (t == nullptr || !on(*t, dev) || t->scalar_type() != at::kBFloat16 || t->dim() != 2 || t->size(0) != T || t->size(1) != q_size ||
          !t->is_contiguous()) {
        if (got != nullptr) PyErr_SetString(PyExc_TypeError, "attend must return contiguous bf16 rows of all heads");
        Py_XDECREF(got);
        Py_XDECREF(keep);
        return nullptr;
      }
      attn = *t;
      Py_DECREF(got);
      no_autograd.emplace();
    } else if (rc == B200_LORA_OK) {
      rc = p_attention(attn.data_ptr(), q_size, qkv.data_ptr(), qkv_width, (int)T, (int)hq, (int)hk, (int)d, cu.data_ptr<int32_t>(),
                       (int)cu.numel() - 1, (int)max_len, 1.0f / std::sqrt((float)d), stream);
    }
    project(l.p[1], y, attn);
    add_norm(*l.ln2);
    if (rc == B200_LORA_OK && silu_in_linear(l.p[2].sl)) {
      const Slices& sl = l.p[2].sl;
      rc = p_linear_silu(act.data_ptr(), inter, normed.data_ptr(), H, (int)T, (int)H, l.p[2].w->data_ptr(), H, (int)(2 * inter),
                         b.tts != nullptr ? sl.n : 0, sl.a, sl.b, sl.out, sl.col, (int)std::max<int64_t>(sl.S, 1), (int)std::max<int64_t>(sl.r, 16),
                         nullptr, b.tts, 1.0f, ws, ws_bytes, stream);
      project(l.p[3], y, act);
      add_norm(i + 1 < layers.size() ? *layers[i + 1].ln1 : last);
      continue;
    }
    project(l.p[2], gate_up, normed);
    if (rc == B200_LORA_OK)
      rc = p_silu(act.data_ptr(), inter, gate_up.data_ptr(), 2 * inter, (int)T, (int)inter, B200_LORA_BF16, stream);
    project(l.p[3], y, act);
    add_norm(i + 1 < layers.size() ? *layers[i + 1].ln1 : last);
  }
  Py_XDECREF(keep);
  return Py_BuildValue("(iN)", rc, THPVariable_Wrap(normed));
  END_HANDLE_TH_ERRORS
}

// An int of a list or tuple; false (error cleared) if the item is none or does not fit.
inline bool as_int32(PyObject* o, int32_t* v) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow;
  const long got = PyLong_AsLongAndOverflow(o, &overflow);
  if (overflow || got < INT32_MIN || got > INT32_MAX) return false;
  *v = (int32_t)got;
  return true;
}

PyObject* list_of(const std::vector<int32_t>& v) {
  PyObject* l = PyList_New((Py_ssize_t)v.size());
  if (l == nullptr) return nullptr;
  for (size_t i = 0; i < v.size(); ++i) PyList_SET_ITEM(l, (Py_ssize_t)i, PyLong_FromLong(v[i]));
  return l;
}

// bucket_lists(token_to_slot) -> (sorted rows, active slots, counts, offsets) as lists, or None: a stable counting sort of
// the rows with slot >= 0. (The numpy form spends 130 us on 4000 rows, most of it in list <-> array conversions.)
PyObject* bucket_lists(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 1) { PyErr_SetString(PyExc_TypeError, "bucket_lists takes 1 argument"); return nullptr; }
  PyObject** it;
  const Py_ssize_t n = items(args[0], &it);
  if (n < 0 || n > INT32_MAX) return not_handled();
  constexpr int32_t kMaxSlot = 1 << 20;
  std::vector<int32_t> slot((size_t)n), start;
  int32_t top = -1;
  for (Py_ssize_t i = 0; i < n; ++i) {
    if (!as_int32(it[i], &slot[i]) || slot[i] > kMaxSlot) return not_handled();
    top = std::max(top, slot[i]);
  }
  start.assign((size_t)top + 2, 0);
  for (int32_t s : slot)
    if (s >= 0) ++start[(size_t)s + 1];
  std::vector<int32_t> active, counts, offsets{0};
  for (int32_t s = 0; s <= top; ++s) {
    const int32_t c = start[(size_t)s + 1];
    if (c > 0) { active.push_back(s); counts.push_back(c); offsets.push_back(offsets.back() + c); }
    start[(size_t)s + 1] += start[s];
  }
  std::vector<int32_t> rows((size_t)offsets.back());
  for (Py_ssize_t i = 0; i < n; ++i)
    if (slot[i] >= 0) rows[(size_t)start[slot[i]]++] = (int32_t)i;
  PyObject* l[4] = {list_of(rows), list_of(active), list_of(counts), list_of(offsets)};
  if (l[0] == nullptr || l[1] == nullptr || l[2] == nullptr || l[3] == nullptr) return nullptr;
  return Py_BuildValue("(NNNN)", l[0], l[1], l[2], l[3]);
  END_HANDLE_TH_ERRORS
}

// pack_lists(lists, device) -> one int32 tensor view per list over ONE device buffer (one pinned buffer, one copy), or None.
// `device` is a CUDA device index, or -1 for host memory.
PyObject* pack_lists(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  PyObject** lists;
  if (nargs != 2) { PyErr_SetString(PyExc_TypeError, "pack_lists takes 2 arguments"); return nullptr; }
  const Py_ssize_t n = items(args[0], &lists);
  const long dev = PyLong_AsLong(args[1]);
  if (PyErr_Occurred()) { PyErr_Clear(); return not_handled(); }
  if (n < 0) return not_handled();
  int64_t total = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject** it;
    const Py_ssize_t m = items(lists[i], &it);
    if (m < 0) return not_handled();
    total += m;
  }
  if (total == 0) return not_handled();
  at::Tensor host = at::empty({total}, at::TensorOptions().dtype(at::kInt).pinned_memory(dev >= 0));
  int32_t* dst = host.data_ptr<int32_t>();
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject** it;
    const Py_ssize_t m = items(lists[i], &it);
    for (Py_ssize_t k = 0; k < m; ++k)
      if (!as_int32(it[k], dst++)) return not_handled();
  }
  const at::Tensor packed = dev >= 0 ? host.to(at::Device(at::kCUDA, (c10::DeviceIndex)dev), /*non_blocking=*/true) : host;
  PyObject* out = PyList_New(n);
  if (out == nullptr) return nullptr;
  int64_t pos = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject** it;
    const Py_ssize_t m = items(lists[i], &it);
    PyList_SET_ITEM(out, i, THPVariable_Wrap(packed.narrow(0, pos, m)));
    pos += m;
  }
  return out;
  END_HANDLE_TH_ERRORS
}

// bind(addresses: dict name -> int, scratch_for)
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2 || !PyDict_Check(args[0])) { PyErr_SetString(PyExc_TypeError, "bind(dict, callable)"); return nullptr; }
  auto address = [&](const char* name) -> void* {
    PyObject* v = PyDict_GetItemString(args[0], name);
    return v == nullptr ? nullptr : PyLong_AsVoidPtr(v);
  };
#define B200_BIND(var, name) \
  if ((var = reinterpret_cast<decltype(var)>(address(#name))) == nullptr) { PyErr_SetString(PyExc_KeyError, #name); return nullptr; }
  B200_BIND(p_add, lora_b200_add)
  B200_BIND(p_delta, lora_b200_delta)
  B200_BIND(p_workspace_bytes, lora_b200_workspace_bytes)
  B200_BIND(p_linear, lora_b200_linear_lora)
  B200_BIND(p_linear_silu, lora_b200_linear_lora_silu)
  B200_BIND(p_rmsnorm, lora_b200_glue_add_rmsnorm)
  B200_BIND(p_silu, lora_b200_glue_silu_mul)
  B200_BIND(p_shrink, lora_b200_shrink_buckets)
  B200_BIND(p_expand, lora_b200_expand_buckets)
  B200_BIND(p_attention, lora_b200_prefill_attention)
  B200_BIND(p_rope, lora_b200_glue_rope_kv_store)
#undef B200_BIND
  Py_INCREF(args[1]);
  Py_XDECREF(scratch_for);
  scratch_for = args[1];
  Py_RETURN_NONE;
}

#define B200_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {B200_METHOD(add), B200_METHOD(shrink), B200_METHOD(expand), B200_METHOD(linear), B200_METHOD(add_rms_norm), B200_METHOD(silu_mul),
                         B200_METHOD(rope_kv_store), B200_METHOD(prefill_layers), B200_METHOD(bucket_lists), B200_METHOD(pack_lists), B200_METHOD(bind), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "b200lora_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_b200lora_binding(void) {
  s_weight = PyUnicode_InternFromString("weight");
  s_lora_a = PyUnicode_InternFromString("lora_A");
  s_tts = PyUnicode_InternFromString("token_to_slot");
  s_sorted = PyUnicode_InternFromString("token_indices_sorted_by_slot");
  s_ids = PyUnicode_InternFromString("active_slot_ids");
  s_counts = PyUnicode_InternFromString("num_tokens_per_slot");
  s_offsets = PyUnicode_InternFromString("slot_start_offsets");
  s_num_active = PyUnicode_InternFromString("num_active_loras");
  return PyModule_Create(&module_def);
}
