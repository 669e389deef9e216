// The host side of the calls whose device work is shorter than the Python that launches it, as a CPython extension over
// the C ABI: checks, output tensors, argument structures and library calls of one step in one native call.
//
// Every function takes only the plain case: exact CUDA tensors of the expected types, shapes and layouts on the current
// device, no dispatch or function mode, no transform wrapper, nothing to convert or to copy.  For anything else it returns
// None before it has done anything, and the Python operator (which converts, copies or raises) runs as if it were not there.
// A library error code comes back as an int.  An allocation that fails comes back as None too, possibly behind launches of the
// same call (outputs are allocated between launches so that the device starts at once): the Python operator then runs the
// whole step again from the same inputs, into other outputs or the same cache rows, and meets the failure as its own.
//
// Host time of a step, us (calls into an empty queue; Python operators -> here): float32 decode step 81 -> 27, ratio-4
// token (prep and sdpa) 72 -> 25, q8 token (append and attention) 69 -> 20.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/moespresso_b200.h"

namespace {

struct Library {
  decltype(&mxb_indexer_scores) indexer_scores;
  decltype(&mxb_topk_workspace_bytes) topk_workspace_bytes;
  decltype(&mxb_topk_select) topk_select;
  decltype(&mxb_sparse_attn_workspace_bytes) sparse_attn_workspace_bytes;
  decltype(&mxb_sparse_attn) sparse_attn;
  decltype(&mxb_fused_decode_prep_workspace_bytes) fused_decode_prep_workspace_bytes;
  decltype(&mxb_fused_decode_prep) fused_decode_prep;
  decltype(&mxb_fused_decode_sdpa_workspace_bytes) fused_decode_sdpa_workspace_bytes;
  decltype(&mxb_fused_decode_sdpa) fused_decode_sdpa;
  decltype(&mxb_affine_q8_append) affine_q8_append;
  decltype(&mxb_sdpa_decode_q8) sdpa_decode_q8;
  decltype(&mxb_merge_partials) merge_partials;
} lib;
bool bound = false;

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return MXB_F32;
    case at::kHalf: return MXB_F16;
    case at::kBFloat16: return MXB_BF16;
    case at::kFloat8_e4m3fn: return MXB_F8E4M3;
    case at::kChar: return MXB_I8;
    default: return -1;
  }
}

// A call's device, stream and output allocations.
struct Call {
  c10::DeviceIndex dev = -1;
  bool ok = true;

  Call() {
    ok = bound && !c10::impl::dispatch_mode_enabled() && !at::impl::torch_function_mode_enabled();
    if (ok) dev = c10::cuda::current_device();
  }
  // The tensor behind `o` if it is a plain one on the current device; an empty reference and ok = false otherwise.
  const at::Tensor& tensor(PyObject* o) {
    static const at::Tensor none;
    if (!ok || !THPVariable_CheckExact(o)) {
      ok = false;
      return none;
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    constexpr c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                           c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize,
                                           c10::DispatchKey::Batched, c10::DispatchKey::Conjugate,
                                           c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
    if (!t.defined() || !t.is_cuda() || t.get_device() != dev || t.layout() != at::kStrided || t.key_set().has_any(wrapped) ||
        !t.has_storage()) {
      ok = false;
      return none;
    }
    return t;
  }
  const at::Tensor& tensor(PyObject* o, at::ScalarType type, int64_t dim) {   // contiguous, of this type and rank
    const at::Tensor& t = tensor(o);
    if (ok) ok = t.scalar_type() == type && t.dim() == dim && t.is_contiguous();
    return t;
  }
  void require(bool c) { ok = ok && c; }
  int64_t integer(PyObject* o) {
    if (!ok || !PyLong_CheckExact(o)) {
      ok = false;
      return 0;
    }
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      ok = false;
    }
    ok = ok && v >= -(1ll << 31) && v < (1ll << 31);
    return v;
  }
  double real(PyObject* o) {
    if (ok && PyFloat_CheckExact(o)) return PyFloat_AS_DOUBLE(o);
    ok = false;
    return 0.0;
  }
  at::Tensor empty(at::IntArrayRef sizes, at::ScalarType type) const {
    return at::empty(sizes, at::TensorOptions().dtype(type).device(at::Device(at::kCUDA, dev)));
  }
  at::Tensor scratch(int64_t bytes) const { return bytes > 0 ? empty({bytes}, at::kByte) : at::Tensor(); }
  void* stream() const { return c10::cuda::getCurrentCUDAStream(dev).stream(); }
};

template <class Args>
int launch(int (*fn)(const Args*, void*), const Args& a, void* stream) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(&a, stream);
  Py_END_ALLOW_THREADS
  return rc;
}

PyObject* tuple_of(std::initializer_list<at::Tensor> ts) {
  PyObject* out = PyTuple_New((Py_ssize_t)ts.size());
  if (!out) return nullptr;
  Py_ssize_t i = 0;
  for (const at::Tensor& t : ts) {
    PyObject* w = THPVariable_Wrap(t);
    if (!w) {
      Py_DECREF(out);
      return nullptr;
    }
    PyTuple_SET_ITEM(out, i++, w);
  }
  return out;
}

// Runs `body(call)`; a C++ exception (an allocation that failed, say) becomes None: the Python operator repeats the step.
template <class F>
PyObject* guarded(F&& body) {
  try {
    Call c;
    if (c.ok) return body(c);
  } catch (const std::exception&) {
    PyErr_Clear();
  }
  Py_RETURN_NONE;
}
#define PLAIN(c) do { if (!(c).ok) Py_RETURN_NONE; } while (0)

PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  void** slots[] = {(void**)&lib.indexer_scores, (void**)&lib.topk_workspace_bytes, (void**)&lib.topk_select,
                    (void**)&lib.sparse_attn_workspace_bytes, (void**)&lib.sparse_attn,
                    (void**)&lib.fused_decode_prep_workspace_bytes, (void**)&lib.fused_decode_prep,
                    (void**)&lib.fused_decode_sdpa_workspace_bytes, (void**)&lib.fused_decode_sdpa,
                    (void**)&lib.affine_q8_append, (void**)&lib.sdpa_decode_q8, (void**)&lib.merge_partials};
  if (n != (Py_ssize_t)(sizeof(slots) / sizeof(slots[0]))) {
    PyErr_SetString(PyExc_TypeError, "bind takes one address per library function");
    return nullptr;
  }
  for (Py_ssize_t i = 0; i < n; ++i) {
    *slots[i] = PyLong_AsVoidPtr(args[i]);
    if (PyErr_Occurred()) return nullptr;
  }
  bound = true;
  Py_RETURN_NONE;
}

// (q, idx_q, idx_w, kv, kv_scales, idx_keys, row_start, row_count, max_rows, k, scale, d_v, sinks, out_dtype, exact_fp32)
// -> (out, ids, scores)
PyObject* decode_step(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 15) Py_RETURN_NONE;
  return guarded([&](Call& c) -> PyObject* {
    const at::Tensor &q = c.tensor(args[0]), &idx_q = c.tensor(args[1]), &idx_w = c.tensor(args[2], at::kFloat, 2);
    const at::Tensor &kv = c.tensor(args[3]), &keys = c.tensor(args[5]);
    const at::Tensor &row_start = c.tensor(args[6], at::kLong, 1), &row_count = c.tensor(args[7], at::kInt, 1);
    const int64_t max_rows = c.integer(args[8]), k = c.integer(args[9]), d_v = c.integer(args[11]);
    const double scale = c.real(args[10]);
    c.require(args[14] == Py_True || args[14] == Py_False);
    c.require(THPDtype_Check(args[13]));
    PLAIN(c);
    const at::ScalarType out_type = reinterpret_cast<THPDtype*>(args[13])->scalar_type;
    const bool exact = args[14] == Py_True;
    c.require(q.dim() == 3 && idx_q.dim() == 3 && kv.dim() == 2 && keys.dim() == 2);
    PLAIN(c);
    const int64_t B = row_start.size(0), H = q.size(1), D = q.size(2), Hi = idx_q.size(1), Di = idx_q.size(2);
    c.require(B > 0 && k > 0 && max_rows > 0 && d_v > 0 && q.size(0) == B && idx_q.size(0) == B && row_count.size(0) == B &&
              idx_w.size(0) == B && idx_w.size(1) == Hi && keys.size(1) == Di && kv.size(1) == D);
    c.require(q.stride(2) == 1 && idx_q.stride(2) == 1 && kv.is_contiguous() && keys.is_contiguous());
    c.require(dtype_code(q.scalar_type()) >= 0 && dtype_code(idx_q.scalar_type()) >= 0 && dtype_code(kv.scalar_type()) >= 0 &&
              dtype_code(keys.scalar_type()) >= 0);
    c.require(out_type == at::kFloat || out_type == at::kHalf || out_type == at::kBFloat16);
    const at::Tensor *scales = nullptr, *sinks = nullptr;
    if (args[4] != Py_None) scales = &c.tensor(args[4], at::kHalf, 1);
    if (args[12] != Py_None) sinks = &c.tensor(args[12], at::kFloat, 1);
    c.require((kv.scalar_type() == at::kChar) == (scales != nullptr));
    PLAIN(c);
    c.require((!scales || scales->size(0) == kv.size(0)) && (!sinks || sinks->size(0) == H));
    PLAIN(c);

    void* st = c.stream();
    const at::Tensor scores = c.empty({keys.size(0)}, at::kFloat), ids = c.empty({B, k}, at::kInt);
    mxb_indexer_scores_args s{};
    s.q = idx_q.data_ptr(); s.q_dtype = dtype_code(idx_q.scalar_type());
    s.q_stride_b = idx_q.stride(0); s.q_stride_h = idx_q.stride(1); s.q_stride_t = Di;
    s.keys = keys.data_ptr(); s.key_dtype = dtype_code(keys.scalar_type());
    s.weights = static_cast<const float*>(idx_w.data_ptr()); s.scores = static_cast<float*>(scores.data_ptr());
    s.row_start = static_cast<const int64_t*>(row_start.data_ptr()); s.row_count = static_cast<const int32_t*>(row_count.data_ptr());
    s.B = (int32_t)B; s.T = 1; s.H = (int32_t)Hi; s.D = (int32_t)Di;
    s.n_rows = max_rows; s.rows_total = keys.size(0);
    s.flags = exact ? MXB_INDEXER_EXACT_FP32 : 0;
    if (const int rc = launch(lib.indexer_scores, s, st)) return PyLong_FromLong(rc);

    mxb_topk_args t{};
    t.scores = s.scores; t.row_start = s.row_start; t.row_count = s.row_count; t.out_ids = static_cast<int32_t*>(ids.data_ptr());
    t.rows = (int32_t)B; t.n = max_rows; t.k = (int32_t)k;
    const at::Tensor topk_ws = c.scratch(lib.topk_workspace_bytes(t.rows, t.n, t.k));
    if (topk_ws.defined()) { t.workspace = topk_ws.data_ptr(); t.workspace_bytes = topk_ws.numel(); }
    if (const int rc = launch(lib.topk_select, t, st)) return PyLong_FromLong(rc);

    const at::Tensor out = c.empty({B, H, d_v}, out_type);
    mxb_sparse_attn_args a{};
    a.q = q.data_ptr(); a.q_dtype = dtype_code(q.scalar_type());
    a.q_stride_b = q.stride(0); a.q_stride_h = q.stride(1); a.q_stride_t = D;
    a.comp_kv = kv.data_ptr(); a.kv_dtype = dtype_code(kv.scalar_type()); a.comp_scales = scales ? scales->data_ptr() : nullptr;
    a.comp_row_start = s.row_start; a.comp_row_count = s.row_count; a.n_comp = max_rows;
    a.topk = t.out_ids; a.k = (int32_t)k; a.sinks = sinks ? static_cast<const float*>(sinks->data_ptr()) : nullptr;
    a.out = out.data_ptr(); a.out_dtype = dtype_code(out_type);
    a.out_stride_b = H * d_v; a.out_stride_h = d_v; a.out_stride_t = d_v;
    a.B = (int32_t)B; a.T = 1; a.H = (int32_t)H; a.Dqk = (int32_t)D; a.Dv = (int32_t)d_v; a.scale = (float)scale;
    a.flags = MXB_SPARSE_AFTER_SELECT;   // (exact_fp32 is about the scores)
    const at::Tensor attn_ws = c.scratch(lib.sparse_attn_workspace_bytes(&a));
    if (attn_ws.defined()) { a.workspace = attn_ws.data_ptr(); a.workspace_bytes = attn_ws.numel(); }
    if (const int rc = launch(lib.sparse_attn, a, st)) return PyLong_FromLong(rc);
    return tuple_of({out, ids, scores});
  });
}

// inv_freq [32] float32 and params (int32 or int64) with at least `need` values, both contiguous
struct Token {
  const at::Tensor& inv_freq;
  const at::Tensor& params;
};
Token token(Call& c, PyObject* inv_freq, PyObject* params, int64_t need) {
  Token t{c.tensor(inv_freq, at::kFloat, 1), c.tensor(params)};
  if (c.ok)
    c.require(t.inv_freq.size(0) == 32 && t.params.numel() >= need && t.params.is_contiguous() &&
              (t.params.scalar_type() == at::kInt || t.params.scalar_type() == at::kLong));
  return t;
}

// (q_idx, pooled_qat, weights, kv_row, inv_freq, params, scale, topk) -> (sel, row, scores)
PyObject* fused_decode_prep(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 8) Py_RETURN_NONE;
  return guarded([&](Call& c) -> PyObject* {
    const at::Tensor &q = c.tensor(args[0]), &pooled = c.tensor(args[1], at::kFloat, 2), &weights = c.tensor(args[2], at::kFloat, 1);
    const at::Tensor& kv_row = c.tensor(args[3], at::kHalf, 1);
    const Token tok = token(c, args[4], args[5], 1);
    const double scale = c.real(args[6]);
    const int64_t topk = c.integer(args[7]);
    PLAIN(c);
    c.require(q.dim() == 2 && q.is_contiguous() &&
              (q.scalar_type() == at::kFloat || q.scalar_type() == at::kHalf || q.scalar_type() == at::kBFloat16));
    PLAIN(c);
    const int64_t heads = q.size(0), rows = pooled.size(0);
    c.require(q.size(1) == 128 && heads > 0 && heads <= 64 && pooled.size(1) == 128 && weights.size(0) == heads &&
              kv_row.size(0) == 512 && topk > 0 && topk < rows);
    PLAIN(c);
    const at::Tensor sel = c.empty({topk}, at::kInt), row = c.empty({512}, at::kHalf), scores = c.empty({rows}, at::kFloat);
    mxb_fused_decode_prep_args a{};
    a.q_idx = q.data_ptr(); a.q_dtype = dtype_code(q.scalar_type());
    a.pooled_qat = static_cast<const float*>(pooled.data_ptr()); a.weights = static_cast<const float*>(weights.data_ptr());
    a.kv_row = kv_row.data_ptr(); a.inv_freq = static_cast<const float*>(tok.inv_freq.data_ptr());
    a.params = tok.params.data_ptr(); a.params_int64 = tok.params.scalar_type() == at::kLong;
    a.scale = (float)scale; a.n_heads = (int32_t)heads; a.topk = (int32_t)topk; a.n_rows = rows;
    const at::Tensor ws = c.scratch(lib.fused_decode_prep_workspace_bytes(&a));
    a.sel = static_cast<int32_t*>(sel.data_ptr()); a.row = row.data_ptr(); a.scores = static_cast<float*>(scores.data_ptr());
    if (ws.defined()) { a.workspace = ws.data_ptr(); a.workspace_bytes = ws.numel(); }
    if (const int rc = launch(lib.fused_decode_prep, a, c.stream())) return PyLong_FromLong(rc);
    return tuple_of({sel, row, scores});
  });
}

// (q, window, row, pooled, sel, sinks, inv_freq, params, scale) -> out
PyObject* fused_decode_sdpa(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 9) Py_RETURN_NONE;
  return guarded([&](Call& c) -> PyObject* {
    const at::Tensor &q = c.tensor(args[0], at::kHalf, 2), &window = c.tensor(args[1], at::kHalf, 2);
    const at::Tensor &row = c.tensor(args[2], at::kHalf, 1), &pooled = c.tensor(args[3], at::kHalf, 2);
    const at::Tensor &sel = c.tensor(args[4], at::kInt, 1), &sinks = c.tensor(args[5], at::kHalf, 1);
    const Token tok = token(c, args[6], args[7], 2);
    const double scale = c.real(args[8]);
    PLAIN(c);
    const int64_t heads = q.size(0);
    c.require(heads > 0 && q.size(1) == 512 && window.size(1) == 512 && row.size(0) == 512 && pooled.size(1) == 512 &&
              sinks.size(0) == heads);
    PLAIN(c);
    const at::Tensor out = c.empty({heads, 512}, at::kHalf);
    mxb_fused_decode_sdpa_args a{};
    a.q = q.data_ptr(); a.window = window.data_ptr(); a.row = row.data_ptr(); a.pooled = pooled.data_ptr();
    a.sel = static_cast<const int32_t*>(sel.data_ptr()); a.sinks = sinks.data_ptr();
    a.inv_freq = static_cast<const float*>(tok.inv_freq.data_ptr());
    a.params = tok.params.data_ptr(); a.params_int64 = tok.params.scalar_type() == at::kLong; a.scale = (float)scale;
    a.n_heads = (int32_t)heads; a.window_rows = (int32_t)window.size(0); a.topk = (int32_t)sel.size(0); a.n_rows = pooled.size(0);
    const at::Tensor ws = c.scratch(lib.fused_decode_sdpa_workspace_bytes(&a));
    a.out = out.data_ptr();
    if (ws.defined()) { a.workspace = ws.data_ptr(); a.workspace_bytes = ws.numel(); }
    if (const int rc = launch(lib.fused_decode_sdpa, a, c.stream())) return PyLong_FromLong(rc);
    return THPVariable_Wrap(out);
  });
}

// Rows between consecutive heads of (packed, scales, biases) x (keys, values), all row-contiguous views [1, Hkv, P, w] of
// one capacity and one row width, scales of one type; 0 when they are not (_q8_head_rows of full_attention.py).
int64_t q8_head_rows(const at::Tensor* const* t) {
  const at::Tensor &kp = *t[0], &ks = *t[1], &vp = *t[3];
  for (int i = 0; i < 6; ++i)
    if (t[i]->dim() != 4) return 0;
  const int64_t heads = kp.size(1), n = kp.size(2), words = kp.size(3), groups = words / 16;
  if (words % 16 || kp.size(0) != 1 || ks.size(0) != 1 || vp.sizes() != kp.sizes() || vp.strides() != kp.strides() ||
      kp.stride(2) != words || kp.stride(3) != 1)
    return 0;
  if (ks.size(1) != heads || ks.size(2) != n || ks.size(3) != groups || ks.stride(2) != groups || ks.stride(3) != 1) return 0;
  for (const int i : {2, 4, 5})
    if (t[i]->sizes() != ks.sizes() || t[i]->strides() != ks.strides() || t[i]->scalar_type() != ks.scalar_type()) return 0;
  if (kp.scalar_type() != at::kInt || vp.scalar_type() != at::kInt) return 0;
  if (heads == 1) return n;
  const int64_t head_rows = kp.stride(1) / words;
  return kp.stride(1) % words == 0 && head_rows >= n && ks.stride(1) == head_rows * groups ? head_rows : 0;
}

// ((packed, scales, biases) of the keys, the same of the values, offset, capacity, keys, values): quantises the new rows into
// the cache -> the prefix including them as two such tuples
PyObject* q8_append(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 6) Py_RETURN_NONE;
  return guarded([&](Call& c) -> PyObject* {
    const at::Tensor* t[6];
    for (int s = 0; s < 2; ++s) {
      if (!PyTuple_CheckExact(args[s]) || PyTuple_GET_SIZE(args[s]) != 3) Py_RETURN_NONE;
      for (int i = 0; i < 3; ++i) t[3 * s + i] = &c.tensor(PyTuple_GET_ITEM(args[s], i));
    }
    const int64_t offset = c.integer(args[2]), capacity = c.integer(args[3]);
    const at::Tensor &k = c.tensor(args[4]), &v = c.tensor(args[5]);
    PLAIN(c);
    const int64_t head_rows = q8_head_rows(t);
    c.require(head_rows > 0 && k.dim() == 4 && k.sizes() == v.sizes() && k.strides() == v.strides());
    PLAIN(c);
    const int64_t heads = t[0]->size(1), rows = t[0]->size(2), width = 4 * t[0]->size(3), L = k.size(2);
    const at::ScalarType type = t[1]->scalar_type();
    c.require(L > 0 && offset >= 0 && offset + L <= capacity && offset + L <= rows && k.size(0) == 1 && k.size(1) == heads &&
              k.size(3) == width && k.stride(3) == 1 && k.scalar_type() == type && v.scalar_type() == type &&
              (type == at::kFloat || type == at::kHalf || type == at::kBFloat16));
    PLAIN(c);
    mxb_affine_q8_pair_args a{};
    a.x[0] = k.data_ptr(); a.x[1] = v.data_ptr();
    for (int s = 0; s < 2; ++s) {
      a.packed[s] = t[3 * s]->data_ptr(); a.scales[s] = t[3 * s + 1]->data_ptr(); a.biases[s] = t[3 * s + 2]->data_ptr();
    }
    a.x_dtype = a.sb_dtype = dtype_code(type);
    a.x_head_stride = k.stride(1); a.x_row_stride = k.stride(2); a.head_rows = head_rows; a.row0 = offset; a.n_rows = L;
    a.heads = (int32_t)heads; a.width = (int32_t)width;
    if (const int rc = launch(lib.affine_q8_append, a, c.stream())) return PyLong_FromLong(rc);
    PyObject* out = PyTuple_New(2);
    if (!out) return nullptr;
    for (int s = 0; s < 2; ++s) {
      PyObject* part = tuple_of({t[3 * s]->slice(2, 0, offset + L), t[3 * s + 1]->slice(2, 0, offset + L),
                                 t[3 * s + 2]->slice(2, 0, offset + L)});
      if (!part) {
        Py_DECREF(out);
        return nullptr;
      }
      PyTuple_SET_ITEM(out, s, part);
    }
    return out;
  });
}

// (queries [1, Hq, 1, 256], packed, scales, biases of keys, the same of values, scale, splits) -> [1, Hq, 1, 256]
PyObject* q8_decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 9) Py_RETURN_NONE;
  return guarded([&](Call& c) -> PyObject* {
    const at::Tensor& q = c.tensor(args[0]);
    const at::Tensor* t[6];
    for (int i = 0; i < 6; ++i) t[i] = &c.tensor(args[1 + i]);
    const double scale = c.real(args[7]);
    int64_t splits = c.integer(args[8]);
    PLAIN(c);
    const int64_t head_rows = q8_head_rows(t);
    const at::ScalarType type = q.scalar_type();
    c.require(head_rows > 0 && q.dim() == 4 && q.is_contiguous() &&
              (type == at::kFloat || type == at::kHalf || type == at::kBFloat16) && dtype_code(t[1]->scalar_type()) >= 0);
    PLAIN(c);
    const int64_t Hq = q.size(1), P = t[0]->size(2);
    c.require(q.size(0) == 1 && q.size(2) == 1 && q.size(3) == 256 && Hq > 0 && P > 0 &&
              t[0]->size(3) == 64);   // rows of 256 features: the library is not told the cache's width
    PLAIN(c);
    splits = std::max<int64_t>(1, std::min(splits, P));
    const at::Tensor parts = c.empty({splits * Hq * 258}, at::kFloat), out = c.empty({1, Hq, 1, 256}, type);
    float* o_parts = static_cast<float*>(parts.data_ptr());
    float* ml_parts = o_parts + splits * Hq * 256;
    void* st = c.stream();
    mxb_sdpa_decode_q8_args a{};
    a.q = q.data_ptr(); a.q_dtype = dtype_code(type);
    a.k_packed = t[0]->data_ptr(); a.k_scales = t[1]->data_ptr(); a.k_biases = t[2]->data_ptr();
    a.v_packed = t[3]->data_ptr(); a.v_scales = t[4]->data_ptr(); a.v_biases = t[5]->data_ptr();
    a.sb_dtype = dtype_code(t[1]->scalar_type()); a.head_stride_rows = head_rows;
    a.P = (int32_t)P; a.Hq = (int32_t)Hq; a.Hkv = (int32_t)t[0]->size(1); a.D = 256; a.scale = (float)scale;
    a.n_splits = (int32_t)splits; a.o_parts = o_parts; a.ml_parts = ml_parts;
    if (const int rc = launch(lib.sdpa_decode_q8, a, st)) return PyLong_FromLong(rc);
    mxb_merge_args m{};
    m.o_parts = o_parts; m.ml_parts = ml_parts; m.out = out.data_ptr(); m.out_dtype = dtype_code(type);
    m.out_stride_b = m.out_stride_t = Hq * 256; m.out_stride_h = 256;
    m.P = (int32_t)splits; m.B = m.T = 1; m.H = (int32_t)Hq; m.Dv = 256;
    if (const int rc = launch(lib.merge_partials, m, st)) return PyLong_FromLong(rc);
    return THPVariable_Wrap(out);
  });
}

#define FAST(name, doc) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, doc}
PyMethodDef methods[] = {
    FAST(bind, "addresses of the library's functions"),
    FAST(decode_step, "scores, selection and attention of one decode step"),
    FAST(fused_decode_prep, "the token operator of that name"),
    FAST(fused_decode_sdpa, "the token operator of that name"),
    FAST(q8_append, "new rows into an affine-q8 cache"),
    FAST(q8_decode, "one token over an affine-q8 cache"),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "native host calls over the C ABI", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
