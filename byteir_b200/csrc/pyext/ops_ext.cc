// Native side of byteir_b200/ops.py: argument checks, output and workspace allocation and the call into the kernel
// ABI (include/b200_kernels.h) for one op, in one step from Python.
//
// Why: an op on a small tensor takes 2-5 us on the GPU, while the same steps written in Python (tensor attributes,
// torch.empty, the current stream, a ctypes call with a dozen converted arguments) took 12-15 us per call, 20-25 us
// with a workspace and 60 us for attention forward + backward, so the host bound every call below ~100 MB.
//
// The GIL is released around the kernel call, as ctypes does: a launch blocks while the stream's queue is full.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <initializer_list>

#include "b200_kernels.h"

extern "C" {
// entry points that pick a code path explicitly (0 = automatic); not in the header
int b200_index_select_path(int path, int elt_bytes, int idx_bytes, const void *in, const void *idx, void *out, int64_t A,
                           int64_t IB, int64_t OB, int64_t C, int *status, cudaStream_t stream);
int b200_transpose_batched_path(int path, int elt_bytes, const void *in, void *out, int64_t batch, int64_t rows,
                                int64_t cols, cudaStream_t stream);
size_t b200_reduce_scratch_bytes(int op, int dtype, int64_t A, int64_t B, int64_t C);
}

namespace {

using at::Tensor;
using Shape = c10::SmallVector<int64_t, 8>;

PyObject *g_check = nullptr; // _native.check(rc, what): raises B200Error

// thrown after a Python exception has been set
struct Raised {};

[[noreturn]] void raise(PyObject *type, const char *msg) {
  PyErr_SetString(type, msg);
  throw Raised();
}

const Tensor &tensor(PyObject *o, const char *what) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a tensor, not %s", what, Py_TYPE(o)->tp_name);
    throw Raised();
  }
  return THPVariable_Unpack(o);
}
const Tensor *optional(PyObject *o, const char *what) { return o == Py_None ? nullptr : &tensor(o, what); }
int64_t integer(PyObject *o) {
  const int64_t v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred())
    throw Raised();
  return v;
}
float real(PyObject *o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred())
    throw Raised();
  return (float)v;
}

int dtype_code(const Tensor &t) {
  switch (t.scalar_type()) {
  case at::kFloat: return B200_F32;
  case at::kHalf: return B200_F16;
  case at::kBFloat16: return B200_BF16;
  default:
    PyErr_Format(PyExc_TypeError, "unsupported element type %s", c10::toString(t.scalar_type()));
    throw Raised();
  }
}

void need_cuda(const Tensor &t) {
  if (!t.is_cuda())
    raise(PyExc_ValueError, "byteir_b200 ops take CUDA tensors; there is no CPU path");
  if (!t.is_contiguous())
    raise(PyExc_ValueError, "tensors must be contiguous (ByRE memrefs are)");
}

Tensor new_empty(at::IntArrayRef shape, at::ScalarType type, const Tensor &like) {
  return at::detail::empty_cuda(shape, type, like.device(), std::nullopt);
}
// torch.empty_like, by the short way where the strides are the plain ones.  is_contiguous() does not say so: it passes over
// dimensions of size 1, whose strides empty_like keeps (the batch of one of x[:, :s]).
Tensor new_like(const Tensor &t) {
  int64_t plain = 1;
  for (int64_t i = t.dim() - 1; i >= 0; --i) {
    if (t.stride(i) != plain)
      return at::empty_like(t);
    plain *= t.size(i);
  }
  return new_empty(t.sizes(), t.scalar_type(), t);
}

// the caller's workspace, or one of `need` bytes from torch's caching allocator (stream-ordered: it may be handed out
// again as soon as this call has been enqueued)
struct Workspace {
  Workspace(const Tensor *given, size_t need, const Tensor &like) {
    if (given) {
      ptr = given->data_ptr();
      bytes = (size_t)given->numel() * given->element_size();
    } else if (need) {
      own = new_empty({(int64_t)need}, at::kByte, like);
      ptr = own.data_ptr();
      bytes = need;
    }
  }
  Tensor own;
  void *ptr = nullptr;
  size_t bytes = 0;
};

cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

template <typename F> void call(const char *what, F &&f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS;
  rc = f();
  Py_END_ALLOW_THREADS;
  if (rc) {
    PyObject *r = PyObject_CallFunction(g_check, "is", rc, what);
    Py_XDECREF(r);
    if (!r)
      throw Raised();
  }
}

int *status_ptr(const Tensor *t) { return t ? static_cast<int *>(t->data_ptr()) : nullptr; }
const void *ptr(const Tensor *t) { return t ? t->data_ptr() : nullptr; }
PyObject *wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject *given_or(PyObject *given, Tensor &made) {
  if (given != Py_None) {
    Py_INCREF(given);
    return given;
  }
  return wrap(std::move(made));
}

// ---- reductions ---------------------------------------------------------------------------------------------------
struct Abc {
  int64_t A, B, C;
  Shape out;
};

// The A x B x C view (reduce_impl.h:28-59) of `x` reduced over `dims`.  Dimensions of size 1 are taken out of the
// shape first, so that reduced dimensions with only such dimensions between them count as consecutive.
Abc reduce_view(const Tensor &x, PyObject *dims) {
  const auto shape = x.sizes();
  const int64_t rank = (int64_t)shape.size();
  c10::SmallVector<bool, 8> reduced(rank, false);
  PyObject *seq = PySequence_Fast(dims, "dimensions must be a sequence of integers");
  if (!seq)
    throw Raised();
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) {
    const int64_t d = PyLong_AsLongLong(PySequence_Fast_GET_ITEM(seq, i));
    if ((d == -1 && PyErr_Occurred()) || d < 0 || d >= rank) {
      Py_DECREF(seq);
      if (!PyErr_Occurred())
        PyErr_SetString(PyExc_IndexError, "reduce dimension out of range");
      throw Raised();
    }
    reduced[d] = true;
  }
  Py_DECREF(seq);
  Abc r{1, 1, 1, {}};
  int state = 0; // 0 in front of the reduced group, 1 inside, 2 behind it
  for (int64_t i = 0; i < rank; ++i) {
    if (!reduced[i])
      r.out.push_back(shape[i]);
    if (shape[i] == 1)
      continue;
    if (reduced[i]) {
      if (state == 2)
        raise(PyExc_ValueError, "Only consecutive dimensions reduction is supported");
      state = 1;
      r.B *= shape[i];
    } else if (state == 0) {
      r.A *= shape[i];
    } else {
      state = 2;
      r.C *= shape[i];
    }
  }
  if (state == 0) { // nothing to reduce: a copy
    r.C = x.numel();
    r.A = r.B = 0;
  }
  return r;
}

// (op, x, dimensions, out, workspace)
PyObject *reduce(PyObject *const *a, Py_ssize_t) {
  const int op = (int)integer(a[0]);
  const Tensor &x = tensor(a[1], "x");
  need_cuda(x);
  const int dt = dtype_code(x);
  const Abc v = reduce_view(x, a[2]);
  const Tensor *given = optional(a[3], "out");
  Tensor made;
  if (!given)
    made = new_empty(v.out, x.scalar_type(), x);
  const Tensor *ws_given = optional(a[4], "workspace");
  Workspace ws(ws_given, ws_given ? 0 : b200_reduce_scratch_bytes(op, dt, v.A, v.B, v.C), x);
  const void *in = x.data_ptr();
  void *out = given ? given->data_ptr() : made.data_ptr();
  cudaStream_t st = stream();
  call("b200_reduce", [&] { return b200_reduce(op, dt, in, out, v.A, v.B, v.C, ws.ptr, ws.bytes, st); });
  return given_or(a[3], made);
}

// (x, dimensions, out, workspace): the unrounded f32 sum, A x C values
PyObject *reduce_sum_to_f32(PyObject *const *a, Py_ssize_t) {
  const Tensor &x = tensor(a[0], "x");
  need_cuda(x);
  const int dt = dtype_code(x);
  const Abc v = reduce_view(x, a[1]);
  const Tensor *given = optional(a[2], "out");
  Tensor made;
  if (!given)
    made = new_empty({v.A * v.C}, at::kFloat, x);
  const Tensor *ws_given = optional(a[3], "workspace");
  Workspace ws(ws_given, ws_given ? 0 : b200_reduce_scratch_bytes(B200_REDUCE_SUM, dt, v.A, v.B, v.C), x);
  const void *in = x.data_ptr();
  float *out = static_cast<float *>(given ? given->data_ptr() : made.data_ptr());
  cudaStream_t st = stream();
  call("b200_reduce_sum_to_f32", [&] { return b200_reduce_sum_to_f32(dt, in, out, v.A, v.B, v.C, ws.ptr, ws.bytes, st); });
  return given_or(a[2], made);
}

// ---- indexing -----------------------------------------------------------------------------------------------------
int64_t checked_dim(const Tensor &x, PyObject *o) {
  const int64_t dim = integer(o);
  if (dim < 0 || dim >= x.dim())
    raise(PyExc_IndexError, "dim out of range");
  return dim;
}

// (x, index, dim, out, status, path)
PyObject *index_select(PyObject *const *a, Py_ssize_t) {
  const Tensor &x = tensor(a[0], "x"), &index = tensor(a[1], "index");
  need_cuda(x);
  need_cuda(index);
  const auto it = index.scalar_type();
  if (it != at::kLong && it != at::kInt && it != at::kUInt32)
    raise(PyExc_TypeError, "index must be i64 or ui32");
  const int64_t dim = checked_dim(x, a[2]);
  const auto shape = x.sizes();
  int64_t A = 1, C = 1;
  for (int64_t i = 0; i < dim; ++i)
    A *= shape[i];
  for (int64_t i = dim + 1; i < x.dim(); ++i)
    C *= shape[i];
  const int64_t IB = shape[dim], OB = index.numel();
  const Tensor *given = optional(a[3], "out"), *status = optional(a[4], "status");
  const int path = (int)integer(a[5]);
  Tensor made;
  if (!given) {
    Shape os(shape.begin(), shape.end());
    os[dim] = OB;
    made = new_empty(os, x.scalar_type(), x);
  }
  const int es = (int)x.element_size(), is = (int)index.element_size();
  const void *in = x.data_ptr(), *idx = index.data_ptr();
  void *out = given ? given->data_ptr() : made.data_ptr();
  cudaStream_t st = stream();
  call("b200_index_select",
       [&] { return b200_index_select_path(path, es, is, in, idx, out, A, IB, OB, C, status_ptr(status), st); });
  return given_or(a[3], made);
}

// (x, index, update, dim, out, workspace, status)
PyObject *index_put_add(PyObject *const *a, Py_ssize_t) {
  const Tensor &x = tensor(a[0], "x"), &index = tensor(a[1], "index"), &update = tensor(a[2], "update");
  need_cuda(x);
  need_cuda(index);
  need_cuda(update);
  if (index.scalar_type() != at::kLong)
    raise(PyExc_TypeError, "index must be i64");
  const int dt = dtype_code(x);
  const int64_t dim = checked_dim(x, a[3]);
  int64_t rows = 1, feature = 1;
  for (int64_t i = 0; i < x.dim(); ++i)
    (i <= dim ? rows : feature) *= x.sizes()[i];
  const int64_t n = index.numel();
  const Tensor *given = optional(a[4], "out"), *ws_given = optional(a[5], "workspace"), *status = optional(a[6], "status");
  Tensor made;
  if (!given)
    made = new_like(x);
  Workspace ws(ws_given, ws_given ? 0 : b200_index_put_workspace_bytes(dt, rows, n, feature), x);
  const void *in = x.data_ptr(), *upd = update.data_ptr();
  const int64_t *idx = static_cast<const int64_t *>(index.data_ptr());
  void *out = given ? given->data_ptr() : made.data_ptr();
  cudaStream_t st = stream();
  call("b200_index_put_add", [&] {
    return b200_index_put_add(dt, in, idx, upd, out, rows, n, feature, ws.ptr, ws.bytes, status_ptr(status), st);
  });
  return given_or(a[4], made);
}

// ---- transposes ---------------------------------------------------------------------------------------------------
// (x, permutation, out)
PyObject *transpose(PyObject *const *a, Py_ssize_t) {
  const Tensor &x = tensor(a[0], "x");
  need_cuda(x);
  const int64_t rank = x.dim();
  Shape perm, os;
  PyObject *seq = PySequence_Fast(a[1], "permutation must be a sequence of integers");
  if (!seq)
    throw Raised();
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i)
    perm.push_back(PyLong_AsLongLong(PySequence_Fast_GET_ITEM(seq, i)));
  Py_DECREF(seq);
  if (PyErr_Occurred())
    throw Raised();
  bool fits = (int64_t)perm.size() == rank;
  for (int64_t p : perm)
    fits = fits && p >= 0 && p < rank;
  if (!fits)
    raise(PyExc_IndexError, "permutation does not fit the rank of x");
  const Tensor *given = optional(a[2], "out");
  Tensor made;
  if (!given) {
    for (int64_t p : perm)
      os.push_back(x.sizes()[p]);
    made = new_empty(os, x.scalar_type(), x);
  }
  const int es = (int)x.element_size();
  const void *in = x.data_ptr();
  void *out = given ? given->data_ptr() : made.data_ptr();
  cudaStream_t st = stream();
  call("b200_permute", [&] { return b200_permute(es, in, out, (int)rank, x.sizes().data(), perm.data(), st); });
  return given_or(a[2], made);
}

// (x, out, path): [batch, rows, cols] -> [batch, cols, rows]
PyObject *transpose_batched(PyObject *const *a, Py_ssize_t) {
  const Tensor &x = tensor(a[0], "x");
  need_cuda(x);
  if (x.dim() != 3)
    raise(PyExc_ValueError, "x must be [batch, rows, cols]");
  const int64_t b = x.size(0), r = x.size(1), c = x.size(2);
  const Tensor *given = optional(a[1], "out");
  const int path = (int)integer(a[2]);
  Tensor made;
  if (!given)
    made = new_empty({b, c, r}, x.scalar_type(), x);
  const int es = (int)x.element_size();
  const void *in = x.data_ptr();
  void *out = given ? given->data_ptr() : made.data_ptr();
  cudaStream_t st = stream();
  call("b200_transpose_batched", [&] { return b200_transpose_batched_path(path, es, in, out, b, r, c, st); });
  return given_or(a[1], made);
}

// ---- attention ----------------------------------------------------------------------------------------------------
int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

void need_rows(std::initializer_list<const Tensor *> ts, const char *msg) {
  for (const Tensor *t : ts) {
    if (!t)
      continue;
    if (!t->is_cuda() || t->dim() != 4 || t->stride(3) != 1)
      raise(PyExc_ValueError, msg);
  }
}

void window_of(PyObject *o, bool causal, int64_t *left, int64_t *right) {
  PyObject *seq = PySequence_Fast(o, "window must be (left, right)");
  if (!seq)
    throw Raised();
  if (PySequence_Fast_GET_SIZE(seq) != 2) {
    Py_DECREF(seq);
    raise(PyExc_ValueError, "window must be (left, right)");
  }
  *left = PyLong_AsLongLong(PySequence_Fast_GET_ITEM(seq, 0));
  *right = PyLong_AsLongLong(PySequence_Fast_GET_ITEM(seq, 1));
  Py_DECREF(seq);
  if (PyErr_Occurred())
    throw Raised();
  if (causal)
    *right = 0;
}

bool truth(PyObject *o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0)
    throw Raised();
  return v != 0;
}

b200_flash_attn_params attn_params(const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &o, PyObject *scale,
                                   PyObject *causal, PyObject *window) {
  b200_flash_attn_params p{};
  p.q_batch_stride = q.stride(0), p.q_row_stride = q.stride(1), p.q_head_stride = q.stride(2);
  p.k_batch_stride = k.stride(0), p.k_row_stride = k.stride(1), p.k_head_stride = k.stride(2);
  p.v_batch_stride = v.stride(0), p.v_row_stride = v.stride(1), p.v_head_stride = v.stride(2);
  p.o_batch_stride = o.stride(0), p.o_row_stride = o.stride(1), p.o_head_stride = o.stride(2);
  p.b = q.size(0), p.seqlen_q = q.size(1), p.h = q.size(2), p.d = q.size(3);
  p.seqlen_k = k.size(1), p.h_k = k.size(2);
  p.d_rounded = round_up(p.d, 32);
  p.seqlen_q_rounded = round_up(p.seqlen_q, 128), p.seqlen_k_rounded = round_up(p.seqlen_k, 128);
  p.softmax_scale = real(scale);
  p.p_dropout = 0.f;
  window_of(window, truth(causal), &p.window_size_left, &p.window_size_right);
  return p;
}

// (q, k, v, softmax_scale, causal, window, out, lse)
PyObject *flash_attn_fwd(PyObject *const *a, Py_ssize_t) {
  const Tensor &q = tensor(a[0], "q"), &k = tensor(a[1], "k"), &v = tensor(a[2], "v");
  need_rows({&q, &k, &v}, "q, k, v must be CUDA tensors with a contiguous last dim");
  const Tensor *out_given = optional(a[6], "out"), *lse_given = optional(a[7], "lse");
  Tensor out_made, lse_made;
  if (!out_given)
    out_made = new_like(q);
  if (!lse_given)
    lse_made = new_empty({q.size(0), q.size(2), q.size(1)}, at::kFloat, q);
  const Tensor &out = out_given ? *out_given : out_made;
  const b200_flash_attn_params p = attn_params(q, k, v, out, a[3], a[4], a[5]);
  const int dt = dtype_code(q);
  const void *qp = q.data_ptr(), *kp = k.data_ptr(), *vp = v.data_ptr();
  void *op = out.data_ptr();
  float *lp = static_cast<float *>(lse_given ? lse_given->data_ptr() : lse_made.data_ptr());
  cudaStream_t st = stream();
  call("b200_flash_attn_fwd", [&] { return b200_flash_attn_fwd(dt, qp, kp, vp, op, lp, &p, st); });
  return Py_BuildValue("NN", given_or(a[6], out_made), given_or(a[7], lse_made));
}

// (dout, q, k, v, out, lse, softmax_scale, causal, window, dq, dk, dv, d_softmax_sum)
PyObject *flash_attn_bwd(PyObject *const *a, Py_ssize_t) {
  const Tensor &dout = tensor(a[0], "dout"), &q = tensor(a[1], "q"), &k = tensor(a[2], "k"), &v = tensor(a[3], "v"),
               &out = tensor(a[4], "out"), &lse = tensor(a[5], "lse");
  need_rows({&dout, &q, &k, &v, &out}, "tensors must be CUDA tensors with a contiguous last dim");
  if (dout.strides() != out.strides())
    raise(PyExc_ValueError, "dout must share out's strides");
  const Tensor *given[4];
  Tensor made[4];
  const char *names[4] = {"dq", "dk", "dv", "d_softmax_sum"};
  for (int i = 0; i < 4; ++i)
    given[i] = optional(a[9 + i], names[i]);
  const Tensor *like[3] = {&q, &k, &v};
  for (int i = 0; i < 3; ++i) {
    // The kernel writes by the strides of q, k and v.  empty_like keeps them only where the tensor is dense, which one
    // part of a packed [B, S, 3, H, D] tensor, for instance, is not.
    if (!given[i])
      made[i] = like[i]->is_non_overlapping_and_dense() ? new_like(*like[i])
                                                        : at::empty_strided(like[i]->sizes(), like[i]->strides(), like[i]->options());
    else if (given[i]->sizes() == like[i]->sizes())
      for (int64_t d = 0; d < 4; ++d)
        if (given[i]->size(d) > 1 && given[i]->stride(d) != like[i]->stride(d))
          raise(PyExc_ValueError, "dq, dk, dv must share the strides of q, k, v");
  }
  const b200_flash_attn_params p = attn_params(q, k, v, out, a[6], a[7], a[8]);
  if (!given[3])
    made[3] = new_empty({p.b, p.h, p.seqlen_q_rounded}, at::kFloat, q);
  void *g[4];
  for (int i = 0; i < 4; ++i)
    g[i] = given[i] ? given[i]->data_ptr() : made[i].data_ptr();
  const int dt = dtype_code(q);
  const void *dp = dout.data_ptr(), *qp = q.data_ptr(), *kp = k.data_ptr(), *vp = v.data_ptr(), *op = out.data_ptr();
  const float *lp = static_cast<const float *>(lse.data_ptr());
  cudaStream_t st = stream();
  call("b200_flash_attn_bwd", [&] {
    return b200_flash_attn_bwd(dt, dp, qp, kp, vp, op, lp, g[0], g[1], g[2], static_cast<float *>(g[3]), nullptr, &p, st);
  });
  return Py_BuildValue("NNN", given_or(a[9], made[0]), given_or(a[10], made[1]), given_or(a[11], made[2]));
}

// (q, kcache, vcache, knew, vnew, seqlens_k, softmax_scale, causal, window, out, lse, workspace)
PyObject *flash_attn_kvcache(PyObject *const *a, Py_ssize_t) {
  const Tensor &q = tensor(a[0], "q"), &kc = tensor(a[1], "kcache"), &vc = tensor(a[2], "vcache");
  const Tensor *kn = optional(a[3], "knew"), *vn = optional(a[4], "vnew"), *lens = optional(a[5], "seqlens_k");
  need_rows({&q, &kc, &vc, kn, vn}, "tensors must be CUDA tensors with a contiguous last dim");
  if (lens && (lens->scalar_type() != at::kInt || !lens->is_contiguous()))
    raise(PyExc_ValueError, "seqlens_k must be a contiguous int32 tensor");
  const Tensor *out_given = optional(a[9], "out"), *lse_given = optional(a[10], "lse"), *ws_given = optional(a[11], "workspace");
  Tensor out_made, lse_made;
  if (!out_given)
    out_made = new_like(q);
  if (!lse_given)
    lse_made = new_empty({q.size(0), q.size(2), q.size(1)}, at::kFloat, q);
  const Tensor &out = out_given ? *out_given : out_made;
  b200_flash_kvcache_params p{};
  p.q_batch_stride = q.stride(0), p.q_row_stride = q.stride(1), p.q_head_stride = q.stride(2);
  p.k_batch_stride = kc.stride(0), p.k_row_stride = kc.stride(1), p.k_head_stride = kc.stride(2);
  p.v_batch_stride = vc.stride(0), p.v_row_stride = vc.stride(1), p.v_head_stride = vc.stride(2);
  if (kn)
    p.knew_batch_stride = kn->stride(0), p.knew_row_stride = kn->stride(1), p.knew_head_stride = kn->stride(2);
  if (vn)
    p.vnew_batch_stride = vn->stride(0), p.vnew_row_stride = vn->stride(1), p.vnew_head_stride = vn->stride(2);
  p.o_batch_stride = out.stride(0), p.o_row_stride = out.stride(1), p.o_head_stride = out.stride(2);
  p.b = q.size(0), p.seqlen_q = q.size(1), p.h = q.size(2), p.d = q.size(3);
  p.seqlen_k = kc.size(1), p.h_k = kc.size(2);
  p.seqlen_knew = kn ? kn->size(1) : 0;
  p.d_rounded = round_up(p.d, 32);
  p.seqlen_q_rounded = round_up(p.seqlen_q, 128), p.seqlen_k_rounded = round_up(p.seqlen_k, 128);
  p.softmax_scale = a[6] == Py_None ? (float)(1.0 / std::sqrt((double)p.d)) : real(a[6]);
  window_of(a[8], truth(a[7]), &p.window_size_left, &p.window_size_right);
  const int dt = dtype_code(q);
  // the workspace comes from torch's allocator; without one the entry point takes it from the stream's memory pool
  const int64_t need = ws_given ? 0 : b200_flash_attn_kvcache_workspace_bytes(&p);
  Workspace ws(ws_given, need > 0 ? (size_t)need : 0, q);
  void *kcp = kc.data_ptr(), *vcp = vc.data_ptr(), *op = out.data_ptr();
  const void *qp = q.data_ptr();
  float *lp = static_cast<float *>(lse_given ? lse_given->data_ptr() : lse_made.data_ptr());
  cudaStream_t st = stream();
  call("b200_flash_attn_kvcache", [&] {
    return b200_flash_attn_kvcache(dt, qp, kcp, vcp, ptr(kn), ptr(vn), static_cast<const int32_t *>(ptr(lens)), op, lp, &p, ws.ptr,
                                   ws.bytes, st);
  });
  return Py_BuildValue("NN", given_or(a[9], out_made), given_or(a[10], lse_made));
}

// ---- module -------------------------------------------------------------------------------------------------------
template <PyObject *(*F)(PyObject *const *, Py_ssize_t), int N> PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
  if (n != N) {
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", N, n);
    return nullptr;
  }
  HANDLE_TH_ERRORS
  try {
    return F(args, n);
  } catch (const Raised &) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

#define OP(name, n) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(&entry<name, n>)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {OP(reduce, 5),
                           OP(reduce_sum_to_f32, 4),
                           OP(index_select, 6),
                           OP(index_put_add, 7),
                           OP(transpose, 3),
                           OP(transpose_batched, 3),
                           OP(flash_attn_fwd, 8),
                           OP(flash_attn_bwd, 13),
                           OP(flash_attn_kvcache, 12),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "byteir_b200._ops_ext", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__ops_ext(void) {
  PyObject *native = PyImport_ImportModule("byteir_b200._native");
  if (!native)
    return nullptr;
  g_check = PyObject_GetAttrString(native, "check");
  Py_DECREF(native);
  if (!g_check)
    return nullptr;
  return PyModule_Create(&g_module);
}
