// The plain form of the decode path's operators as one native call each: tensors in, tensors out.
//
// A decode step is a chain of kernels of 3 to 25 us, and what a call of ops.py costs on the host (argument checks,
// allocations and a ctypes call, each through Python) is about as much.  These functions do the same checks, allocate the
// results and enter the C ABI of libinferop_b200.so without coming back to Python in between.  Quantiser and GEMM of
// 32 x 1024 x 1024, called one after the other: 21.8 -> 9.2 us; of 64 x 24576 x 1536, where the kernels are about as long: 22.1 ->
// 18.4; an attention step of a few short sequences 72 -> 41.
//
// Each takes the arguments of its namesake in ops.py that a plain call has and returns
//   the result(s)   the call was made,
//   an int          the C ABI refused it (status; nothing was launched),
//   None            not the plain case (another device, a view that is not contiguous, a subclass, a wrong type or shape):
//                   ops.py makes the call, or refuses it with its own message.
// Tensors are allocated through torch's dispatcher as torch.empty does; its errors come out as the Python exceptions they
// are there.  The interpreter lock is released from the first allocation to the end of the call, as ctypes does.
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include "inferop_b200.h"

namespace {

const at::Tensor* tensor(PyObject* o) {
  return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr;
}
// Whether `t` is a contiguous tensor on the current CUDA device, which it names.  (A CPU tensor asks CUDA nothing.)
bool leads(const at::Tensor* t, c10::DeviceIndex* dev) {
  if (!t || !t->is_cuda() || !t->is_contiguous()) return false;
  *dev = c10::cuda::current_device();
  return t->device().index() == *dev;
}
// the other tensors of the call
bool plain(const at::Tensor* t, c10::DeviceIndex dev) {
  return t && t->is_cuda() && t->device().index() == dev && t->is_contiguous();
}
int code_of(at::ScalarType t) {   // element type codes of the C ABI, -1: none
  return t == at::kFloat ? 0 : t == at::kHalf ? 1 : t == at::kBFloat16 ? 2 : -1;
}
int out_code(PyObject* o, at::ScalarType* t) {
  if (!THPDtype_Check(o)) return -1;
  *t = reinterpret_cast<THPDtype*>(o)->scalar_type;
  return code_of(*t);
}
bool number(PyObject* o, float* v) {
  if (!PyFloat_CheckExact(o) && !PyLong_CheckExact(o)) return false;
  const double d = PyFloat_AsDouble(o);
  if (d == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  *v = static_cast<float>(d);
  return true;
}
void* stream_of(c10::DeviceIndex dev) { return c10::cuda::getCurrentCUDAStream(dev).stream(); }
at::Tensor make(at::IntArrayRef sizes, const at::Tensor& like, at::ScalarType t) {
  return at::empty(sizes, like.options().dtype(t).requires_grad(false).memory_format(std::nullopt));
}
// b_q uint8 [n, k], b_scales fp32 [ceil(n / 128), k / 128]
bool weights_ok(const at::Tensor& bq, const at::Tensor& bs, int64_t k) {
  return bq.dim() == 2 && bq.scalar_type() == at::kByte && bq.size(1) == k && bs.dim() == 2 &&
         bs.scalar_type() == at::kFloat && bs.size(0) == (bq.size(0) + 127) / 128 && bs.size(1) == k / 128;
}
PyObject* pair(at::Tensor&& a, at::Tensor&& b) {
  PyObject* t = PyTuple_New(2);
  if (!t) return nullptr;
  PyObject* x = THPVariable_Wrap(std::move(a));
  PyObject* y = THPVariable_Wrap(std::move(b));
  if (!x || !y) {
    Py_XDECREF(x);
    Py_XDECREF(y);
    Py_DECREF(t);
    return nullptr;
  }
  PyTuple_SET_ITEM(t, 0, x);
  PyTuple_SET_ITEM(t, 1, y);
  return t;
}

// quant(x)
PyObject* quant(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 1) Py_RETURN_NONE;
  const at::Tensor* x = tensor(a[0]);
  c10::DeviceIndex dev;
  if (!leads(x, &dev) || x->dim() != 2) Py_RETURN_NONE;
  const int dt = code_of(x->scalar_type());
  const int64_t rows = x->size(0), cols = x->size(1);
  if (dt < 0 || rows == 0 || cols % 128 != 0) Py_RETURN_NONE;
  at::Tensor q, s;
  int rc;
  {
    pybind11::gil_scoped_release unlocked;
    q = make({rows, cols}, *x, at::kByte);
    s = make({rows, cols / 128}, *x, at::kFloat);
    rc = inferop_quant_fp8_per_token_group(q.data_ptr(), s.data_ptr(), x->data_ptr(), dt, rows, cols, 128, stream_of(dev));
  }
  if (rc != INFEROP_OK) return PyLong_FromLong(rc);
  return pair(std::move(q), std::move(s));
  END_HANDLE_TH_ERRORS
}

// gemm(a_q, a_scales, b_q, b_scales, out_dtype)
PyObject* gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5) Py_RETURN_NONE;
  const at::Tensor *aq = tensor(a[0]), *as = tensor(a[1]), *bq = tensor(a[2]), *bs = tensor(a[3]);
  at::ScalarType ot;
  const int od = out_code(a[4], &ot);
  c10::DeviceIndex dev;
  if (od < 0 || !leads(aq, &dev) || !plain(as, dev) || !plain(bq, dev) || !plain(bs, dev)) Py_RETURN_NONE;
  if (aq->dim() != 2 || aq->scalar_type() != at::kByte || as->dim() != 2 || as->scalar_type() != at::kFloat) Py_RETURN_NONE;
  const int64_t m = aq->size(0), k = aq->size(1);
  if (k % 128 != 0 || as->size(0) != m || as->size(1) != k / 128 || !weights_ok(*bq, *bs, k)) Py_RETURN_NONE;
  const int64_t nn = bq->size(0);
  at::Tensor c;
  int rc;
  {
    pybind11::gil_scoped_release unlocked;
    c = make({m, nn}, *aq, ot);
    rc = inferop_w8a8_block_fp8_gemm(c.data_ptr(), aq->data_ptr(), as->data_ptr(), bq->data_ptr(), bs->data_ptr(), m, nn, k,
                                     128, 128, od, stream_of(dev));
  }
  if (rc != INFEROP_OK) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(c));
  END_HANDLE_TH_ERRORS
}

// gemm_fused_quant(a, b_q, b_scales, out_dtype)
PyObject* gemm_fused_quant(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4) Py_RETURN_NONE;
  const at::Tensor *x = tensor(a[0]), *bq = tensor(a[1]), *bs = tensor(a[2]);
  at::ScalarType ot;
  const int od = out_code(a[3], &ot);
  c10::DeviceIndex dev;
  if (od < 0 || !leads(x, &dev) || !plain(bq, dev) || !plain(bs, dev) || x->dim() != 2) Py_RETURN_NONE;
  const int dt = code_of(x->scalar_type());
  const int64_t m = x->size(0), k = x->size(1);
  if (dt < 1 || k % 128 != 0 || !weights_ok(*bq, *bs, k)) Py_RETURN_NONE;
  const int64_t nn = bq->size(0);
  at::Tensor c;
  int rc;
  {
    pybind11::gil_scoped_release unlocked;
    c = make({m, nn}, *x, ot);
    rc = inferop_w8a8_block_fp8_gemm_fused_quant(c.data_ptr(), x->data_ptr(), dt, bq->data_ptr(), bs->data_ptr(), m, nn, k, 128,
                                                 128, od, stream_of(dev));
  }
  if (rc != INFEROP_OK) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(c));
  END_HANDLE_TH_ERRORS
}

// rmsnorm_quant(x, weight, eps, residual or None)
PyObject* rmsnorm_quant(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  float eps;
  if (n != 4 || !number(a[2], &eps)) Py_RETURN_NONE;
  const bool add = a[3] != Py_None;
  const at::Tensor *x = tensor(a[0]), *w = tensor(a[1]), *r = add ? tensor(a[3]) : nullptr;
  c10::DeviceIndex dev;
  if (!leads(x, &dev) || !plain(w, dev) || (add && !plain(r, dev)) || x->dim() != 2) Py_RETURN_NONE;
  const int dt = code_of(x->scalar_type());
  const int64_t rows = x->size(0), cols = x->size(1);
  if (dt < 1 || cols % 128 != 0 || w->scalar_type() != x->scalar_type() || w->dim() != 1 || w->size(0) != cols) Py_RETURN_NONE;
  if (add && (r->scalar_type() != x->scalar_type() || r->sizes() != x->sizes())) Py_RETURN_NONE;
  at::Tensor q, s;
  int rc;
  {
    pybind11::gil_scoped_release unlocked;
    q = make({rows, cols}, *x, at::kByte);
    s = make({rows, cols / 128}, *x, at::kFloat);
    rc = inferop_rmsnorm_quant(q.data_ptr(), s.data_ptr(), add ? r->data_ptr() : nullptr, x->data_ptr(), w->data_ptr(), dt, rows,
                               cols, 128, eps, stream_of(dev));
  }
  if (rc != INFEROP_OK) return PyLong_FromLong(rc);
  return pair(std::move(q), std::move(s));
  END_HANDLE_TH_ERRORS
}

// rope_neox(qkv, positions, rotary_dim, base, yarn_factor): in place; True when done
PyObject* rope_neox(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  float base, yarn;
  if (n != 5 || !PyLong_CheckExact(a[2]) || !number(a[3], &base) || !number(a[4], &yarn)) Py_RETURN_NONE;
  int overflow = 0;
  const long rotary = PyLong_AsLongAndOverflow(a[2], &overflow);
  const at::Tensor *x = tensor(a[0]), *pos = tensor(a[1]);
  c10::DeviceIndex dev;
  if (overflow || rotary < 0 || rotary > 0x7FFFFFFF || !leads(x, &dev) || !plain(pos, dev) || x->dim() != 3) Py_RETURN_NONE;
  const int dt = code_of(x->scalar_type());
  if (dt < 0 || pos->scalar_type() != at::kLong || pos->numel() != x->size(0) || x->size(1) > 0x7FFFFFFF ||
      x->size(2) > 0x7FFFFFFF) {
    Py_RETURN_NONE;
  }
  int rc;
  {
    pybind11::gil_scoped_release unlocked;
    rc = inferop_rope_neox(x->data_ptr(), static_cast<const int64_t*>(pos->data_ptr()), dt, x->size(0),
                           static_cast<int32_t>(x->size(1)), static_cast<int32_t>(x->size(2)), static_cast<int32_t>(rotary), base,
                           yarn, stream_of(dev));
  }
  if (rc != INFEROP_OK) return PyLong_FromLong(rc);
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// paged_attn_decode(q, k_cache, v_cache, block_tables, seq_lens, scale)
PyObject* paged_attn_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  float scale;
  if (n != 6 || !number(a[5], &scale)) Py_RETURN_NONE;
  const at::Tensor *q = tensor(a[0]), *kc = tensor(a[1]), *vc = tensor(a[2]), *bt = tensor(a[3]), *sl = tensor(a[4]);
  c10::DeviceIndex dev;
  if (!leads(q, &dev) || !plain(kc, dev) || !plain(vc, dev) || !plain(bt, dev) || !plain(sl, dev)) Py_RETURN_NONE;
  const at::ScalarType t = q->scalar_type();
  const int dt = code_of(t);
  if (dt < 0 || q->dim() != 3 || kc->dim() != 4 || vc->sizes() != kc->sizes() || kc->scalar_type() != t ||
      vc->scalar_type() != t || kc->size(3) != q->size(2)) {
    Py_RETURN_NONE;
  }
  if (bt->scalar_type() != at::kInt || sl->scalar_type() != at::kInt || bt->dim() != 2 || bt->size(0) != q->size(0) ||
      sl->numel() != q->size(0)) {
    Py_RETURN_NONE;
  }
  for (const int64_t v : {q->size(0), q->size(1), kc->size(1), kc->size(2), q->size(2), bt->size(1)})
    if (v > 0x7FFFFFFF) Py_RETURN_NONE;
  at::Tensor out;
  int rc;
  {
    pybind11::gil_scoped_release unlocked;
    out = make(q->sizes(), *q, t);
    rc = inferop_paged_attn_decode(out.data_ptr(), q->data_ptr(), kc->data_ptr(), vc->data_ptr(),
                                   static_cast<const int32_t*>(bt->data_ptr()), static_cast<const int32_t*>(sl->data_ptr()), dt,
                                   static_cast<int32_t>(q->size(0)), static_cast<int32_t>(q->size(1)),
                                   static_cast<int32_t>(kc->size(2)), static_cast<int32_t>(q->size(2)),
                                   static_cast<int32_t>(kc->size(1)), static_cast<int32_t>(bt->size(1)), scale, stream_of(dev));
  }
  if (rc != INFEROP_OK) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

#define FAST(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(quant), FAST(gemm), FAST(gemm_fused_quant), FAST(rmsnorm_quant), FAST(rope_neox),
                         FAST(paged_attn_decode), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall() { return PyModule_Create(&module); }
