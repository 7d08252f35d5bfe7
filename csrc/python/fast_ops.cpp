// The single-GPU ops as Python calls them, for the calls that ask for nothing: checks, output and launch in one native call.
//
// Why: the kernel of a small call is done before Python has prepared the next.  On the host such a call took, in Python and with this
// (B200, microseconds): residual + RMSNorm of 4 x 1024 7.6 and 4.9, GEMM of 16 x 1024 x 1024 9.6 and 4.4, SwiGLU projection 11.7 and
// 4.4, QKV projection 15.6 and 4.6, decode attention 11.0 and 4.4; the launch itself takes 2.3 of these, an output 0.9.
//
// Every function answers None for a call that is not plainly of that kind (an option set, another type, layout, device or number of
// dimensions than the kernels take, a tensor that is a subclass or wrapped by a transform, a mode that wants to see every call):
// the Python implementation beside it then does what it always did, errors included.  An error of the library is raised here as the
// Python path raises it.  The Python lock is not held while memory is allocated and kernels are launched.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/PythonTorchFunctionTLS.h>

#include <climits>
#include <cmath>

#include "../api/oob.h"
#include "../api/oob_model.h"

namespace {

PyObject* g_check = nullptr;  // ooverlap_b200._lib.check

// Releases the Python lock for a scope, also when an exception leaves it.
struct NoLock {
  PyThreadState* state = PyEval_SaveThread();
  ~NoLock() { PyEval_RestoreThread(state); }
};

PyObject* none() { Py_RETURN_NONE; }

// The library's error `rc` as an exception.
PyObject* fail(int rc) {
  PyObject* r = PyObject_CallFunction(g_check, "i", rc);
  Py_XDECREF(r);
  if (r != nullptr) PyErr_SetString(PyExc_RuntimeError, "the native library reported an error");
  return nullptr;
}

bool modes_on() {
  return c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled();
}

// A strided tensor of this device without anything wrapped around it, or null.
const at::Tensor* plain(PyObject* o, c10::DeviceIndex dev) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.device().index() != dev) return nullptr;
  static const c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::Functionalize,
                                            c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                            c10::DispatchKey::Conjugate, c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
  if (t.unsafeGetTensorImpl()->key_set().has_any(wrapped) || !t.has_storage()) return nullptr;
  return &t;
}

bool half(const at::Tensor& t) { return t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16; }
int dtype_code(const at::Tensor& t) { return t.scalar_type() == at::kBFloat16 ? OOB_BF16 : OOB_F16; }
bool fits(int64_t v) { return v >= INT_MIN && v <= INT_MAX; }
bool dense_rows(const at::Tensor& t) { return t.dim() == 2 && t.stride(1) == 1 && t.stride(0) == t.size(1); }

// The current device, if `o` is a tensor on a GPU at all.
bool device(PyObject* o, c10::DeviceIndex* dev) {
  if (!THPVariable_CheckExact(o) || !THPVariable_Unpack(o).is_cuda()) return false;
  *dev = c10::cuda::current_device();
  return true;
}
void* stream(c10::DeviceIndex dev) { return c10::cuda::getCurrentCUDAStream(dev).stream(); }
// An int that is one and fits, not a subclass (bool).
bool whole(PyObject* o, int* v) {
  if (!PyLong_CheckExact(o)) return false;
  int over = 0;
  const long long x = PyLong_AsLongLongAndOverflow(o, &over);
  if (over != 0 || !fits(x)) return false;
  *v = static_cast<int>(x);
  return true;
}

// What is promised about B (oob_gemm_args_t::b_static); anything else: nothing.
int promise(PyObject* o) {
  int v = 0;
  if (PyBool_Check(o)) return o == Py_True;
  return whole(o, &v) && v >= 0 && v <= 2 ? v : 0;
}

// The operands of a GEMM that the kernels take as they are; false: not for this path.
bool operands(const at::Tensor& a, const at::Tensor& b, int b_static, oob_gemm_args_t* g) {
  if (!half(a) || a.scalar_type() != b.scalar_type() || a.dim() != 2 || b.dim() != 2) return false;
  if (a.size(1) != b.size(1) || a.stride(1) != 1 || b.stride(1) != 1) return false;
  if (!fits(a.size(0)) || !fits(a.size(1)) || !fits(b.size(0)) || !fits(a.stride(0)) || !fits(b.stride(0))) return false;
  *g = oob_gemm_args_t{};
  g->mode = OOB_GEMM_PLAIN;
  g->dtype = dtype_code(a);
  g->M = static_cast<int>(a.size(0));
  g->N = static_cast<int>(b.size(0));
  g->K = static_cast<int>(a.size(1));
  g->A = a.data_ptr();
  g->lda = static_cast<int>(a.stride(0));
  g->B = b.data_ptr();
  g->ldb = static_cast<int>(b.stride(0));
  g->b_static = b_static;
  return true;
}

// rmsnorm(x, weight, eps, residual)
PyObject* py_rmsnorm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  c10::DeviceIndex dev;
  if (n != 4 || !PyFloat_CheckExact(args[2]) || modes_on() || !device(args[0], &dev)) return none();
  const at::Tensor *x = plain(args[0], dev), *w = plain(args[1], dev), *r = nullptr;
  if (args[3] != Py_None && (r = plain(args[3], dev)) == nullptr) return none();
  if (x == nullptr || w == nullptr || !half(*x) || !dense_rows(*x) || w->scalar_type() != x->scalar_type() || w->dim() != 1 ||
      w->size(0) != x->size(1) || w->stride(0) != 1 || !fits(x->size(0)) || !fits(x->size(1)))
    return none();
  if (r != nullptr && (r->scalar_type() != x->scalar_type() || !dense_rows(*r) || r->size(0) != x->size(0) || r->size(1) != x->size(1)))
    return none();
  const float eps = static_cast<float>(PyFloat_AS_DOUBLE(args[2]));
  at::Tensor y, res_out;
  int rc;
  {
    NoLock unlocked;
    y = at::empty({x->size(0), x->size(1)}, x->options());
    if (r != nullptr) res_out = at::empty({x->size(0), x->size(1)}, x->options());
    oob_norm_args_t a{};
    a.dtype = dtype_code(*x);
    a.rows = static_cast<int>(x->size(0));
    a.hidden = static_cast<int>(x->size(1));
    a.eps = eps;
    a.x_off = reinterpret_cast<uint64_t>(x->data_ptr());  // no communicator: the address
    a.residual = r != nullptr ? r->data_ptr() : nullptr;
    a.weight = w->data_ptr();
    a.y_local = y.data_ptr();
    a.res_out_reg = -1;
    a.res_out_local = r != nullptr ? res_out.data_ptr() : nullptr;
    rc = oob_fused_norm(nullptr, OOB_NORM_LOCAL, &a, 0, stream(dev));
  }
  if (rc != 0) return fail(rc);
  PyObject* py = THPVariable_Wrap(std::move(y));
  if (r == nullptr || py == nullptr) return py;
  PyObject* pr = THPVariable_Wrap(std::move(res_out));
  PyObject* both = pr != nullptr ? PyTuple_Pack(2, py, pr) : nullptr;
  Py_DECREF(py);
  Py_XDECREF(pr);
  return both;
  END_HANDLE_TH_ERRORS
}

// gemm(a, b, b_static)
PyObject* py_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  c10::DeviceIndex dev;
  if (n != 3 || modes_on() || !device(args[0], &dev)) return none();
  const at::Tensor *a = plain(args[0], dev), *b = plain(args[1], dev);
  oob_gemm_args_t g;
  if (a == nullptr || b == nullptr || !operands(*a, *b, promise(args[2]), &g)) return none();
  at::Tensor out;
  int rc;
  {
    NoLock unlocked;
    out = at::empty({g.M, g.N}, a->options());
    g.C = out.data_ptr();
    g.ldc = g.N;
    rc = oob_gemm(nullptr, &g, stream(dev));
  }
  return rc != 0 ? fail(rc) : THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// gemm_swiglu(a, b, b_static); None also where no kernel that has the sums may apply the activation.
PyObject* py_gemm_swiglu(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  c10::DeviceIndex dev;
  if (n != 3 || modes_on() || !device(args[0], &dev)) return none();
  const at::Tensor *a = plain(args[0], dev), *b = plain(args[1], dev);
  oob_gemm_args_t g;
  if (a == nullptr || b == nullptr || !operands(*a, *b, promise(args[2]), &g) || g.N % 16 != 0) return none();
  at::Tensor out;
  int rc;
  bool split;
  {
    NoLock unlocked;
    split = oob_gemm_plan_splits(g.M, g.N, g.K, 0, 0) > 1;
    out = at::empty({g.M, g.N / 2}, a->options());
    g.C = out.data_ptr();
    g.ldc = g.N / 2;
    oob_gemm_epilogue_swiglu_t epi{};
    epi.F = g.N / 2;
    g.epilogue = split ? OOB_EPILOGUE_SWIGLU : OOB_EPILOGUE_SWIGLU_TILE;
    g.epilogue_args = &epi;
    rc = oob_gemm(nullptr, &g, stream(dev));
  }
  if (rc == OOB_ERR_UNSUPPORTED && !split) return none();
  return rc != 0 ? fail(rc) : THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// gemm_rope_kv_write(x, wqkv, B, T, heads, kv_heads, k_cache, v_cache, cos, sin, pos, batch0, b_static)
PyObject* py_gemm_rope_kv_write(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  c10::DeviceIndex dev;
  if (n != 13 || modes_on() || !device(args[0], &dev)) return none();
  const at::Tensor *x = plain(args[0], dev), *w = plain(args[1], dev), *kc = plain(args[6], dev), *vc = plain(args[7], dev),
                   *cos = plain(args[8], dev), *sin = plain(args[9], dev), *pos = nullptr;
  oob_gemm_args_t g;
  if (x == nullptr || w == nullptr || kc == nullptr || vc == nullptr || cos == nullptr || sin == nullptr ||
      !operands(*x, *w, promise(args[12]), &g))
    return none();
  oob_rope_args_t r{};
  if (!whole(args[2], &r.B) || !whole(args[3], &r.T) || !whole(args[4], &r.H) || !whole(args[5], &r.KV) || !whole(args[11], &r.batch0) ||
      r.B <= 0 || r.T <= 0 || r.H <= 0 || r.KV <= 0 || r.batch0 < 0)
    return none();
  if (THPVariable_Check(args[10])) {
    pos = plain(args[10], dev);
    if (pos == nullptr || pos->scalar_type() != at::kLong || pos->numel() != 1) return none();
    r.pos_dev = static_cast<const int64_t*>(pos->data_ptr());
  } else if (!whole(args[10], &r.pos0)) {
    return none();
  }
  const int64_t heads = static_cast<int64_t>(r.H) + 2 * static_cast<int64_t>(r.KV);
  if (static_cast<int64_t>(r.B) * r.T != g.M || g.N % heads != 0 || g.N / heads % 8 != 0) return none();
  const int64_t hd = g.N / heads;
  if (kc->dim() != 4 || kc->scalar_type() != x->scalar_type() || vc->scalar_type() != x->scalar_type() || kc->sizes() != vc->sizes() ||
      kc->strides() != vc->strides() || kc->size(1) != r.KV || kc->size(3) != hd || kc->stride(3) != 1 || kc->stride(2) != hd ||
      kc->stride(1) != kc->size(2) * hd || static_cast<int64_t>(r.batch0) + r.B > kc->size(0) || !fits(kc->size(2)))
    return none();
  for (const at::Tensor* t : {cos, sin})
    if (t->scalar_type() != at::kFloat || t->dim() != 2 || t->size(0) != kc->size(2) || t->size(1) != hd / 2 || !t->is_contiguous()) return none();
  r.dtype = g.dtype;
  r.hd = static_cast<int>(hd);
  r.k_cache = kc->data_ptr();
  r.v_cache = vc->data_ptr();
  r.cache_batch_stride = kc->stride(0);
  r.max_len = static_cast<int>(kc->size(2));
  r.cos_table = static_cast<const float*>(cos->data_ptr());
  r.sin_table = static_cast<const float*>(sin->data_ptr());
  at::Tensor q, qkv;
  int rc;
  {
    NoLock unlocked;
    const bool split = oob_gemm_plan_splits(g.M, g.N, g.K, 0, 0) > 1;
    if (split) {
      q = at::empty({g.M, r.H * hd}, x->options());
      r.q_out = q.data_ptr();
      g.C = r.q_out;  // not written; a valid aligned pointer keeps the checks uniform
      g.ldc = g.N;
      g.epilogue = OOB_EPILOGUE_ROPE_KV;
      g.epilogue_args = &r;
      rc = oob_gemm(nullptr, &g, stream(dev));
    } else {
      qkv = at::empty({g.M, g.N}, x->options());
      g.C = qkv.data_ptr();
      g.ldc = g.N;
      rc = oob_gemm(nullptr, &g, stream(dev));
      if (rc == 0) {
        q = at::empty({g.M, r.H * hd}, x->options());
        r.q_out = q.data_ptr();
        r.qkv = qkv.data_ptr();
        rc = oob_rope_kv_write(&r, stream(dev));
      }
    }
  }
  return rc != 0 ? fail(rc) : THPVariable_Wrap(std::move(q));
  END_HANDLE_TH_ERRORS
}

// attn_decode(q, k_cache, v_cache, pos, batch0, splits, len_bound, cache_ready), the default scale
PyObject* py_attn_decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  c10::DeviceIndex dev;
  if (n != 8 || modes_on() || !device(args[0], &dev)) return none();
  const at::Tensor *q = plain(args[0], dev), *kc = plain(args[1], dev), *vc = plain(args[2], dev);
  if (q == nullptr || kc == nullptr || vc == nullptr || !half(*q) || kc->scalar_type() != q->scalar_type() ||
      vc->scalar_type() != q->scalar_type() || q->dim() != 3 || q->size(2) != 128 || !q->is_contiguous() || kc->dim() != 4 ||
      kc->sizes() != vc->sizes() || kc->strides() != vc->strides())
    return none();
  oob_attn_decode_args_t a{};
  if (!PyBool_Check(args[7]) || !whole(args[4], &a.batch0) || !whole(args[5], &a.splits) || !whole(args[6], &a.len_bound) || a.batch0 < 0 || a.splits < 0 ||
      a.len_bound < 0)
    return none();
  const int64_t B = q->size(0), H = q->size(1), KV = kc->size(1), max_len = kc->size(2);
  if (KV <= 0 || H % KV != 0 || H / KV > 16 || kc->size(3) != 128 || kc->stride(3) != 1 || kc->stride(2) != 128 || kc->stride(1) != max_len * 128 ||
      a.batch0 + B > kc->size(0) || !fits(B) || !fits(H) || !fits(max_len))
    return none();
  if (THPVariable_Check(args[3])) {
    const at::Tensor* pos = plain(args[3], dev);
    if (pos == nullptr || pos->scalar_type() != at::kLong || pos->numel() != 1) return none();
    a.pos_dev = static_cast<const int64_t*>(pos->data_ptr());
  } else {
    int p;
    if (!whole(args[3], &p) || p == INT_MAX) return none();
    a.len = p + 1;
  }
  a.dtype = dtype_code(*q);
  a.B = static_cast<int>(B);
  a.H = static_cast<int>(H);
  a.KV = static_cast<int>(KV);
  a.q = q->data_ptr();
  a.k_cache = kc->data_ptr();
  a.v_cache = vc->data_ptr();
  a.cache_batch_stride = kc->stride(0);
  a.max_len = static_cast<int>(max_len);
  a.scale = static_cast<float>(1.0 / std::sqrt(128.0));
  a.ahead = args[7] == Py_True;
  if (a.len_bound == 0) a.len_bound = a.max_len;
  at::Tensor out, ws;
  int rc;
  {
    NoLock unlocked;
    out = at::empty({B, H * 128}, q->options());
    a.out = out.data_ptr();
    if (a.splits == 0) a.splits = oob_attn_decode_auto_splits(a.B, a.KV, a.len_bound);
    if (a.splits > 1) {  // of this call alone, in stream order
      ws = at::empty({static_cast<int64_t>(oob_attn_decode_workspace_bytes(a.B, a.H, a.splits))}, q->options().dtype(at::kByte));
      a.workspace = static_cast<float*>(ws.data_ptr());
    }
    rc = oob_attn_decode(&a, stream(dev));
  }
  return rc != 0 ? fail(rc) : THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

}  // namespace

PyMODINIT_FUNC PyInit__fast_ops() {
  using Fast = PyObject* (*)(PyObject*, PyObject* const*, Py_ssize_t);
  auto method = [](const char* name, Fast f) {
    return PyMethodDef{name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr};
  };
  static PyMethodDef methods[] = {method("rmsnorm", py_rmsnorm), method("gemm", py_gemm), method("gemm_swiglu", py_gemm_swiglu),
                                  method("gemm_rope_kv_write", py_gemm_rope_kv_write), method("attn_decode", py_attn_decode),
                                  PyMethodDef{}};
  static PyModuleDef def = {PyModuleDef_HEAD_INIT, "_fast_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};
  PyObject* lib = PyImport_ImportModule("ooverlap_b200._lib");
  if (lib == nullptr) return nullptr;
  g_check = PyObject_GetAttrString(lib, "check");
  Py_DECREF(lib);
  return g_check != nullptr ? PyModule_Create(&def) : nullptr;
}
