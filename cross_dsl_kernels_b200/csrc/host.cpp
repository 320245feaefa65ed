// The eager calls of ops.py and w4a16.py in native code: check the tensors, allocate the outputs, launch.
//
// A decode step called eagerly is bound by the host: the checks and the ctypes call of one op took 17 - 75 us of Python,
// several times the kernel.  Here they take 5 (a BF16 norm of 16 x 4096: 18.7 -> 5.9 us a call; an append of few tokens:
// 76 -> 5.3; two eager decode layers of 4 tokens, 14 calls: 492 -> 120).  Each function here takes the arguments of the
// Python op by position, repeats the op's conditions on the tensors' metadata, and launches through the same C ABI entry
// point on torch's current stream.  It takes the ordinary call only: where a condition fails, or an argument has another
// form than the ordinary one (a tensor subclass, an odd type), it returns None and the Python function decides -- and words
// the error -- as before.
// Outputs come from torch's allocator (at::empty), so streams, graph capture and dispatch modes see what they saw.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <cmath>
#include <limits>

#include "../../include/xdk_b200.h"

namespace {

PyObject* g_check = nullptr;  // _native.check(status, what): raises

// the tensor behind `o`, or nullptr: a plain torch.Tensor on the GPU
const at::Tensor* tensor_of(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided ? &t : nullptr;
}
bool sm100(const at::Tensor& t) {
  constexpr int kMax = 64;
  static std::atomic<signed char> known[kMax];  // 0 not asked, 1 yes, -1 no: a property of the device
  const int d = t.get_device();
  if (d < 0 || d >= kMax) return false;
  if (known[d] == 0) {
    int major = 0;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, d) != cudaSuccess) {
      (void)cudaGetLastError();
      return false;
    }
    known[d] = major == 10 ? 1 : -1;
  }
  return known[d] == 1;
}
bool int_of(PyObject* o, int64_t& v) {  // exactly an int
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0 && !(v == -1 && PyErr_Occurred());
}
bool flag_of(PyObject* o, bool& v) {  // exactly a bool
  if (!PyBool_Check(o)) return false;
  v = o == Py_True;
  return true;
}
int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return XDK_F32;
    case at::kBFloat16: return XDK_BF16;
    case at::kHalf: return XDK_F16;
    default: return -1;
  }
}
// "NHD" 0, "HND" 1, anything else -1
int layout_of(PyObject* o) {
  if (!PyUnicode_CheckExact(o)) return -1;
  if (PyUnicode_CompareWithASCIIString(o, "NHD") == 0) return 0;
  return PyUnicode_CompareWithASCIIString(o, "HND") == 0 ? 1 : -1;
}
bool overlaps(const at::Tensor& a, const at::Tensor& b) {  // of byte spans, as contracts.storage_overlaps
  auto span = [](const at::Tensor& t, uintptr_t& lo, uintptr_t& hi) {
    lo = reinterpret_cast<uintptr_t>(t.data_ptr());
    int64_t reach = 0;
    for (int64_t d = 0; d < t.dim(); ++d) reach += (t.size(d) - 1) * t.stride(d);
    hi = lo + static_cast<uintptr_t>((reach + 1) * static_cast<int64_t>(t.element_size()));
  };
  if (a.numel() == 0 || b.numel() == 0) return false;
  uintptr_t a0, a1, b0, b1;
  span(a, a0, a1);
  span(b, b0, b1);
  return a0 < b1 && b0 < a1;
}
void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// the output, or the exception that _native.check makes of the status
PyObject* finish(int status, const char* what, PyObject* result) {
  if (status == XDK_OK) return result;
  Py_XDECREF(result);
  PyObject* r = PyObject_CallFunction(g_check, "is", status, what);
  if (r) {
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, what);
  }
  return nullptr;
}
unsigned launch_flags(bool dependent) { return dependent ? XDK_DEPENDENT_LAUNCH : 0u; }

// The interpreter lock is given up while torch allocates and CUDA launches, as ctypes does for a foreign call.
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

#define NOT_MINE Py_RETURN_NONE
#define NEED(cond) \
  if (!(cond)) NOT_MINE

// (x, residual, weight, eps, return_residual, dependent_launch)
PyObject* rmsnorm(PyObject*, PyObject* const* arg, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  NEED(n == 6);
  const at::Tensor *x = tensor_of(arg[0]), *r = tensor_of(arg[1]), *w = tensor_of(arg[2]);
  bool ret, dep;
  NEED(x && r && w && PyFloat_CheckExact(arg[3]) && flag_of(arg[4], ret) && flag_of(arg[5], dep));
  const double eps = PyFloat_AS_DOUBLE(arg[3]);
  const int code = dtype_code(x->scalar_type());
  NEED(code >= 0 && std::isfinite(eps) && eps > 0.0 && sm100(*x));
  NEED(r->scalar_type() == x->scalar_type() && w->scalar_type() == x->scalar_type() && x->dim() == 2 && r->sizes() == x->sizes());
  NEED(w->dim() == 1 && w->size(0) == x->size(1) && x->numel() > 0 && r->device() == x->device() && w->device() == x->device());
  NEED(x->is_contiguous() && r->is_contiguous() && w->is_contiguous());
  at::Tensor y, out;
  int st;
  {
    Unlocked unlocked;
    c10::cuda::CUDAGuard guard(x->device());
    y = at::empty_like(*x), out = at::empty_like(*r);
    st = xdk_rmsnorm_v2(x->data_ptr(), r->data_ptr(), w->data_ptr(), y.data_ptr(), out.data_ptr(), x->size(0), x->size(1),
                                  static_cast<float>(eps), code, launch_flags(dep), stream_of(*x));
  }
  PyObject* second = ret ? THPVariable_Wrap(std::move(out)) : Py_NewRef(Py_None);
  return finish(st, "xdk_rmsnorm", Py_BuildValue("NN", THPVariable_Wrap(std::move(y)), second));
  END_HANDLE_TH_ERRORS
}

// (x, weight, bias or None, weight_layout, split_k, dependent_launch)
PyObject* linear(PyObject*, PyObject* const* arg, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  NEED(n == 6);
  const at::Tensor *x = tensor_of(arg[0]), *w = tensor_of(arg[1]), *b = arg[2] == Py_None ? nullptr : tensor_of(arg[2]);
  int64_t split;
  bool dep;
  NEED(x && w && (b || arg[2] == Py_None) && PyUnicode_CheckExact(arg[3]) && int_of(arg[4], split) && flag_of(arg[5], dep));
  const bool nk = PyUnicode_CompareWithASCIIString(arg[3], "NK") == 0;
  NEED(nk || PyUnicode_CompareWithASCIIString(arg[3], "KN") == 0);
  NEED(split == 0 || split == 1 || split == 2 || split == 4 || split == 8);
  NEED(x->dim() == 2 && w->dim() == 2 && x->scalar_type() == at::kFloat && w->scalar_type() == at::kFloat && w->device() == x->device());
  const int64_t m = x->size(0), k = x->size(1), cols = w->size(nk ? 0 : 1);
  NEED(m > 0 && k > 0 && cols > 0 && w->size(nk ? 1 : 0) == k && x->is_contiguous() && w->is_contiguous() && sm100(*x));
  NEED(!b || (b->device() == x->device() && b->scalar_type() == at::kFloat && b->dim() == 1 && b->size(0) == cols && b->is_contiguous()));
  at::Tensor y;
  int st;
  {
    Unlocked unlocked;
    c10::cuda::CUDAGuard guard(x->device());
    y = at::empty({m, cols}, x->options());
    st = xdk_gemv_f32_v2(x->const_data_ptr<float>(), w->const_data_ptr<float>(), b ? b->const_data_ptr<float>() : nullptr,
                                   y.mutable_data_ptr<float>(), m, k, cols, nk, static_cast<int>(split), nullptr, 0,
                                   launch_flags(dep), stream_of(*x));
  }
  return finish(st, "xdk_gemv_f32", THPVariable_Wrap(std::move(y)));
  END_HANDLE_TH_ERRORS
}

// (x, packed, scales, bias or None, group_size, out or None, dependent_launch)
PyObject* w4a16(PyObject*, PyObject* const* arg, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  NEED(n == 7);
  const at::Tensor *x = tensor_of(arg[0]), *p = tensor_of(arg[1]), *s = tensor_of(arg[2]);
  const at::Tensor *b = arg[3] == Py_None ? nullptr : tensor_of(arg[3]), *o = arg[5] == Py_None ? nullptr : tensor_of(arg[5]);
  int64_t group;
  bool dep;
  NEED(x && p && s && (b || arg[3] == Py_None) && (o || arg[5] == Py_None) && int_of(arg[4], group) && flag_of(arg[6], dep));
  NEED(group == 32 || group == 64 || group == 128 || group == 256);
  NEED(x->dim() == 2 && x->scalar_type() == at::kHalf && p->dim() == 2 && p->scalar_type() == at::kByte);
  const int64_t m = x->size(0), k = x->size(1), cols = p->size(0);
  NEED(m >= 1 && m <= 16 && k >= 1 && cols >= 1 && p->size(1) == (k + 1) / 2);
  NEED(s->dim() == 2 && s->scalar_type() == at::kHalf && s->size(0) == cols && s->size(1) == (k + group - 1) / group);
  NEED(!b || (b->dim() == 1 && b->scalar_type() == at::kHalf && b->size(0) == cols));
  NEED(!o || (o->dim() == 2 && o->scalar_type() == at::kHalf && o->size(0) == m && o->size(1) == cols));
  const at::Tensor* all[5] = {x, p, s, b, o};
  for (const at::Tensor* t : all)
    NEED(!t || (t->device() == x->device() && t->is_contiguous() && !t->requires_grad() &&
                t->numel() <= std::numeric_limits<int32_t>::max()));
  NEED(k <= std::numeric_limits<int32_t>::max() && sm100(*x));
  if (o)
    for (int i = 0; i < 4; ++i) NEED(!all[i] || !overlaps(*o, *all[i]));
  at::Tensor y;
  int st;
  {
    Unlocked unlocked;
    c10::cuda::CUDAGuard guard(x->device());
    y = o ? *o : at::empty({m, cols}, x->options());
    st = xdk_w4a16_v2(x->data_ptr(), static_cast<const uint8_t*>(p->data_ptr()), s->data_ptr(), b ? b->data_ptr() : nullptr,
                                y.data_ptr(), m, k, cols, static_cast<int>(group), launch_flags(dep), stream_of(*x));
  }
  return finish(st, "xdk_w4a16", o ? Py_NewRef(arg[5]) : THPVariable_Wrap(std::move(y)));
  END_HANDLE_TH_ERRORS
}

// (q, k, v, cos, sin, positions, page_table, sequence_ids, k_cache, v_cache, page_size, rope_dim, interleaved, kv_layout,
//  dependent_launch)
PyObject* append(PyObject*, PyObject* const* arg, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  NEED(n == 15);
  const at::Tensor* t[10];
  for (int i = 0; i < 10; ++i) NEED((t[i] = tensor_of(arg[i])) != nullptr);
  const at::Tensor &q = *t[0], &k = *t[1], &v = *t[2], &cos = *t[3], &sin = *t[4], &pos = *t[5], &table = *t[6], &seq = *t[7],
                   &kc = *t[8], &vc = *t[9];
  int64_t page, rope;
  bool interleaved, dep;
  NEED(int_of(arg[10], page) && int_of(arg[11], rope) && flag_of(arg[12], interleaved) && flag_of(arg[14], dep));
  const int hnd = layout_of(arg[13]), code = dtype_code(q.scalar_type());
  NEED(hnd >= 0 && code >= 0 && page > 0 && rope > 0 && rope % 2 == 0 && sm100(q));
  for (int i = 1; i < 10; ++i) {
    const at::ScalarType want = i <= 2 || i >= 8 ? q.scalar_type() : (i <= 4 ? at::kFloat : at::kLong);
    NEED(t[i]->device() == q.device() && t[i]->scalar_type() == want && (i <= 2 || t[i]->is_contiguous()));
  }
  for (int i = 0; i < 3; ++i) {
    NEED(t[i]->dim() == 3);
    NEED(t[i]->is_contiguous() || (t[i]->stride(2) == 1 && t[i]->stride(1) == t[i]->size(2) && t[i]->stride(0) >= t[i]->size(1) * t[i]->size(2)));
  }
  NEED(cos.dim() == 2 && sin.dim() == 2 && pos.dim() == 1 && seq.dim() == 1 && table.dim() == 2 && kc.dim() == 4 && vc.dim() == 4);
  const int64_t tokens = q.size(0), hq = q.size(1), dim = q.size(2), hkv = k.size(1);
  NEED(tokens > 0 && hq > 0 && hkv > 0 && dim > 0 && hq % hkv == 0 && rope <= dim);
  NEED(k.size(0) == tokens && v.size(0) == tokens && k.size(2) == dim && v.size(2) == dim && v.size(1) == hkv);
  NEED(pos.size(0) == tokens && seq.size(0) == tokens && cos.size(1) >= rope / 2 && sin.sizes() == cos.sizes() && table.size(1) > 0);
  NEED(kc.sizes() == vc.sizes() && kc.size(hnd ? 2 : 1) == page && kc.size(hnd ? 1 : 2) == hkv && kc.size(3) == dim);
  NEED(!overlaps(kc, vc));
  for (int i = 0; i < 8; ++i) NEED(!overlaps(kc, *t[i]) && !overlaps(vc, *t[i]));
  at::Tensor out;
  int st;
  {
    Unlocked unlocked;
    c10::cuda::CUDAGuard guard(q.device());
    out = at::empty(q.sizes(), q.options());
    xdk_peer_out dst = {};
    dst.ptr[0] = out.data_ptr(), dst.world = 1, dst.ld = hq * dim, dst.col0 = 0;
    st = xdk_rope_kv_append_peer(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), cos.const_data_ptr<float>(), sin.const_data_ptr<float>(), pos.const_data_ptr<int64_t>(),
        table.const_data_ptr<int64_t>(), seq.const_data_ptr<int64_t>(), &dst, kc.data_ptr(), vc.data_ptr(), tokens, hq, hkv, dim,
        cos.size(1), table.size(1), page, rope, tokens > 1 ? q.stride(0) : hq * dim, tokens > 1 ? k.stride(0) : hkv * dim,
        tokens > 1 ? v.stride(0) : hkv * dim, interleaved, hnd, code, launch_flags(dep), stream_of(q));
  }
  return finish(st, "xdk_rope_kv_append", THPVariable_Wrap(std::move(out)));
  END_HANDLE_TH_ERRORS
}

// (q, k_cache, v_cache, positions, page_table, sequence_ids, page_size, kv_layout, scale or None, context_hint,
//  dependent_launch)
PyObject* attention(PyObject*, PyObject* const* arg, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  NEED(n == 11);
  const at::Tensor* t[6];
  for (int i = 0; i < 6; ++i) NEED((t[i] = tensor_of(arg[i])) != nullptr);
  const at::Tensor &q = *t[0], &kc = *t[1], &vc = *t[2], &pos = *t[3], &table = *t[4], &seq = *t[5];
  int64_t page, hint;
  bool dep;
  NEED(int_of(arg[6], page) && (arg[8] == Py_None || PyFloat_CheckExact(arg[8])) && int_of(arg[9], hint) && flag_of(arg[10], dep));
  const int hnd = layout_of(arg[7]), code = dtype_code(q.scalar_type());
  NEED(hnd >= 0 && code >= 0 && page > 0 && sm100(q));
  for (int i = 0; i < 6; ++i)
    NEED(t[i]->device() == q.device() && t[i]->is_contiguous() && t[i]->scalar_type() == (i <= 2 ? q.scalar_type() : at::kLong));
  NEED(q.dim() == 3 && kc.dim() == 4 && kc.sizes() == vc.sizes() && pos.dim() == 1 && seq.dim() == 1 && table.dim() == 2);
  const int64_t tokens = q.size(0), hq = q.size(1), dim = q.size(2), hkv = kc.size(hnd ? 1 : 2);
  NEED(tokens > 0 && hq > 0 && hkv > 0 && kc.size(hnd ? 2 : 1) == page && kc.size(3) == dim && hq % hkv == 0);
  const int64_t g = hq / hkv;
  NEED((g == 1 || g == 2 || g == 4 || g == 8) && (dim == 64 || dim == 128 || dim == 256));
  NEED(pos.size(0) == tokens && seq.size(0) == tokens);
  const double scale = arg[8] == Py_None ? std::pow(static_cast<double>(dim), -0.5) : PyFloat_AS_DOUBLE(arg[8]);
  NEED(std::isfinite(scale));
  if (hint <= 0 && __builtin_mul_overflow(table.size(1), page, &hint)) hint = 0;  // no bound: that of a page table row
  at::Tensor out;
  int st;
  {
    Unlocked unlocked;
    c10::cuda::CUDAGuard guard(q.device());
    out = at::empty_like(q);
    const size_t need = xdk_paged_decode_attention_scratch_bytes(tokens, hq, hkv, dim, hint, code);
    at::Tensor scratch;
    if (need) scratch = at::empty({static_cast<int64_t>(need)}, q.options().dtype(at::kByte));
    xdk_peer_out dst = {};
    dst.ptr[0] = out.data_ptr(), dst.world = 1, dst.ld = hq * dim, dst.col0 = 0;
    st = xdk_paged_decode_attention_ws(
        q.data_ptr(), kc.data_ptr(), vc.data_ptr(), pos.const_data_ptr<int64_t>(), table.const_data_ptr<int64_t>(),
        seq.const_data_ptr<int64_t>(), &dst, tokens, hq, hkv, dim, table.size(1), page, hnd, static_cast<float>(scale), hint, code,
        need ? scratch.data_ptr() : nullptr, need, launch_flags(dep), stream_of(q));
  }
  return finish(st, "xdk_paged_decode_attention", THPVariable_Wrap(std::move(out)));
  END_HANDLE_TH_ERRORS
}

// (upgate, dependent_launch)
PyObject* swiglu(PyObject*, PyObject* const* arg, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  NEED(n == 2);
  const at::Tensor* u = tensor_of(arg[0]);
  bool dep;
  NEED(u && flag_of(arg[1], dep));
  const int code = dtype_code(u->scalar_type());
  NEED(code >= 0 && u->dim() == 2 && u->size(1) % 2 == 0 && u->size(0) > 0 && u->size(1) > 0 && u->stride(1) == 1 &&
       u->stride(0) >= u->size(1) && sm100(*u));
  const int64_t rows = u->size(0), width = u->size(1) / 2;
  at::Tensor out;
  int st;
  {
    Unlocked unlocked;
    c10::cuda::CUDAGuard guard(u->device());
    out = at::empty({rows, width}, u->options());
    st = xdk_swiglu(u->data_ptr(), out.data_ptr(), rows, width, rows > 1 ? u->stride(0) : 2 * width, width, code,
                              launch_flags(dep), stream_of(*u));
  }
  return finish(st, "xdk_swiglu", THPVariable_Wrap(std::move(out)));
  END_HANDLE_TH_ERRORS
}

PyObject* set_check(PyObject*, PyObject* fn) {
  Py_XSETREF(g_check, Py_NewRef(fn));
  Py_RETURN_NONE;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FAST(rmsnorm), FAST(linear), FAST(w4a16), FAST(append), FAST(attention), FAST(swiglu),
                           {"set_check", set_check, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&g_module); }
