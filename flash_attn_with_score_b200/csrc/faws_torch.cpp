// The operators' plain calls from Python: checks, output tensors, the problem struct and the C entry point in one native
// call.  A call is plain when every tensor is an ordinary strided CUDA tensor that TMA can address, on the current device,
// outside of torch's function and dispatch modes, and the shapes fit; for any other the function returns None and the caller goes
// through the Python path, which words the errors.  What a call computes is the same either way.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstring>

#include "faws.h"

namespace {

constexpr int kOpScoresOnly = 100;  // compute_attention_scores, which has no workspace and no operator id

bool plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  const c10::DispatchKeySet keys = t.key_set();
  static const c10::DispatchKeySet usual =
      c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) |
      c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA) | c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView);
  if ((keys.raw_repr() & ~usual.raw_repr()) != 0 || !keys.has(c10::DispatchKey::CUDA)) return false;
  if (t.dim() != 4 || (t.scalar_type() != at::kHalf && t.scalar_type() != at::kBFloat16)) return false;
  if (t.numel() == 0 || t.stride(3) != 1 || reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 != 0) return false;
  return t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0;
}

faws_tensor view(const at::Tensor& t) {
  return faws_tensor{const_cast<void*>(t.const_data_ptr()), t.stride(0), t.stride(1), t.stride(2)};
}

// call(op, q, k, v, causal, sm_scale, split, per_q_head) -> (out, extra), out, extra or None
PyObject* call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8) {
    PyErr_SetString(PyExc_TypeError, "call takes eight arguments");
    return nullptr;
  }
  const long op = PyLong_AsLong(a[0]);
  if (op == -1 && PyErr_Occurred()) return nullptr;
  if (!plain(a[1]) || !plain(a[2]) || !plain(a[3]) || at::impl::torch_function_mode_enabled() ||
      c10::impl::TorchDispatchModeTLS::any_modes_set())
    Py_RETURN_NONE;
  const at::Tensor &q = THPVariable_Unpack(a[1]), &k = THPVariable_Unpack(a[2]), &v = THPVariable_Unpack(a[3]);
  const int64_t B = q.size(0), H = q.size(1), M = q.size(2), D = q.size(3), Hk = k.size(1), N = k.size(2);
  if (k.size(3) != D || v.size(3) != D || (D != 16 && D != 32 && D != 64 && D != 128)) Py_RETURN_NONE;
  if (v.size(1) != Hk || H % Hk != 0 || k.size(0) != B || v.size(0) != B || v.size(2) != N) Py_RETURN_NONE;
  if (k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) Py_RETURN_NONE;
  if (B > INT32_MAX || H > INT32_MAX || M > INT32_MAX || N > INT32_MAX) Py_RETURN_NONE;
  const c10::Device dev = q.device();
  if (k.device() != dev || v.device() != dev || dev.index() != c10::cuda::current_device()) Py_RETURN_NONE;
  const int causal = PyObject_IsTrue(a[4]);
  if (causal < 0) return nullptr;
  double sm_scale = 1.0 / std::sqrt((double)D);
  if (a[5] != Py_None) {
    sm_scale = PyFloat_AsDouble(a[5]);
    if (sm_scale == -1.0 && PyErr_Occurred()) {  // what Python's float() takes, or refuses in words of its own
      PyErr_Clear();
      Py_RETURN_NONE;
    }
  }
  const long split = PyLong_AsLong(a[6]);
  if (split == -1 && PyErr_Occurred()) return nullptr;
  const int per_q_head = PyObject_IsTrue(a[7]);
  if (per_q_head < 0) return nullptr;

  faws_problem p{};
  p.B = (int32_t)B; p.Hq = (int32_t)H; p.Hk = (int32_t)Hk; p.M = (int32_t)M; p.N = (int32_t)N; p.D = (int32_t)D;
  p.dtype = q.scalar_type() == at::kHalf ? FAWS_FP16 : FAWS_BF16;
  p.causal = causal;
  p.sm_scale = (float)sm_scale;
  p.m_end = (int32_t)M;
  p.q = view(q); p.k = view(k); p.v = view(v);
  at::Tensor out;
  if (op != kOpScoresOnly) {
    out = at::empty_like(q);
    p.out = view(out);
  } else {
    p.out = p.q;
  }
  const auto f32 = q.options().dtype(at::kFloat).requires_grad(false);
  at::Tensor extra, ws;
  size_t ws_bytes = 0;
  auto scratch = [&](int32_t which, int32_t arg) {
    ws_bytes = faws_workspace_bytes(which, &p, arg);
    if (ws_bytes > 0) ws = at::empty({(int64_t)ws_bytes}, q.options().dtype(at::kByte).requires_grad(false));
  };
  auto ws_ptr = [&]() -> void* { return ws_bytes > 0 ? ws.data_ptr() : nullptr; };
  int32_t n_splits = 1;
  const char* name = "";
  switch (op) {
    case FAWS_OP_ATTENTION:
      n_splits = faws_split_kv_plan(&p);
      name = n_splits > 1 ? "faws_attention_split_kv" : "faws_attention";
      if (n_splits > 1) scratch(FAWS_OP_ATTENTION_SPLIT_KV, n_splits);
      break;
    case FAWS_OP_SCORES: name = "faws_attention_with_scores"; extra = at::empty({B, H, M, N}, f32); break;
    case kOpScoresOnly:
      name = "faws_compute_attention_scores";
      extra = at::empty({B, H, M, N}, q.options().requires_grad(false));
      break;
    case FAWS_OP_ROW_SUM: name = "faws_attention_with_row_sum"; extra = at::empty({B, H, M}, f32); break;
    default:
      extra = at::empty({B, per_q_head ? H : Hk, split > 0 ? split : N}, f32);
      scratch((int32_t)op, (int32_t)split);
  }
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  float* sums = extra.defined() && extra.scalar_type() == at::kFloat ? extra.data_ptr<float>() : nullptr;
  int st = FAWS_EINVAL;
  Py_BEGIN_ALLOW_THREADS
  switch (op) {
    case FAWS_OP_ATTENTION:
      st = n_splits > 1 ? faws_attention_split_kv(&p, n_splits, ws_ptr(), ws_bytes, stream) : faws_attention(&p, stream);
      break;
    case FAWS_OP_SCORES: st = faws_attention_with_scores(&p, sums, FAWS_SCORES_F32, 0xff800000u, stream); break;
    case kOpScoresOnly: st = faws_compute_attention_scores(&p, extra.data_ptr(), FAWS_SCORES_INPUT, stream); break;
    case FAWS_OP_ROW_SUM: st = faws_attention_with_row_sum(&p, sums, stream); break;
    case FAWS_OP_COL_SUM:
      name = "faws_attention_with_col_sum";
      st = faws_attention_with_col_sum(&p, sums, per_q_head, ws_ptr(), ws_bytes, stream);
      break;
    case FAWS_OP_COL_SUM_SEQUENTIAL:
      name = "faws_attention_with_col_sum_sequential";
      st = faws_attention_with_col_sum_sequential(&p, sums, per_q_head, ws_ptr(), ws_bytes, stream);
      break;
    case FAWS_OP_SOFTMAX_COL_SUM:
      name = "faws_attention_with_softmax_col_sum";
      st = faws_attention_with_softmax_col_sum(&p, sums, per_q_head, ws_ptr(), ws_bytes, stream);
      break;
    case FAWS_OP_CROSS_QK_SUM:
      name = "faws_attention_cross_token_qk_sum";
      st = faws_attention_cross_token_qk_sum(&p, (int32_t)split, sums, per_q_head, ws_ptr(), ws_bytes, stream);
      break;
    case FAWS_OP_CROSS_SOFTMAX_SUM:
      name = "faws_attention_cross_token_softmax_sum";
      st = faws_attention_cross_token_softmax_sum(&p, (int32_t)split, sums, per_q_head, ws_ptr(), ws_bytes, stream);
      break;
    case FAWS_OP_CROSS_SOFTMAX_SUM_BUFFERED:
      name = "faws_attention_cross_token_softmax_sum_buffered";
      st = faws_attention_cross_token_softmax_sum_buffered(&p, (int32_t)split, sums, per_q_head, ws_ptr(), ws_bytes, stream);
      break;
    default: break;
  }
  Py_END_ALLOW_THREADS
  if (st != FAWS_OK) {
    PyErr_Format(PyExc_RuntimeError, "%s: libfaws status %d: %s", name, st, faws_strerror(st));
    return nullptr;
  }
  if (!extra.defined()) return THPVariable_Wrap(std::move(out));
  if (!out.defined()) return THPVariable_Wrap(std::move(extra));
  PyObject* first = THPVariable_Wrap(std::move(out));
  if (first == nullptr) return nullptr;
  PyObject* second = THPVariable_Wrap(std::move(extra));
  if (second == nullptr) {
    Py_DECREF(first);
    return nullptr;
  }
  PyObject* both = PyTuple_New(2);
  if (both == nullptr) {
    Py_DECREF(first);
    Py_DECREF(second);
    return nullptr;
  }
  PyTuple_SET_ITEM(both, 0, first);
  PyTuple_SET_ITEM(both, 1, second);
  return both;
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call)), METH_FASTCALL,
     "call(op, q, k, v, causal, sm_scale, split, per_q_head): a plain call, or None where it is not one"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_plain", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// Tensors are read by the layout of the torch that this was compiled against, so no other one may load it, and no other
// Python.
PyMODINIT_FUNC PyInit__plain() {
#define FAWS_STR2(x) #x
#define FAWS_STR(x) FAWS_STR2(x)
  static const char python[] = FAWS_STR(PY_MAJOR_VERSION) "." FAWS_STR(PY_MINOR_VERSION) ".";
  if (std::strncmp(Py_GetVersion(), python, sizeof(python) - 1) != 0) {
    PyErr_Format(PyExc_ImportError, "_plain.so was built for Python %s, this is %s", python, Py_GetVersion());
    return nullptr;
  }
  PyObject* torch = PyImport_ImportModule("torch");
  if (torch == nullptr) return nullptr;
  PyObject* version = PyObject_GetAttrString(torch, "__version__");
  Py_DECREF(torch);
  if (version == nullptr) return nullptr;
  const bool same = PyUnicode_Check(version) && PyUnicode_CompareWithASCIIString(version, FAWS_TORCH_VERSION) == 0;
  if (!same) PyErr_Format(PyExc_ImportError, "_plain.so was built for torch " FAWS_TORCH_VERSION ", this is %S", version);
  Py_DECREF(version);
  return same ? PyModule_Create(&kModule) : nullptr;
}
