// CPython binding of the hot entry points: tensors in, tensor out, one call per linear.
//
// What it replaces and why.  A decode step of a small model is bound by the host: with the checks,
// the output allocation, the workspace look-up and the ctypes conversion of a dozen arguments in
// Python, one W8A8 linear cost 30 us of host time for two kernels of 2-3 us each.  Here the same
// steps are native, the arguments travel as borrowed references (METH_FASTCALL, no argument
// tuple), outputs are allocated without a trip through the dispatcher, and the codes and scales of
// a dynamically quantised linear share one allocation.
//
// Contract with quantization/cuda.py: a function returns None when it does not take its arguments
// as they are (not contiguous, a wrong type, shapes that do not fit, tensors not on one GPU);
// the Python function then names the error or makes the tensors contiguous and calls again.
// A failing library call raises through the handler that _lib.py installs (set_error_handler).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <climits>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/b200q.h"

namespace {

PyObject* g_on_error = nullptr;  // _lib.check(code, where, detail)

// ------------------------------------------------------------------- argument helpers
inline const at::Tensor* tensor_of(PyObject* o) {
  return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr;
}
// a CUDA tensor on `device` of the given type, dense
inline bool dense(const at::Tensor* t, at::ScalarType type, const at::Device& device) {
  return t != nullptr && t->scalar_type() == type && t->device() == device && t->is_contiguous();
}
inline int dtype_id(at::ScalarType t) {
  return t == at::kHalf ? B200Q_DTYPE_F16 : t == at::kBFloat16 ? B200Q_DTYPE_BF16 : -1;
}
inline at::Tensor empty_on(at::IntArrayRef shape, at::ScalarType type, const at::Device& device) {
  return at::detail::empty_cuda(shape, type, device, std::nullopt);
}
inline void* stream_of(const at::Device& device) {
  return c10::cuda::getCurrentCUDAStream(device.index()).stream();
}
// weights [N, K], scales [N], optional bias [N] of type `type`
struct Weights {
  const at::Tensor *w, *s, *b;
  int64_t N, K;
};
inline bool weights_of(PyObject* w, PyObject* s, PyObject* b, at::ScalarType type,
                       const at::Device& device, Weights* out) {
  out->w = tensor_of(w);
  out->s = tensor_of(s);
  out->b = b == Py_None ? nullptr : tensor_of(b);
  if (!dense(out->w, at::kChar, device) || out->w->dim() != 2) return false;
  out->N = out->w->size(0);
  out->K = out->w->size(1);
  if (out->N == 0 || out->K == 0) return false;
  if (!dense(out->s, at::kFloat, device) || out->s->dim() != 1 || out->s->size(0) != out->N) return false;
  if (b != Py_None && (!dense(out->b, type, device) || out->b->dim() != 1 || out->b->size(0) != out->N))
    return false;
  return true;
}
inline void* ptr(const at::Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }
inline bool fits_int(int64_t v) { return v >= 0 && v <= INT_MAX; }

// x [..., K] -> the output shape [..., N]
inline c10::SmallVector<int64_t, 5> out_shape(const at::Tensor& x, int64_t N) {
  c10::SmallVector<int64_t, 5> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = N;
  return shape;
}

PyObject* fail(int rc, const char* where, int64_t M, int64_t N, int64_t K) {
  const std::string detail =
      "M=" + std::to_string(M) + " N=" + std::to_string(N) + " K=" + std::to_string(K);
  if (g_on_error != nullptr) {
    PyObject* r = PyObject_CallFunction(g_on_error, "iss", rc, where, detail.c_str());
    if (r == nullptr) return nullptr;
    Py_DECREF(r);
  }
  PyErr_Format(PyExc_RuntimeError, "%s: error %d [%s]", where, rc, detail.c_str());
  return nullptr;
}

// ------------------------------------------------------------------------- workspace
// One zero-filled scratch buffer per device, shared by every call there (calls of one model runner
// are stream-ordered; the split-K kernels leave their counters at zero).  It is allocated once,
// large enough for a decode step, so that nothing is allocated while a graph is captured.
constexpr int kMaxDevices = 64;
std::mutex g_ws_mutex;
at::Tensor* const g_ws = new at::Tensor[kMaxDevices];  // never destroyed: CUDA may be gone at exit
// Outgrown buffers: a captured graph may go on writing to the one that it was captured with.  A buffer grows
// by half at least, so what is kept here is at most twice the current one.
std::vector<at::Tensor>* const g_ws_outgrown = new std::vector<at::Tensor>;
int64_t g_ws_floor = 64ll << 20;

// The buffer as it is; undefined before the first call that needed one.
at::Tensor current_workspace(const at::Device& device) {
  std::lock_guard<std::mutex> lock(g_ws_mutex);
  return g_ws[device.index()];
}

// A reference to the buffer of at least `bytes` bytes; throws std::runtime_error during capture.
at::Tensor workspace(const at::Device& device, int64_t bytes) {
  std::lock_guard<std::mutex> lock(g_ws_mutex);
  at::Tensor& ws = g_ws[device.index()];
  if (!ws.defined() || ws.numel() < bytes) {
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None)
      throw std::runtime_error(
          "b200q workspace of " + std::to_string(bytes) +
          " bytes requested during CUDA graph capture; run the shape once eagerly first or call "
          "reserve_workspace() before capture");
    // a buffer of this process must be an ordinary tensor whatever mode the first caller is in
    c10::InferenceMode normal(false);
    const int64_t least = ws.defined() ? ws.numel() / 2 * 3 : 0;
    at::Tensor larger =
        at::zeros({std::max({bytes, g_ws_floor, least})}, at::TensorOptions().dtype(at::kByte).device(device));
    if (ws.defined()) g_ws_outgrown->push_back(ws);
    ws = std::move(larger);
  }
  return ws;
}

#define B200Q_NEEDS(n)                                                        \
  if (nargs != (n)) {                                                         \
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments");            \
    return nullptr;                                                           \
  }

// Runs one library call with the interpreter lock released (a launch can block on a full queue).
template <typename F>
inline int unlocked(F&& call) {
  PyThreadState* state = PyEval_SaveThread();
  const int rc = call();
  PyEval_RestoreThread(state);
  return rc;
}

// call(workspace, bytes) -> return code.  Most calls need no workspace: it is allocated only for one that asks for
// it (and then has launched nothing), so that a capture is refused only for such a call.
template <typename F>
inline int with_workspace(const at::Device& device, int op, int m, int n, int k, F&& call) {
  at::Tensor ws = current_workspace(device);
  auto once = [&] {
    return unlocked([&] { return call(ws.defined() ? ws.data_ptr() : nullptr, ws.defined() ? ws.numel() : 0); });
  };
  int rc = once();
  if (rc == B200Q_ERR_WORKSPACE) {
    ws = workspace(device, static_cast<int64_t>(b200q_workspace_bytes(op, m, n, k)));
    rc = once();
  }
  return rc;
}

// ------------------------------------------------------------------------- functions
// w8a16(x, qweight, scales, bias | None) -> y
PyObject* w8a16(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  B200Q_NEEDS(4)
  const at::Tensor* x = tensor_of(args[0]);
  if (x == nullptr || !x->is_cuda() || !x->is_contiguous() || x->dim() == 0) Py_RETURN_NONE;
  const int dt = dtype_id(x->scalar_type());
  const at::Device device = x->device();
  Weights p;
  if (dt < 0 || !weights_of(args[1], args[2], args[3], x->scalar_type(), device, &p)) Py_RETURN_NONE;
  if (x->size(-1) != p.K || x->numel() == 0) Py_RETURN_NONE;
  const int64_t M = x->numel() / p.K;
  if (!fits_int(M) || !fits_int(p.N) || !fits_int(p.K)) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(device);
  const int m = static_cast<int>(M), n = static_cast<int>(p.N), k = static_cast<int>(p.K);
  at::Tensor y = empty_on(out_shape(*x, p.N), x->scalar_type(), device);
  const int rc = with_workspace(device, B200Q_OP_W8A16, m, n, k, [&](void* ws, size_t bytes) {
    return b200q_w8a16_gemm(x->data_ptr(), static_cast<const int8_t*>(ptr(p.w)),
                            static_cast<const float*>(ptr(p.s)), ptr(p.b), y.data_ptr(), m, n, k, dt, ws, bytes,
                            stream_of(device));
  });
  if (rc != B200Q_OK) return fail(rc, "b200q_w8a16_gemm", M, p.N, p.K);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// w8a8_dynamic(x, qweight, w_scales, bias | None) -> y: per-token quantisation and the GEMM
PyObject* w8a8_dynamic(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  B200Q_NEEDS(4)
  const at::Tensor* x = tensor_of(args[0]);
  if (x == nullptr || !x->is_cuda() || !x->is_contiguous() || x->dim() == 0) Py_RETURN_NONE;
  const int dt = dtype_id(x->scalar_type());
  const at::Device device = x->device();
  Weights p;
  if (dt < 0 || !weights_of(args[1], args[2], args[3], x->scalar_type(), device, &p)) Py_RETURN_NONE;
  if (x->size(-1) != p.K || x->numel() == 0) Py_RETURN_NONE;
  if (reinterpret_cast<uintptr_t>(x->data_ptr()) % 16 != 0 || p.K % 8 != 0) Py_RETURN_NONE;
  const int64_t M = x->numel() / p.K;
  if (!fits_int(M) || !fits_int(p.N) || !fits_int(p.K)) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(device);
  const int m = static_cast<int>(M);
  at::Tensor y = empty_on(out_shape(*x, p.N), x->scalar_type(), device);
  const int n = static_cast<int>(p.N), k = static_cast<int>(p.K);
  at::Tensor quant;
  const size_t scratch = b200q_w8a8_dynamic_scratch_bytes(m, n, k);
  if (scratch > 0) quant = empty_on({static_cast<int64_t>(scratch)}, at::kByte, device);
  const int rc = with_workspace(device, B200Q_OP_W8A8, m, n, k, [&](void* ws, size_t bytes) {
    return b200q_w8a8_dynamic_gemm(
        x->data_ptr(), static_cast<const int8_t*>(ptr(p.w)), static_cast<const float*>(ptr(p.s)),
        ptr(p.b), y.data_ptr(), m, n, k, dt, scratch > 0 ? quant.data_ptr() : nullptr, scratch, ws, bytes,
        stream_of(device));
  });
  if (rc != B200Q_OK) return fail(rc, "b200q_w8a8_dynamic_gemm", M, p.N, p.K);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

int run_w8a8(const at::Device& device, const int8_t* xq, const float* a_s, const Weights& p, void* y,
             int m, int out_dt) {
  const int n = static_cast<int>(p.N), k = static_cast<int>(p.K);
  return with_workspace(device, B200Q_OP_W8A8, m, n, k, [&](void* ws, size_t bytes) {
    return b200q_w8a8_gemm(xq, a_s, static_cast<const int8_t*>(ptr(p.w)), static_cast<const float*>(ptr(p.s)),
                           ptr(p.b), y, m, n, k, out_dt, ws, bytes, stream_of(device));
  });
}

// w8a8(x_q, a_scales, qweight, w_scales, bias | None, dtype id, shape | None, out | None) -> y
PyObject* w8a8(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  B200Q_NEEDS(8)
  const at::Tensor* xq = tensor_of(args[0]);
  const at::Tensor* a_s = tensor_of(args[1]);
  if (xq == nullptr || !xq->is_cuda() || xq->dim() != 2 || !dense(xq, at::kChar, xq->device()))
    Py_RETURN_NONE;
  const at::Device device = xq->device();
  const long dt = PyLong_AsLong(args[5]);
  if (dt != B200Q_DTYPE_F16 && dt != B200Q_DTYPE_BF16) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const at::ScalarType type = dt == B200Q_DTYPE_F16 ? at::kHalf : at::kBFloat16;
  const int64_t M = xq->size(0);
  Weights p;
  if (!dense(a_s, at::kFloat, device) || a_s->dim() != 1 || a_s->size(0) != M || M == 0 ||
      !weights_of(args[2], args[3], args[4], type, device, &p) || xq->size(1) != p.K || !fits_int(M) ||
      !fits_int(p.N) || !fits_int(p.K))
    Py_RETURN_NONE;
  c10::SmallVector<int64_t, 5> shape = {M, p.N};
  if (args[6] != Py_None) {
    PyObject* want = args[6];  // a tuple (torch.Size is one) of M * N elements
    if (!PyTuple_Check(want)) Py_RETURN_NONE;
    shape.clear();
    int64_t count = 1;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(want); ++i) {
      const long long d = PyLong_AsLongLong(PyTuple_GET_ITEM(want, i));
      if (d <= 0) {  // also -1 ("infer") and a conversion error: the general route
        PyErr_Clear();
        Py_RETURN_NONE;
      }
      shape.push_back(d);
      count *= d;
    }
    if (count != M * p.N) Py_RETURN_NONE;
  }
  c10::cuda::CUDAGuard guard(device);
  at::Tensor y;
  if (args[7] == Py_None) {
    y = empty_on(shape, type, device);
  } else {
    const at::Tensor* out = tensor_of(args[7]);
    if (!dense(out, type, device) || out->dim() != 2 || out->size(0) != M || out->size(1) != p.N ||
        args[6] != Py_None)
      Py_RETURN_NONE;
    y = *out;
  }
  const int rc = run_w8a8(device, static_cast<const int8_t*>(xq->data_ptr()),
                          static_cast<const float*>(a_s->data_ptr()), p, y.data_ptr(),
                          static_cast<int>(M), static_cast<int>(dt));
  if (rc != B200Q_OK) return fail(rc, "b200q_w8a8_gemm", M, p.N, p.K);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// w8a8_i32(x_q, qweight) -> int32 accumulators
PyObject* w8a8_i32(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  B200Q_NEEDS(2)
  const at::Tensor *xq = tensor_of(args[0]), *w = tensor_of(args[1]);
  if (xq == nullptr || !xq->is_cuda() || !dense(xq, at::kChar, xq->device()) || xq->dim() != 2 ||
      !dense(w, at::kChar, xq->device()) || w->dim() != 2 || w->size(1) != xq->size(1) ||
      !fits_int(xq->size(0)) || !fits_int(xq->size(1)) || !fits_int(w->size(0)))
    Py_RETURN_NONE;
  const at::Device device = xq->device();
  c10::cuda::CUDAGuard guard(device);
  const int m = static_cast<int>(xq->size(0)), n = static_cast<int>(w->size(0)),
            k = static_cast<int>(w->size(1));
  at::Tensor acc = empty_on({m, n}, at::kInt, device);
  const int rc = with_workspace(device, B200Q_OP_W8A8, m, n, k, [&](void* ws, size_t bytes) {
    return b200q_w8a8_gemm_i32(static_cast<const int8_t*>(xq->data_ptr()),
                               static_cast<const int8_t*>(w->data_ptr()),
                               static_cast<int32_t*>(acc.data_ptr()), m, n, k, ws, bytes, stream_of(device));
  });
  if (rc != B200Q_OK) return fail(rc, "b200q_w8a8_gemm_i32", m, n, k);
  return THPVariable_Wrap(std::move(acc));
  END_HANDLE_TH_ERRORS
}

// quantize(x [M, K]) -> (x_q, a_scales)
PyObject* quantize(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  B200Q_NEEDS(1)
  const at::Tensor* x = tensor_of(args[0]);
  if (x == nullptr || !x->is_cuda() || x->dim() != 2 || x->numel() == 0) Py_RETURN_NONE;
  const int dt = dtype_id(x->scalar_type());
  const int64_t M = x->size(0), K = x->size(1);
  // rows may be further apart than K, on 16-byte boundaries
  if (dt < 0 || x->stride(1) != 1 || x->stride(0) < K || x->stride(0) % 8 != 0 ||
      reinterpret_cast<uintptr_t>(x->data_ptr()) % 16 != 0 || !fits_int(M) || !fits_int(K))
    Py_RETURN_NONE;
  const at::Device device = x->device();
  c10::cuda::CUDAGuard guard(device);
  at::Tensor xq = empty_on({M, K}, at::kChar, device);
  at::Tensor a_s = empty_on({M}, at::kFloat, device);
  const int rc = unlocked([&] {
    return b200q_act_quant_i8(x->data_ptr(), x->stride(0), dt, static_cast<int8_t*>(xq.data_ptr()),
                              static_cast<float*>(a_s.data_ptr()), static_cast<int>(M),
                              static_cast<int>(K), stream_of(device));
  });
  if (rc != B200Q_OK) return fail(rc, "b200q_act_quant_i8", M, 0, K);
  return Py_BuildValue("NN", THPVariable_Wrap(std::move(xq)), THPVariable_Wrap(std::move(a_s)));
  END_HANDLE_TH_ERRORS
}

PyObject* or_none(at::Tensor&& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(t));
}

// rmsnorm_quant(x, weight, eps, residual | None, return_normed)
//   -> (x_q, a_scales, new_residual | None, normed | None)
PyObject* rmsnorm_quant(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  B200Q_NEEDS(5)
  const at::Tensor *x = tensor_of(args[0]), *w = tensor_of(args[1]);
  if (x == nullptr || !x->is_cuda() || !x->is_contiguous() || x->dim() == 0 || x->numel() == 0)
    Py_RETURN_NONE;
  const at::ScalarType type = x->scalar_type();
  const int dt = dtype_id(type);
  const at::Device device = x->device();
  const int64_t K = x->size(-1), M = x->numel() / K;
  if (dt < 0 || !dense(w, type, device) || w->dim() != 1 || w->numel() != K || !fits_int(M) ||
      !fits_int(K))
    Py_RETURN_NONE;
  const at::Tensor* res = args[3] == Py_None ? nullptr : tensor_of(args[3]);
  if (args[3] != Py_None && (!dense(res, type, device) || res->sizes() != x->sizes())) Py_RETURN_NONE;
  const double eps = PyFloat_AsDouble(args[2]);
  if (eps == -1.0 && PyErr_Occurred()) return nullptr;
  const int normed_wanted = PyObject_IsTrue(args[4]);
  if (normed_wanted < 0) return nullptr;
  c10::cuda::CUDAGuard guard(device);
  at::Tensor xq = empty_on({M, K}, at::kChar, device);
  at::Tensor a_s = empty_on({M}, at::kFloat, device);
  at::Tensor new_res, normed;
  if (res != nullptr) new_res = empty_on(x->sizes(), type, device);
  if (normed_wanted) normed = empty_on(x->sizes(), type, device);
  const int rc = unlocked([&] {
    return b200q_add_rmsnorm_quant_i8(
        x->data_ptr(), ptr(res), w->data_ptr(), static_cast<float>(eps),
        res != nullptr ? new_res.data_ptr() : nullptr, normed_wanted ? normed.data_ptr() : nullptr,
        static_cast<int8_t*>(xq.data_ptr()), static_cast<float*>(a_s.data_ptr()), static_cast<int>(M),
        static_cast<int>(K), dt, stream_of(device));
  });
  if (rc != B200Q_OK) return fail(rc, "b200q_add_rmsnorm_quant_i8", M, 0, K);
  return Py_BuildValue("NNNN", THPVariable_Wrap(std::move(xq)), THPVariable_Wrap(std::move(a_s)),
                       or_none(std::move(new_res)), or_none(std::move(normed)));
  END_HANDLE_TH_ERRORS
}

// silu_mul_quant(gate_up [..., 2 I], return_act) -> (x_q, a_scales, act | None)
PyObject* silu_mul_quant(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  B200Q_NEEDS(2)
  const at::Tensor* x = tensor_of(args[0]);
  if (x == nullptr || !x->is_cuda() || !x->is_contiguous() || x->dim() == 0 || x->numel() == 0)
    Py_RETURN_NONE;
  const at::ScalarType type = x->scalar_type();
  const int dt = dtype_id(type);
  const at::Device device = x->device();
  const int64_t two_i = x->size(-1), I = two_i / 2, M = x->numel() / two_i;
  if (dt < 0 || two_i % 2 != 0 || !fits_int(M) || !fits_int(two_i)) Py_RETURN_NONE;
  const int act_wanted = PyObject_IsTrue(args[1]);
  if (act_wanted < 0) return nullptr;
  c10::cuda::CUDAGuard guard(device);
  at::Tensor xq = empty_on({M, I}, at::kChar, device);
  at::Tensor a_s = empty_on({M}, at::kFloat, device);
  at::Tensor act;
  if (act_wanted) act = empty_on(out_shape(*x, I), type, device);
  const int rc = unlocked([&] {
    return b200q_silu_mul_quant_i8(x->data_ptr(), two_i, act_wanted ? act.data_ptr() : nullptr,
                                   static_cast<int8_t*>(xq.data_ptr()),
                                   static_cast<float*>(a_s.data_ptr()), static_cast<int>(M),
                                   static_cast<int>(I), dt, stream_of(device));
  });
  if (rc != B200Q_OK) return fail(rc, "b200q_silu_mul_quant_i8", M, 0, I);
  return Py_BuildValue("NNN", THPVariable_Wrap(std::move(xq)), THPVariable_Wrap(std::move(a_s)),
                       or_none(std::move(act)));
  END_HANDLE_TH_ERRORS
}

// reserve(bytes, device index | -1): raises the floor of the workspace size; with a device the
// buffer is allocated now
PyObject* reserve(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  long long bytes;
  int index;
  if (!PyArg_ParseTuple(args, "Li", &bytes, &index)) return nullptr;
  {
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    g_ws_floor = std::max<int64_t>(g_ws_floor, bytes);
  }
  if (index >= 0 && bytes > 0) {
    const at::Device device(at::kCUDA, static_cast<c10::DeviceIndex>(index));
    c10::cuda::CUDAGuard guard(device);
    workspace(device, bytes);
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject* set_error_handler(PyObject*, PyObject* f) {
  Py_XINCREF(f);
  Py_XSETREF(g_on_error, f);
  Py_RETURN_NONE;
}

#define B200Q_FAST(f) \
  { #f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)), METH_FASTCALL, nullptr }
PyMethodDef g_methods[] = {B200Q_FAST(w8a16),
                           B200Q_FAST(w8a8_dynamic),
                           B200Q_FAST(w8a8),
                           B200Q_FAST(w8a8_i32),
                           B200Q_FAST(quantize),
                           B200Q_FAST(rmsnorm_quant),
                           B200Q_FAST(silu_mul_quant),
                           {"reserve", reserve, METH_VARARGS, nullptr},
                           {"set_error_handler", set_error_handler, METH_O, nullptr},
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_b200q_torch", nullptr, -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200q_torch(void) { return PyModule_Create(&g_module); }
