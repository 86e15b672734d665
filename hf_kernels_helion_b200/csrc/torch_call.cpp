// The short way from a Python call to the C ABI (include/b200fp8.h): for ordinary eager CUDA tensors one
// native function checks the operands, takes the result and the scratch from torch's caching allocator and
// enqueues the launches, without the interpreter lock. What it does not know to be that case (another layout, a
// tensor subclass, a grad or a dual tensor, tracing, an active torch mode or profiler, a bad argument) makes it
// return None, and the Python path - registered torch op, argument errors, copies of unusual layouts - handles
// the call as it would without this file. A call through the registered op and ctypes costs 30-50 us of host
// time, more than the kernels of most decode and small-matrix calls take.
//
// Scratch belongs to one call: it comes from the caching allocator of the current stream, is given back when
// the call returns (stream order keeps it safe) and is never shared between threads, streams or graphs.
//
// The file reads torch's and Python's own structures, so what it compiles to works with the torch and the Python it
// was built for and no others: `built_for` names them, and _lib.load_native compares it before it calls anything here.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/record_function.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <cstdlib>

#include "../../include/b200fp8.h"

#ifndef B200FP8_BUILT_FOR
#error "B200FP8_BUILT_FOR: a string that names the torch and the Python this is built for"
#endif

namespace {

struct Abi {
  decltype(&b200fp8_gemm) gemm = nullptr;
  decltype(&b200fp8_gemm_workspace_bytes) gemm_ws = nullptr;
  decltype(&b200fp8_gemm_rowscale) rowscale = nullptr;
  decltype(&b200fp8_gemm_rowscale_workspace_bytes) rowscale_ws = nullptr;
  decltype(&b200fp8_linear) linear = nullptr;
  decltype(&b200fp8_linear_workspace_bytes) linear_ws = nullptr;
  decltype(&b200fp8_quant_act) quant_act = nullptr;
  decltype(&b200fp8_quant_weight) quant_weight = nullptr;
} g_abi;
std::atomic<bool> g_bound{false};

// Status word of each device, owned by the Python side (runtime.status_word), which tells this file its address.
constexpr int kMaxDevices = 64;
std::atomic<uint32_t*> g_status[kMaxDevices];

// No tracing, no functorch transform, no Python dispatch or function mode, no profiler.
bool plain_state() {
  const auto tls = c10::impl::tls_local_dispatch_key_set();
  if ((tls.included_.raw_repr() & ~c10::default_included_set.raw_repr()) != 0) return false;
  return !at::impl::torch_function_mode_enabled() && !at::hasCallbacks();
}

bool auto_variant() { return std::getenv("B200FP8_VARIANT") == nullptr; }

// A tensor with nothing but CUDA storage behind it and nothing that autograd or forward mode would record.
const at::Tensor* plain_cuda(PyObject* o, at::ScalarType type) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  static const uint64_t allowed =
      c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView,
                           c10::DispatchKey::AutocastCUDA})   // (every CUDA tensor has it; autocast that is switched on shows in plain_state)
          .raw_repr();
  if ((t.key_set().raw_repr() & ~allowed) != 0 || !t.is_cuda() || t.scalar_type() != type) return nullptr;
  if (t.requires_grad() && c10::GradMode::is_enabled()) return nullptr;
  if (t.unsafeGetTensorImpl()->_fw_grad(0, t).defined()) return nullptr;
  return &t;
}

struct Mat {
  const void* p;
  int64_t rows, cols, ld;
};

// The row-major view the kernels can address as it is: unit inner stride, pitch and base address multiples of
// `align` elements.
bool as_mat(const at::Tensor& t, int64_t align, Mat& m) {
  if (t.dim() != 2) return false;
  m.rows = t.size(0);
  m.cols = t.size(1);
  if (m.rows < 1 || m.cols < 1) return false;
  if (m.cols > 1 && t.stride(1) != 1) return false;
  m.ld = m.rows > 1 ? t.stride(0) : m.cols;
  if (m.ld < m.cols || m.ld % align != 0) return false;
  m.p = t.data_ptr();
  return reinterpret_cast<uintptr_t>(m.p) % (align * t.element_size()) == 0;
}

int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

// -1: not a type that the kernels write
int out_code(PyObject* dtype, at::ScalarType& type) {
  if (!THPDtype_Check(dtype)) return -1;
  type = reinterpret_cast<THPDtype*>(dtype)->scalar_type;
  return type == at::kBFloat16 ? B200FP8_OUT_BF16 : type == at::kFloat ? B200FP8_OUT_FP32 : -1;
}

bool is_128(PyObject* o) {
  int overflow = 0;
  return PyLong_CheckExact(o) && PyLong_AsLongAndOverflow(o, &overflow) == 128 && overflow == 0;
}

// [128, 128] or (128, 128)
bool is_block_128(PyObject* o) {
  if (PyList_CheckExact(o)) return PyList_GET_SIZE(o) == 2 && is_128(PyList_GET_ITEM(o, 0)) && is_128(PyList_GET_ITEM(o, 1));
  if (PyTuple_CheckExact(o))
    return PyTuple_GET_SIZE(o) == 2 && is_128(PyTuple_GET_ITEM(o, 0)) && is_128(PyTuple_GET_ITEM(o, 1));
  return false;
}

// One call's device, stream, status word and scratch.
struct Launch {
  c10::cuda::CUDAGuard guard;
  void* stream;
  uint32_t* status;
  at::Tensor ws;
  const at::TensorOptions options;

  explicit Launch(const at::Tensor& t)
      : guard(t.device()),
        stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()),
        status(t.device().index() < kMaxDevices ? g_status[t.device().index()].load(std::memory_order_acquire) : nullptr),
        options(t.options().requires_grad(false)) {}
  bool scratch(int64_t bytes) {
    if (bytes < 0 || status == nullptr) return false;
    if (bytes > 0) ws = at::empty({bytes}, options.dtype(at::kByte));
    return true;
  }
  void* ws_ptr() const { return ws.defined() ? ws.data_ptr() : nullptr; }
  size_t ws_bytes() const { return ws.defined() ? static_cast<size_t>(ws.numel()) : 0; }
};

PyObject* none() { Py_RETURN_NONE; }

// Gives the interpreter lock up for its lifetime (also when an exception leaves the scope). An allocation or a launch may
// wait - for the driver, for room in the queue - and what it waits for may be another Python thread's to do.
// Taking the lock back costs nothing that shows (512 x 512 x 2048 fp32 8.14 us a call both ways, 4 x 2560 x 2048 7.96 and 8.06).
struct WithoutGil {
  PyThreadState* const state = PyEval_SaveThread();
  WithoutGil() = default;
  WithoutGil(const WithoutGil&) = delete;
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

// The result of a call: `out`, or None where it was not taken. Needs the interpreter lock.
PyObject* wrap(bool taken, at::Tensor&& out) { return taken ? THPVariable_Wrap(std::move(out)) : none(); }

struct GemmOperands {
  const at::Tensor *A, *B, *As, *Bs;
  Mat a, b, as, bs;
};

bool gemm_operands(PyObject* const* args, bool row_scaled, GemmOperands& g) {
  g.A = plain_cuda(args[0], at::kFloat8_e4m3fn);
  g.B = g.A ? plain_cuda(args[1], at::kFloat8_e4m3fn) : nullptr;
  g.As = g.B ? plain_cuda(args[2], at::kFloat) : nullptr;
  g.Bs = g.As ? plain_cuda(args[3], at::kFloat) : nullptr;
  if (g.Bs == nullptr) return false;
  const auto dev = g.A->device();
  if (g.B->device() != dev || g.As->device() != dev || g.Bs->device() != dev) return false;
  if (!as_mat(*g.A, 16, g.a) || !as_mat(*g.B, 16, g.b) || !as_mat(*g.As, 1, g.as) || !as_mat(*g.Bs, 1, g.bs)) return false;
  const int64_t kblocks = cdiv(g.a.cols, 128);
  return g.a.cols == g.b.cols && g.as.rows == g.a.rows && g.as.cols == kblocks && g.bs.cols == kblocks &&
         g.bs.rows == (row_scaled ? g.b.rows : cdiv(g.b.rows, 128));
}

// Status of a block-scaled product into `out`.
int run_gemm(Launch& l, const Mat& a, const Mat& b, const Mat& as, const Mat& bs, at::Tensor& out, int code) {
  const int64_t N = b.rows;
  return g_abi.gemm(a.p, b.p, static_cast<const float*>(as.p), static_cast<const float*>(bs.p), out.data_ptr(), a.rows, N,
                    a.cols, a.ld, b.ld, as.ld, bs.ld, N, code, B200FP8_VARIANT_AUTO, l.ws_ptr(), l.ws_bytes(), l.status,
                    l.stream);
}

// matmul(A, B, As, Bs, block_size, output_dtype) -> Tensor or None
PyObject* matmul(PyObject*, PyObject* const* args, Py_ssize_t n) {
  try {
    if (n != 6 || !g_bound.load(std::memory_order_acquire) || !plain_state() || !auto_variant()) return none();
    at::ScalarType type;
    const int code = out_code(args[5], type);
    const bool row_scaled = is_128(args[4]);
    if (code < 0 || !(row_scaled || is_block_128(args[4]))) return none();
    GemmOperands g;
    if (!gemm_operands(args, row_scaled, g)) return none();
    const int64_t M = g.a.rows, N = g.b.rows, K = g.a.cols;
    at::Tensor out;
    bool taken = false;
    {
      WithoutGil unlocked;
      Launch l(*g.A);
      if (l.scratch(row_scaled ? g_abi.rowscale_ws(M, N, K) : g_abi.gemm_ws(M, N, K, B200FP8_VARIANT_AUTO))) {
        out = at::empty({M, N}, l.options.dtype(type));
        int st;
        if (row_scaled)
          st = g_abi.rowscale(g.a.p, g.b.p, static_cast<const float*>(g.as.p), static_cast<const float*>(g.bs.p),
                              out.data_ptr(), M, N, K, g.a.ld, g.b.ld, g.as.ld, g.bs.ld, N, code, l.ws_ptr(),
                              l.ws_bytes(), l.status, l.stream);
        else
          st = run_gemm(l, g.a, g.b, g.as, g.bs, out, code);
        taken = st == B200FP8_OK;
      }
    }
    return wrap(taken, std::move(out));
  } catch (const std::exception&) {
    return none();   // (out of memory and the like: the Python path meets and reports it)
  }
}

// linear(x, weight, weight_scale, output_dtype) -> Tensor or None
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
  try {
    if (n != 4 || !g_bound.load(std::memory_order_acquire) || !plain_state() || !auto_variant()) return none();
    at::ScalarType type;
    const int code = out_code(args[3], type);
    if (code < 0) return none();
    const at::Tensor* x = plain_cuda(args[0], at::kBFloat16);
    const at::Tensor* B = x ? plain_cuda(args[1], at::kFloat8_e4m3fn) : nullptr;
    const at::Tensor* Bs = B ? plain_cuda(args[2], at::kFloat) : nullptr;
    if (Bs == nullptr || B->device() != x->device() || Bs->device() != x->device()) return none();
    Mat a, b, bs;
    if (!as_mat(*B, 16, b) || !as_mat(*Bs, 1, bs)) return none();
    const int64_t N = b.rows, K = b.cols;
    if (x->dim() == 2) {
      if (!as_mat(*x, 8, a)) return none();
    } else {
      if (x->dim() < 1 || !x->is_contiguous() || x->numel() == 0) return none();
      a = {x->data_ptr(), x->numel() / x->size(-1), x->size(-1), x->size(-1)};
      if (reinterpret_cast<uintptr_t>(a.p) % 16 != 0) return none();
    }
    const int64_t M = a.rows;
    if (a.cols != K || K % 16 != 0 || bs.cols != cdiv(K, 128) || bs.rows != cdiv(N, 128)) return none();
    at::DimVector shape(x->sizes().begin(), x->sizes().end());
    shape.back() = N;
    const bool fused = M <= 256 && K % 128 == 0;
    at::Tensor out;
    bool taken = false;
    {
      WithoutGil unlocked;
      Launch l(*x);
      if (l.scratch((fused ? g_abi.linear_ws : g_abi.gemm_ws)(M, N, K, B200FP8_VARIANT_AUTO))) {
        out = at::empty(shape, l.options.dtype(type));
        int st;
        if (fused) {
          st = g_abi.linear(a.p, b.p, static_cast<const float*>(bs.p), out.data_ptr(), M, N, K, a.ld, b.ld, bs.ld, N, code,
                            B200FP8_VARIANT_AUTO, l.ws_ptr(), l.ws_bytes(), l.status, l.stream);
        } else {
          at::Tensor q = at::empty({M, K}, l.options.dtype(at::kFloat8_e4m3fn));
          at::Tensor s = at::empty({M, cdiv(K, 128)}, l.options.dtype(at::kFloat));
          st = g_abi.quant_act(a.p, q.data_ptr(), s.data_ptr<float>(), M, K, a.ld, K, s.size(1), l.stream);
          if (st == B200FP8_OK)
            st = run_gemm(l, {q.data_ptr(), M, K, K}, b, {s.data_ptr(), M, s.size(1), s.size(1)}, bs, out, code);
        }
        taken = st == B200FP8_OK;
      }
    }
    return wrap(taken, std::move(out));
  } catch (const std::exception&) {
    return none();
  }
}

PyObject* quantise(PyObject* const* args, Py_ssize_t n, bool weight) {
  try {
    if (n != 2 || !g_bound.load(std::memory_order_acquire) || !plain_state() || !is_128(args[1])) return none();
    const at::Tensor* x = plain_cuda(args[0], at::kBFloat16);
    Mat m;
    if (x == nullptr || !as_mat(*x, 8, m) || m.cols % 8 != 0) return none();
    at::Tensor q, s;
    int st;
    {
      WithoutGil unlocked;
      Launch l(*x);
      q = at::empty({m.rows, m.cols}, l.options.dtype(at::kFloat8_e4m3fn));
      s = at::empty({weight ? cdiv(m.rows, 128) : m.rows, cdiv(m.cols, 128)}, l.options.dtype(at::kFloat));
      st = (weight ? g_abi.quant_weight : g_abi.quant_act)(m.p, q.data_ptr(), s.data_ptr<float>(), m.rows, m.cols, m.ld,
                                                           m.cols, s.size(1), l.stream);
    }
    if (st != B200FP8_OK) return none();
    PyObject* a = THPVariable_Wrap(std::move(q));
    PyObject* b = a ? THPVariable_Wrap(std::move(s)) : nullptr;
    PyObject* r = b ? PyTuple_Pack(2, a, b) : nullptr;
    Py_XDECREF(a);
    Py_XDECREF(b);
    return r;
  } catch (const std::exception&) {
    return none();
  }
}

PyObject* act_quant(PyObject*, PyObject* const* args, Py_ssize_t n) { return quantise(args, n, false); }
PyObject* weight_quant(PyObject*, PyObject* const* args, Py_ssize_t n) { return quantise(args, n, true); }

// bind(gemm, gemm_workspace_bytes, rowscale, rowscale_workspace_bytes, linear, linear_workspace_bytes, quant_act,
// quant_weight): addresses of the loaded library's functions
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  void* p[8];
  if (n != 8) {
    PyErr_SetString(PyExc_TypeError, "bind takes eight function addresses");
    return nullptr;
  }
  for (int i = 0; i < 8; ++i) {
    p[i] = PyLong_AsVoidPtr(args[i]);
    if (p[i] == nullptr) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null function address");
      return nullptr;
    }
  }
  g_abi.gemm = reinterpret_cast<decltype(g_abi.gemm)>(p[0]);
  g_abi.gemm_ws = reinterpret_cast<decltype(g_abi.gemm_ws)>(p[1]);
  g_abi.rowscale = reinterpret_cast<decltype(g_abi.rowscale)>(p[2]);
  g_abi.rowscale_ws = reinterpret_cast<decltype(g_abi.rowscale_ws)>(p[3]);
  g_abi.linear = reinterpret_cast<decltype(g_abi.linear)>(p[4]);
  g_abi.linear_ws = reinterpret_cast<decltype(g_abi.linear_ws)>(p[5]);
  g_abi.quant_act = reinterpret_cast<decltype(g_abi.quant_act)>(p[6]);
  g_abi.quant_weight = reinterpret_cast<decltype(g_abi.quant_weight)>(p[7]);
  g_bound.store(true, std::memory_order_release);
  return none();
}

// set_status(device index, address of its status word)
PyObject* set_status(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "set_status takes a device index and an address");
    return nullptr;
  }
  const long dev = PyLong_AsLong(args[0]);
  void* p = PyLong_AsVoidPtr(args[1]);
  if (PyErr_Occurred()) return nullptr;
  if (dev >= 0 && dev < kMaxDevices) g_status[dev].store(static_cast<uint32_t*>(p), std::memory_order_release);
  return none();
}

#define B200FP8_METHOD(name) \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {B200FP8_METHOD(bind),   B200FP8_METHOD(set_status), B200FP8_METHOD(matmul),
                          B200FP8_METHOD(linear), B200FP8_METHOD(act_quant),  B200FP8_METHOD(weight_quant),
                          {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_call", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_call(void) {
  PyObject* m = PyModule_Create(&kModule);
  if (m != nullptr && PyModule_AddStringConstant(m, "built_for", B200FP8_BUILT_FOR) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
