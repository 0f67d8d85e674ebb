// Host side of the composed calls for plain tensors: argument checks, allocations and the autograd node of the INT8
// linear without the Python interpreter in between.  Small calls are bound by it: 128x1024x1024 forward 47 us a call in
// Python against 18 us on the device, forward and backward of 512x1024x1024 205 us against 58.
//
// Everything here handles one case, contiguous bf16 CUDA tensors of matching shapes outside of tracing, transforms and
// modes, and returns None for any other: the callers in kernels.py and linear.py then take the Python path, which
// accepts or refuses it.  The entry points of libi8linear.so are passed in by address (setup), so that the library in
// use is the one that _lib.py has loaded.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/PythonFallbackKernel.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <atomic>

#include "../../include/i8linear.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

decltype(&i8l_quant_gemm) lib_quant_gemm = nullptr;
decltype(&i8l_linear_backward_bias) lib_linear_backward = nullptr;
decltype(&i8l_status_peek) lib_status_peek = nullptr;
PyObject* on_error = nullptr;       // (entry point, code, device index): raises
PyObject* on_timeout = nullptr;     // (device index): raises, or returns where there is nothing to report now
PyObject* open_status = nullptr;    // (device index) -> (status word, poller), as integers
PyObject* py_backward = nullptr;    // the Python path of the backward pass

class WithGil {
 public:
  WithGil() : state_(PyGILState_Ensure()) {}
  ~WithGil() { PyGILState_Release(state_); }

 private:
  PyGILState_STATE state_;
};
class WithoutGil {
 public:
  WithoutGil() : state_(PyEval_SaveThread()) {}
  ~WithoutGil() { PyEval_RestoreThread(state_); }

 private:
  PyThreadState* state_;
};

[[noreturn]] void throw_python_error() {   // the Python error that is set, carried through C++ frames and threads
  python_error e;
  e.persist();
  throw e;
}

struct Status {
  std::atomic<int32_t*> word{nullptr};
  std::atomic<void*> poller{nullptr};
};
constexpr int MAX_DEVICES = 64;
std::array<Status, MAX_DEVICES> statuses;

Status& status_of(int dev) {
  Status& s = statuses[dev];
  if (!s.word.load(std::memory_order_acquire)) {
    const WithGil gil;
    PyObject* r = PyObject_CallFunction(open_status, "i", dev);
    if (!r) throw_python_error();
    unsigned long long word = 0, poller = 0;
    const int ok = PyArg_ParseTuple(r, "KK", &word, &poller);
    Py_DECREF(r);
    if (!ok) throw_python_error();
    s.poller.store(reinterpret_cast<void*>(poller), std::memory_order_relaxed);   // the same pair for every thread that comes here
    s.word.store(reinterpret_cast<int32_t*>(word), std::memory_order_release);
  }
  return s;
}

void check(const char* name, int rc, int dev) {
  if (rc == I8L_OK) return;
  const WithGil gil;
  PyObject* r = PyObject_CallFunction(on_error, "sii", name, rc, dev);
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s failed with code %d", name, rc);
  throw_python_error();
}

void report_timeout(int dev) {   // an earlier GEMM gave up a wait
  if (lib_status_peek(status_of(dev).poller.load(std::memory_order_relaxed)) == I8L_OK) return;
  const WithGil gil;
  PyObject* r = PyObject_CallFunction(on_timeout, "i", dev);
  if (!r) throw_python_error();
  Py_DECREF(r);
}

// A dense bf16 CUDA tensor with its own memory and nothing that a dispatcher would have to see.
bool plain(const Tensor& t) {
  const auto ks = t.key_set();
  return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.layout() == at::kStrided && t.is_contiguous() &&
         t.get_device() < MAX_DEVICES &&
         !ks.has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot,
                                          c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate,
                                          c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor,
                                          c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                          c10::DispatchKey::FuncTorchBatchedDecomposition, c10::DispatchKey::BatchedNestedTensor,
                                          c10::DispatchKey::Batched}));
}
// No mode, transform or tracer looks at what this thread does.
bool plain_thread() {
  const auto inc = c10::impl::tls_local_dispatch_key_set().included_;
  return !c10::impl::dispatch_mode_enabled() && !at::impl::torch_function_mode_enabled() &&
         !inc.has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchDynamicLayerFrontMode,
                                           c10::DispatchKey::FuncTorchDynamicLayerBackMode, c10::DispatchKey::FuncTorchVmapMode,
                                           c10::DispatchKey::VmapMode, c10::DispatchKey::Tracer, c10::DispatchKey::Python,
                                           c10::DispatchKey::Functionalize}));
}

int64_t pad(int64_t n) { return (n + 255) & -256; }
int64_t scale_count(int gran, int64_t batch, int64_t rows, int64_t cols) {
  switch (gran) {
    case I8L_GRAN_TILE128: return batch * (rows / 128) * (cols / 128);
    case I8L_GRAN_TILE128X256: return batch * (rows / 128) * (cols / 256);
    case I8L_GRAN_GROUP128: return batch * rows * (cols / 128);
    default: return batch * rows;
  }
}
Tensor bytes(int64_t n, const Tensor& like) { return at::empty({n}, like.options().dtype(at::kChar)); }

struct Transposed {
  Tensor q, scale;
};

// a [B, M, K] x b [N, K] or [B, N, K], as [B, M, N]; the caller has checked shapes and tensors.
Tensor quant_gemm(const Tensor& a, int64_t B, int64_t M, const Tensor& b, bool b_batched, int a_gran, int b_gran, int qmode,
                  int hadamard, const Tensor* bias, double post, int flags, Transposed* at_out) {
  const int64_t K = b.size(-1), N = b.size(-2), nb = b_batched ? B : 1;
  const int dev = a.get_device();
  const c10::cuda::CUDAGuard guard(dev);
  Status& status = status_of(dev);
  Tensor out = at::empty({B, M, N}, a.options().dtype(flags & I8L_GEMM_OUT_F32 ? at::kFloat : at::kBFloat16));
  const int64_t size = pad(B * M * K) + pad(nb * N * K) + pad(4 * scale_count(a_gran, B, M, K)) +
                       pad(4 * scale_count(b_gran, nb, N, K)) + (at_out ? pad(4 * K) : 0);
  const Tensor ws = bytes(size, a);
  int8_t* qt = nullptr;
  float* st = nullptr;
  if (at_out) {
    at_out->q = at::empty({B, K, M}, a.options().dtype(at::kChar));
    const auto f32 = a.options().dtype(at::kFloat);
    at_out->scale = a_gran == I8L_GRAN_TILE128 ? at::empty({B, K / 128, M / 128}, f32)
                    : a_gran == I8L_GRAN_ROW   ? at::empty({B, K}, f32)
                                               : at::empty({B, K, M / 128}, f32);
    qt = static_cast<int8_t*>(at_out->q.data_ptr());
    st = static_cast<float*>(at_out->scale.data_ptr());
  }
  check("i8l_quant_gemm",
        lib_quant_gemm(a.data_ptr(), b.data_ptr(), bias ? bias->data_ptr() : nullptr, out.data_ptr(), qt, st, B, M, N, K, b_batched,
                       a_gran, b_gran, qmode, hadamard, (float)post, flags, ws.data_ptr(), size,
                       status.word.load(std::memory_order_relaxed), c10::cuda::getCurrentCUDAStream(dev).stream()),
        dev);
  return out;
}

bool plain_bias(const Tensor& bias, const Tensor& a, int64_t N) {
  return plain(bias) && bias.device() == a.device() && bias.numel() >= N;
}

// What a linear layer needs to know of its Int8Config.
struct Config {
  int gran, qmode, hadamard, flags;
  bool whole_k;
  double post(int64_t) const { return hadamard ? 1.0 / hadamard : 1.0; }
  int64_t code() const { return gran | qmode << 8 | flags << 16 | (int64_t)whole_k << 31 | (int64_t)hadamard << 32; }
  static Config from(int64_t c) {
    return Config{(int)(c & 0xff), (int)(c >> 8 & 0xff), (int)(c >> 32), (int)(c >> 16 & 0xff), (bool)(c >> 31 & 1)};
  }
};

Tensor linear_forward(const Tensor& x, const Tensor& weight, const Tensor* bias, const Config& c, Transposed* xt) {
  const int64_t K = weight.size(1), M = x.numel() / K;
  const int b_gran = I8L_GRAN_ROW, a_gran = c.whole_k ? I8L_GRAN_ROW : c.gran;
  const Tensor y = quant_gemm(x, 1, M, weight, false, a_gran, b_gran, c.whole_k ? I8L_QMODE_ROWRCP : c.qmode, c.hadamard, bias,
                              c.post(K), c.whole_k ? 0 : c.flags, xt);
  auto shape = x.sizes().vec();
  shape.back() = weight.size(0);
  return y.select(0, 0).view(shape);   // a view, as the Python path returns it
}

// The Python path of the backward pass, for what the native one does not take.
void backward_in_python(const Tensor& dy, const Tensor& weight, const Tensor& q, const Tensor& s, const Config& c, bool need_dx,
                        bool need_dw, Tensor& dx, Tensor& dw) {
  const WithGil gil;
  PyObject *pd = THPVariable_Wrap(dy), *pw = THPVariable_Wrap(weight), *pq = THPVariable_Wrap(q), *ps = THPVariable_Wrap(s);
  PyObject* r = PyObject_CallFunction(py_backward, "NNNNiiiiiii", pd, pw, pq, ps, c.gran, c.qmode, c.hadamard, c.flags, (int)c.whole_k,
                                      (int)need_dx, (int)need_dw);
  if (!r) throw_python_error();
  PyObject *px = nullptr, *pdw = nullptr;
  const int ok = PyArg_ParseTuple(r, "OO", &px, &pdw);
  if (ok && THPVariable_Check(px)) dx = THPVariable_Unpack(px);
  if (ok && THPVariable_Check(pdw)) dw = THPVariable_Unpack(pdw);
  Py_DECREF(r);
  if (!ok) throw_python_error();
}

void linear_backward(const Tensor& dy, const Tensor& weight, const Tensor& q, const Tensor& s, const Config& c, bool need_dx,
                     bool need_dw, bool need_db, Tensor& dx, Tensor& dw, Tensor& db) {
  const int64_t M = dy.size(0), N = dy.size(1), K = weight.size(1);
  const int gran = c.whole_k ? I8L_GRAN_ROW : c.gran;
  bool ok = plain_thread() && plain(dy) && plain(weight) && weight.size(0) == N && weight.device() == dy.device();
  if (ok && need_dw) {
    ok = q.defined() && s.defined() && q.device() == dy.device() && s.device() == dy.device() && q.scalar_type() == at::kChar &&
         s.scalar_type() == at::kFloat && q.is_contiguous() && s.is_contiguous() && q.sizes() == at::IntArrayRef({1, K, M}) &&
         s.numel() == scale_count(gran, 1, K, M);
  }
  // torch's sum where its graph is wanted (create_graph), and where the kernel's 16-byte loads do not fit
  const bool own_sum = need_db && ok && !at::GradMode::is_enabled() && reinterpret_cast<uintptr_t>(dy.data_ptr()) % 16 == 0;
  if (need_db && !own_sum) db = dy.sum(0);
  if (!ok) {
    if (need_dx || need_dw) backward_in_python(dy, weight, q, s, c, need_dx, need_dw, dx, dw);
    return;
  }
  if (!need_dx && !need_dw && !own_sum) return;
  const int dev = dy.get_device();
  const c10::cuda::CUDAGuard guard(dev);
  Status& status = status_of(dev);
  if (need_dx) dx = at::empty({M, K}, dy.options());
  if (need_dw) dw = at::empty({N, K}, dy.options());
  if (own_sum) db = at::empty({N}, dy.options());
  int64_t size = pad(4 * std::max(K, N));
  if (need_dx) size += pad(M * N) + pad(4 * scale_count(gran, 1, M, N)) + pad(4 * K) + (need_dw ? 0 : pad(K * N));
  if (need_dw) size += pad(N * M) + pad(4 * scale_count(gran, 1, N, M));
  const Tensor ws = bytes(size, dy);
  check("i8l_linear_backward_bias",
        lib_linear_backward(dy.data_ptr(), weight.data_ptr(), need_dw ? static_cast<const int8_t*>(q.data_ptr()) : nullptr,
                            need_dw ? static_cast<const float*>(s.data_ptr()) : nullptr, need_dx ? dx.data_ptr() : nullptr,
                            need_dw ? dw.data_ptr() : nullptr, own_sum ? db.data_ptr() : nullptr, M, N, K, gran, c.whole_k ? I8L_QMODE_ROWRCP : c.qmode, c.hadamard,
                            (float)c.post(N), (float)c.post(M), c.whole_k ? 0 : c.flags, ws.data_ptr(), size,
                            status.word.load(std::memory_order_relaxed), c10::cuda::getCurrentCUDAStream(dev).stream()),
        dev);
}

struct Int8LinearNode : torch::autograd::Function<Int8LinearNode> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const std::optional<Tensor>& bias, int64_t config,
                        bool need_w) {
    Transposed xt;
    const Tensor y = linear_forward(x, weight, bias ? &*bias : nullptr, Config::from(config), need_w ? &xt : nullptr);
    ctx->saved_data["config"] = config;
    ctx->saved_data["bias"] = bias.has_value();
    ctx->saved_data["shape"] = x.sizes().vec();
    if (need_w) ctx->save_for_backward({weight, xt.q, xt.scale});
    else ctx->save_for_backward({weight});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Config c = Config::from(ctx->saved_data["config"].toInt());
    const bool has_bias = ctx->saved_data["bias"].toBool();
    const Tensor& dy = grads[0];
    const Tensor dy2 = dy.reshape({-1, dy.size(-1)}).contiguous();
    Tensor dx, dw, db;
    linear_backward(dy2, saved[0], saved.size() > 1 ? saved[1] : Tensor(), saved.size() > 1 ? saved[2] : Tensor(), c,
                    ctx->needs_input_grad(0), ctx->needs_input_grad(1), has_bias && ctx->needs_input_grad(2), dx, dw, db);
    if (dx.defined()) dx = dx.view(ctx->saved_data["shape"].toIntVector());
    return {dx, dw, db, Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------ Python
bool exact_tensor(PyObject* o) { return THPVariable_CheckExact(o); }

// linear(x, weight, bias or None, gran, qmode, hadamard, flags, whole_k) -> y, or None
PyObject* py_linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8) {
    PyErr_SetString(PyExc_TypeError, "linear takes 8 arguments");
    return nullptr;
  }
  if (!exact_tensor(args[0]) || !exact_tensor(args[1]) || (args[2] != Py_None && !exact_tensor(args[2]))) Py_RETURN_NONE;
  const Tensor x = THPVariable_Unpack(args[0]), weight = THPVariable_Unpack(args[1]);
  std::optional<Tensor> bias;
  if (args[2] != Py_None) bias = THPVariable_Unpack(args[2]);
  const Config c{(int)PyLong_AsLong(args[3]), (int)PyLong_AsLong(args[4]), (int)PyLong_AsLong(args[5]), (int)PyLong_AsLong(args[6]),
                 args[7] == Py_True};
  if (PyErr_Occurred()) return nullptr;
  if ((c.hadamard != 0 && c.hadamard != 128) || !plain_thread() || !plain(x) || !plain(weight) || x.dim() < 1 || weight.dim() != 2 ||
      x.numel() == 0 || weight.numel() == 0 || x.size(-1) != weight.size(1) || weight.device() != x.device() ||
      (bias && !plain_bias(*bias, x, weight.size(0))) || x._fw_grad(0).defined() || weight._fw_grad(0).defined() ||
      (bias && bias->_fw_grad(0).defined()))
    Py_RETURN_NONE;
  Tensor y;
  {
    const WithoutGil no_gil;
    report_timeout(x.get_device());
    const bool grad = at::GradMode::is_enabled();
    if (grad && (x.requires_grad() || weight.requires_grad() || (bias && bias->requires_grad())))
      y = Int8LinearNode::apply(x, weight, bias, c.code(), weight.requires_grad());
    else {
      const at::AutoGradMode off(false);   // as inside the node: a view made here is one made without gradients
      y = linear_forward(x, weight, bias ? &*bias : nullptr, c, nullptr);
    }
  }
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

// quant_gemm(a, b, a_gran, b_gran, qmode, hadamard, bias or None, post_scale, flags, want_at) -> (out, (qt, st)), or None
PyObject* py_quant_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 10) {
    PyErr_SetString(PyExc_TypeError, "quant_gemm takes 10 arguments");
    return nullptr;
  }
  if (!exact_tensor(args[0]) || !exact_tensor(args[1]) || (args[6] != Py_None && !exact_tensor(args[6]))) Py_RETURN_NONE;
  const Tensor a = THPVariable_Unpack(args[0]), b = THPVariable_Unpack(args[1]);
  Tensor bias;
  if (args[6] != Py_None) bias = THPVariable_Unpack(args[6]);
  const int a_gran = (int)PyLong_AsLong(args[2]), b_gran = (int)PyLong_AsLong(args[3]), qmode = (int)PyLong_AsLong(args[4]),
            hadamard = (int)PyLong_AsLong(args[5]), flags = (int)PyLong_AsLong(args[8]), want = PyObject_IsTrue(args[9]);
  const double post = PyFloat_AsDouble(args[7]);
  if (PyErr_Occurred()) return nullptr;
  if (!plain_thread() || !plain(a) || !plain(b) || a.dim() != 3 || (b.dim() != 2 && b.dim() != 3) || a.numel() == 0 || b.numel() == 0 ||
      b.size(-1) != a.size(2) || (b.dim() == 3 && b.size(0) != a.size(0)) || b.device() != a.device() ||
      (bias.defined() && !plain_bias(bias, a, b.size(-2))))
    Py_RETURN_NONE;
  Transposed t;
  Tensor out;
  {
    const WithoutGil no_gil;
    out = quant_gemm(a, a.size(0), a.size(1), b, b.dim() == 3, a_gran, b_gran, qmode, hadamard, bias.defined() ? &bias : nullptr, post,
                     flags, want ? &t : nullptr);
  }
  if (!want) return Py_BuildValue("N(OO)", THPVariable_Wrap(out), Py_None, Py_None);
  return Py_BuildValue("N(NN)", THPVariable_Wrap(out), THPVariable_Wrap(t.q), THPVariable_Wrap(t.scale));
  END_HANDLE_TH_ERRORS
}

// setup(address of i8l_quant_gemm, of i8l_linear_backward_bias, of i8l_status_peek, on_error, on_timeout, open_status, py_backward)
PyObject* py_setup(PyObject*, PyObject* args) {
  unsigned long long qg = 0, lb = 0, sp = 0;
  PyObject *err = nullptr, *timeout = nullptr, *open = nullptr, *bwd = nullptr;
  if (!PyArg_ParseTuple(args, "KKKOOOO", &qg, &lb, &sp, &err, &timeout, &open, &bwd)) return nullptr;
  lib_quant_gemm = reinterpret_cast<decltype(lib_quant_gemm)>(qg);
  lib_linear_backward = reinterpret_cast<decltype(lib_linear_backward)>(lb);
  lib_status_peek = reinterpret_cast<decltype(lib_status_peek)>(sp);
  Py_INCREF(err);
  Py_INCREF(timeout);
  Py_INCREF(open);
  Py_INCREF(bwd);
  on_error = err;
  on_timeout = timeout;
  open_status = open;
  py_backward = bwd;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"setup", py_setup, METH_VARARGS, nullptr},
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_linear)), METH_FASTCALL, nullptr},
    {"quant_gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(py_quant_gemm)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "abi", I8L_HOST_ABI)) Py_CLEAR(m);   // see host_abi in build.py
  return m;
}
