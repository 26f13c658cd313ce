// Host path of the calls an inference program makes most, as one native function per call: the linear
// layers' forwards, the row kernels and the attention entry points.
//
// A layer of a few sequences takes the GPU about ten microseconds; the same call marshalled in Python (device
// and stream look-ups through context managers, two ctypes calls of a dozen arguments, four or five output
// tensors) took the host fifty.  Here it is a METH_FASTCALL function that checks the tensors, allocates the
// results through ATen and calls the C ABI: one crossing of the language border for one call.  A pass over a
// 4864 x 896 layer went from 53 to 11 us (int8, 16 tokens; 9.5 since its GEMM quantizes), a 28-layer 4-bit model's step
// from 9.4 to 4.2 ms (2.7 with fewer launches, 1.0 with a block's step as one call).
//
// The checks are those of the Python wrappers before it (ops.py, glue.py, attention.py), with the same exceptions; the
// attention calls also check caches and lengths against the query's batch.
// Nothing is kept between calls but the devices' workspaces, which the package owns for the life of the
// process.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <algorithm>
#include <atomic>
#include <optional>

#include "../../include/llmqrt_b200.h"

namespace {

using at::Tensor;

Tensor tensor_arg(PyObject* o, const char* what) {
  if (o == Py_None) return Tensor();
  TORCH_CHECK_TYPE(THPVariable_Check(o), "llmqrt_b200: ", what, " must be a tensor, not ", Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
// int(o) and float(o): whatever converts to a number is one.
int64_t int_arg(PyObject* o) {
  THPObjectPtr n(PyNumber_Long(o));
  if (!n) throw python_error();
  const long long v = PyLong_AsLongLong(n.get());
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
double float_arg(PyObject* o) {
  THPObjectPtr f(PyNumber_Float(o));
  if (!f) throw python_error();
  return PyFloat_AS_DOUBLE(f.get());
}
bool bool_arg(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}
PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
template <typename... Ts> PyObject* wrap_tuple(const Ts&... ts) {
  PyObject* items[] = {wrap(ts)...};
  PyObject* tup = PyTuple_New(sizeof...(Ts));
  for (size_t i = 0; i < sizeof...(Ts); ++i) {
    if (!tup || !items[i]) throw python_error();
    PyTuple_SET_ITEM(tup, i, items[i]);
  }
  return tup;
}

void check(int rc) {
  TORCH_CHECK(rc == LLMQRT_OK, "llmqrt_b200: ", llmqrt_last_error(), " (status ", rc, ")");
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return LLMQRT_F16;
    case at::kBFloat16: return LLMQRT_BF16;
    case at::kFloat: return LLMQRT_F32;
    case at::kFloat8_e4m3fn: return LLMQRT_E4M3;
    case at::kFloat8_e5m2: return LLMQRT_E5M2;
    default: TORCH_CHECK_TYPE(false, "llmqrt_b200: unsupported dtype ", t);
  }
}

c10::Device same_device(std::initializer_list<const Tensor*> ts) {
  c10::Device dev(c10::DeviceType::CPU);
  bool first = true;
  for (const Tensor* t : ts) {
    if (!t->defined()) continue;
    TORCH_CHECK(t->is_cuda(), "llmqrt_b200: tensors must live on a CUDA device (there is no CPU path)");
    if (first) dev = t->device();
    else TORCH_CHECK(t->device() == dev, "llmqrt_b200: all tensors must be on the same device");
    first = false;
  }
  return dev;
}

// The package's workspaces (one per device, made by the Python side on first use and never freed).
constexpr int kMaxDevices = 64;
std::atomic<void*> g_workspace[kMaxDevices];
PyObject* g_make_workspace = nullptr;                  // device index -> tensor

// The interpreter lock is given up between the reading of the arguments and the wrapping of the results, as
// a launch may wait for room in the stream's queue.
class GilRelease {
 public:
  GilRelease() : state_(PyEval_SaveThread()) {}
  ~GilRelease() { done(); }
  void done() {
    if (state_) PyEval_RestoreThread(state_);
    state_ = nullptr;
  }

 private:
  PyThreadState* state_;
};

// Device guard, stream and workspace of one call.
struct Call {
  explicit Call(c10::Device dev) : guard(dev), index(dev.index()) {
    stream = c10::cuda::getCurrentCUDAStream(index).stream();
  }
  void* workspace() {
    TORCH_CHECK(index >= 0 && index < kMaxDevices, "llmqrt_b200: device index out of range");
    void* ws = g_workspace[index].load(std::memory_order_acquire);
    if (!ws) {
      const PyGILState_STATE gil = PyGILState_Ensure();
      PyObject* t = PyObject_CallFunction(g_make_workspace, "i", (int)index);
      python_error err;
      if (t) {
        ws = THPVariable_Unpack(t).data_ptr();
        Py_DECREF(t);
      } else {
        err.persist();
      }
      PyGILState_Release(gil);
      if (!ws) throw err;
      g_workspace[index].store(ws, std::memory_order_release);
    }
    return ws;
  }
  c10::cuda::CUDAGuard guard;
  c10::DeviceIndex index;
  cudaStream_t stream;
};

const void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
void* mptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// [M, K] with unit inner stride (copying only if it must).
Tensor rows(const Tensor& x) {
  Tensor r = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
  return r.stride(-1) == 1 ? r : r.contiguous();
}
Tensor empty(const Tensor& like, at::IntArrayRef shape, at::ScalarType dt) {
  return at::empty(shape, like.options().dtype(dt).requires_grad(false));
}
c10::SmallVector<int64_t, 6> out_shape(const Tensor& x, int64_t n) {
  c10::SmallVector<int64_t, 6> s(x.sizes().begin(), x.sizes().end());
  s.back() = n;
  return s;
}
Tensor f32_vector(const Tensor& t) { return t.to(at::kFloat).reshape({-1}).contiguous(); }

// One scratch allocation: M x K quantized bytes, then `scales` floats on a 16-byte boundary.
struct QuantScratch {
  QuantScratch(const Tensor& x, int64_t M, int64_t K, int64_t scales) {
    const int64_t bytes = (M * K + 15) / 16 * 16;
    buf = empty(x, {bytes + 4 * scales}, at::kByte);
    q = static_cast<uint8_t*>(buf.data_ptr());
    scale = reinterpret_cast<float*>(q + bytes);
  }
  Tensor buf;
  uint8_t* q;
  float* scale;
};

// Sizes and rows that the GEMM quantizes itself.
bool few_tokens(const Tensor& x2, int64_t N) {
  return x2.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(x2.data_ptr()) % 16 == 0 && x2.size(1) % 16 == 0 &&
         x2.stride(0) >= x2.size(1) && (x2.scalar_type() == at::kHalf || x2.scalar_type() == at::kBFloat16) &&
         llmqrt_w8a8_dynamic_fits(x2.size(0), N, x2.size(1));
}

#define FAST_FN(name) PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n)
#define FAST_BEGIN(count)                                                                               \
  HANDLE_TH_ERRORS                                                                                      \
  TORCH_CHECK_TYPE(n == (count), "llmqrt_b200: expected ", (count), " arguments, got ", (int64_t)n);     \
  at::NoGradGuard no_grad;
#define FAST_END END_HANDLE_TH_ERRORS

// ---- linear layers ---------------------------------------------------------------------------------

// (x, qweight, bias or None, weight_scale [N] fp32) -> y in x's dtype: per-token x per-channel int8.
FAST_FN(sq_per_channel) {
  FAST_BEGIN(4)
  const Tensor x = tensor_arg(a[0], "x"), w = tensor_arg(a[1], "qweight"), bias = tensor_arg(a[2], "bias");
  const Tensor ws = tensor_arg(a[3], "weight_scale");
  GilRelease gil;
  const Tensor x2 = rows(x);
  const int64_t M = x2.size(0), K = x2.size(1), N = w.size(0);
  if (M == 0) {
    const Tensor z = at::zeros(out_shape(x, N), x.options().requires_grad(false));
    gil.done();
    return wrap(z);
  }
  Call c(same_device({&x, &w, &bias, &ws}));
  const Tensor w_s = f32_vector(ws);
  TORCH_CHECK(w_s.numel() == N, "per-channel int8 linear: a_scale must have M elements and w_scale N elements");
  const int xd = dtype_code(x.scalar_type()), bd = bias.defined() ? dtype_code(bias.scalar_type()) : LLMQRT_F16;
  Tensor out = empty(x, out_shape(x, N), x.scalar_type());
  if (few_tokens(x2, N)) {
    check(llmqrt_w8a8_linear_dynamic(0, ptr(x2), xd, x2.stride(0), ptr(w), w.stride(0), ptr(bias), bd,
                                     static_cast<const float*>(ptr(w_s)), mptr(out), xd, N, M, N, K, c.stream));
    gil.done();
    return wrap(out);
  }
  QuantScratch s(x, M, K, M);
  check(llmqrt_quantize_int8(ptr(x2), xd, M, K, x2.stride(0), 1, reinterpret_cast<int8_t*>(s.q), nullptr, s.scale, 1.f,
                             c.workspace(), c.stream));
  check(llmqrt_w8a8_int8_linear_per_channel(reinterpret_cast<const int8_t*>(s.q), K, static_cast<const int8_t*>(ptr(w)),
                                            w.stride(0), ptr(bias), bd, s.scale, static_cast<const float*>(ptr(w_s)),
                                            mptr(out), xd, N, M, N, K, c.workspace(), c.stream,
                                            LLMQRT_GEMM_STATIC_WEIGHT));
  gil.done();
  return wrap(out);
  FAST_END
}

// (x, qweight, bias fp16, weight_scale float) -> y in x's dtype: per-tensor x per-tensor int8.
FAST_FN(sq_per_tensor) {
  FAST_BEGIN(4)
  const Tensor x = tensor_arg(a[0], "x"), w = tensor_arg(a[1], "qweight"), bias = tensor_arg(a[2], "bias");
  const float weight_scale = (float)float_arg(a[3]);
  GilRelease gil;
  const Tensor x2 = rows(x);
  const int64_t M = x2.size(0), K = x2.size(1), N = w.size(0);
  if (M == 0) {
    const Tensor z = at::zeros(out_shape(x, N), x.options().requires_grad(false));
    gil.done();
    return wrap(z);
  }
  Call c(same_device({&x, &w, &bias}));
  const int xd = dtype_code(x.scalar_type());
  QuantScratch s(x, M, K, 1);
  Tensor out = empty(x, out_shape(x, N), at::kHalf);
  check(llmqrt_quantize_int8(ptr(x2), xd, M, K, x2.stride(0), 0, reinterpret_cast<int8_t*>(s.q), nullptr, s.scale,
                             weight_scale, c.workspace(), c.stream));
  check(llmqrt_w8a8_int8_linear_per_tensor(reinterpret_cast<const int8_t*>(s.q), K, static_cast<const int8_t*>(ptr(w)),
                                           w.stride(0), ptr(bias), 0.f, s.scale, 1.f, mptr(out), N, M, N, K,
                                           c.workspace(), c.stream, LLMQRT_GEMM_STATIC_WEIGHT));
  out = out.to(x.scalar_type());
  gil.done();
  return wrap(out);
  FAST_END
}

// (x, weight e4m3, bias or None, weight_scale) -> y in x's dtype: per-token x per-channel fp8, a bf16 result.
FAST_FN(fp8_per_token) {
  FAST_BEGIN(4)
  const Tensor x = tensor_arg(a[0], "x"), w = tensor_arg(a[1], "weight"), bias = tensor_arg(a[2], "bias");
  const Tensor ws = tensor_arg(a[3], "weight_scale");
  GilRelease gil;
  const Tensor x2 = rows(x);
  const int64_t M = x2.size(0), K = x2.size(1), N = w.size(0);
  Call c(same_device({&x, &w, &bias, &ws}));
  const int xd = dtype_code(x.scalar_type()), bd = bias.defined() ? dtype_code(bias.scalar_type()) : LLMQRT_BF16;
  Tensor out = empty(x, out_shape(x, N), at::kBFloat16);
  const Tensor w_s = f32_vector(ws);
  if (few_tokens(x2, N)) {
    check(llmqrt_w8a8_linear_dynamic(1, ptr(x2), xd, x2.stride(0), ptr(w), w.stride(0), ptr(bias), bd,
                                     static_cast<const float*>(ptr(w_s)), mptr(out), LLMQRT_BF16, N, M, N, K, c.stream));
    out = out.to(x.scalar_type());
    gil.done();
    return wrap(out);
  }
  QuantScratch s(x, M, K, M);
  check(llmqrt_quantize_fp8(ptr(x2), xd, M, K, x2.stride(0), 1, s.q, s.scale, 1.f, c.workspace(), c.stream));
  check(llmqrt_f8f8bf16_rowwise(s.q, LLMQRT_E4M3, K, static_cast<const uint8_t*>(ptr(w)), w.stride(0), ptr(bias), bd,
                                s.scale, static_cast<const float*>(ptr(w_s)), mptr(out), N, M, N, K, c.workspace(),
                                c.stream, LLMQRT_GEMM_STATIC_WEIGHT));
  out = out.to(x.scalar_type());
  gil.done();
  return wrap(out);
  FAST_END
}

// (x, weight e4m3, bias in the out dtype or None, weight_scale [1], input_scale [1] or None (dynamic), out
// dtype) -> y in that dtype: per-tensor fp8.
FAST_FN(fp8_per_tensor) {
  FAST_BEGIN(6)
  const Tensor x = tensor_arg(a[0], "x"), w = tensor_arg(a[1], "weight"), bias = tensor_arg(a[2], "bias");
  const Tensor ws = tensor_arg(a[3], "weight_scale"), in_scale = tensor_arg(a[4], "input_scale");
  TORCH_CHECK_TYPE(THPDtype_Check(a[5]), "llmqrt_b200: the result's dtype must be a torch.dtype");
  const at::ScalarType od = reinterpret_cast<THPDtype*>(a[5])->scalar_type;
  GilRelease gil;
  const Tensor x2 = rows(x);
  const int64_t M = x2.size(0), K = x2.size(1), N = w.size(0);
  Call c(same_device({&x, &w, &bias, &ws, &in_scale}));
  const int xd = dtype_code(x.scalar_type());
  TORCH_CHECK(ws.numel() == 1 && (!in_scale.defined() || in_scale.numel() == 1), "fp8 per-tensor linear: the scales must be scalars");
  const Tensor w_s = f32_vector(ws), x_s = in_scale.defined() ? f32_vector(in_scale) : Tensor();
  QuantScratch s(x, M, K, 1);
  Tensor out = empty(x, out_shape(x, N), od);
  check(llmqrt_quantize_fp8_alpha(ptr(x2), xd, M, K, x2.stride(0), static_cast<const float*>(ptr(x_s)),
                                  static_cast<const float*>(ptr(w_s)), s.q, s.scale, c.workspace(), c.stream));
  check(llmqrt_f8f8_tensorwise(s.q, LLMQRT_E4M3, K, static_cast<const uint8_t*>(ptr(w)), w.stride(0), ptr(bias), 0.f,
                               s.scale, 1.f, mptr(out), dtype_code(od), N, M, N, K, c.workspace(), c.stream,
                               LLMQRT_GEMM_STATIC_WEIGHT));
  gil.done();
  return wrap(out);
  FAST_END
}

// (x fp16, wq_t, sz_t, bias or None, K, N, G) -> y fp16 [..., N].
FAST_FN(awq_linear) {
  FAST_BEGIN(7)
  const Tensor x = tensor_arg(a[0], "x"), wq = tensor_arg(a[1], "wq_t"), sz = tensor_arg(a[2], "sz_t");
  const Tensor bias = tensor_arg(a[3], "bias");
  const int64_t K = int_arg(a[4]), N = int_arg(a[5]), G = int_arg(a[6]);
  GilRelease gil;
  const Tensor x2 = rows(x);
  const int64_t M = x2.size(0);
  Call c(same_device({&x, &wq, &bias}));
  TORCH_CHECK(x2.size(1) == K, "awq_gemm: x has K=", x2.size(1), ", layer has K=", K);
  Tensor out = empty(x, out_shape(x, N), at::kHalf);
  check(llmqrt_awq_gemm(ptr(x2), x2.stride(0), static_cast<const uint32_t*>(ptr(wq)), static_cast<const uint32_t*>(ptr(sz)),
                        ptr(bias), mptr(out), N, M, N, K, G, c.workspace(), c.stream));
  gil.done();
  return wrap(out);
  FAST_END
}

// (x fp16 of at most 16 tokens, wq_t, sz_t, bias or None, residual or None, K, N, G) -> residual + y, or without a
// residual silu(first half of y) * second half.
FAST_FN(awq_tail) {
  FAST_BEGIN(8)
  const Tensor x = tensor_arg(a[0], "x"), wq = tensor_arg(a[1], "wq_t"), sz = tensor_arg(a[2], "sz_t");
  const Tensor bias = tensor_arg(a[3], "bias"), res = tensor_arg(a[4], "residual");
  const int64_t K = int_arg(a[5]), N = int_arg(a[6]), G = int_arg(a[7]);
  GilRelease gil;
  const Tensor x2 = rows(x);
  const int64_t M = x2.size(0), cols = res.defined() ? N : N / 2;
  Call c(same_device({&x, &wq, &bias, &res}));
  TORCH_CHECK(x2.size(1) == K, "awq_gemm: x has K=", x2.size(1), ", layer has K=", K);
  Tensor r2;
  if (res.defined()) {
    r2 = rows(res);
    TORCH_CHECK(res.scalar_type() == at::kHalf && r2.size(0) == M && r2.size(1) == N, "awq_gemm: residual must be fp16 [M, N]");
  }
  Tensor out = empty(x, out_shape(x, cols), at::kHalf);
  check(llmqrt_awq_gemm_tail(ptr(x2), x2.stride(0), static_cast<const uint32_t*>(ptr(wq)),
                             static_cast<const uint32_t*>(ptr(sz)), ptr(bias), ptr(r2), res.defined() ? r2.stride(0) : 0,
                             mptr(out), cols, M, N, K, G, c.stream));
  gil.done();
  return wrap(out);
  FAST_END
}

// ---- row kernels -----------------------------------------------------------------------------------

// (x, weight, eps, residual or None, quantize, want_y) -> (y, h, q, scale), absent ones None.
FAST_FN(rmsnorm) {
  FAST_BEGIN(6)
  const Tensor x = tensor_arg(a[0], "x"), w = tensor_arg(a[1], "weight"), res = tensor_arg(a[3], "residual");
  const float eps = (float)float_arg(a[2]);
  const bool quantize = bool_arg(a[4]), want_y = bool_arg(a[5]);
  GilRelease gil;
  Call c(same_device({&x, &w, &res}));
  const int64_t H = x.size(-1);
  const Tensor x2 = x.reshape({-1, H}).contiguous();
  const int64_t M = x2.size(0);
  const Tensor r2 = res.defined() ? res.reshape({-1, H}).contiguous() : Tensor();
  TORCH_CHECK(!r2.defined() || r2.size(0) == M, "rmsnorm: x and residual must have the same number of rows");
  Tensor h, y, q, s;
  if (res.defined()) h = empty(x, x.sizes(), x.scalar_type());
  if (want_y) y = empty(x, x.sizes(), x.scalar_type());
  if (quantize) {
    q = empty(x, {M, H}, at::kChar);
    s = empty(x, {M}, at::kFloat);
  }
  check(llmqrt_rmsnorm(ptr(x2), ptr(r2), mptr(h), ptr(w), eps, mptr(y), static_cast<int8_t*>(mptr(q)),
                       static_cast<float*>(mptr(s)), dtype_code(x.scalar_type()), M, H, c.stream));
  gil.done();
  return wrap_tuple(y, h, q, s);
  FAST_END
}

// (gate_up, quantize, want_y) -> (h, q, scale), absent ones None.
FAST_FN(silu_mul) {
  FAST_BEGIN(3)
  const Tensor gu = tensor_arg(a[0], "gate_up");
  const bool quantize = bool_arg(a[1]), want_y = bool_arg(a[2]);
  GilRelease gil;
  Call c(same_device({&gu}));
  const int64_t I = gu.size(-1) / 2;
  Tensor g2 = gu.reshape({-1, 2 * I});
  if (g2.stride(1) != 1) g2 = g2.contiguous();
  const int64_t M = g2.size(0);
  Tensor y, q, s;
  if (want_y) y = empty(gu, out_shape(gu, I), gu.scalar_type());
  if (quantize) {
    q = empty(gu, {M, I}, at::kChar);
    s = empty(gu, {M}, at::kFloat);
  }
  check(llmqrt_silu_mul(ptr(g2), g2.stride(0), mptr(y), static_cast<int8_t*>(mptr(q)), static_cast<float*>(mptr(s)),
                        dtype_code(gu.scalar_type()), M, I, c.stream));
  gil.done();
  return wrap_tuple(y, q, s);
  FAST_END
}

// (q, k, v or None, cos, sin, pos0, pos_dev or None, k_cache or None, v_cache or None), in place.
FAST_FN(rope_kv_write) {
  FAST_BEGIN(9)
  const Tensor q = tensor_arg(a[0], "q"), k = tensor_arg(a[1], "k"), v = tensor_arg(a[2], "v");
  const Tensor cos = tensor_arg(a[3], "cos"), sin = tensor_arg(a[4], "sin"), pos_dev = tensor_arg(a[6], "pos_dev");
  const Tensor kc = tensor_arg(a[7], "k_cache"), vc = tensor_arg(a[8], "v_cache");
  const int64_t pos0 = int_arg(a[5]);
  GilRelease gil;
  Call c(same_device({&q, &k, &v, &cos, &sin, &pos_dev, &kc, &vc}));
  const int64_t B = q.size(0), S = q.size(1), Hq = q.size(2), d = q.size(3), Hkv = k.size(2);
  for (const Tensor* t : {&q, &k, &v})
    TORCH_CHECK(!t->defined() || (t->stride(3) == 1 && t->stride(2) == d && t->stride(0) == S * t->stride(1)),
                "rope_kv_write: tensors must be [B, S, H, d] with heads and d contiguous");
  TORCH_CHECK(!v.defined() || v.stride(1) == k.stride(1), "rope_kv_write: k and v must share the token stride");
  check(llmqrt_rope_kv_write(mptr(q), q.stride(1), mptr(k), ptr(v), k.stride(1), mptr(kc), mptr(vc),
                             kc.defined() ? kc.stride(0) : 0, kc.defined() ? kc.stride(1) : 0, (int32_t)pos0,
                             static_cast<const int32_t*>(ptr(pos_dev)), static_cast<const float*>(ptr(cos)),
                             static_cast<const float*>(ptr(sin)), cos.size(0), dtype_code(q.scalar_type()), B, S, Hq, Hkv,
                             d, c.stream));
  gil.done();
  Py_RETURN_NONE;
  FAST_END
}

// ---- attention -------------------------------------------------------------------------------------

// [B, S, H, d] with heads and d contiguous and batches back to back; copies only if it must.
Tensor token_strided(const Tensor& x) {
  const int64_t S = x.size(1), d = x.size(3);
  const bool ok = x.stride(3) == 1 && x.stride(2) == d && x.stride(0) == S * x.stride(1) && x.stride(1) % 8 == 0 &&
                  reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0;
  return ok ? x : x.contiguous();
}

// Key and value caches of at least B sequences, [B, rows, Hkv, d] with heads and d contiguous and one set of strides.
// Returns the rows that both have.  The kernels index them by what the caller says, so nothing is launched before this
// holds; the checks of shapes come before those of devices.
int64_t check_caches(const Tensor& kc, const Tensor& vc, int64_t B, int64_t d, const char* what) {
  TORCH_CHECK(kc.dim() == 4 && vc.dim() == 4 && kc.size(3) == d && vc.size(3) == d && vc.size(2) == kc.size(2) &&
              kc.stride(3) == 1 && kc.stride(2) == d && vc.strides() == kc.strides(),
              what, ": caches must be [B, S, Hkv, d] with heads and d contiguous");
  TORCH_CHECK(kc.size(0) >= B && vc.size(0) >= B, what, ": the caches hold ", std::min(kc.size(0), vc.size(0)),
              " sequences, the call has ", B);
  return std::min(kc.size(1), vc.size(1));
}
// Lengths of B sequences, back to back.
Tensor check_lens(const Tensor& lens, int64_t B, const char* what) {
  if (!lens.defined()) return lens;
  TORCH_CHECK_TYPE(lens.scalar_type() == at::kInt, what, ": sequence lengths must be int32");
  TORCH_CHECK(lens.numel() >= B, what, ": ", lens.numel(), " sequence lengths for ", B, " sequences");
  return lens.contiguous();
}

// (q, k, v, causal, softcap) -> out
FAST_FN(attn_prefill) {
  FAST_BEGIN(5)
  Tensor q = tensor_arg(a[0], "q"), k = tensor_arg(a[1], "k"), v = tensor_arg(a[2], "v");
  const bool causal = bool_arg(a[3]);
  const float softcap = (float)float_arg(a[4]);
  GilRelease gil;
  TORCH_CHECK_TYPE(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(),
                   "flash_attn_func: q, k and v must share one dtype");
  Call c(same_device({&q, &k, &v}));
  TORCH_CHECK(q.dim() == 4 && k.dim() == 4 && k.size(1) == q.size(1) && v.sizes() == k.sizes() && k.size(0) == q.size(0) &&
              k.size(3) == q.size(3), "flash_attn_func: q, k, v must share batch, sequence length and head_dim");
  const int64_t B = q.size(0), S = q.size(1), Hq = q.size(2), d = q.size(3), Hkv = k.size(2);
  q = token_strided(q);
  k = token_strided(k);
  v = token_strided(v);
  if (k.stride(1) != v.stride(1)) {
    v = v.contiguous();
    k = k.contiguous();
  }
  Tensor out = empty(q, {B, S, Hq, d}, q.scalar_type());
  check(llmqrt_attn_prefill(ptr(q), q.stride(1), ptr(k), ptr(v), k.stride(1), mptr(out), out.stride(1),
                            dtype_code(q.scalar_type()), B, S, Hq, Hkv, d, causal ? 1 : 0, softcap, c.stream));
  gil.done();
  return wrap(out);
  FAST_END
}

// (k_cache, v_cache, k, v, cache_seqlens or None, start_pos), in place.
FAST_FN(kv_append) {
  FAST_BEGIN(6)
  const Tensor kc = tensor_arg(a[0], "k_cache"), vc = tensor_arg(a[1], "v_cache"), k0 = tensor_arg(a[2], "k");
  const Tensor v0 = tensor_arg(a[3], "v"), lens0 = tensor_arg(a[4], "cache_seqlens");
  const int64_t start = int_arg(a[5]);
  GilRelease gil;
  TORCH_CHECK(k0.dim() == 4 && v0.sizes() == k0.sizes(), "kv_append: k and v must be [B, S, Hkv, d]");
  TORCH_CHECK_TYPE(k0.scalar_type() == kc.scalar_type() && v0.scalar_type() == kc.scalar_type() &&
                   vc.scalar_type() == kc.scalar_type(), "kv_append: k, v and the caches must share one dtype");
  const int64_t B = k0.size(0), S = k0.size(1), Hkv = k0.size(2), d = k0.size(3);
  const int64_t cache_rows = check_caches(kc, vc, B, d, "kv_append");
  TORCH_CHECK(kc.size(2) >= Hkv, "kv_append: the caches have ", kc.size(2), " heads, k has ", Hkv);
  const Tensor lens = check_lens(lens0, B, "kv_append");
  Call c(same_device({&kc, &vc, &k0, &v0, &lens}));
  const Tensor k = k0.contiguous(), v = v0.contiguous();
  check(llmqrt_kv_append(mptr(kc), mptr(vc), kc.stride(0), kc.stride(1), ptr(k), ptr(v),
                         static_cast<const int32_t*>(ptr(lens)), (int32_t)start, dtype_code(kc.scalar_type()), B, S, Hkv, d,
                         cache_rows, c.stream));
  gil.done();
  Py_RETURN_NONE;
  FAST_END
}

// Batch stride of a [B, H, d] tensor whose heads and d are contiguous (a slice of a fused row).
int64_t rows_stride(const Tensor& t, int64_t B, int64_t H, int64_t d, const char* what) {
  TORCH_CHECK(t.dim() == 3 && t.size(0) == B && t.size(1) == H && t.size(2) == d && t.stride(2) == 1 && t.stride(1) == d &&
              reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 &&
              !(B > 1 && (t.stride(0) < H * d || t.stride(0) % 8)),
              "attn_decode: ", what, " must be [B, H, d] with heads and d contiguous, 16-byte aligned");
  return B > 1 ? t.stride(0) : H * d;
}

// (q, k_cache, v_cache, seqlens, max_seqlen, softcap, quantize, k_new, v_new, cos, sin) -> (out, out_q, scale)
FAST_FN(attn_decode) {
  FAST_BEGIN(11)
  Tensor q = tensor_arg(a[0], "q");
  const Tensor kc = tensor_arg(a[1], "k_cache"), vc = tensor_arg(a[2], "v_cache"), lens0 = tensor_arg(a[3], "seqlens");
  const int64_t max_seqlen0 = int_arg(a[4]);
  const float softcap = (float)float_arg(a[5]);
  const bool quantize = bool_arg(a[6]);
  const Tensor kn = tensor_arg(a[7], "k_new"), vn = tensor_arg(a[8], "v_new");
  const Tensor cos = tensor_arg(a[9], "cos"), sin = tensor_arg(a[10], "sin");
  GilRelease gil;
  TORCH_CHECK(q.dim() == 3, "attn_decode: q must be [B, Hq, d] and the caches [B, S, Hkv, d]");
  const int64_t B = q.size(0), Hq = q.size(1), d = q.size(2);
  const int64_t max_seqlen = std::min(max_seqlen0, check_caches(kc, vc, B, d, "attn_decode")), Hkv = kc.size(2);
  TORCH_CHECK_TYPE(lens0.defined(), "attn_decode: seqlens must be int32");
  const Tensor lens = check_lens(lens0, B, "attn_decode");
  Call c(same_device({&q, &kc, &vc, &lens, &kn, &vn, &cos, &sin}));
  TORCH_CHECK_TYPE(kc.scalar_type() == q.scalar_type() && vc.scalar_type() == q.scalar_type(),
                   "attn_decode: q and the caches must share one dtype");
  if (B > 0 && (q.stride(2) != 1 || q.stride(1) != d || (B > 1 && (q.stride(0) < Hq * d || q.stride(0) % 8)) ||
                reinterpret_cast<uintptr_t>(q.data_ptr()) % 16))
    q = q.contiguous();
  Tensor out = empty(q, {B, Hq, d}, q.scalar_type()), out_q, scale;
  if (quantize) {
    out_q = empty(q, {B, Hq * d}, at::kChar);
    scale = empty(q, {B}, at::kFloat);
  }
  const int64_t q_stride = B > 1 ? q.stride(0) : Hq * d;
  int64_t kv_stride = 0;
  if (kn.defined()) {
    TORCH_CHECK(vn.defined() && kn.scalar_type() == q.scalar_type() && vn.scalar_type() == q.scalar_type(),
                "attn_decode: k_new and v_new go together, in q's dtype");
    kv_stride = rows_stride(kn, B, Hkv, d, "k_new");
    TORCH_CHECK(rows_stride(vn, B, Hkv, d, "v_new") == kv_stride, "attn_decode: k_new and v_new must share one batch stride");
  }
  if (cos.defined())
    TORCH_CHECK(sin.defined() && cos.scalar_type() == at::kFloat && sin.scalar_type() == at::kFloat &&
                cos.sizes() == sin.sizes() && cos.size(-1) == d / 2 && cos.is_contiguous() && sin.is_contiguous(),
                "attn_decode: cos / sin must be contiguous fp32 [rows, d/2]");
  check(llmqrt_attn_decode_append(ptr(q), q_stride, ptr(kn), ptr(vn), kv_stride, static_cast<const float*>(ptr(cos)),
                                  static_cast<const float*>(ptr(sin)), cos.defined() ? cos.size(0) : 0, mptr(kc), mptr(vc),
                                  kc.stride(0), kc.stride(1), static_cast<const int32_t*>(ptr(lens)), mptr(out),
                                  static_cast<int8_t*>(mptr(out_q)), static_cast<float*>(mptr(scale)),
                                  dtype_code(q.scalar_type()), B, Hq, Hkv, d, max_seqlen, softcap, c.workspace(), c.stream));
  gil.done();
  return wrap_tuple(out, out_q, scale);
  FAST_END
}

// (q [B, 1, Hq, d], k_cache, v_cache, k, v (one new token [B, 1, Hkv, d], or None), cache_seqlens or None, length added
// to those, max_seqlen, softcap, cos or None, sin or None, write the row twice) -> out [B, 1, Hq, d]
FAST_FN(attn_decode_step) {
  FAST_BEGIN(12)
  const Tensor q4 = tensor_arg(a[0], "q"), kc = tensor_arg(a[1], "k_cache"), vc = tensor_arg(a[2], "v_cache");
  const Tensor k4 = tensor_arg(a[3], "k"), v4 = tensor_arg(a[4], "v"), lens0 = tensor_arg(a[5], "cache_seqlens");
  const int64_t len_add = int_arg(a[6]), max_seqlen0 = int_arg(a[7]);
  const float softcap = (float)float_arg(a[8]);
  const Tensor cos = tensor_arg(a[9], "cos"), sin = tensor_arg(a[10], "sin");
  const bool twice = bool_arg(a[11]);
  GilRelease gil;
  TORCH_CHECK(q4.dim() == 4 && q4.size(1) == 1, "attn_decode: q must be [B, 1, Hq, d] and the caches [B, S, Hkv, d]");
  const int64_t B = q4.size(0), Hq = q4.size(2), d = q4.size(3);
  const int64_t cache_rows = check_caches(kc, vc, B, d, "attn_decode"), Hkv = kc.size(2);
  const int64_t max_seqlen = std::min(max_seqlen0, cache_rows);
  const Tensor lens = check_lens(lens0, B, "attn_decode");
  Call c(same_device({&q4, &kc, &vc, &k4, &v4, &lens, &cos, &sin}));
  TORCH_CHECK_TYPE(kc.scalar_type() == q4.scalar_type() && vc.scalar_type() == q4.scalar_type(),
                   "attn_decode: q and the caches must share one dtype");
  auto usable = [&](const Tensor& t, int64_t H) {
    return t.stride(3) == 1 && t.stride(2) == d && (B <= 1 || (t.stride(0) >= H * d && t.stride(0) % 8 == 0)) &&
           reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  };
  const Tensor q = B == 0 || usable(q4, Hq) ? q4 : q4.contiguous();
  Tensor k, v;
  if (k4.defined()) {
    TORCH_CHECK(k4.dim() == 4 && v4.defined() && v4.sizes() == k4.sizes() && k4.size(0) == B && k4.size(1) == 1 &&
                k4.size(2) == Hkv && k4.size(3) == d, "attn_decode: k and v must be [B, 1, Hkv, d]");
    k = k4.to(kc.scalar_type());
    v = v4.to(vc.scalar_type());
    if (B > 0 && !(usable(k, Hkv) && usable(v, Hkv) && (B == 1 || k.stride(0) == v.stride(0)))) {
      k = k.contiguous();
      v = v.contiguous();
      // (contiguous storage may still start off a 16-byte boundary)
      if (!usable(k, Hkv)) k = k.clone();
      if (!usable(v, Hkv)) v = v.clone();
    }
  }
  if (cos.defined())
    TORCH_CHECK(sin.defined() && cos.scalar_type() == at::kFloat && sin.scalar_type() == at::kFloat &&
                cos.sizes() == sin.sizes() && cos.size(-1) == d / 2 && cos.is_contiguous() && sin.is_contiguous(),
                "attn_decode: cos / sin must be contiguous fp32 [rows, d/2]");
  Tensor out = empty(q4, q4.sizes(), q4.scalar_type());
  check(llmqrt_attn_decode_step(ptr(q), B > 1 ? q.stride(0) : Hq * d, ptr(k), ptr(v), k.defined() && B > 1 ? k.stride(0) : Hkv * d,
                                static_cast<const float*>(ptr(cos)), static_cast<const float*>(ptr(sin)),
                                cos.defined() ? cos.size(0) : 0, twice ? 1 : 0, mptr(kc), mptr(vc), kc.stride(0), kc.stride(1), cache_rows,
                                static_cast<const int32_t*>(ptr(lens)), (int32_t)len_add, mptr(out),
                                dtype_code(q4.scalar_type()), B, Hq, Hkv, d, max_seqlen, softcap, c.workspace(), c.stream));
  gil.done();
  return wrap(out);
  FAST_END
}

// Identity and in-place version of a tensor, appended to a key.
using Key = c10::SmallVector<int64_t, 32>;
void key_of(const Tensor& t, Key& k) {
  if (!t.defined()) return;
  k.push_back((int64_t)reinterpret_cast<intptr_t>(t.data_ptr()));
  k.push_back(t._version());
  k.push_back((int64_t)t.scalar_type());
  k.push_back((int64_t)t.device().type() * 256 + t.device().index());
  k.push_back(t.dim());
  for (int64_t s : t.sizes()) k.push_back(s);
}

// (tensor or None, ...) -> identity and in-place version of the tensors, as one tuple of integers.
FAST_FN(tensor_key) {
  HANDLE_TH_ERRORS
  Key k;
  for (Py_ssize_t i = 0; i < n; ++i) key_of(tensor_arg(a[i], "buffer"), k);
  PyObject* tup = PyTuple_New((Py_ssize_t)k.size());
  if (!tup) throw python_error();
  for (size_t i = 0; i < k.size(); ++i) PyTuple_SET_ITEM(tup, i, PyLong_FromLongLong(k[i]));
  return tup;
  FAST_END
}

// ---- a 4-bit decoder block's step ------------------------------------------------------------------

// A block of a few tokens is seven kernels of 2 to 9 us; as eight calls of Python modules it took the host 90 us.  The call
// below does the whole step or, wherever anything about the block is not as these classes made it, nothing: it returns
// None, having changed nothing, and the caller goes on with the modules, whose behaviour (and errors) this one has.

PyObject* g_plain = nullptr;                           // ((class, attribute, the function it was defined with), ...)
PyObject* g_hooks = nullptr;                           // the dictionaries of hooks on all modules
PyTypeObject *g_norm = nullptr, *g_attn = nullptr, *g_mlp = nullptr, *g_linear = nullptr, *g_cache = nullptr;

// (RMSNorm, QuantAttentionFused, FusedGateUpMLP, WQLinear_GEMM, WindowedCache, plain, hooks)
FAST_FN(set_block_classes) {
  FAST_BEGIN(7)
  for (int i = 0; i < 7; ++i) Py_INCREF(a[i]);         // (for the life of the process)
  g_norm = reinterpret_cast<PyTypeObject*>(a[0]);
  g_attn = reinterpret_cast<PyTypeObject*>(a[1]);
  g_mlp = reinterpret_cast<PyTypeObject*>(a[2]);
  g_linear = reinterpret_cast<PyTypeObject*>(a[3]);
  g_cache = reinterpret_cast<PyTypeObject*>(a[4]);
  g_plain = a[5];
  g_hooks = a[6];
  Py_RETURN_NONE;
  FAST_END
}

struct NotPlain {};                                    // whatever the step does not cover

PyObject* name_of(const char* text) {
  PyObject* s = PyUnicode_InternFromString(text);
  if (!s) throw python_error();
  return s;
}
#define NAME(text) ([]() { static PyObject* const s = name_of(text); return s; }())

// Reads an object's own attributes: straight from its dictionary, a module's registered tensors and children included.
class Fields {
 public:
  explicit Fields(PyObject* o) : owner_(PyObject_GenericGetDict(o, nullptr)), dict_(owner_.get()) {
    if (dict_) return;
    PyErr_Clear();                                     // (an object without a dictionary)
    throw NotPlain();
  }
  PyObject* find(PyObject* name) const {               // borrowed; null if there is none
    PyObject* v = PyDict_GetItemWithError(dict_, name);
    if (!v && PyErr_Occurred()) throw python_error();
    return v;
  }
  PyObject* get(PyObject* name) const {
    PyObject* v = find(name);
    if (!v) throw NotPlain();
    return v;
  }
  PyObject* in(PyObject* group, PyObject* name) const {   // of _modules, _buffers or _parameters
    PyObject* d = find(group);
    if (!d || !PyDict_Check(d)) return nullptr;
    PyObject* v = PyDict_GetItemWithError(d, name);
    if (!v && PyErr_Occurred()) throw python_error();
    return v;
  }
  PyObject* child(PyObject* name) const {
    PyObject* v = in(NAME("_modules"), name);
    if (!v || find(name)) throw NotPlain();
    return v;
  }
  Tensor tensor(PyObject* name) const {                // attribute, buffer or parameter; undefined if it is None
    PyObject* v = find(name);
    if (!v) v = in(NAME("_buffers"), name);
    if (!v) v = in(NAME("_parameters"), name);
    if (!v) throw NotPlain();
    if (v == Py_None) return Tensor();
    if (!THPVariable_Check(v)) throw NotPlain();
    return THPVariable_Unpack(v);
  }
  bool none(PyObject* name) const {
    PyObject* v = find(name);
    if (!v) v = in(NAME("_modules"), name);
    return v == Py_None;
  }
  int64_t integer(PyObject* name) const {
    PyObject* v = get(name);
    if (!PyLong_CheckExact(v)) throw NotPlain();
    const long long i = PyLong_AsLongLong(v);
    if (i == -1 && PyErr_Occurred()) { PyErr_Clear(); throw NotPlain(); }
    return i;
  }
  double number(PyObject* name) const {
    PyObject* v = get(name);
    if (PyFloat_CheckExact(v)) return PyFloat_AS_DOUBLE(v);
    if (!PyLong_CheckExact(v)) throw NotPlain();
    return PyLong_AsDouble(v);
  }
  bool empty(PyObject* name) const {
    PyObject* v = get(name);
    return PyDict_Check(v) && PyDict_GET_SIZE(v) == 0;
  }
  PyObject* dict() const { return dict_; }

 private:
  THPObjectPtr owner_;
  PyObject* dict_;
};

// obj.name, through the class where the instance has none.
bool flag(PyObject* obj, PyObject* name) {
  THPObjectPtr v(PyObject_GetAttr(obj, name));
  if (!v) throw python_error();
  return bool_arg(v.get());
}

// An object of exactly this class that has none of the class's functions replaced on itself.
Fields plain_object(PyObject* o, PyTypeObject* cls) {
  if (Py_TYPE(o) != cls) throw NotPlain();
  Fields f(o);
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(g_plain); ++i) {
    PyObject* p = PyTuple_GET_ITEM(g_plain, i);
    if (PyTuple_GET_ITEM(p, 0) == reinterpret_cast<PyObject*>(cls) && f.find(PyTuple_GET_ITEM(p, 1))) throw NotPlain();
  }
  return f;
}

// A module whose call is its class's forward and nothing else.
Fields plain_module(PyObject* m, PyTypeObject* cls, bool called = true) {
  Fields f = plain_object(m, cls);
  if (called) {
    PyObject* compiled = f.find(NAME("_compiled_call_impl"));
    if (!f.empty(NAME("_forward_hooks")) || !f.empty(NAME("_forward_pre_hooks")) || !f.empty(NAME("_backward_hooks")) ||
        !f.empty(NAME("_backward_pre_hooks")) || (compiled && compiled != Py_None))
      throw NotPlain();
  }
  return f;
}

// One WQLinear_GEMM whose packed weights are those of its buffers as they are now.
struct PlainLinear {
  PlainLinear(PyObject* m, c10::Device dev) {
    const Fields f = plain_module(m, g_linear);
    PyObject* packed = f.get(NAME("_packed"));
    PyObject* key = f.get(NAME("_packed_key"));
    if (packed == Py_None || !PyTuple_CheckExact(key)) throw NotPlain();
    Key now;
    const Tensor qw = f.tensor(NAME("qweight"));
    if (!qw.defined() || qw.device() != dev) throw NotPlain();
    key_of(qw, now);
    key_of(f.tensor(NAME("qzeros")), now);
    key_of(f.tensor(NAME("scales")), now);
    if ((size_t)PyTuple_GET_SIZE(key) != now.size()) throw NotPlain();
    for (size_t i = 0; i < now.size(); ++i)
      if (PyLong_AsLongLong(PyTuple_GET_ITEM(key, i)) != now[i]) throw NotPlain();
    wq = tensor_of(packed, NAME("wq_t"));
    sz = tensor_of(packed, NAME("sz_t"));
    K = int_of(packed, NAME("K"));
    N = int_of(packed, NAME("N"));
    G = int_of(packed, NAME("G"));
    bias = f.tensor(NAME("bias"));
    if (bias.defined() && (bias.device() != dev || bias.scalar_type() != at::kHalf || bias.numel() != N || !bias.is_contiguous()))
      throw NotPlain();
    if (f.integer(NAME("in_features")) != K || f.integer(NAME("out_features")) != N || K % 32 || G % 32 || N % 8) throw NotPlain();
  }
  void run(const void* x, void* out, int64_t M, Call& c) const {
    check(llmqrt_awq_gemm(x, K, words(wq), words(sz), ptr(bias), out, N, M, N, K, G, c.workspace(), c.stream));
  }
  void run_tail(const void* x, const void* residual, void* out, int64_t M, Call& c) const {
    check(llmqrt_awq_gemm_tail(x, K, words(wq), words(sz), ptr(bias), residual, residual ? N : 0, out, residual ? N : N / 2, M, N,
                               K, G, c.stream));
  }
  Tensor wq, sz, bias;
  int64_t K, N, G;

 private:
  static const uint32_t* words(const Tensor& t) { return static_cast<const uint32_t*>(ptr(t)); }
  static Tensor tensor_of(PyObject* o, PyObject* name) {
    THPObjectPtr v(PyObject_GetAttr(o, name));
    if (!v) throw python_error();
    return tensor_arg(v.get(), "packed weights");
  }
  static int64_t int_of(PyObject* o, PyObject* name) {
    THPObjectPtr v(PyObject_GetAttr(o, name));
    if (!v) throw python_error();
    return int_arg(v.get());
  }
};

struct PlainNorm {
  PlainNorm(PyObject* m, c10::Device dev, int64_t hidden) {
    const Fields f = plain_module(m, g_norm);
    w = f.tensor(NAME("weight"));
    eps = (float)f.number(NAME("variance_epsilon"));
    if (!w.defined() || w.device() != dev || w.scalar_type() != at::kHalf || w.numel() != hidden || !w.is_contiguous()) throw NotPlain();
  }
  void run(const void* x, const void* residual, void* h, void* y, int64_t M, Call& c) const {
    check(llmqrt_rmsnorm(x, residual, h, ptr(w), eps, y, nullptr, nullptr, LLMQRT_F16, M, w.numel(), c.stream));
  }
  Tensor w;
  float eps;
};

Tensor plain_cache(const Fields& cache, PyObject* name, const Tensor& x) {
  const Tensor t = cache.tensor(name);
  if (!t.defined() || t.dim() != 4 || t.scalar_type() != at::kHalf || t.device() != x.device() || t.stride(3) != 1 ||
      t.stride(2) != t.size(3) || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16)
    throw NotPlain();
  return t;
}

// Everything the step reads, gathered before anything is launched.
struct BlockStep {
  BlockStep(PyObject* block, const Tensor& x)
      : me(block), attn_o(me.child(NAME("attn"))), mlp(plain_module(me.child(NAME("mlp")), g_mlp, false)),
        attn(plain_module(attn_o, g_attn, false)), dev(x.device()), B(x.size(0)), hidden(x.size(2)),
        norm1(me.child(NAME("norm_1")), dev, hidden), norm2(me.child(NAME("norm_2")), dev, hidden),
        qkv(attn.child(NAME("qkv_proj")), dev), o(attn.child(NAME("o_proj")), dev), gate_up(mlp.child(NAME("gate_up")), dev),
        down(mlp.child(NAME("down_proj")), dev) {
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(g_plain); ++i) {
      PyObject* p = PyTuple_GET_ITEM(g_plain, i);
      THPObjectPtr now(PyObject_GetAttr(PyTuple_GET_ITEM(p, 0), PyTuple_GET_ITEM(p, 1)));
      if (!now) throw python_error();
      if (now.get() != PyTuple_GET_ITEM(p, 2)) throw NotPlain();
    }
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(g_hooks); ++i)
      if (PyObject_Size(PyTuple_GET_ITEM(g_hooks, i)) != 0) throw NotPlain();
    if (!attn.none(NAME("q_proj")) || !attn.none(NAME("q_norm")) || !attn.none(NAME("k_norm"))) throw NotPlain();
    Hq = attn.integer(NAME("n_heads"));
    Hkv = attn.integer(NAME("n_kv_heads"));
    if (!Hkv) Hkv = Hq;
    d = attn.integer(NAME("head_dim"));
    pos = attn.integer(NAME("start_pos"));
    softcap = (float)attn.number(NAME("attn_logit_softcapping"));
    const Fields cache = plain_object(attn.get(NAME("cache")), g_cache);
    kc = plain_cache(cache, NAME("k"), x);
    vc = plain_cache(cache, NAME("v"), x);
    const Fields rope(attn.child(NAME("rope")));
    cos = rope.tensor(NAME("cos"));
    sin = rope.tensor(NAME("sin"));
    if (attn.integer(NAME("cache_batch_size")) != B || kc.size(0) < B || vc.sizes() != kc.sizes() || vc.strides() != kc.strides() ||
        kc.size(2) != Hkv || kc.size(3) != d || (d != 64 && d != 128) || Hq <= 0 || Hkv <= 0 || Hq % Hkv || pos < 0 || pos >= kc.size(1))
      throw NotPlain();
    for (const Tensor* t : {&cos, &sin})
      if (!t->defined() || t->device() != dev || t->scalar_type() != at::kFloat || t->dim() != 2 || t->size(1) != d / 2 ||
          !t->is_contiguous() || t->size(0) <= pos)
        throw NotPlain();
    if (cos.sizes() != sin.sizes() || qkv.K != hidden || qkv.N != (Hq + 2 * Hkv) * d || o.K != Hq * d || o.N != hidden ||
        gate_up.K != hidden || gate_up.N % 16 || down.K != gate_up.N / 2 || down.N != hidden)
      throw NotPlain();
    twice = flag(attn_o, NAME("REFERENCE_DOUBLE_APPEND")) && pos + 1 < kc.size(1);
    rewind = flag(attn_o, NAME("is_hf_transformers"));
  }

  Tensor run(const Tensor& x0) {
    Call c(dev);
    const Tensor x = x0.contiguous();
    const int64_t M = B, sizes[] = {hidden, qkv.N, o.K, hidden, hidden, hidden, down.K};
    int64_t at[8] = {0};                               // the intermediate results, each on a boundary of 256 bytes
    for (int i = 0; i < 7; ++i) at[i + 1] = at[i] + (M * sizes[i] * 2 + 255) / 256 * 256;
    const Tensor scratch = empty(x, {at[7]}, at::kByte);
    Tensor out = empty(x, {B, 1, hidden}, at::kHalf);
    uint8_t* base = static_cast<uint8_t*>(scratch.data_ptr());
    auto* y1 = base + at[0]; auto* p = base + at[1]; auto* w = base + at[2]; auto* ao = base + at[3];
    auto* h = base + at[4]; auto* y2 = base + at[5]; auto* g = base + at[6];
    norm1.run(ptr(x), nullptr, nullptr, y1, M, c);
    qkv.run(y1, p, M, c);
    const int64_t len = pos + (twice ? 2 : 1);
    check(llmqrt_attn_decode_step(p, B > 1 ? qkv.N : Hq * d, p + Hq * d * 2, p + (Hq + Hkv) * d * 2, B > 1 ? qkv.N : Hkv * d,
                                  static_cast<const float*>(ptr(cos)), static_cast<const float*>(ptr(sin)), cos.size(0), twice ? 1 : 0,
                                  mptr(kc), mptr(vc), kc.stride(0), kc.stride(1), kc.size(1), nullptr, (int32_t)len, w, LLMQRT_F16, B,
                                  Hq, Hkv, d, std::min(len, kc.size(1)), softcap, c.workspace(), c.stream));
    o.run(w, ao, M, c);
    norm2.run(ptr(x), ao, h, y2, M, c);
    gate_up.run_tail(y2, nullptr, g, M, c);
    down.run_tail(g, h, mptr(out), M, c);
    return out;
  }
  void advance() {
    THPObjectPtr next(PyLong_FromLongLong(rewind ? 0 : pos + 1));
    if (!next || PyDict_SetItem(attn.dict(), NAME("start_pos"), next.get()) < 0) throw python_error();
  }

  Fields me;
  PyObject* attn_o;
  Fields mlp, attn;
  c10::Device dev;
  int64_t B, hidden;
  PlainNorm norm1, norm2;
  PlainLinear qkv, o, gate_up, down;
  int64_t Hq, Hkv, d, pos;
  float softcap;
  Tensor kc, vc, cos, sin;
  bool twice, rewind;
};

// (block, hidden_states [B, 1, hidden]) -> the block's output and its start_pos moved on, or None.
FAST_FN(awq_block_step) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_TYPE(n == 2, "llmqrt_b200: expected 2 arguments, got ", (int64_t)n);
  if (!g_plain || !THPVariable_CheckExact(a[1])) Py_RETURN_NONE;
  const Tensor x = THPVariable_Unpack(a[1]);
  if (!x.is_cuda() || x.scalar_type() != at::kHalf || x.dim() != 3 || x.size(1) != 1 || x.size(0) < 1 || x.size(0) > 16 ||
      (at::GradMode::is_enabled() && x.requires_grad()))
    Py_RETURN_NONE;
  at::NoGradGuard no_grad;
  std::optional<BlockStep> step;
  try {
    step.emplace(a[0], x);
  } catch (const NotPlain&) {
    Py_RETURN_NONE;
  }
  Tensor out;
  {
    GilRelease gil;
    out = step->run(x);
  }
  step->advance();
  return wrap(out);
  FAST_END
}

FAST_FN(set_workspace_maker) {
  FAST_BEGIN(1)
  Py_INCREF(a[0]);
  Py_XSETREF(g_make_workspace, a[0]);
  Py_RETURN_NONE;
  FAST_END
}

#define FAST_DEF(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST_DEF(sq_per_channel), FAST_DEF(sq_per_tensor), FAST_DEF(fp8_per_token), FAST_DEF(fp8_per_tensor),
                         FAST_DEF(awq_linear), FAST_DEF(awq_tail), FAST_DEF(rmsnorm), FAST_DEF(silu_mul), FAST_DEF(rope_kv_write),
                         FAST_DEF(attn_prefill), FAST_DEF(kv_append), FAST_DEF(attn_decode), FAST_DEF(attn_decode_step), FAST_DEF(tensor_key),
                         FAST_DEF(set_block_classes), FAST_DEF(awq_block_step),
                         FAST_DEF(set_workspace_maker), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fast", "Native host path of llmqrt_b200.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fast() { return PyModule_Create(&module); }
