// PyTorch side of the library: argument checks, allocation, the autograd node and the calls
// into the C ABI (include/fa_sm100.h), all in C++.
//
// What bounds small problems is the host: through a Python autograd.Function and ctypes a
// forward + backward of a (2, 128, 4, 64) problem took 167 us of interpreter time next to 16 us
// of kernels.  Here the forward is one C call and the backward a native graph node, which runs
// in the autograd engine's own thread without the interpreter lock.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/FuncTorchTLS.h>
#include <ATen/SavedTensorHooks.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <mutex>
#include <string>
#include <tuple>

#include "../../include/fa_sm100.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// ---------------------------------------------------------------------------- errors
// An argument error with the Python exception type the public interface promises.
struct ArgError : public std::exception {
  PyObject* type;
  std::string msg;
  ArgError(PyObject* t, std::string m) : type(t), msg(std::move(m)) {}
  const char* what() const noexcept override { return msg.c_str(); }
};
[[noreturn]] void fail(PyObject* type, std::string msg) { throw ArgError(type, std::move(msg)); }

void check_code(int code, const char* what) {
  if (code != FA_OK)
    throw std::runtime_error(std::string(what) + " failed: " + fa_status_string(code) + " (code " +
                             std::to_string(code) + ")");
}

// ---------------------------------------------------------------------------- device health
// Host copies of the per-device status words (pinned memory that the Python side owns and
// registers on first use): a kernel that abandoned a wait wrote its record there, and every call
// looks before it launches.
constexpr int kMaxDevices = 64;
std::atomic<const volatile int32_t*> g_health[kMaxDevices];
PyObject* g_register_health = nullptr;  // callable(device) -> address

void require_health_words(int device) {  // interpreter lock held
  if (device < 0 || device >= kMaxDevices || g_health[device].load(std::memory_order_acquire)) return;
  PyObject* r = PyObject_CallFunction(g_register_health, "i", device);
  if (!r) throw python_error();
  const unsigned long long addr = PyLong_AsUnsignedLongLong(r);
  Py_DECREF(r);
  if (PyErr_Occurred()) throw python_error();
  g_health[device].store(reinterpret_cast<const volatile int32_t*>(addr), std::memory_order_release);
}

void raise_if_unhealthy(int device) {
  if (device < 0 || device >= kMaxDevices) return;
  const volatile int32_t* w = g_health[device].load(std::memory_order_acquire);
  if (w && w[0] != 0)
    throw std::runtime_error("a kernel on cuda:" + std::to_string(device) + " abandoned a bounded wait (kernel " +
                             std::to_string(w[1]) + ", block " + std::to_string(w[2]) + ", site " +
                             std::to_string(w[4]) + ", iteration " + std::to_string(w[5]) +
                             "); later kernels do no work until _cabi.reset_device_status() is called");
}

// ---------------------------------------------------------------------------- operands
// A (B, S, H, D) operand as the kernels take it: address and the strides over B, S, H.
struct View {
  void* ptr;
  int64_t s[3];
};

bool strides_ok(int64_t s0, int64_t s1, int64_t s2, int64_t s3, const void* ptr) {
  return s3 == 1 && s0 > 0 && s1 > 0 && s2 > 0 && (s0 | s1 | s2) % 8 == 0 &&
         reinterpret_cast<uintptr_t>(ptr) % 16 == 0;
}
bool tile_ok(const Tensor& t) {
  const auto st = t.strides();
  return strides_ok(st[0], st[1], st[2], st[3], t.const_data_ptr());
}
// Unit inner stride, every other stride and the base address a multiple of 16 bytes; copies only
// when needed.
Tensor tile_ready(const Tensor& t) { return tile_ok(t) ? t : t.contiguous(); }

View view_of(const Tensor& t) {
  const auto st = t.strides();
  return View{const_cast<void*>(t.const_data_ptr()), {st[0], st[1], st[2]}};
}
// q, k or v inside a (B, S, 3, H, D) tensor
View slice_of(const Tensor& qkv, int i) {
  const auto st = qkv.strides();
  return View{static_cast<char*>(const_cast<void*>(qkv.const_data_ptr())) + i * st[2] * 2, {st[0], st[1], st[3]}};
}

void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream(); }

Tensor empty_on(const Tensor& like, at::IntArrayRef size, at::ScalarType dtype) {
  return at::detail::empty_cuda(size, dtype, like.device(), std::nullopt);
}

// (B, H, M, N) tensor whose row pitch is a multiple of 16 bytes: dense when N allows it, else a
// view of a padded buffer.
Tensor pitched_empty(const Tensor& like, at::IntArrayRef size, at::ScalarType dtype, bool zero) {
  const int64_t per16 = 16 / static_cast<int64_t>(at::elementSize(dtype));
  const int64_t n_pad = (size[3] + per16 - 1) / per16 * per16;
  Tensor buf = empty_on(like, {size[0], size[1], size[2], n_pad}, dtype);
  if (zero) buf.zero_();
  return n_pad == size[3] ? buf : buf.narrow(3, 0, size[3]);
}

// What the tile kernels need of a bias: unit inner stride, 16-byte aligned pitches and address.
bool bias_ok(const Tensor& bias) {
  const int64_t eb = static_cast<int64_t>(bias.element_size());
  const auto st = bias.strides();
  return st[3] == 1 && st[2] > 0 && (st[0] * eb) % 16 == 0 && (st[1] * eb) % 16 == 0 && (st[2] * eb) % 16 == 0 &&
         reinterpret_cast<uintptr_t>(bias.const_data_ptr()) % 16 == 0;
}

// Bias / mask with unit inner stride and 16-byte aligned pitches.  Expanded views (stride 0 over B
// or H) pass through untouched.  Otherwise a copy is made, with its rows padded to 32 bytes (the
// kernels then fetch whole sectors) and its expanded B and H dimensions kept folded: a key-padding
// mask (B, 1, 1, N) expanded over heads and rows is written once per batch element, not per head.
Tensor bias_ready(const Tensor& bias) {
  if (bias_ok(bias)) return bias;
  const auto st = bias.strides();
  const auto sz = bias.sizes();
  const int64_t align = 32 / static_cast<int64_t>(bias.element_size());
  const int64_t n_pad = (sz[3] + align - 1) / align * align;
  const int64_t b = st[0] == 0 ? 1 : sz[0], h = st[1] == 0 ? 1 : sz[1];
  Tensor out = empty_on(bias, {b, h, sz[2], n_pad}, bias.scalar_type()).narrow(3, 0, sz[3]);
  const int eb = static_cast<int>(bias.element_size());
  if (st[3] != 1 || eb > 4 || sz[2] > INT32_MAX || sz[3] > INT32_MAX ||
      fa_pad_rows(out.mutable_data_ptr(), out.strides().data(), bias.const_data_ptr(), st.data(), eb, static_cast<int>(b),
                  static_cast<int>(h), static_cast<int>(sz[2]), static_cast<int>(sz[3]), bias.get_device(),
                  stream_of(bias.get_device())) != FA_OK)
    out.copy_(bias.narrow(0, 0, b).narrow(1, 0, h));  // another inner stride, or too large for it
  return out.expand(sz);
}

struct Shape {
  int64_t B, M, N, H, D;
  at::ScalarType dtype;
  int device;
};

struct Bias {
  Tensor t;  // what the kernels read; undefined without a bias
  int kind = FA_BIAS_NONE;
};

// `any_layout`: the reader takes it with any strides but the innermost
Bias classify_bias(const Tensor& bias, at::ScalarType q_dtype, bool any_layout = false) {
  if (!bias.defined()) return {};
  const auto dt = bias.scalar_type();
  const auto ready = [&](const Tensor& t) { return any_layout && t.stride(3) == 1 ? t : bias_ready(t); };
  if (dt == at::kBool) return {ready(bias), FA_BIAS_BOOL};
  if (!at::isFloatingType(dt))
    fail(PyExc_TypeError, std::string("bias must be a bool or floating tensor, got ") + toString(dt));
  if (dt == q_dtype) return {ready(bias), FA_BIAS_SAME};
  // Any other float dtype is streamed as fp32 (the reference also adds the bias in fp32,
  // flash_attention.py 52, 292): nothing is rounded to 16 bits, the gradient comes back in fp32.
  return {ready(dt == at::kFloat ? bias : bias.to(at::kFloat)), FA_BIAS_F32};
}
// Short sequences: the kernels read the bias and write its gradient in any layout.
bool is_small(const Shape& s) {
  return fa_small_takes(static_cast<int>(s.M), static_cast<int>(s.N), static_cast<int>(s.D)) != 0;
}
bool few_rows(const Shape& s) { return fa_fwd_takes_any_bias(static_cast<int>(s.M), static_cast<int>(s.D)) != 0; }
Bias forward_bias(const Shape& s, const Tensor& bias) { return classify_bias(bias, s.dtype, few_rows(s) || is_small(s)); }

// ---------------------------------------------------------------------------- argument checks
std::string shape_text(at::IntArrayRef s) {
  std::string t = "(";
  for (size_t i = 0; i < s.size(); ++i) t += (i ? ", " : "") + std::to_string(s[i]);
  return t + (s.size() == 1 ? ",)" : ")");
}

void check_bias(const Shape& s, const Tensor& bias, const Tensor& q) {
  if (!bias.defined()) return;
  const int64_t want[4] = {s.B, s.H, s.M, s.N};
  if (bias.sizes() != at::IntArrayRef(want, 4))
    fail(PyExc_ValueError, "bias must have shape (B, H, M, N) = " + shape_text(at::IntArrayRef(want, 4)) + ", got " +
                               shape_text(bias.sizes()));
  if (bias.device() != q.device()) fail(PyExc_ValueError, "bias must live on q's device");
}

void check_head_dim(int64_t D) {
  if (D != 16 && D != 32 && D != 64 && D != 128 && D != 256)
    fail(PyExc_AssertionError, "head dimension must be one of 16, 32, 64, 128, 256");
}
void check_dtype(at::ScalarType a, at::ScalarType b, at::ScalarType c) {
  if ((a != at::kHalf && a != at::kBFloat16) || b != a || c != a)
    fail(PyExc_TypeError, "q, k, v must share one dtype: torch.float16 or torch.bfloat16");
}

Shape check_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& bias) {
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4)
    fail(PyExc_ValueError, "q, k, v must be 4-D: (B, M, H, D) / (B, N, H, D)");
  const Shape s{q.size(0), q.size(1), k.size(1), q.size(2), q.size(3), q.scalar_type(),
                q.is_cuda() ? q.get_device() : -1};
  if (k.size(3) != s.D) fail(PyExc_AssertionError, "q and k must share the head dimension");
  check_head_dim(s.D);
  if (v.sizes() != k.sizes())
    fail(PyExc_ValueError, "v must have the shape of k (value head dim == query/key head dim)");
  if (k.size(0) != s.B || k.size(2) != s.H) fail(PyExc_ValueError, "q and k/v disagree on batch or heads");
  check_dtype(s.dtype, k.scalar_type(), v.scalar_type());
  if (!q.is_cuda() || k.device() != q.device() || v.device() != q.device())
    fail(PyExc_ValueError, "q, k, v must live on the same CUDA device (there is no CPU path)");
  check_bias(s, bias, q);
  return s;
}

Shape check_packed(const Tensor& qkv, const Tensor& bias) {
  if (qkv.dim() != 5 || qkv.size(2) != 3) fail(PyExc_ValueError, "qkv must be (B, S, 3, H, D)");
  const Shape s{qkv.size(0), qkv.size(1), qkv.size(1), qkv.size(3), qkv.size(4), qkv.scalar_type(),
                qkv.is_cuda() ? qkv.get_device() : -1};
  check_head_dim(s.D);
  check_dtype(s.dtype, s.dtype, s.dtype);
  if (!qkv.is_cuda()) fail(PyExc_ValueError, "q, k, v must live on the same CUDA device (there is no CPU path)");
  check_bias(s, bias, qkv);
  return s;
}

// qkv such that its three slices are tile ready.  (A copy and not contiguous(): a dense tensor may lie at an address
// that is no multiple of 16 bytes.)
Tensor packed_ready(const Tensor& qkv) {
  const auto st = qkv.strides();
  if (strides_ok(st[0], st[1], st[3], st[4], qkv.const_data_ptr()) && st[2] % 8 == 0) return qkv;
  return qkv.clone(at::MemoryFormat::Contiguous);
}

// ---------------------------------------------------------------------------- C ABI calls
void set_stride(int64_t (&dst)[3], const int64_t* src) {
  for (int i = 0; i < 3; ++i) dst[i] = src[i];
}

fa_params common_params(const Shape& s, const View& q, const View& k, const View& v, const View& o, const Tensor& lse,
                        const Bias& bias, bool causal, double scale) {
  fa_params p{};
  p.struct_size = sizeof(fa_params);
  p.device = s.device;
  p.B = static_cast<int32_t>(s.B);
  p.H = static_cast<int32_t>(s.H);
  p.M = static_cast<int32_t>(s.M);
  p.N = static_cast<int32_t>(s.N);
  p.D = static_cast<int32_t>(s.D);
  p.dtype = s.dtype == at::kBFloat16 ? FA_BF16 : FA_F16;
  p.bias_kind = bias.kind;
  p.causal = causal ? 1 : 0;
  p.sm_scale = static_cast<float>(scale);
  p.q = q.ptr;
  p.k = k.ptr;
  p.v = v.ptr;
  p.o = o.ptr;
  set_stride(p.q_stride, q.s);
  set_stride(p.k_stride, k.s);
  set_stride(p.v_stride, v.s);
  set_stride(p.o_stride, o.s);
  p.lse = lse.mutable_data_ptr<float>();
  if (bias.t.defined()) {
    p.bias = const_cast<void*>(bias.t.const_data_ptr());
    set_stride(p.bias_stride, bias.t.strides().data());
  }
  return p;
}

// Forward launch: (out (B, M, H, D), log2-domain log-sum-exp (B, H, M) fp32).  Replaces
// _flash_attn_fwd of the reference (flash_attention.py 649-685).
std::tuple<Tensor, Tensor> forward(const Shape& s, const Tensor& like, const View& q, const View& k, const View& v,
                                   const Bias& bias, bool causal, double scale) {
  raise_if_unhealthy(s.device);
  Tensor o = empty_on(like, {s.B, s.M, s.H, s.D}, s.dtype);
  Tensor lse = empty_on(like, {s.B, s.H, s.M}, at::kFloat);
  const fa_params p = common_params(s, q, k, v, view_of(o), lse, bias, causal, scale);
  check_code(!few_rows(s) && is_small(s) ? fa_small_fwd(&p, stream_of(s.device)) : fa_fwd(&p, stream_of(s.device)), "fa_fwd");
  return {std::move(o), std::move(lse)};
}

// Backward launches; fills dq, dk, dv and - when defined - dbias.  Replaces _flash_attn_bwd of the
// reference (flash_attention.py 688-763).  `any_layout`: the bias and dbias may be laid out as only the kernels for
// short sequences take them (these sequences are).
void backward(const Shape& s, const Tensor& grad, const View& q, const View& k, const View& v, const Tensor& out,
              const Tensor& lse, const Bias& bias, bool causal, double scale, const View& dq, const View& dk,
              const View& dv, const Tensor& dbias, bool any_layout) {
  raise_if_unhealthy(s.device);
  const Tensor o = tile_ready(out), g = tile_ready(grad);
  Tensor delta = empty_on(o, {s.B, s.H, s.M}, at::kFloat);
  fa_params p = common_params(s, q, k, v, view_of(o), lse, bias, causal, scale);
  const View gv = view_of(g);
  p.d_o = gv.ptr;
  set_stride(p.do_stride, gv.s);
  p.dq = dq.ptr;
  p.dk = dk.ptr;
  p.dv = dv.ptr;
  set_stride(p.dq_stride, dq.s);
  set_stride(p.dk_stride, dk.s);
  set_stride(p.dv_stride, dv.s);
  p.delta = delta.mutable_data_ptr<float>();
  if (dbias.defined()) {
    p.write_dbias = 1;
    p.dbias = dbias.mutable_data_ptr();
    set_stride(p.dbias_stride, dbias.strides().data());
  }
  if (any_layout) {
    check_code(fa_small_bwd(&p, stream_of(s.device)), "fa_bwd");
    return;
  }
  // Scratch for dS where it has no tensor of its own.  Without the memory for all the library asks
  // for, one problem's share; without that, the scores are recomputed where the kernels can.
  uint64_t bytes = fa_bwd_workspace_bytes(&p);
  Tensor ws;
  if (bytes > 0) {
    const uint64_t one = static_cast<uint64_t>((s.N + 7) / 8 * 8 * s.M * 2);
    try {
      ws = empty_on(o, {static_cast<int64_t>(bytes)}, at::kByte);
    } catch (const c10::OutOfMemoryError&) {
      bytes = one;
      try {
        ws = empty_on(o, {static_cast<int64_t>(bytes)}, at::kByte);
      } catch (const c10::OutOfMemoryError&) {
        if (s.D == 256 || bias.kind == FA_BIAS_F32) throw;
        bytes = 0;
      }
    }
  }
  check_code(fa_bwd_workspace(&p, bytes ? ws.mutable_data_ptr() : nullptr, bytes, stream_of(s.device)), "fa_bwd");
}

// empty_like (strides preserved, as the reference's flash_attention.py 796-798) when the kernels
// can write through those strides, else a dense tensor
Tensor grad_like(const Tensor& t) {
  if (t.is_contiguous()) return empty_on(t, t.sizes(), t.scalar_type());
  Tensor g = at::empty_like(t);
  return tile_ok(g) ? g : empty_on(t, t.sizes(), t.scalar_type());
}

// Gradient buffer for the bias as the kernels write it: q's dtype when the bias has it, else fp32.
// Zero-filled where the kernels skip the causally masked tiles without writing them (fp32
// gradients; every gradient at head dim 256).
Tensor new_dbias(const Shape& s, const Tensor& bias, bool causal) {
  const bool same = bias.scalar_type() == s.dtype;
  if (is_small(s)) return empty_on(bias, {s.B, s.H, s.M, s.N}, same ? s.dtype : at::kFloat);  // dense, all of it is written
  return pitched_empty(bias, {s.B, s.H, s.M, s.N}, same ? s.dtype : at::kFloat, causal && (!same || s.D == 256));
}
// Gradient as the reference returns it (flash_attention.py 799): dense, in the bias's own dtype.
Tensor finish_dbias(const Tensor& dbias, at::ScalarType dtype) {
  if (dbias.scalar_type() != dtype) return dbias.to(dtype);  // also compacts a padded buffer
  if (dbias.is_contiguous()) return dbias;
  const auto sz = dbias.sizes();
  Tensor out = empty_on(dbias, sz, dtype);
  if (sz[3] > INT32_MAX ||
      fa_pack_rows(out.mutable_data_ptr(), dbias.const_data_ptr(), dbias.stride(2), static_cast<int>(dbias.element_size()),
                   sz[0] * sz[1] * sz[2], static_cast<int>(sz[3]), dbias.get_device(), stream_of(dbias.get_device())) != FA_OK)
    out.copy_(dbias);
  return out;
}

// ---------------------------------------------------------------------------- autograd
// A copy of the bias that the forward had to make is kept for the backward up to this size; a larger
// one is made again there, so that many layers do not hold two copies of a big bias each.  Under
// saved-tensor hooks (checkpointing, offloading) none is kept: what the hooks see is all that stays.
constexpr int64_t kKeepBiasCopyBytes = 64ll << 20;

// Backward node of one attention call: inputs (q, k, v, bias), or (qkv, bias) when packed.
struct AttentionBackward : public torch::autograd::Node {
  SavedVariable a_, k_, v_, bias_, out_, lse_;  // a_: q, or qkv
  Tensor bias_copy_;                            // the padded copy made in forward, if any
  bool packed_ = false, causal_ = false, has_bias_ = false, train_bias_ = false;
  double scale_ = 1.0;

  std::string name() const override { return packed_ ? "FlashAttentionQKVPackedFnBackward" : "FlashAttentionFnBackward"; }

  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    a_.reset_data();
    k_.reset_data();
    v_.reset_data();
    bias_.reset_data();
    out_.reset_data();
    lse_.reset_data();
    bias_copy_.reset();
  }

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list res(packed_ ? 2 : 4);
    const Tensor a0 = a_.unpack(), out = out_.unpack(shared_from_this()), lse = lse_.unpack();
    const Tensor bias = has_bias_ ? bias_.unpack() : Tensor();
    at::AutoDispatchBelowADInplaceOrView guard;
    // an upstream function that returned no gradient counts as zeros, as for a Python autograd function
    const Tensor grad = grads[0].defined() ? grads[0] : at::zeros_like(out);
    const auto bias_for = [&](at::ScalarType dt, bool any_layout) {
      return bias_copy_.defined() ? Bias{bias_copy_, bias.scalar_type() == at::kBool ? FA_BIAS_BOOL
                                                     : bias.scalar_type() == dt      ? FA_BIAS_SAME
                                                                                     : FA_BIAS_F32}
                                  : classify_bias(bias, dt, any_layout);
    };
    if (packed_) {
      const Shape s = check_packed(a0, bias);
      const c10::cuda::CUDAGuard device(static_cast<c10::DeviceIndex>(s.device));
      const Tensor qkv = packed_ready(a0);
      Tensor dqkv = empty_on(qkv, qkv.sizes(), s.dtype);
      Tensor dbias = train_bias_ ? new_dbias(s, bias, causal_) : Tensor();
      backward(s, grad, slice_of(qkv, 0), slice_of(qkv, 1), slice_of(qkv, 2), out, lse, bias_for(s.dtype, is_small(s)),
               causal_, scale_, slice_of(dqkv, 0), slice_of(dqkv, 1), slice_of(dqkv, 2), dbias, is_small(s));
      res[0] = std::move(dqkv);
      if (train_bias_) res[1] = finish_dbias(dbias, bias.scalar_type());
      return res;
    }
    const Tensor k0 = k_.unpack(), v0 = v_.unpack();
    const Shape s = check_inputs(a0, k0, v0, bias);
    const c10::cuda::CUDAGuard device(static_cast<c10::DeviceIndex>(s.device));
    const Tensor q = tile_ready(a0), k = tile_ready(k0), v = tile_ready(v0);
    Tensor dq = grad_like(a0), dk = grad_like(k0), dv = grad_like(v0);
    Tensor dbias = train_bias_ ? new_dbias(s, bias, causal_) : Tensor();
    backward(s, grad, view_of(q), view_of(k), view_of(v), out, lse, bias_for(s.dtype, is_small(s)), causal_, scale_,
             view_of(dq), view_of(dk), view_of(dv), dbias, is_small(s));
    res[0] = std::move(dq);
    res[1] = std::move(dk);
    res[2] = std::move(dv);
    if (train_bias_) res[3] = finish_dbias(dbias, bias.scalar_type());
    return res;
  }
};

double scale_of(PyObject* obj, int64_t D) {
  if (obj == Py_None) return 1.0 / std::sqrt(static_cast<double>(D));
  THPObjectPtr number(PyNumber_Float(obj));  // whatever float() takes
  if (!number) throw python_error();
  return PyFloat_AsDouble(number.get());
}

// One attention call with its graph node when a gradient is wanted.  `k`, `v` undefined: packed.
Tensor attention(const Tensor& a, const Tensor& k, const Tensor& v, const Tensor& bias, bool causal, PyObject* scale_obj) {
  // No rule for torch.func transforms exists either (RuntimeError): under one, what looks like a plain tensor may be
  // a batch or a differentiation level of its own.
  if (const auto& transforms = at::functorch::functorchTLSAccessor()) transforms->checkSupportsCppAutogradFunction();
  const bool packed = !k.defined();
  const bool train_bias = bias.defined() && bias.requires_grad();
  if (train_bias && bias.scalar_type() == at::kBool) fail(PyExc_TypeError, "a bool mask cannot require grad");
  // The node has no forward-mode rule; without this the tangents would be dropped silently.
  for (const Tensor* t : {&a, &k, &v, &bias})
    if (t->defined() && t->_fw_grad(0).defined())
      fail(PyExc_NotImplementedError, "attention has no forward-mode derivative (jvp)");
  const Shape s = packed ? check_packed(a, bias) : check_inputs(a, k, v, bias);
  const double scale = scale_of(scale_obj, s.D);
  require_health_words(s.device);

  pybind11::gil_scoped_release no_gil;
  const c10::cuda::CUDAGuard device(static_cast<c10::DeviceIndex>(s.device));
  const bool wants_grad = at::GradMode::is_enabled() &&
                          (a.requires_grad() || train_bias || (!packed && (k.requires_grad() || v.requires_grad())));
  Tensor out, lse;
  Bias b;
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    b = forward_bias(s, bias);
    if (packed) {
      const Tensor t = packed_ready(a);
      std::tie(out, lse) = forward(s, t, slice_of(t, 0), slice_of(t, 1), slice_of(t, 2), b, causal, scale);
    } else {
      const Tensor tq = tile_ready(a), tk = tile_ready(k), tv = tile_ready(v);
      std::tie(out, lse) = forward(s, tq, view_of(tq), view_of(tk), view_of(tv), b, causal, scale);
    }
  }
  if (!wants_grad) return out;
  auto node = std::shared_ptr<AttentionBackward>(new AttentionBackward(), torch::autograd::deleteNode);
  if (packed)
    node->set_next_edges(torch::autograd::collect_next_edges(a, bias));
  else
    node->set_next_edges(torch::autograd::collect_next_edges(a, k, v, bias));
  node->packed_ = packed;
  node->causal_ = causal;
  node->scale_ = scale;
  node->has_bias_ = bias.defined();
  node->train_bias_ = train_bias;
  node->a_ = SavedVariable(a, false);
  if (!packed) {
    node->k_ = SavedVariable(k, false);
    node->v_ = SavedVariable(v, false);
  }
  if (bias.defined()) {
    node->bias_ = SavedVariable(bias, false);
    // (a converted bias that only the kernel for few rows can read is made again for the backward)
    if (!b.t.is_same(bias) && (bias_ok(b.t) || is_small(s)) && static_cast<int64_t>(b.t.storage().nbytes()) <= kKeepBiasCopyBytes &&
        !at::SavedTensorDefaultHooks::get_hooks().has_value())
      node->bias_copy_ = std::move(b.t);
  }
  node->lse_ = SavedVariable(lse, false);
  torch::autograd::set_history(out, node);
  node->out_ = SavedVariable(out, true);
  return out;
}

// ---------------------------------------------------------------------------- Python entry points
Tensor tensor_arg(PyObject* o, const char* name, bool optional = false) {
  if (optional && o == Py_None) return Tensor();
  if (!THPVariable_Check(o))
    fail(PyExc_TypeError, std::string(name) + " must be a torch.Tensor, got " + Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
bool truth(PyObject* o) {
  const int r = PyObject_IsTrue(o);
  if (r < 0) throw python_error();
  return r != 0;
}
void want_args(Py_ssize_t n, Py_ssize_t want, const char* name) {
  if (n != want)
    fail(PyExc_TypeError, std::string(name) + " takes " + std::to_string(want) + " arguments, got " + std::to_string(n));
}

// Runs `f` with C++ exceptions turned into Python ones.
template <typename F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const ArgError& e) {
    PyErr_SetString(e.type, e.msg.c_str());
    return nullptr;
  } catch (python_error& e) {
    e.restore();
    return nullptr;
  } catch (const c10::Error& e) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// attention(q, k, v, bias | None, causal, sm_scale | None) -> out
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    want_args(n, 6, "attention");
    return THPVariable_Wrap(attention(tensor_arg(a[0], "q"), tensor_arg(a[1], "k"), tensor_arg(a[2], "v"),
                                      tensor_arg(a[3], "bias", true), truth(a[4]), a[5]));
  });
}

// attention_packed(qkv, bias | None, causal, sm_scale | None) -> out
PyObject* py_attention_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    want_args(n, 4, "attention_packed");
    return THPVariable_Wrap(attention(tensor_arg(a[0], "qkv"), Tensor(), Tensor(), tensor_arg(a[1], "bias", true),
                                      truth(a[2]), a[3]));
  });
}

// fwd(q, k, v, bias | None, causal, sm_scale) -> (out, lse2), no autograd
PyObject* py_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    want_args(n, 6, "fwd");
    const Tensor q0 = tensor_arg(a[0], "q"), k0 = tensor_arg(a[1], "k"), v0 = tensor_arg(a[2], "v");
    const Tensor bias = tensor_arg(a[3], "bias", true);
    const bool causal = truth(a[4]);
    const Shape s = check_inputs(q0, k0, v0, bias);
    const double scale = scale_of(a[5], s.D);
    require_health_words(s.device);
    const c10::cuda::CUDAGuard device(static_cast<c10::DeviceIndex>(s.device));
    at::AutoDispatchBelowADInplaceOrView guard;
    const Tensor q = tile_ready(q0), k = tile_ready(k0), v = tile_ready(v0);
    Tensor out, lse;
    std::tie(out, lse) =
        forward(s, q, view_of(q), view_of(k), view_of(v), forward_bias(s, bias), causal, scale);
    return PyTuple_Pack(2, THPObjectPtr(THPVariable_Wrap(out)).get(), THPObjectPtr(THPVariable_Wrap(lse)).get());
  });
}

// bwd(do, q, k, v, o, bias | None, causal, sm_scale, lse, dq, dk, dv, dbias | None): fills the gradients
PyObject* py_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want_args(n, 13, "bwd");
    const Tensor g = tensor_arg(a[0], "do"), q0 = tensor_arg(a[1], "q"), k0 = tensor_arg(a[2], "k");
    const Tensor v0 = tensor_arg(a[3], "v"), o = tensor_arg(a[4], "o"), bias = tensor_arg(a[5], "bias", true);
    const bool causal = truth(a[6]);
    const Tensor lse = tensor_arg(a[8], "lse"), dq = tensor_arg(a[9], "dq"), dk = tensor_arg(a[10], "dk");
    const Tensor dv = tensor_arg(a[11], "dv"), dbias = tensor_arg(a[12], "dbias", true);
    const Shape s = check_inputs(q0, k0, v0, bias);
    const double scale = scale_of(a[7], s.D);
    require_health_words(s.device);
    const c10::cuda::CUDAGuard device(static_cast<c10::DeviceIndex>(s.device));
    at::AutoDispatchBelowADInplaceOrView guard;
    const Tensor q = tile_ready(q0), k = tile_ready(k0), v = tile_ready(v0);
    // (the caller's gradient has to meet the tile kernels' rule at any size)
    const bool any_layout = is_small(s) && (!dbias.defined() || bias_ok(dbias));
    backward(s, g, view_of(q), view_of(k), view_of(v), o, lse, classify_bias(bias, s.dtype, any_layout), causal, scale,
             view_of(dq), view_of(dk), view_of(dv), dbias, any_layout);
    Py_RETURN_NONE;
  });
}

// classify_bias(bias | None, q) -> (tensor the kernels read | None, kind)
PyObject* py_classify_bias(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    want_args(n, 2, "classify_bias");
    const Tensor bias = tensor_arg(a[0], "bias", true), q = tensor_arg(a[1], "q");
    at::NoGradGuard no_grad;
    const Bias b = classify_bias(bias, q.scalar_type());
    return Py_BuildValue("(Ni)", THPVariable_Wrap(b.t), b.kind);  // an undefined tensor becomes None
  });
}

// set_health_registrar(callable(device) -> address of the int32[8] host words)
PyObject* py_set_health_registrar(PyObject*, PyObject* cb) {
  Py_INCREF(cb);
  Py_XDECREF(g_register_health);
  g_register_health = cb;
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_attention)), METH_FASTCALL, nullptr},
    {"attention_packed", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_attention_packed)), METH_FASTCALL, nullptr},
    {"fwd", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_fwd)), METH_FASTCALL, nullptr},
    {"bwd", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_bwd)), METH_FASTCALL, nullptr},
    {"classify_bias", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_classify_bias)), METH_FASTCALL, nullptr},
    {"set_health_registrar", py_set_health_registrar, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fa_torch", "Native launch path of the attention kernels.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fa_torch(void) { return PyModule_Create(&kModule); }
