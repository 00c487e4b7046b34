// Host path of the public operators in C++: argument checks, output allocation, autograd node and the call into the
// C ABI (include/b200attn.h) for the ordinary call of flash_attention (no dropout, no auxiliary results),
// flash_attention_split_kv and paged_attention. Small calls are bound by host work: the same steps in Python
// (autograd.Function, ctypes structures, stride loops) took about 35 us for a forward whose kernel takes 6 us.
//
// Every entry returns None when the call is not an ordinary one (a copy is needed first, an argument is wrong, a tensor
// subclass, a functorch transform, a dispatch mode or a tracer is active, ...); the Python implementation then handles
// it or raises what it has always raised.
#include <ATen/ATen.h>
#include <ATen/FuncTorchTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <chrono>
#include <cmath>
#include <optional>

#include "../../include/b200attn.h"

namespace {

// Entry points of libb200attn.so, handed over by the loader that opened it (bind() below).
struct Api {
  decltype(&b200attn_fwd) fwd = nullptr;
  decltype(&b200attn_bwd_stages) bwd_stages = nullptr;
  decltype(&b200attn_bwd_workspace_bytes) bwd_workspace_bytes = nullptr;
  decltype(&b200attn_fwd_splitkv) fwd_splitkv = nullptr;
  decltype(&b200attn_splitkv_num_splits) splitkv_num_splits = nullptr;
  decltype(&b200attn_paged_attention) paged = nullptr;
  decltype(&b200attn_last_error) last_error = nullptr;
} api;
PyObject* poll_fn = nullptr;  // status.poll_pointer(device index) -> address of the device's status word

void check(int rc, const char* what) {
  static const char* names[] = {"OK", "EINVAL", "EUNSUPPORTED", "ECUDA", "ETIMEOUT"};
  TORCH_CHECK(rc == 0, what, " failed (", rc <= 0 && rc >= -4 ? names[-rc] : "?", "): ", api.last_error());
}

// The device's status word. status.poll looks at what earlier launches reported (and may raise); it runs at most
// once a millisecond and device here, so a failure surfaces at one of the next calls, as before.
int32_t* status_word(int device) {
  constexpr int MAX = 64;
  static std::atomic<int64_t> last_poll[MAX];
  static std::atomic<int32_t*> words[MAX];
  TORCH_CHECK(device >= 0 && device < MAX, "device ordinal out of range");
  const int64_t now = std::chrono::steady_clock::now().time_since_epoch() / std::chrono::microseconds(1);
  int32_t* word = words[device].load(std::memory_order_acquire);
  if (word != nullptr && now - last_poll[device].load(std::memory_order_relaxed) < 1000) return word;
  pybind11::gil_scoped_acquire gil;
  pybind11::object r = pybind11::reinterpret_steal<pybind11::object>(PyObject_CallFunction(poll_fn, "i", device));
  if (!r) {
    python_error failed;   // carries the Python exception to whichever thread reports it
    failed.persist();
    throw failed;
  }
  word = static_cast<int32_t*>(PyLong_AsVoidPtr(r.ptr()));
  words[device].store(word, std::memory_order_release);
  last_poll[device].store(now, std::memory_order_relaxed);
  return word;
}

// Lets go of the GIL. (pybind11::gil_scoped_release also looks up and updates its own thread state, a part of a
// microsecond that shows in a call of five.)
class NoGil {
 public:
  NoGil() : state_(PyEval_SaveThread()) {}
  ~NoGil() { PyEval_RestoreThread(state_); }
  NoGil(const NoGil&) = delete;
  NoGil& operator=(const NoGil&) = delete;

 private:
  PyThreadState* state_;
};

// A plain strided CUDA tensor of `dims` dimensions that TMA can describe as it is.
bool ready(const at::Tensor& x, int dims) {
  using c10::DispatchKey;
  const auto ks = x.key_set();
  if (!x.defined() || !x.is_cuda() || x.dim() != dims || x.layout() != at::kStrided || ks.has(DispatchKey::Python) ||
      ks.has(DispatchKey::FuncTorchBatched) || ks.has(DispatchKey::FuncTorchGradWrapper) ||
      ks.has(DispatchKey::Functionalize) || ks.has(DispatchKey::ZeroTensor) || !x.has_storage())
    return false;
  const void* ptr = x.const_data_ptr();
  if (ptr == nullptr || reinterpret_cast<uintptr_t>(ptr) % 16 != 0) return false;
  const auto sizes = x.sizes(), strides = x.strides();
  if (strides[dims - 1] != 1) return false;
  const int64_t esize = static_cast<int64_t>(x.element_size());
  for (int i = 0; i < dims - 1; ++i)
    if (sizes[i] > 1 && (strides[i] <= 0 || (strides[i] * esize) % 16 != 0)) return false;
  return true;
}

// Whether a functorch transform is active on this thread. A thread that has ever used functorch, also through
// torch.compile, keeps its functorch state; the state itself knows whether a transform is active and then refuses C++
// autograd functions. (The key test only spares the exception in the usual case.)
bool transform_active() {
  const auto& state = at::functorch::functorchTLSAccessor();
  if (!state) return false;
  if (c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode)) return true;
  try {
    state->checkSupportsCppAutogradFunction();
  } catch (const c10::Error&) {
    return true;
  }
  return false;
}

bool ordinary_mode() {
  return !transform_active() && !c10::impl::TorchDispatchModeTLS::any_modes_set() && !torch::jit::tracer::isTracing();
}

bool head_dim_ok(int64_t d) { return d == 16 || d == 32 || d == 64 || d == 128; }
int32_t dtype_code(at::ScalarType t) { return t == at::kHalf ? B200ATTN_F16 : t == at::kBFloat16 ? B200ATTN_BF16 : B200ATTN_F32; }

b200attn_tensor tensor4(const at::Tensor& t) {
  b200attn_tensor r;
  r.ptr = t.data_ptr();
  for (int i = 0; i < 4; ++i) r.stride[i] = t.stride(i);
  return r;
}

// q [B, Hq, M, D], k and v [B, Hkv, N, D] of one 16-bit type on one device, as they are.
bool qkv_ok(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v) {
  if (!ready(q, 4) || !ready(k, 4) || !ready(v, 4)) return false;
  const auto dt = q.scalar_type();
  if ((dt != at::kHalf && dt != at::kBFloat16) || k.scalar_type() != dt || v.scalar_type() != dt) return false;
  if (k.device() != q.device() || v.device() != q.device()) return false;
  if (!head_dim_ok(q.size(3)) || k.size(3) != q.size(3) || k.sizes() != v.sizes() || k.size(0) != q.size(0)) return false;
  if (q.numel() == 0 || k.numel() == 0 || q.size(1) % k.size(1) != 0) return false;
  for (int i = 0; i < 3; ++i)
    if (q.size(i) > INT32_MAX || k.size(i) > INT32_MAX) return false;
  return true;
}

// split_kv.choose_num_splits: whether flash_attention takes the split-KV branch.
bool takes_split_branch(int64_t B, int64_t H, int64_t M, int64_t N, int sms) {
  const int64_t ctas = B * H * ((M + 15) / 16), n_blocks = (N + 127) / 128;
  if (static_cast<double>(ctas) >= 0.8 * sms) return false;
  const int64_t limit = std::min<int64_t>({sms, n_blocks, 128});
  auto admissible = [&](int64_t s) {
    const int64_t per = (n_blocks + s - 1) / s;
    return s == 1 || per * s - n_blocks < per;
  };
  auto efficiency = [&](int64_t s) {
    const double waves = static_cast<double>(ctas * s) / sms;
    return waves / std::ceil(waves);
  };
  double best = 0.;
  for (int64_t s = 1; s <= limit; ++s)
    if (admissible(s)) best = std::max(best, efficiency(s));
  for (int64_t s = 1; s <= limit; ++s)
    if (admissible(s) && efficiency(s) >= 0.85 * best) return s > 1;
  return false;
}

int sm_count(const at::Tensor& q) { return at::cuda::getDeviceProperties(q.get_device())->multiProcessorCount; }
void* current_stream(const at::Tensor& q) { return c10::cuda::getCurrentCUDAStream(q.get_device()).stream(); }

void fill_fwd(b200attn_fwd_params& p, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o,
              const at::Tensor& lse, bool causal, double scale, int32_t* status) {
  p.q = tensor4(q); p.k = tensor4(k); p.v = tensor4(v); p.o = tensor4(o);
  p.lse = lse.data_ptr<float>();
  p.B = q.size(0); p.Hq = q.size(1); p.Hkv = k.size(1); p.M = q.size(2); p.N = k.size(2); p.D = q.size(3);
  p.dtype = p.o_dtype = dtype_code(q.scalar_type());
  p.causal = causal;
  p.sm_scale = static_cast<float>(scale);
  p.status = status;
}

// Forward over split keys: (o in q's type, log-normaliser).
std::pair<at::Tensor, at::Tensor> split_kv_forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, bool causal,
                                                   double scale) {
  const int64_t B = q.size(0), H = q.size(1), M = q.size(2), D = q.size(3), Hk = k.size(1), N = k.size(2);
  const int S = api.splitkv_num_splits(B, H, Hk, M, N, D, sm_count(q));
  at::Tensor o = at::empty({B, H, M, D}, q.options());
  at::Tensor lse = at::empty({B, H, M}, q.options().dtype(at::kFloat));
  int32_t* status = status_word(q.get_device());
  if (S <= 1 && H / Hk * M > 2) {
    b200attn_fwd_params p{};
    fill_fwd(p, q, k, v, o, lse, causal, scale, status);
    check(api.fwd(&p, current_stream(q)), "b200attn_fwd");
    return {o, lse};
  }
  // one scratch allocation: per-split outputs, then per-split normalisers (unused by the single-split streaming kernel).
  // The log-normaliser is a tensor of its own: autograd saves it, which must not keep the partial outputs alive.
  const int64_t rows = B * H * M;
  at::Tensor parts = S > 1 ? at::empty({rows * (S * D + S)}, lse.options()) : lse;
  b200attn_splitkv_params p{};
  p.q = tensor4(q); p.k = tensor4(k); p.v = tensor4(v); p.o = tensor4(o);
  p.lse = lse.data_ptr<float>();
  p.part_o = parts.data_ptr<float>();
  p.part_lse = S > 1 ? p.part_o + rows * S * D : p.part_o;
  p.B = B; p.Hq = H; p.Hkv = Hk; p.M = M; p.N = N; p.D = D;
  p.num_splits = S;
  p.dtype = dtype_code(q.scalar_type());
  p.causal = causal;
  p.sm_scale = static_cast<float>(scale);
  p.status = status;
  check(api.fwd_splitkv(&p, current_stream(q)), "b200attn_fwd_splitkv");
  return {o, lse};
}

// The tensor, or a contiguous copy that TMA can describe.
at::Tensor made_ready(const at::Tensor& x) { return ready(x, 4) ? x : x.contiguous(); }
at::Tensor empty_ready_like(const at::Tensor& x) {
  at::Tensor r = at::empty_like(x);
  return ready(r, 4) ? r : at::empty(x.sizes(), x.options());
}

struct FlashAttention : torch::autograd::Function<FlashAttention> {
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                            bool causal, double scale) {
    at::Tensor o, lse;
    if (takes_split_branch(q.size(0), q.size(1), q.size(2), k.size(2), sm_count(q))) {
      std::tie(o, lse) = split_kv_forward(q, k, v, causal, scale);
    } else {
      lse = at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat));
      o = empty_ready_like(q);
      b200attn_fwd_params p{};
      fill_fwd(p, q, k, v, o, lse, causal, scale, status_word(q.get_device()));
      check(api.fwd(&p, current_stream(q)), "b200attn_fwd");
    }
    ctx->save_for_backward({q, k, v, o, lse});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return o;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &q = saved[0], &k = saved[1], &v = saved[2], &o = saved[3], &lse = saved[4];
    const int64_t B = q.size(0), H = q.size(1), M = q.size(2), D = q.size(3), Hk = k.size(1), N = k.size(2);
    const c10::cuda::CUDAGuard guard(q.device());
    const at::Tensor d_o = made_ready(grads[0].scalar_type() == q.scalar_type() ? grads[0] : grads[0].to(q.scalar_type()));
    at::Tensor dq = empty_ready_like(q);
    at::Tensor dk = at::empty({B, Hk, N, D}, k.options()), dv = at::empty({B, Hk, N, D}, v.options());
    const int64_t work = static_cast<int64_t>(std::max<size_t>(api.bwd_workspace_bytes(B, H, Hk, M, N, D), 16)) / 4;
    // workspace, then the row sums dot(O, dO)
    at::Tensor scratch = at::empty({work + B * H * M}, lse.options());
    b200attn_bwd_params p{};
    p.q = tensor4(q); p.k = tensor4(k); p.v = tensor4(v); p.o = tensor4(o); p.d_o = tensor4(d_o);
    p.dq = tensor4(dq); p.dk = tensor4(dk); p.dv = tensor4(dv);
    p.lse = lse.data_ptr<float>();
    p.workspace = scratch.data_ptr<float>();
    p.delta = scratch.data_ptr<float>() + work;
    p.B = B; p.Hq = H; p.Hkv = Hk; p.M = M; p.N = N; p.D = D;
    p.dtype = p.o_dtype = dtype_code(q.scalar_type());
    p.causal = ctx->saved_data["causal"].toBool();
    p.sm_scale = static_cast<float>(ctx->saved_data["scale"].toDouble());
    p.status = status_word(q.get_device());
    // dQ is summed by fp32 reductions in global memory unless reproducible results are asked for
    const int stages = B200ATTN_BWD_STAGE_ALL | (at::globalContext().deterministicAlgorithms() ? B200ATTN_BWD_STAGE_UNFUSED : 0);
    check(api.bwd_stages(&p, current_stream(q), stages), "b200attn_bwd_stages");
    return {dq, dk, dv, at::Tensor(), at::Tensor()};
  }
};

// Exactly torch.Tensor or nn.Parameter: another subclass may define its own results, through __torch_function__ too.
bool plain_tensors(PyObject* const* args, int n) {
  for (int i = 0; i < n; ++i)
    if (!THPVariable_CheckExact(args[i])) return false;
  return true;
}

// sm_scale argument: None means 1 / sqrt(D).
bool scale_of(PyObject* arg, int64_t d, double* out) {
  if (arg == Py_None) {
    *out = 1.0 / std::sqrt(static_cast<double>(d));
    return true;
  }
  *out = PyFloat_AsDouble(arg);
  return !(*out == -1.0 && PyErr_Occurred());
}

// flash(q, k, v, causal, sm_scale) and split_kv(q, k, v, causal, sm_scale)
template <bool SPLIT>
PyObject* attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 5 || !plain_tensors(args, 3) || !ordinary_mode()) Py_RETURN_NONE;
  const at::Tensor q = THPVariable_Unpack(args[0]), k = THPVariable_Unpack(args[1]), v = THPVariable_Unpack(args[2]);
  if (!qkv_ok(q, k, v)) Py_RETURN_NONE;
  const int causal = PyObject_IsTrue(args[3]);
  double scale;
  if (causal < 0 || !scale_of(args[4], q.size(3), &scale)) return nullptr;
  at::Tensor o;
  {
    // Allocations and launches may block (a full launch queue, a cudaMalloc), and a host callback of the stream may
    // need the GIL before the queue moves on.
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    if constexpr (SPLIT) {
      const at::NoGradGuard no_grad;
      o = split_kv_forward(q, k, v, causal != 0, scale).first;
    } else {
      o = FlashAttention::apply(q, k, v, causal != 0, scale);
    }
  }
  return THPVariable_Wrap(std::move(o));
  END_HANDLE_TH_ERRORS
}

// paged(query, key_cache, value_cache, context_lens, block_tables, attn_scale, max_context_len, num_splits)
PyObject* paged(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8 || !plain_tensors(args, 5) || !ordinary_mode()) Py_RETURN_NONE;
  const at::Tensor q = THPVariable_Unpack(args[0]), kc = THPVariable_Unpack(args[1]), vc = THPVariable_Unpack(args[2]),
                   lens = THPVariable_Unpack(args[3]), tables = THPVariable_Unpack(args[4]);
  if (!ready(q, 3) || !ready(kc, 4) || !ready(vc, 4)) Py_RETURN_NONE;
  const auto dt = q.scalar_type();
  if ((dt != at::kHalf && dt != at::kBFloat16) || kc.scalar_type() != dt || vc.scalar_type() != dt ||
      kc.sizes() != vc.sizes() || kc.size(3) != q.size(2) || !head_dim_ok(q.size(2)) || q.numel() == 0 || kc.numel() == 0 ||
      q.size(1) % kc.size(1) != 0 || kc.device() != q.device() || vc.device() != q.device())
    Py_RETURN_NONE;
  if (!lens.is_cuda() || !tables.is_cuda() || lens.device() != q.device() || tables.device() != q.device() ||
      lens.scalar_type() != at::kInt || tables.scalar_type() != at::kInt || lens.dim() != 1 || tables.dim() != 2 ||
      !lens.is_contiguous() || tables.stride(1) != 1 || lens.size(0) != q.size(0) || tables.size(0) != q.size(0))
    Py_RETURN_NONE;
  for (int i = 0; i < 3; ++i)
    if (q.size(i) > INT32_MAX || kc.size(i) > INT32_MAX) Py_RETURN_NONE;
  double scale;
  if (args[5] == Py_None || !scale_of(args[5], q.size(2), &scale)) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  if (!PyLong_CheckExact(args[6]) || !PyLong_CheckExact(args[7])) Py_RETURN_NONE;
  const long long longest = PyLong_AsLongLong(args[6]), asked = PyLong_AsLongLong(args[7]);
  if (PyErr_Occurred() || longest < 1 || longest > INT32_MAX || asked < 0 || asked > INT32_MAX) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  at::Tensor out;
  {
    const NoGil no_gil;  // as above
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    const at::NoGradGuard no_grad;
    const int64_t seqs = q.size(0), H = q.size(1), D = q.size(2), rows = seqs * H;
    const int64_t S = asked > 0 ? asked : api.splitkv_num_splits(seqs, H, kc.size(1), 1, longest, D, sm_count(q));
    out = at::empty({seqs, H, D}, q.options());
    at::Tensor parts = at::empty({rows * (S * D + S + 1)}, q.options().dtype(at::kFloat));
    b200attn_paged_params p{};
    auto rows4 = [](const at::Tensor& t) {  // [seqs, heads, D] described as [seqs, heads, 1, D]
      b200attn_tensor r;
      r.ptr = t.data_ptr();
      r.stride[0] = t.stride(0); r.stride[1] = t.stride(1); r.stride[2] = t.size(2); r.stride[3] = t.stride(2);
      return r;
    };
    p.q = rows4(q); p.o = rows4(out);
    p.key_cache = tensor4(kc); p.value_cache = tensor4(vc);
    p.block_table = tables.data_ptr<int32_t>();
    p.block_table_stride = tables.stride(0);
    p.context_lens = lens.data_ptr<int32_t>();
    p.part_o = parts.data_ptr<float>();
    p.part_lse = p.part_o + rows * S * D;
    p.lse = p.part_lse + rows * S;
    p.num_seqs = seqs; p.Hq = H; p.Hkv = kc.size(1); p.D = D; p.block_size = kc.size(2); p.num_blocks = kc.size(0);
    p.max_context_len = longest;
    p.num_splits = S;
    p.dtype = dtype_code(dt);
    p.sm_scale = static_cast<float>(scale);
    p.status = status_word(q.get_device());
    check(api.paged(&p, current_stream(q)), "b200attn_paged_attention");
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// bind(addresses of the entry points in the order of Api, poll function)
PyObject* bind(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  unsigned long long a[7];
  PyObject* poll;
  if (!PyArg_ParseTuple(args, "(KKKKKKK)O", &a[0], &a[1], &a[2], &a[3], &a[4], &a[5], &a[6], &poll)) return nullptr;
  api.fwd = reinterpret_cast<decltype(api.fwd)>(a[0]);
  api.bwd_stages = reinterpret_cast<decltype(api.bwd_stages)>(a[1]);
  api.bwd_workspace_bytes = reinterpret_cast<decltype(api.bwd_workspace_bytes)>(a[2]);
  api.fwd_splitkv = reinterpret_cast<decltype(api.fwd_splitkv)>(a[3]);
  api.splitkv_num_splits = reinterpret_cast<decltype(api.splitkv_num_splits)>(a[4]);
  api.paged = reinterpret_cast<decltype(api.paged)>(a[5]);
  api.last_error = reinterpret_cast<decltype(api.last_error)>(a[6]);
  Py_INCREF(poll);
  Py_XSETREF(poll_fn, poll);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// takes_split_branch(B, H, M, N, sms): the rule by itself, for comparison with split_kv.choose_num_splits
PyObject* split_branch(PyObject*, PyObject* args) {
  long long b, h, m, n;
  int sms;
  if (!PyArg_ParseTuple(args, "LLLLi", &b, &h, &m, &n, &sms)) return nullptr;
  return PyBool_FromLong(takes_split_branch(b, h, m, n, sms));
}

// ordinary_mode(): that rule by itself
PyObject* mode_is_ordinary(PyObject*, PyObject*) {
  HANDLE_TH_ERRORS
  return PyBool_FromLong(ordinary_mode());
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"ordinary_mode", &mode_is_ordinary, METH_NOARGS, nullptr},
    {"takes_split_branch", &split_branch, METH_VARARGS, nullptr},
    {"flash", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&attention<false>)), METH_FASTCALL, nullptr},
    {"split_kv", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&attention<true>)), METH_FASTCALL, nullptr},
    {"paged", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&paged)), METH_FASTCALL, nullptr},
    {"bind", &bind, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native host path of the operators", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
