// Host side of the library (module avelang_b200._host), in C++: the operators torch.ops.avelang_gdn.* and the public functions.
//
// An operator's CUDA kernel fills the C argument block and calls into libave_gdn_b200.so on torch's current stream.  A public
// function takes the positional arguments its Python wrapper passes (METH_FASTCALL: no tuple, no keyword parsing), checks
// them, raises ValueError with the wording of the Python API, allocates what it returns and calls the operator through the
// dispatcher, so dispatch modes, tensor subclasses and the profiler see every call.
//
// A decode step of a few sequences runs for 5 to 30 us on the GPU; with the checks and the argument block filled from Python
// (attribute by attribute through ctypes, behind a boxed dispatcher round trip) a call cost 45 to 75 us of host time and the
// GPU idled between steps.  Here a call costs a few microseconds (back-to-back steps on one sequence of 32 heads:
// 51.0 -> 5.0 us; 37 sequences with the gated norm: 57.6 -> 30.1 us, now bound by the kernel).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <c10/core/InferenceMode.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>

#include <atomic>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <sstream>
#include <string>
#include <utility>
#include <vector>

#include "ave_gdn.h"

namespace {

using at::Tensor;

// ---------------------------------------------------------------------------------------------- errors
template <class... Parts>
std::string text(const Parts&... parts) {
  std::ostringstream s;
  (void)std::initializer_list<int>{(s << parts, 0)...};
  return s.str();
}
// argument problems raise ValueError, from a public function and from an operator alike
#define BAD_ARGUMENT(...) throw c10::ValueError({__func__, __FILE__, static_cast<uint32_t>(__LINE__)}, text(__VA_ARGS__))
#define REQ(cond, ...)                                            \
  do {                                                            \
    if (__builtin_expect(!(cond), 0)) BAD_ARGUMENT(__VA_ARGS__);  \
  } while (0)

std::string shape_of(at::IntArrayRef s) {  // as Python prints a tuple
  std::ostringstream o;
  o << "(";
  for (size_t i = 0; i < s.size(); ++i) o << (i ? ", " : "") << s[i];
  o << (s.size() == 1 ? ",)" : ")");
  return o.str();
}
std::string dtype_name(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return "torch.float32";
    case at::kDouble: return "torch.float64";
    case at::kHalf: return "torch.float16";
    case at::kBFloat16: return "torch.bfloat16";
    case at::kInt: return "torch.int32";
    case at::kLong: return "torch.int64";
    case at::kBool: return "torch.bool";
    case at::kByte: return "torch.uint8";
    case at::kChar: return "torch.int8";
    case at::kShort: return "torch.int16";
    default: return std::string("torch.") + c10::toString(t.scalar_type());
  }
}

// ---------------------------------------------------------------------------------------------- the C library
struct Api {
  decltype(&ave_gdn_chunk_prefill) chunk_prefill = nullptr;
  decltype(&ave_gdn_prefill_workspace_bytes) prefill_workspace_bytes = nullptr;
  decltype(&ave_gdn_decode_step) decode_step = nullptr;
  decltype(&ave_gdn_mixed_step) mixed_step = nullptr;
  decltype(&ave_gdn_gated_rmsnorm) gated_rmsnorm = nullptr;
  decltype(&ave_gemm_bf16_nt) gemm_bf16_nt = nullptr;
  decltype(&ave_gdn_conv1d_silu) conv1d_silu = nullptr;
  decltype(&ave_gdn_conv1d_update) conv1d_update = nullptr;
  decltype(&ave_gdn_gate_beta) gate_beta = nullptr;
  decltype(&ave_gdn_decode_layer_step) decode_layer_step = nullptr;
  decltype(&ave_gdn_recurrent_backward) recurrent_backward = nullptr;
  decltype(&ave_gdn_backward_workspace_bytes) backward_workspace_bytes = nullptr;
  decltype(&ave_gdn_status_string) status_string = nullptr;
  decltype(&ave_gdn_last_cuda_error) last_cuda_error = nullptr;
} api;

// Argument problems raise ValueError, device problems RuntimeError.
void check(int rc, const char* what) {
  if (__builtin_expect(rc == AVE_GDN_OK, 1)) return;
  const std::string msg = text(what, ": ", api.status_string(rc));
  if (rc == AVE_GDN_CUDA_ERROR) throw c10::Error({__func__, __FILE__, static_cast<uint32_t>(__LINE__)}, text(msg, " (cudaError ", api.last_cuda_error(), ")"));
  BAD_ARGUMENT(msg);
}
// an operator reached before the Python layer has loaded the library
void loaded() { TORCH_CHECK(api.chunk_prefill != nullptr, "libave_gdn_b200.so is not loaded: run `python -m avelang_b200.build`; there is no fallback implementation"); }

// ---------------------------------------------------------------------------------------------- arguments
const Tensor* opt_tensor(PyObject* o, const char* name) {
  if (o == Py_None) return nullptr;
  REQ(THPVariable_Check(o), name, " must be a tensor");
  return &THPVariable_Unpack(o);
}
const Tensor& tensor(PyObject* o, const char* name) {
  REQ(THPVariable_Check(o), name, " must be a tensor");
  return THPVariable_Unpack(o);
}
bool truth(PyObject* o) {
  if (o == Py_True) return true;
  if (o == Py_False || o == Py_None) return false;
  const int r = PyObject_IsTrue(o);
  if (r < 0) throw python_error();
  return r != 0;
}
double number(PyObject* o) {
  const double x = PyFloat_AsDouble(o);
  if (x == -1.0 && PyErr_Occurred()) throw python_error();
  return x;
}
int64_t integer(PyObject* o) {
  PyObject* i = PyNumber_Long(o);
  if (i == nullptr) throw python_error();
  const int64_t x = PyLong_AsLongLong(i);
  Py_DECREF(i);
  if (x == -1 && PyErr_Occurred()) throw python_error();
  return x;
}
PyObject* wrap(const Tensor& t) { return THPVariable_Wrap(t); }
PyObject* wrap_pair(const Tensor& a, const Tensor& b) {
  PyObject* r = PyTuple_New(2);
  if (r == nullptr) throw python_error();
  PyTuple_SET_ITEM(r, 0, wrap(a));
  if (b.defined()) {
    PyTuple_SET_ITEM(r, 1, wrap(b));
  } else {
    Py_INCREF(Py_None);
    PyTuple_SET_ITEM(r, 1, Py_None);
  }
  return r;
}

const void* ptr(const Tensor* t) { return t != nullptr && t->numel() > 0 ? t->data_ptr() : nullptr; }
template <class T>
T* ptr_as(const Tensor* t) { return reinterpret_cast<T*>(const_cast<void*>(ptr(t))); }
Tensor empty(at::IntArrayRef shape, at::ScalarType dt, const Tensor& like) {
  return at::empty(shape, like.options().dtype(dt).requires_grad(false));
}
// fp32, contiguous; the tensor itself when it is both already
Tensor f32(const Tensor& t) { return (t.requires_grad() ? t.detach() : t).to(at::kFloat).contiguous(); }

// ---------------------------------------------------------------------------------------------- scratch and status word
const Tensor& status_word(const at::Device& dev) {  // one a device, never destroyed: the CUDA context may be gone at exit
  static std::atomic<Tensor*> words[C10_COMPILE_TIME_MAX_GPUS];
  static std::mutex mu;
  const int idx = dev.has_index() ? dev.index() : c10::cuda::current_device();
  std::atomic<Tensor*>& w = words[idx];
  Tensor* t = w.load(std::memory_order_acquire);
  if (t == nullptr) {
    const c10::InferenceMode ordinary(false);  // a word made in inference mode could not be reset outside it
    auto made = std::make_unique<Tensor>(at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::Device(at::kCUDA, idx))));
    std::lock_guard<std::mutex> lock(mu);
    t = w.load(std::memory_order_acquire);
    if (t == nullptr) w.store(t = made.release(), std::memory_order_release);
  }
  return *t;
}
// Scratch.  A call owns its block from the moment it asks for one until all that uses it is enqueued, and then leaves it for the
// next call on the same stream: two host threads on one stream never work on one block, and since the stream orders the
// calls, a block left behind may still be in use on the GPU.  While the stream is being captured the block comes from the
// graph's own memory and is not kept, so a replay finds what it was captured with whatever ran in between.  Kept blocks are
// bounded in number and bytes, the least recently used going first, and go back to torch's allocator when that runs short.
constexpr size_t KEPT_BLOCKS = 8;             // a device
constexpr int64_t KEPT_BYTES = 12ll << 30;    // a device; the largest prefill measured (262144 tokens, 32 heads) takes 9
class ScratchPool {
 public:
  Tensor take(int device, cudaStream_t stream, int64_t bytes) {
    Tensor t;
    {
      std::lock_guard<std::mutex> lock(mu_);
      const auto it = blocks_.find({device, stream});
      if (it != blocks_.end()) {
        t = std::move(it->second.t);
        blocks_.erase(it);
      }
    }
    if (t.defined() && t.numel() < bytes) t.reset();  // (before the larger one is asked for)
    if (!t.defined()) t = at::empty({bytes}, at::TensorOptions().dtype(at::kByte).device(at::Device(at::kCUDA, device)));
    return t;
  }
  void give(int device, cudaStream_t stream, Tensor t) {
    std::vector<Tensor> out;  // outlives the lock: freeing a block may call release()
    out.push_back(std::move(t));
    if (out[0].numel() > KEPT_BYTES) return;
    std::lock_guard<std::mutex> lock(mu_);
    Block& own = blocks_[{device, stream}];
    if (!own.t.defined() || own.t.numel() < out[0].numel()) std::swap(own.t, out[0]);  // (another thread may have left a larger one)
    own.used = ++clock_;
    for (;;) {
      size_t count = 0;
      int64_t bytes = 0;
      auto oldest = blocks_.end();
      for (auto it = blocks_.begin(); it != blocks_.end(); ++it) {
        if (it->first.first != device) continue;
        ++count;
        bytes += it->second.t.numel();
        if (oldest == blocks_.end() || it->second.used < oldest->second.used) oldest = it;
      }
      if (count <= KEPT_BLOCKS && bytes <= KEPT_BYTES) break;
      out.push_back(std::move(oldest->second.t));
      blocks_.erase(oldest);
    }
  }
  bool release(int device) {  // whether there was anything to give back
    std::vector<Tensor> out;
    std::lock_guard<std::mutex> lock(mu_);
    for (auto it = blocks_.begin(); it != blocks_.end();) {
      if (it->first.first != device) { ++it; continue; }
      out.push_back(std::move(it->second.t));
      it = blocks_.erase(it);
    }
    return !out.empty();
  }

 private:
  struct Block {
    Tensor t;
    uint64_t used = 0;
  };
  std::mutex mu_;
  std::map<std::pair<int, cudaStream_t>, Block> blocks_;
  uint64_t clock_ = 0;
};
ScratchPool& scratch_pool() {
  static auto* pool = new ScratchPool();  // never destroyed: the CUDA context may be gone at exit
  return *pool;
}
// Called by torch's allocator, before it gives up, on the thread that asked it for memory (with that thread's device current).
class ReleaseScratch : public c10::FreeMemoryCallback {
 public:
  bool Execute() override { return scratch_pool().release(c10::cuda::current_device()); }
};

class Scratch {  // one call's block
 public:
  Scratch(const Tensor& like, cudaStream_t stream, size_t bytes)
      : device_(like.get_device()), stream_(stream),
        captured_(c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) {
    const int64_t n = bytes > 0 ? (int64_t)bytes : 1;
    t_ = captured_ ? at::empty({n}, at::TensorOptions().dtype(at::kByte).device(like.device())) : scratch_pool().take(device_, stream, n);
  }
  ~Scratch() {
    if (!captured_) scratch_pool().give(device_, stream_, std::move(t_));
  }
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
  void* data() const { return t_.data_ptr(); }
  uint64_t size() const { return (uint64_t)t_.numel(); }

 private:
  int device_;
  cudaStream_t stream_;
  bool captured_;
  Tensor t_;
};
struct Launch {  // device of the tensors made current, its current stream, no GIL while the library enqueues
  c10::cuda::OptionalCUDAGuard guard;
  cudaStream_t stream;
  explicit Launch(const Tensor& t) {
    if (t.get_device() != c10::cuda::current_device()) guard.set_index(t.get_device());
    stream = c10::cuda::getCurrentCUDAStream(t.get_device()).stream();
  }
  template <class F>
  int operator()(F f) {
    if (PyGILState_Check() == 0) return f();  // an operator called without it
    PyThreadState* ts = PyEval_SaveThread();
    const int rc = f();
    PyEval_RestoreThread(ts);
    return rc;
  }
};

// ---------------------------------------------------------------------------------------------- shared checks
struct Shape {
  int64_t B, T, Hk, Hv, dk, dv, n;
};
bool share_strides(const Tensor& a, const Tensor& b) { return a.strides() == b.strides(); }

Shape check_common(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor* z,
                   const Tensor* cu) {
  const std::pair<const char*, const Tensor*> qkv[] = {{"q", &q}, {"k", &k}, {"v", &v}};
  for (const auto& [name, t] : qkv) {
    REQ(t->dim() == 4, name, " must be a 4-D tensor [B, T, H, d]");
    REQ(t->scalar_type() == at::kBFloat16, name, " must have dtype torch.bfloat16, got ", dtype_name(*t), ".");
    REQ(t->is_cuda(), name, " must be a CUDA tensor");
    REQ(t->stride(3) == 1, name, " must be contiguous in its last dimension");
    REQ(t->device() == q.device(), name, " must be on device ", q.device(), ", got ", t->device(), ".");
  }
  Shape s;
  s.B = q.size(0); s.T = q.size(1); s.Hk = q.size(2); s.dk = q.size(3);
  REQ(k.sizes() == q.sizes(), "k must have shape ", shape_of(q.sizes()), ", got ", shape_of(k.sizes()), ".");
  REQ(v.size(0) == s.B && v.size(1) == s.T, "v must have leading shape ", shape_of(q.sizes().slice(0, 2)), ", got ",
      shape_of(v.sizes().slice(0, 2)), ".");
  s.Hv = v.size(2); s.dv = v.size(3);
  REQ(s.Hk > 0 && s.Hv % s.Hk == 0, "value heads (", s.Hv, ") must be a multiple of key heads (", s.Hk, ").");
  REQ((s.dk == 128 && s.dv == 128) || (s.dk == 64 && s.dv == 64), "head dims (dk, dv) must be (128, 128) or (64, 64), got (", s.dk,
      ", ", s.dv, ").");
  const std::pair<const char*, const Tensor*> gb[] = {{"g", &g}, {"beta", &beta}};
  for (const auto& [name, t] : gb) {
    REQ(t->scalar_type() == at::kFloat, name, " must have dtype torch.float32, got ", dtype_name(*t), ".");
    REQ(t->dim() == 3 && t->size(0) == s.B && t->size(1) == s.T && t->size(2) == s.Hv, name, " must have shape ",
        shape_of({s.B, s.T, s.Hv}), ", got ", shape_of(t->sizes()), ".");
    REQ(t->device() == q.device(), name, " must be on device ", q.device(), ", got ", t->device(), ".");
    REQ(t->stride(2) == 1 || s.Hv == 1, name, " must be contiguous in its last dimension");
  }
  REQ(share_strides(g, beta), "g and beta must share strides");
  if (z != nullptr)
    REQ(z->scalar_type() == at::kBFloat16 && z->sizes() == v.sizes() && z->device() == q.device() && z->stride(3) == 1,
        "z must be a bf16 tensor of shape ", shape_of(v.sizes()), " on ", q.device());
  s.n = s.B;
  if (cu != nullptr) {
    REQ(s.B == 1, "cu_seqlens requires B == 1 (packed layout)");
    REQ(cu->scalar_type() == at::kInt && cu->dim() == 1 && cu->numel() >= 1, "cu_seqlens must be a 1-D int32 tensor [N+1]");
    REQ(cu->device() == q.device() && cu->is_contiguous(), "cu_seqlens must be contiguous on ", q.device());
    s.n = cu->numel() - 1;
  }
  return s;
}

Tensor prep_out(const Tensor* out, const Tensor& v) {
  if (out == nullptr) return empty(v.sizes(), at::kBFloat16, v);
  REQ(out->sizes() == v.sizes(), "out must have shape ", shape_of(v.sizes()), ", got ", shape_of(out->sizes()), ".");
  REQ(out->scalar_type() == at::kBFloat16, "out must have dtype torch.bfloat16, got ", dtype_name(*out), ".");
  REQ(out->device() == v.device(), "out must be on device ", v.device(), ", got ", out->device(), ".");
  REQ(out->stride(3) == 1, "out must be contiguous in its last dimension");
  return *out;
}

Tensor prep_norm_weight(const Tensor* w, const Tensor* z, const Shape& s, const at::Device& dev) {
  if (w == nullptr) return Tensor();
  REQ(z != nullptr, "norm_weight needs z (the gate of the fused RMSNorm)");
  REQ(w->numel() == s.dv && w->device() == dev, "norm_weight must have ", s.dv, " elements on ", dev);
  return f32(*w);
}

// final states to write (undefined when none are wanted)
Tensor prep_states(const Tensor* s0, const Tensor* idx, const Shape& s, const Tensor& like, bool want_final,
                                       bool inplace) {
  int64_t slots = s.n;
  if (s0 != nullptr) {
    REQ(s0->scalar_type() == at::kFloat, "initial_state must have dtype torch.float32, got ", dtype_name(*s0), ".");
    REQ(s0->dim() == 4 && s0->size(1) == s.Hv && s0->size(2) == s.dk && s0->size(3) == s.dv, "initial_state must have shape [N, ",
        s.Hv, ", ", s.dk, ", ", s.dv, "], got ", shape_of(s0->sizes()), ".");
    REQ(s0->is_contiguous() && s0->device() == like.device(), "initial_state must be contiguous on ", like.device());
    slots = s0->size(0);
  }
  if (idx != nullptr) {
    REQ(s0 != nullptr, "state_indices needs initial_state (the state pool)");
    REQ(idx->scalar_type() == at::kInt && idx->dim() == 1 && idx->size(0) == s.n, "state_indices must be int32 of shape (", s.n, ",)");
    REQ(idx->device() == like.device() && idx->is_contiguous(), "state_indices must be contiguous on ", like.device());
  } else {
    REQ(s0 == nullptr || slots == s.n, "initial_state must hold one state per sequence (", s.n, "), got ", slots, ".");
  }
  Tensor final;
  if (want_final) {
    if (idx != nullptr) final = inplace ? *s0 : s0->clone();
    else if (s.T == 0) final = s0 != nullptr ? s0->clone() : at::zeros({s.n, s.Hv, s.dk, s.dv}, like.options().dtype(at::kFloat));  // no kernel runs
    else final = empty({s.n, s.Hv, s.dk, s.dv}, at::kFloat, like);
  }
  return final;
}

#define STRIDES4(dst, name, t) \
  (dst).name##_stride_b = (t).stride(0), (dst).name##_stride_t = (t).stride(1), (dst).name##_stride_h = (t).stride(2)

AveGdnArgs fill_args(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor* z,
                     const Tensor* norm_weight, double norm_eps, const Tensor& o, double scale, const Tensor* s0,
                     const Tensor* final, const Tensor* cu, const Tensor* idx, int64_t slots, int64_t n, bool l2norm) {
  AveGdnArgs a{};
  a.struct_size = sizeof(a);
  a.flags = l2norm ? AVE_GDN_FLAG_QK_L2NORM : 0;
  a.q = ptr(&q); a.k = ptr(&k); a.v = ptr(&v);
  a.g = ptr_as<float>(&g); a.beta = ptr_as<float>(&beta);
  a.z = ptr(z); a.o = const_cast<void*>(ptr(&o));
  a.norm_weight = ptr_as<float>(norm_weight);
  a.initial_state = ptr_as<float>(s0); a.final_state = ptr_as<float>(final);
  a.cu_seqlens = ptr_as<int32_t>(cu); a.state_indices = ptr_as<int32_t>(idx);
  a.status = reinterpret_cast<uint32_t*>(status_word(q.device()).data_ptr());
  a.B = (int32_t)q.size(0); a.T = (int32_t)q.size(1); a.Hk = (int32_t)q.size(2); a.Hv = (int32_t)v.size(2);
  a.dk = (int32_t)q.size(3); a.dv = (int32_t)v.size(3);
  a.n_seqs = (int32_t)n; a.num_slots = (int32_t)slots; a.chunk = 64;
  STRIDES4(a, q, q); STRIDES4(a, k, k); STRIDES4(a, v, v); STRIDES4(a, o, o);
  if (z != nullptr) STRIDES4(a, z, *z);
  a.g_stride_b = g.stride(0); a.g_stride_t = g.stride(1);
  a.scale = (float)scale; a.norm_eps = (float)norm_eps;
  return a;
}

// ---------------------------------------------------------------------------------------------- operators
// The CUDA kernels of torch.ops.avelang_gdn.* (schemas: torch_ops.py).  They take tensors the caller has laid out; the library
// checks what they pass on.
using OptTensor = std::optional<Tensor>;
const Tensor* some(const Tensor& t) { return t.defined() ? &t : nullptr; }
const Tensor* some(const OptTensor& t) { return t.has_value() && t->defined() ? &*t : nullptr; }
OptTensor opt(const Tensor* t) { return t != nullptr ? OptTensor(*t) : OptTensor(); }
OptTensor opt(const Tensor& t) { return opt(some(t)); }
int64_t n_sequences(const Tensor& q, const Tensor* cu) { return cu != nullptr ? cu->numel() - 1 : q.size(0); }
int64_t n_slots(const Tensor* s0, const Tensor* final, int64_t n) {
  const Tensor* pool = final != nullptr ? final : s0;
  return pool != nullptr ? pool->size(0) : n;
}

void enqueue_prefill(AveGdnArgs& a, const Tensor& q, const AveGdnArgs* decode = nullptr) {  // with the single-token part of a mixed step
  Launch launch(q);
  const Scratch ws(q, launch.stream, api.prefill_workspace_bytes(&a));
  a.workspace = ws.data(); a.workspace_bytes = ws.size();
  if (decode != nullptr) return check(launch([&] { return api.mixed_step(decode, &a, launch.stream); }), "mixed_prefill_decode_step");
  check(launch([&] { return api.chunk_prefill(&a, launch.stream); }), "chunk_gated_delta_rule");
}
void enqueue_decode(AveGdnArgs& a, const Tensor& q) {
  Launch launch(q);
  check(launch([&] { return api.decode_step(&a, launch.stream); }), "fused_recurrent_gated_delta_rule");
}

void op_prefill(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& out, double scale,
                const OptTensor& initial_state, const OptTensor& final_state, const OptTensor& cu_seqlens, const OptTensor& state_indices,
                const OptTensor& z, const OptTensor& norm_weight, double norm_eps, bool l2norm, int64_t max_seqlen, const OptTensor& out_peers) {
  loaded();
  const Tensor *s0 = some(initial_state), *sf = some(final_state), *cu = some(cu_seqlens), *peers = some(out_peers);
  const int64_t n = n_sequences(q, cu);
  AveGdnArgs a = fill_args(q, k, v, g, beta, some(z), some(norm_weight), norm_eps, out, scale, s0, sf, cu, some(state_indices),
                           n_slots(s0, sf, n), n, l2norm);
  a.max_seqlen = (int32_t)max_seqlen;
  if (peers != nullptr) { a.o_peers = reinterpret_cast<const void* const*>(peers->data_ptr()); a.n_peers = (int32_t)peers->numel(); }
  enqueue_prefill(a, q);
}

void op_decode(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& out, double scale,
               const OptTensor& initial_state, const OptTensor& final_state, const OptTensor& cu_seqlens, const OptTensor& state_indices,
               const OptTensor& z, const OptTensor& norm_weight, double norm_eps, bool l2norm) {
  loaded();
  const Tensor *s0 = some(initial_state), *sf = some(final_state), *cu = some(cu_seqlens);
  const int64_t n = n_sequences(q, cu);
  AveGdnArgs a = fill_args(q, k, v, g, beta, some(z), some(norm_weight), norm_eps, out, scale, s0, sf, cu, some(state_indices),
                           n_slots(s0, sf, n), n, l2norm);
  enqueue_decode(a, q);
}

void op_mixed(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& out, double scale,
              const Tensor& state_pool, const Tensor& cu_seqlens, const Tensor& state_indices, int64_t n_decode, const OptTensor& z,
              const OptTensor& norm_weight, double norm_eps, bool l2norm) {
  loaded();
  const int64_t n = cu_seqlens.numel() - 1;
  REQ(n_decode >= 0 && n_decode <= n && n_decode <= q.size(1), "n_decode must lie in [0, ", std::min(n, q.size(1)), "], got ", n_decode, ".");
  AveGdnArgs a = fill_args(q, k, v, g, beta, some(z), some(norm_weight), norm_eps, out, scale, &state_pool, &state_pool, &cu_seqlens, &state_indices,
                           state_pool.size(0), n, l2norm);
  AveGdnArgs d = a;
  if (n_decode > 0) {  // one single-token sequence per row: the token stride becomes the batch stride
    d.B = d.n_seqs = (int32_t)n_decode;
    d.T = 1;
    d.cu_seqlens = nullptr;
    d.q_stride_b = a.q_stride_t; d.k_stride_b = a.k_stride_t; d.v_stride_b = a.v_stride_t; d.z_stride_b = a.z_stride_t;
    d.o_stride_b = a.o_stride_t; d.g_stride_b = a.g_stride_t;
    if (n_decode == n) return enqueue_decode(d, q);
  }
  if (n_decode < n) {
    a.cu_seqlens += n_decode;  // offsets stay absolute: the tables use differences, the tokens are addressed from the packed base
    a.state_indices += n_decode;
    a.n_seqs = (int32_t)(n - n_decode);
    a.token_begin = (int32_t)n_decode;
    enqueue_prefill(a, q, n_decode > 0 ? &d : nullptr);
  }
}

// [rows, H, d] views
void op_rmsnorm(const Tensor& x, const Tensor& z, const OptTensor& weight, double eps, bool gate_first, const Tensor& out) {
  loaded();
  AveGdnNormArgs a{};
  a.struct_size = sizeof(a);
  a.flags = gate_first ? AVE_GDN_FLAG_GATE_FIRST : 0;
  a.x = x.data_ptr(); a.z = z.data_ptr(); a.y = out.data_ptr();
  a.weight = ptr_as<float>(some(weight));
  a.rows = x.size(0) * x.size(1); a.heads = (int32_t)x.size(1); a.d = (int32_t)x.size(2);
  a.x_stride_t = x.stride(0); a.x_stride_h = x.stride(1);
  a.z_stride_t = z.stride(0); a.z_stride_h = z.stride(1);
  a.y_stride_t = out.stride(0); a.y_stride_h = out.stride(1);
  a.eps = (float)eps;
  Launch launch(x);
  check(launch([&] { return api.gated_rmsnorm(&a, launch.stream); }), "gated_rmsnorm");
}

void op_conv(const Tensor& x, const Tensor& w, const OptTensor& bias, const OptTensor& cu_seqlens, const Tensor& out) {
  loaded();
  const Tensor* cu = some(cu_seqlens);
  REQ(out.data_ptr() != x.data_ptr() || x.numel() == 0, "out must not alias x (later tokens read earlier inputs)");
  AveConvArgs a{};
  a.struct_size = sizeof(a);
  a.x = x.data_ptr(); a.w = w.data_ptr(); a.y = out.data_ptr(); a.bias = ptr(some(bias));
  a.B = (int32_t)x.size(0); a.T = (int32_t)x.size(1); a.C = (int32_t)x.size(2); a.width = (int32_t)w.size(1);
  if (cu != nullptr) { a.cu_seqlens = reinterpret_cast<const int32_t*>(cu->data_ptr()); a.n_seqs = (int32_t)cu->numel() - 1; }
  a.x_stride_b = x.stride(0); a.x_stride_t = x.stride(1); a.y_stride_b = out.stride(0); a.y_stride_t = out.stride(1);
  Launch launch(x);
  check(launch([&] { return api.conv1d_silu(&a, launch.stream); }), "causal_conv1d_silu");
}

void op_conv_update(const Tensor& x, const Tensor& conv_state, const Tensor& w, const OptTensor& bias, const OptTensor& state_indices, const Tensor& out) {
  loaded();
  AveConvUpdateArgs a{};
  a.struct_size = sizeof(a);
  a.x = x.data_ptr(); a.w = w.data_ptr(); a.y = out.data_ptr(); a.conv_state = conv_state.data_ptr(); a.bias = ptr(some(bias));
  a.state_indices = ptr_as<int32_t>(some(state_indices));
  a.n_seqs = (int32_t)x.size(0); a.C = (int32_t)x.size(1); a.width = (int32_t)w.size(1); a.num_slots = (int32_t)conv_state.size(0);
  a.x_stride = x.stride(0); a.y_stride = out.stride(0);
  a.status = reinterpret_cast<uint32_t*>(status_word(x.device()).data_ptr());
  Launch launch(x);
  check(launch([&] { return api.conv1d_update(&a, launch.stream); }), "causal_conv1d_update");
}

// a, b: [rows, Hv] views
void op_gate(const Tensor& a, const Tensor& b, const Tensor& A_log, const Tensor& dt_bias, const Tensor& g, const Tensor& beta) {
  loaded();
  AveGateArgs s{};
  s.struct_size = sizeof(s);
  s.a = a.data_ptr(); s.b = b.data_ptr(); s.A_log = ptr_as<float>(&A_log); s.dt_bias = ptr_as<float>(&dt_bias);
  s.g = ptr_as<float>(&g); s.beta = ptr_as<float>(&beta);
  s.rows = a.size(0); s.Hv = (int32_t)a.size(1);
  s.a_stride_row = a.stride(0); s.b_stride_row = b.stride(0);
  Launch launch(a);
  check(launch([&] { return api.gate_beta(&s, launch.stream); }), "gate_beta");
}

void op_gemm(const Tensor& A, const Tensor& B, const Tensor& out) {
  loaded();
  AveGemmArgs a{};
  a.struct_size = sizeof(a);
  a.a = A.data_ptr(); a.b = B.data_ptr(); a.c = out.data_ptr();
  a.M = A.size(0); a.N = B.size(0); a.K = A.size(1);
  a.lda = A.stride(0); a.ldb = B.stride(0); a.ldc = out.stride(0);
  a.status = reinterpret_cast<uint32_t*>(status_word(A.device()).data_ptr());
  Launch launch(A);
  check(launch([&] { return api.gemm_bf16_nt(&a, launch.stream); }), "gemm_pipeline_transposed_b");
}

// The checks of a decode layer step, for the operator and the public function.
void check_layer(const Tensor& proj, const Tensor& cw, const Tensor* cb, const Tensor& cs, const Tensor& A_log, const Tensor& dt_bias,
                 const Tensor* w, const Tensor& pool, const Tensor* idx, int64_t Hk, int64_t Hv) {
  constexpr int64_t d = 128;
  REQ(proj.scalar_type() == at::kBFloat16 && proj.dim() == 2 && proj.is_cuda() && proj.stride(1) == 1,
      "proj must be a bf16 CUDA tensor [N, columns]");
  const int64_t N = proj.size(0);
  REQ(Hk > 0 && Hv > 0 && Hv % Hk == 0, "value heads (", Hv, ") must be a multiple of key heads (", Hk, ").");
  const int64_t Cn = 2 * Hk * d + Hv * d, cols = 2 * Hk * d + 2 * Hv * d + 2 * Hv;
  REQ(proj.size(1) >= cols, "proj must have at least ", cols, " columns, got ", proj.size(1), ".");
  REQ(cw.scalar_type() == at::kBFloat16 && cw.dim() == 2 && cw.size(0) == Cn && cw.size(1) >= 2 && cw.size(1) <= 4 &&
          cw.device() == proj.device(),
      "conv_weight must be a bf16 tensor [", Cn, ", W] with W in 2..4 on ", proj.device());
  const int64_t W = cw.size(1);
  REQ(cs.scalar_type() == at::kBFloat16 && cs.dim() == 3 && cs.size(1) == W - 1 && cs.size(2) == Cn && cs.is_contiguous() &&
          cs.device() == proj.device(),
      "conv_state must be a contiguous bf16 tensor [slots, ", W - 1, ", ", Cn, "] on ", proj.device());
  REQ(pool.scalar_type() == at::kFloat && pool.dim() == 4 && pool.size(1) == Hv && pool.size(2) == d && pool.size(3) == d &&
          pool.is_contiguous() && pool.device() == proj.device(),
      "state_pool must be a contiguous fp32 tensor [slots, ", Hv, ", ", d, ", ", d, "] on ", proj.device());
  REQ(pool.size(0) == cs.size(0), "conv_state and state_pool must have the same number of slots");
  if (idx != nullptr)
    REQ(idx->scalar_type() == at::kInt && idx->dim() == 1 && idx->size(0) == N && idx->device() == proj.device() && idx->is_contiguous(),
        "state_indices must be a contiguous int32 tensor (", N, ",) on ", proj.device());
  else
    REQ(pool.size(0) >= N, "the pools need one slot per sequence when state_indices is not given");
  REQ(A_log.numel() == Hv && dt_bias.numel() == Hv && A_log.device() == proj.device(), "A_log and dt_bias must have ", Hv, " elements on ",
      proj.device());
  if (w != nullptr) REQ(w->numel() == d && w->device() == proj.device(), "norm_weight must have ", d, " elements on ", proj.device());
  if (cb != nullptr)
    REQ(cb->scalar_type() == at::kBFloat16 && cb->numel() == Cn && cb->device() == proj.device(), "conv_bias must be bf16 [", Cn, "]");
}

void op_decode_layer(const Tensor& proj, const Tensor& conv_w, const OptTensor& conv_bias, const Tensor& conv_state, const Tensor& A_log_in,
                     const Tensor& dt_bias_in, const OptTensor& norm_weight, const Tensor& state_pool, const OptTensor& state_indices,
                     const Tensor& out, int64_t Hk, int64_t Hv, double scale, double norm_eps, bool gate_first) {
  loaded();
  constexpr int64_t d = 128;
  const Tensor *cb = some(conv_bias), *w = some(norm_weight), *idx = some(state_indices);
  check_layer(proj, conv_w, cb, conv_state, A_log_in, dt_bias_in, w, state_pool, idx, Hk, Hv);
  const int64_t N = proj.size(0);
  REQ(out.dim() == 3 && out.size(0) == N && out.size(1) == Hv && out.size(2) == d && out.scalar_type() == at::kBFloat16 &&
          out.device() == proj.device() && out.stride(2) == 1 && out.stride(1) == d,
      "out must be a bf16 tensor (", N, ", ", Hv, ", ", d, ") with contiguous rows on ", proj.device());
  const Tensor A_log = f32(A_log_in), dt_bias = f32(dt_bias_in), cw = conv_w.contiguous();
  const Tensor nw = w != nullptr ? f32(*w) : Tensor(), bias = cb != nullptr ? cb->contiguous() : Tensor();
  AveGdnDecodeLayerArgs a{};
  a.struct_size = sizeof(a);
  a.flags = gate_first ? AVE_GDN_FLAG_GATE_FIRST : 0;
  a.proj = proj.data_ptr(); a.conv_w = cw.data_ptr(); a.conv_bias = ptr(some(bias)); a.conv_state = conv_state.data_ptr();
  a.A_log = ptr_as<float>(&A_log); a.dt_bias = ptr_as<float>(&dt_bias); a.norm_weight = ptr_as<float>(some(nw));
  a.state_pool = ptr_as<float>(&state_pool); a.state_indices = ptr_as<int32_t>(idx); a.o = out.data_ptr();
  a.status = reinterpret_cast<uint32_t*>(status_word(proj.device()).data_ptr());
  a.n_seqs = (int32_t)N; a.Hk = (int32_t)Hk; a.Hv = (int32_t)Hv; a.dk = a.dv = (int32_t)d; a.width = (int32_t)cw.size(1);
  a.num_slots = (int32_t)state_pool.size(0);
  a.proj_stride = proj.stride(0); a.o_stride = out.stride(0);
  a.norm_eps = (float)norm_eps; a.scale = (float)scale;
  Launch launch(proj);
  check(launch([&] { return api.decode_layer_step(&a, launch.stream); }), "decode_layer_step");
}

// dq, dk and dv: fp32 per value head, or all bf16 with dq and dk summed over the value heads of a key head; contiguous
void op_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& d_o, double scale,
                 const OptTensor& initial_state, const OptTensor& d_final_state, const OptTensor& cu_seqlens, const Tensor& dq, const Tensor& dk,
                 const Tensor& dv, const Tensor& dg, const Tensor& dbeta, const OptTensor& d_initial_state) {
  loaded();
  const bool summed = dq.scalar_type() == at::kBFloat16;
  const at::ScalarType dt = summed ? at::kBFloat16 : at::kFloat;
  REQ(dq.scalar_type() == dt && dk.scalar_type() == dt && dv.scalar_type() == dt, "dq, dk and dv must be all fp32 or all bf16");
  const Tensor *s0 = some(initial_state), *ds = some(d_final_state), *cu = some(cu_seqlens), *ds0 = some(d_initial_state);
  AveGdnBwdArgs a{};
  a.struct_size = sizeof(a);
  a.flags = summed ? AVE_GDN_FLAG_BWD_SUMMED : 0;
  a.q = ptr(&q); a.k = ptr(&k); a.v = ptr(&v); a.g = ptr_as<float>(&g); a.beta = ptr_as<float>(&beta); a.d_o = ptr(&d_o);
  a.initial_state = ptr_as<float>(s0); a.d_final_state = ptr_as<float>(ds); a.cu_seqlens = ptr_as<int32_t>(cu);
  a.d_q = ptr_as<float>(&dq); a.d_k = ptr_as<float>(&dk); a.d_v = ptr_as<float>(&dv);
  a.d_g = ptr_as<float>(&dg); a.d_beta = ptr_as<float>(&dbeta); a.d_initial_state = ptr_as<float>(ds0);
  a.status = reinterpret_cast<uint32_t*>(status_word(q.device()).data_ptr());
  a.B = (int32_t)q.size(0); a.T = (int32_t)q.size(1); a.Hk = (int32_t)q.size(2); a.Hv = (int32_t)v.size(2);
  a.dk = (int32_t)q.size(3); a.dv = (int32_t)v.size(3);
  a.n_seqs = (int32_t)(cu != nullptr ? cu->numel() - 1 : q.size(0));
  STRIDES4(a, q, q); STRIDES4(a, k, k); STRIDES4(a, v, v); STRIDES4(a, do, d_o);
  a.g_stride_b = g.stride(0); a.g_stride_t = g.stride(1); a.scale = (float)scale;
  Launch launch(q);
  // Scratch for all key heads at once; where that does not fit, for half of them, a quarter, ...: the call then takes as many
  // passes.  (Two sequences of 4096 tokens, 32 value heads: 0.82 ms in one pass of 1.03 GB, 1.12 in two, 1.78 in four: with half
  // the heads the scans use half the SMs.)
  std::optional<Scratch> ws;
  for (int heads = a.Hk;; heads = (heads + 1) / 2) {
    AveGdnBwdArgs part = a;
    part.Hk = heads; part.Hv = a.Hk > 0 ? heads * (a.Hv / a.Hk) : a.Hv;
    try {
      ws.emplace(q, launch.stream, api.backward_workspace_bytes(&part));
      break;
    } catch (const c10::OutOfMemoryError&) {
      if (heads <= 1) throw;
    }
  }
  a.workspace = ws->data(); a.workspace_bytes = ws->size();
  check(launch([&] { return api.recurrent_backward(&a, launch.stream); }), "gated_delta_rule_backward");
}

#define OPERATORS(X)                                                                                                        \
  X("chunk_prefill", op_prefill) X("decode_step", op_decode) X("mixed_step", op_mixed) X("decode_layer_step", op_decode_layer) \
  X("gated_rmsnorm", op_rmsnorm) X("conv1d_silu", op_conv) X("conv1d_update", op_conv_update) X("gate_beta", op_gate)          \
  X("gemm_bf16_nt", op_gemm) X("recurrent_backward", op_backward)
TORCH_LIBRARY_IMPL(avelang_gdn, CUDA, m) {
#define CUDA_KERNEL(name, f) m.impl(name, f);
  OPERATORS(CUDA_KERNEL)
}
// The operators return nothing and write into what they are given, so torch's stand-in for a missing autograd kernel, which
// goes through a boxed call (0.4 us), has nothing to do for them.
TORCH_LIBRARY_IMPL(avelang_gdn, Autograd, m) {
#define NO_AUTOGRAD(name, f) m.impl(name, torch::CppFunction::makeFallthrough());
  OPERATORS(NO_AUTOGRAD)
}

double scale_or(PyObject* o, int64_t dk) { return o == Py_None ? 1.0 / std::sqrt((double)dk) : number(o); }

// ---------------------------------------------------------------------------------------------- public functions
// The operator F, through the dispatcher.
template <auto F, class... Args>
void call(const char* name, Args&&... args) {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<std::remove_pointer_t<decltype(F)>>();
  op.call(std::forward<Args>(args)...);
}

// prefill(q, k, v, g, beta, scale, initial_state, output_final_state, l2norm, cu_seqlens, z, norm_weight, norm_eps,
//         state_indices, inplace_state, chunk_size, out, out_peers, max_seqlen) -> (o, final or None)
PyObject* prefill(PyObject* const* p) {
  const Tensor &q = tensor(p[0], "q"), &k = tensor(p[1], "k"), &v = tensor(p[2], "v"), &g = tensor(p[3], "g"), &beta = tensor(p[4], "beta");
  const Tensor *s0 = opt_tensor(p[6], "initial_state"), *cu = opt_tensor(p[9], "cu_seqlens"), *z = opt_tensor(p[10], "z"),
               *w = opt_tensor(p[11], "norm_weight"), *idx = opt_tensor(p[13], "state_indices"), *out = opt_tensor(p[16], "out"),
               *peers = opt_tensor(p[17], "out_peers");
  const Shape s = check_common(q, k, v, g, beta, z, cu);
  const int64_t chunk = integer(p[15]);
  REQ(chunk == 64, "chunk_size must be 64, got ", chunk, ".");
  int64_t bound = 0;
  if (p[18] != Py_None) {
    const int64_t m = integer(p[18]);
    REQ(m >= 0, "max_seqlen must be non-negative, got ", m, ".");
    if (cu != nullptr) bound = std::min(m, s.T);
  }
  const Tensor o = prep_out(out, v);
  const Tensor nw = prep_norm_weight(w, z, s, q.device());
  const Tensor final = prep_states(s0, idx, s, q, truth(p[7]), truth(p[14]));
  if (peers != nullptr) {
    REQ(z != nullptr, "out_peers needs z (the stores are fused into the gated norm)");
    REQ(peers->scalar_type() == at::kLong && peers->dim() == 1 && peers->device() == q.device() && peers->is_contiguous(),
        "out_peers must be a contiguous 1-D int64 tensor on ", q.device());
  }
  call<op_prefill>("avelang_gdn::chunk_prefill", q, k, v, g, beta, o, scale_or(p[5], s.dk), opt(s0), opt(final), opt(cu), opt(idx), opt(z), opt(nw),
                   number(p[12]), truth(p[8]), bound, opt(peers));
  return wrap_pair(o, final);
}

// decode(q, k, v, g, beta, scale, initial_state, output_final_state, l2norm, cu_seqlens, state_indices, inplace_state, z,
//        norm_weight, norm_eps, out) -> (o, final or None)
PyObject* decode(PyObject* const* p) {
  const Tensor &q = tensor(p[0], "q"), &k = tensor(p[1], "k"), &v = tensor(p[2], "v"), &g = tensor(p[3], "g"), &beta = tensor(p[4], "beta");
  const Tensor *s0 = opt_tensor(p[6], "initial_state"), *cu = opt_tensor(p[9], "cu_seqlens"), *idx = opt_tensor(p[10], "state_indices"),
               *z = opt_tensor(p[12], "z"), *w = opt_tensor(p[13], "norm_weight"), *out = opt_tensor(p[15], "out");
  const Shape s = check_common(q, k, v, g, beta, z, cu);
  const Tensor o = prep_out(out, v);
  const Tensor nw = prep_norm_weight(w, z, s, q.device());
  const Tensor final = prep_states(s0, idx, s, q, truth(p[7]), truth(p[11]));
  call<op_decode>("avelang_gdn::decode_step", q, k, v, g, beta, o, scale_or(p[5], s.dk), opt(s0), opt(final), opt(cu), opt(idx), opt(z), opt(nw),
                  number(p[14]), truth(p[8]));
  return wrap_pair(o, final);
}

// mixed(q, k, v, g, beta, cu_seqlens, n_decode, state_pool, state_indices, scale, l2norm, z, norm_weight, norm_eps, out) -> o
PyObject* mixed(PyObject* const* p) {
  const Tensor &q = tensor(p[0], "q"), &k = tensor(p[1], "k"), &v = tensor(p[2], "v"), &g = tensor(p[3], "g"), &beta = tensor(p[4], "beta");
  const Tensor *cu = opt_tensor(p[5], "cu_seqlens"), *pool = opt_tensor(p[7], "state_pool"), *idx = opt_tensor(p[8], "state_indices"),
               *z = opt_tensor(p[11], "z"), *w = opt_tensor(p[12], "norm_weight"), *out = opt_tensor(p[14], "out");
  const Shape s = check_common(q, k, v, g, beta, z, cu);
  REQ(cu != nullptr && s.B == 1, "mixed_prefill_decode_step takes a packed batch: B == 1 with cu_seqlens");
  const int64_t nd = integer(p[6]);
  REQ(nd >= 0 && nd <= s.n && nd <= s.T, "n_decode must lie in [0, ", std::min(s.n, s.T), "], got ", nd, ".");
  REQ(pool != nullptr && idx != nullptr, "mixed_prefill_decode_step needs state_pool and state_indices");
  const Tensor o = prep_out(out, v);
  const Tensor nw = prep_norm_weight(w, z, s, q.device());
  prep_states(pool, idx, s, q, true, true);  // its checks
  call<op_mixed>("avelang_gdn::mixed_step", q, k, v, g, beta, o, scale_or(p[9], s.dk), *pool, *cu, *idx, nd, opt(z), opt(nw), number(p[13]), truth(p[10]));
  return wrap(o);
}

// decode_layer(proj, conv_weight, conv_state, A_log, dt_bias, state_pool, state_indices, Hk, Hv, conv_bias, norm_weight,
//              norm_eps, scale, gate_first, out) -> o
PyObject* decode_layer(PyObject* const* p) {
  const Tensor &proj = tensor(p[0], "proj"), &cw = tensor(p[1], "conv_weight"), &cs = tensor(p[2], "conv_state"), &A_log = tensor(p[3], "A_log"),
               &dt_bias = tensor(p[4], "dt_bias"), &pool = tensor(p[5], "state_pool");
  const Tensor *idx = opt_tensor(p[6], "state_indices"), *cb = opt_tensor(p[9], "conv_bias"), *w = opt_tensor(p[10], "norm_weight"),
               *out = opt_tensor(p[14], "out");
  const int64_t Hk = integer(p[7]), Hv = integer(p[8]);
  check_layer(proj, cw, cb, cs, A_log, dt_bias, w, pool, idx, Hk, Hv);
  const Tensor o = out != nullptr ? *out : empty({proj.size(0), Hv, 128}, at::kBFloat16, proj);
  call<op_decode_layer>("avelang_gdn::decode_layer_step", proj, cw, opt(cb), cs, A_log, dt_bias, opt(w), pool, opt(idx), o, Hk, Hv, scale_or(p[12], 128),
                        number(p[11]), truth(p[13]));
  return wrap(o);
}

// rmsnorm(x, z, weight, eps, gate_first, out) -> out
PyObject* rmsnorm(PyObject* const* p) {
  const Tensor &x = tensor(p[0], "x"), &z = tensor(p[1], "z");
  const Tensor *w = opt_tensor(p[2], "weight"), *out = opt_tensor(p[5], "out");
  REQ(x.scalar_type() == at::kBFloat16, "x must have dtype torch.bfloat16, got ", dtype_name(x), ".");
  REQ(z.scalar_type() == at::kBFloat16, "z must have dtype torch.bfloat16, got ", dtype_name(z), ".");
  REQ(x.is_cuda() && z.device() == x.device(), "z must be on device ", x.device(), ", got ", z.device(), ".");
  REQ(z.sizes() == x.sizes(), "z must have shape ", shape_of(x.sizes()), ", got ", shape_of(z.sizes()), ".");
  const int64_t nd = x.dim();
  REQ(nd >= 2 && (x.size(-1) == 64 || x.size(-1) == 128), "last dimension must be 64 or 128, got ", nd > 0 ? x.size(-1) : 0, ".");
  const int64_t d = x.size(-1), H = x.size(-2);
  const Tensor y = out != nullptr ? *out : empty(x.sizes(), at::kBFloat16, x);
  REQ(y.sizes() == x.sizes() && y.scalar_type() == at::kBFloat16 && y.device() == x.device(), "out must be a bf16 tensor of shape ",
      shape_of(x.sizes()), " on ", x.device());
  const auto rows = [&](const Tensor& t) { return t.dim() == 3 ? t : t.reshape({-1, H, d}); };
  const Tensor x3 = rows(x), z3 = rows(z), y3 = rows(y);
  REQ(y3.is_alias_of(y), "out must be viewable as [rows, H, d] without a copy");
  REQ(x3.stride(2) == 1 && z3.stride(2) == 1 && y3.stride(2) == 1, "tensors must be contiguous in their last dimension");
  Tensor nw;
  if (w != nullptr) {
    REQ(w->numel() == d && w->device() == x.device(), "weight must have ", d, " elements on ", x.device());
    nw = f32(*w);
  }
  call<op_rmsnorm>("avelang_gdn::gated_rmsnorm", x3, z3, opt(nw), number(p[3]), truth(p[4]), y3);
  return wrap(y);
}

// conv(x, weight, bias, cu_seqlens, out) -> out
PyObject* conv(PyObject* const* p) {
  const Tensor &x = tensor(p[0], "x"), &w = tensor(p[1], "weight");
  const Tensor *bias = opt_tensor(p[2], "bias"), *cu = opt_tensor(p[3], "cu_seqlens"), *out = opt_tensor(p[4], "out");
  REQ(x.scalar_type() == at::kBFloat16 && x.dim() == 3 && x.is_cuda(), "x must be a bf16 CUDA tensor [B, T, C]");
  REQ(x.stride(2) == 1, "x must be contiguous in its last dimension");
  const int64_t Cn = x.size(2);
  REQ(w.scalar_type() == at::kBFloat16 && w.dim() == 2 && w.size(0) == Cn && w.device() == x.device(), "weight must be a bf16 tensor [", Cn,
      ", W] on ", x.device());
  REQ(w.size(1) >= 2 && w.size(1) <= 4, "kernel width must be 2, 3 or 4, got ", w.size(1), ".");
  REQ(Cn % 8 == 0, "channels must be a multiple of 8, got ", Cn, ".");
  const Tensor wc = w.contiguous();
  Tensor bc;
  if (bias != nullptr) {
    REQ(bias->scalar_type() == at::kBFloat16 && bias->numel() == Cn && bias->device() == x.device(), "bias must be bf16 [", Cn, "] on ", x.device());
    bc = bias->contiguous();
  }
  const Tensor y = out != nullptr ? *out : empty(x.sizes(), at::kBFloat16, x);
  REQ(y.sizes() == x.sizes() && y.scalar_type() == at::kBFloat16 && y.device() == x.device() && y.stride(2) == 1,
      "out must be a bf16 tensor of shape ", shape_of(x.sizes()), " on ", x.device());
  REQ(!y.is_alias_of(x) || y.storage_offset() != x.storage_offset() || x.numel() == 0, "out must not alias x (later tokens read earlier inputs)");
  if (cu != nullptr)
    REQ(x.size(0) == 1 && cu->scalar_type() == at::kInt && cu->device() == x.device() && cu->is_contiguous(),
        "cu_seqlens must be a contiguous int32 tensor on the device of x, with B == 1");
  call<op_conv>("avelang_gdn::conv1d_silu", x, wc, opt(bc), opt(cu), y);
  return wrap(y);
}

// conv_update(x, conv_state, weight, bias, state_indices, out) -> out
PyObject* conv_update(PyObject* const* p) {
  const Tensor &x = tensor(p[0], "x"), &cs = tensor(p[1], "conv_state"), &w = tensor(p[2], "weight");
  const Tensor *bias = opt_tensor(p[3], "bias"), *idx = opt_tensor(p[4], "state_indices"), *out = opt_tensor(p[5], "out");
  REQ(x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.is_cuda() && x.stride(1) == 1, "x must be a bf16 CUDA tensor [N, C]");
  const int64_t N = x.size(0), Cn = x.size(1);
  REQ(w.scalar_type() == at::kBFloat16 && w.dim() == 2 && w.size(0) == Cn && w.device() == x.device() && w.size(1) >= 2 && w.size(1) <= 4,
      "weight must be a bf16 tensor [", Cn, ", W] with W in 2..4 on ", x.device());
  const int64_t W = w.size(1);
  REQ(Cn % 8 == 0, "channels must be a multiple of 8, got ", Cn, ".");
  REQ(cs.scalar_type() == at::kBFloat16 && cs.dim() == 3 && cs.size(1) == W - 1 && cs.size(2) == Cn && cs.is_contiguous() && cs.device() == x.device(),
      "conv_state must be a contiguous bf16 tensor [slots, ", W - 1, ", ", Cn, "] on ", x.device());
  if (idx != nullptr)
    REQ(idx->scalar_type() == at::kInt && idx->dim() == 1 && idx->size(0) == N && idx->device() == x.device() && idx->is_contiguous(),
        "state_indices must be a contiguous int32 tensor (", N, ",) on ", x.device());
  else
    REQ(cs.size(0) >= N, "conv_state needs one slot per sequence when state_indices is not given");
  const Tensor wc = w.contiguous();
  const Tensor y = out != nullptr ? *out : empty({N, Cn}, at::kBFloat16, x);
  REQ(y.sizes() == x.sizes() && y.scalar_type() == at::kBFloat16 && y.device() == x.device() && y.stride(1) == 1,
      "out must be a bf16 tensor of shape ", shape_of(x.sizes()), " on ", x.device());
  const Tensor bc = bias != nullptr ? bias->contiguous() : Tensor();
  call<op_conv_update>("avelang_gdn::conv1d_update", x, cs, wc, opt(bc), opt(idx), y);
  return wrap(y);
}

// gate(a, b, A_log, dt_bias) -> (g, beta)
PyObject* gate(PyObject* const* p) {
  const Tensor &a = tensor(p[0], "a"), &b = tensor(p[1], "b");
  REQ(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16 && a.is_cuda(), "a and b must be bf16 CUDA tensors");
  REQ(a.dim() >= 1 && a.sizes() == b.sizes() && a.stride(-1) == 1 && b.stride(-1) == 1, "a and b must share a shape [..., Hv]");
  const int64_t Hv = a.size(-1);
  const Tensor a2 = a.dim() != 2 ? a.reshape({-1, Hv}) : a, b2 = b.dim() != 2 ? b.reshape({-1, Hv}) : b;
  REQ(a2.is_alias_of(a) && b2.is_alias_of(b), "a and b must be viewable as [rows, Hv]");
  const Tensor A_log = f32(tensor(p[2], "A_log")), dt_bias = f32(tensor(p[3], "dt_bias"));
  REQ(A_log.numel() == Hv && dt_bias.numel() == Hv && A_log.device() == a.device(), "A_log and dt_bias must have ", Hv, " elements");
  const Tensor g = empty(a.sizes(), at::kFloat, a), beta = empty(a.sizes(), at::kFloat, a);
  call<op_gate>("avelang_gdn::gate_beta", a2, b2, A_log, dt_bias, g, beta);
  return wrap_pair(g, beta);
}

// gemm(A, B, out) -> out
PyObject* gemm(PyObject* const* p) {
  const Tensor &A = tensor(p[0], "A"), &B = tensor(p[1], "B");
  const Tensor* out = opt_tensor(p[2], "out");
  REQ(A.scalar_type() == at::kBFloat16, "A must have dtype torch.bfloat16, got ", dtype_name(A), ".");
  REQ(B.scalar_type() == at::kBFloat16, "B must have dtype torch.bfloat16, got ", dtype_name(B), ".");
  REQ(A.dim() == 2 && B.dim() == 2 && A.size(1) == B.size(1), "A [M, K] and B [N, K] must share K, got ", shape_of(A.sizes()), " and ",
      shape_of(B.sizes()), ".");
  REQ(A.is_cuda() && B.device() == A.device(), "A and B must be CUDA tensors on one device, got ", A.device(), " and ", B.device(), ".");
  const int64_t m = A.size(0), k = A.size(1), n = B.size(0);
  REQ(k % 8 == 0 && k != 0, "K must be a positive multiple of 8, got ", k, ".");
  REQ(A.stride(1) == 1 && B.stride(1) == 1, "A and B must be contiguous in their last dimension.");
  if (out != nullptr) {
    REQ(out->dim() == 2 && out->size(0) == m && out->size(1) == n, "out must have shape ", shape_of({m, n}), ", got ", shape_of(out->sizes()), ".");
    REQ(out->scalar_type() == at::kBFloat16, "out must have dtype torch.bfloat16, got ", dtype_name(*out), ".");
    REQ(out->device() == A.device(), "out must be on device ", A.device(), ", got ", out->device(), ".");
    REQ(out->stride(1) == 1, "out must be contiguous in its last dimension.");
  }
  const Tensor c = out != nullptr ? *out : empty({m, n}, at::kBFloat16, A);
  call<op_gemm>("avelang_gdn::gemm_bf16_nt", A, B, c);
  return wrap(c);
}

// backward(q, k, v, g, beta, d_o, scale, initial_state, d_final_state, cu_seqlens) -> (dq, dk, dv, dg, dbeta, ds0 or None)
PyObject* backward(PyObject* const* p) {
  const Tensor &q = tensor(p[0], "q"), &k = tensor(p[1], "k"), &v = tensor(p[2], "v"), &g = tensor(p[3], "g"), &beta = tensor(p[4], "beta"),
               &d_o = tensor(p[5], "d_o");
  const Tensor *s0 = opt_tensor(p[7], "initial_state"), *ds = opt_tensor(p[8], "d_final_state"), *cu = opt_tensor(p[9], "cu_seqlens");
  const Shape s = check_common(q, k, v, g, beta, nullptr, cu);
  REQ(s.dk == 128 && s.dv == 128, "the backward pass is built for head dims (128, 128), got (", s.dk, ", ", s.dv, ").");
  REQ(d_o.scalar_type() == at::kBFloat16 && d_o.sizes() == v.sizes() && d_o.device() == q.device() && d_o.stride(3) == 1,
      "d_o must be a bf16 tensor of shape ", shape_of(v.sizes()), " on ", q.device());
  const std::pair<const char*, const Tensor*> states[] = {{"initial_state", s0}, {"d_final_state", ds}};
  for (const auto& [name, t] : states)
    if (t != nullptr)
      REQ(t->scalar_type() == at::kFloat && t->dim() == 4 && t->size(0) == s.n && t->size(1) == s.Hv && t->size(2) == s.dk &&
              t->size(3) == s.dv && t->is_contiguous() && t->device() == q.device(),
          name, " must be a contiguous fp32 tensor (", s.n, ", ", s.Hv, ", ", s.dk, ", ", s.dv, ") on ", q.device());
  const Tensor dq = empty(q.sizes(), at::kBFloat16, q), dk = empty(q.sizes(), at::kBFloat16, q), dv = empty(v.sizes(), at::kBFloat16, v);
  const Tensor dg = empty(g.sizes(), at::kFloat, q), dbeta = empty(g.sizes(), at::kFloat, q);
  Tensor ds0;
  if (s0 != nullptr) {
    ds0 = empty({s.n, s.Hv, s.dk, s.dv}, at::kFloat, q);
    if (s.T == 0 && ds != nullptr) ds0.copy_(*ds);  // no kernel runs: the gradient of the states passes through
    else if (s.T == 0) ds0.zero_();
  }
  call<op_backward>("avelang_gdn::recurrent_backward", q, k, v, g, beta, d_o, scale_or(p[6], s.dk), opt(s0), opt(ds), opt(cu), dq, dk, dv, dg, dbeta, opt(ds0));
  PyObject* r = PyTuple_New(6);
  if (r == nullptr) throw python_error();
  const Tensor* out[] = {&dq, &dk, &dv, &dg, &dbeta, &ds0};
  for (int i = 0; i < 6; ++i) {
    if (!out[i]->defined()) Py_INCREF(Py_None);
    PyTuple_SET_ITEM(r, i, out[i]->defined() ? wrap(*out[i]) : Py_None);
  }
  return r;
}

PyObject* none() { Py_RETURN_NONE; }
// status_word(device_index) -> the device status word; workspace-independent
PyObject* py_status_word(PyObject* const* p) { return wrap(status_word(at::Device(at::kCUDA, (c10::DeviceIndex)integer(p[0])))); }

// bind(path): resolves the entry points of the C library (already loaded by the Python layer)
PyObject* bind(PyObject* const* p) {
  const char* path = PyUnicode_AsUTF8(p[0]);
  if (path == nullptr) throw python_error();
  void* lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  REQ(lib != nullptr, "cannot load ", path);
#define RESOLVE(field, symbol)                                                 \
  api.field = reinterpret_cast<decltype(api.field)>(dlsym(lib, #symbol));      \
  REQ(api.field != nullptr, path, " has no ", #symbol)
  RESOLVE(chunk_prefill, ave_gdn_chunk_prefill);
  RESOLVE(prefill_workspace_bytes, ave_gdn_prefill_workspace_bytes);
  RESOLVE(decode_step, ave_gdn_decode_step);
  RESOLVE(mixed_step, ave_gdn_mixed_step);
  RESOLVE(gated_rmsnorm, ave_gdn_gated_rmsnorm);
  RESOLVE(gemm_bf16_nt, ave_gemm_bf16_nt);
  RESOLVE(conv1d_silu, ave_gdn_conv1d_silu);
  RESOLVE(conv1d_update, ave_gdn_conv1d_update);
  RESOLVE(gate_beta, ave_gdn_gate_beta);
  RESOLVE(decode_layer_step, ave_gdn_decode_layer_step);
  RESOLVE(recurrent_backward, ave_gdn_recurrent_backward);
  RESOLVE(backward_workspace_bytes, ave_gdn_backward_workspace_bytes);
  RESOLVE(status_string, ave_gdn_status_string);
  RESOLVE(last_cuda_error, ave_gdn_last_cuda_error);
#undef RESOLVE
  return none();
}

// ---------------------------------------------------------------------------------------------- module
template <PyObject* (*F)(PyObject* const*), int N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != N) {
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", N, n);
    return nullptr;
  }
  return F(args);
  END_HANDLE_TH_ERRORS
}
#define ENTRY(name, fn, n) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<fn, n>)), METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    ENTRY("bind", bind, 1),
    ENTRY("status_word", py_status_word, 1),
    ENTRY("prefill", prefill, 19),
    ENTRY("decode", decode, 16),
    ENTRY("mixed", mixed, 15),
    ENTRY("decode_layer", decode_layer, 15),
    ENTRY("rmsnorm", rmsnorm, 6),
    ENTRY("conv", conv, 5),
    ENTRY("conv_update", conv_update, 6),
    ENTRY("gate", gate, 4),
    ENTRY("gemm", gemm, 3),
    ENTRY("backward", backward, 10),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  c10::FreeCudaMemoryCallbacksRegistry()->Register(text("avelang_gdn_scratch ", &scratch_pool()), [] { return std::make_unique<ReleaseScratch>(); }, "");
  return PyModule_Create(&module);
}
