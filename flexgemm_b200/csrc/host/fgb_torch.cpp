// The torch side of the library in C++: tensor checks, allocation, autograd nodes and the calls into the C ABI
// (include/flexgemm_b200.h) for the convolutions and their neighbour caches.
//
// A small layer is bound by the host: its kernels take some ten microseconds each, and a Python wrapper per kernel
// (tensor allocation, ctypes call, event or memset) costs as much again.  Here one Python call runs a whole forward
// pass, and the backward pass runs inside the autograd engine without entering Python at all.
//
// The functions take the fast way or none: where an argument is not what the kernels take directly (another device, a
// dtype, a layout, an empty input) they return None and the Python code beside them, which knows every case and raises
// the documented errors, does the call.
//
// The CUDA library is not linked: its entry points are looked up in the handle that the ctypes binding has loaded, so
// that both sides always run the same file.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <atomic>
#include <memory>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "../../../include/flexgemm_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// ------------------------------------------------------------------ the CUDA library
#define FGB_TORCH_API(X)                                                                                            \
  X(fgb_error_string) X(fgb_status_set_mirror) X(fgb_conv_call_workspace_bytes) X(fgb_conv_call_fprop)                \
  X(fgb_conv_call_dgrad) X(fgb_wgrad_call_workspace_bytes) X(fgb_wgrad_call_run) X(fgb_resize_rows)                   \
  X(fgb_bias_grad_workspace_bytes) X(fgb_subm_conv_bias_grad) X(fgb_subm_cache_scratch_bytes)                         \
  X(fgb_subm_cache_build) X(fgb_pp_valid_signal) X(fgb_hash_table_bytes)                                    \
  X(fgb_strided_grid_bytes) X(fgb_strided_mark) X(fgb_strided_build_bytes) X(fgb_strided_build)                       \
  X(fgb_grid_sample_fused) X(fgb_indice_weighted_sum_grad_full_bytes) X(fgb_indice_weighted_sum_grad)
struct Api {
#define X(f) decltype(&::f) f = nullptr;
  FGB_TORCH_API(X)
#undef X
} api;

void check(int64_t rc, const char* what) {  // as _cabi.check: arguments -> ValueError, launches -> RuntimeError
  if (rc >= 0 && rc < FGB_E_CUDA_BASE) return;
  const std::string msg = std::string(what) + " failed: " + api.fgb_error_string(static_cast<int>(rc)) + " (code " + std::to_string(rc) + ")";
  TORCH_CHECK_VALUE(rc >= 0, msg);
  throw std::runtime_error(msg);
}
int64_t check_bytes(int64_t n, const char* what) {
  if (n < 0) check(n, what);
  return n;
}

// ------------------------------------------------------------------ per-device state
constexpr int kMaxDevices = 64;
struct DeviceState {
  std::mutex mu;
  Tensor status;                       // int32 [1]: the device status word of the conv kernels
  std::atomic<volatile int32_t*> mirror{nullptr};  // its copy in mapped host memory
};
DeviceState g_device[kMaxDevices];

DeviceState& device_state(c10::DeviceIndex d) {
  TORCH_CHECK(d >= 0 && d < kMaxDevices, "device index out of range");
  DeviceState& s = g_device[d];
  if (s.mirror.load(std::memory_order_acquire) != nullptr) return s;
  std::lock_guard<std::mutex> lock(s.mu);
  if (s.mirror.load(std::memory_order_relaxed) == nullptr) {
    c10::cuda::CUDAGuard guard(d);
    void *host = nullptr, *dev = nullptr;
    C10_CUDA_CHECK(cudaHostAlloc(&host, 64, cudaHostAllocMapped | cudaHostAllocPortable));
    *static_cast<volatile int32_t*>(host) = 0;
    C10_CUDA_CHECK(cudaHostGetDevicePointer(&dev, host, 0));
    s.status = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, d));
    C10_CUDA_CHECK(cudaStreamSynchronize(c10::cuda::getCurrentCUDAStream(d)));  // once: usable from every stream
    check(api.fgb_status_set_mirror(static_cast<const int32_t*>(s.status.data_ptr()), static_cast<int32_t*>(dev)), "fgb_status_set_mirror");
    s.mirror.store(static_cast<volatile int32_t*>(host), std::memory_order_release);
  }
  return s;
}

[[noreturn]] void throw_soft_error(int code) {
  const char* what = code == FGB_S_TABLE_FULL     ? "hash table full (raise the hashmap ratio)"
                     : code == FGB_S_WAIT_TIMEOUT ? "a bounded barrier wait ran out inside a kernel"
                                                  : nullptr;
  throw std::runtime_error("flexgemm_b200 device-side error: " + (what != nullptr ? std::string(what) : "code " + std::to_string(code)));
}

// A soft error that a kernel has reported: the word is cleared, so that the calls after the exception run normally, and
// the error raised.  Costs a read of host memory when there is none.
void poll(DeviceState& s, c10::cuda::CUDAStream stream) {
  volatile int32_t* mirror = s.mirror.load(std::memory_order_acquire);
  const int code = *mirror;
  if (code == 0) return;
  C10_CUDA_CHECK(cudaDeviceSynchronize());  // kernels that still see the word would store it again
  C10_CUDA_CHECK(cudaMemsetAsync(s.status.data_ptr(), 0, 4, stream));
  C10_CUDA_CHECK(cudaStreamSynchronize(stream));
  *mirror = 0;
  throw_soft_error(code);
}

// Zeroed device words, handed out once each: a slice of a buffer that is zeroed 4096 words at a time on the stream that
// uses it.  One buffer per stream, dropped when it is used up and all of them when streams come and go.  Whoever takes
// words holds their buffer until the work on them is queued: another thread on the same stream may drop it from the pool
// meanwhile, and from then on only the allocator's stream order keeps later users of the memory behind that work.
struct ZeroPool {
  Tensor buf;
  int64_t used = 0;
};
std::mutex g_zero_mu;
std::unordered_map<uint64_t, ZeroPool> g_zero;
constexpr int64_t kZeroPoolWords = 4096;
constexpr size_t kMaxZeroPools = 64;
struct ZeroedWords {
  Tensor buf;  // holds the words
  uint32_t* words = nullptr;
};

// None while the stream is being captured: a graph runs its calls again and must zero their words itself, each time, in
// memory that is its own (the library does so in a call's workspace), and what a capture allocates stays out of the pool.
ZeroedWords zeroed_words(c10::cuda::CUDAStream stream, int64_t words) {
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return {};
  words = (words + 7) & ~int64_t(7);
  std::lock_guard<std::mutex> lock(g_zero_mu);
  const uint64_t key = reinterpret_cast<uint64_t>(stream.stream()) * 64 + static_cast<uint64_t>(stream.device_index());
  auto it = g_zero.find(key);
  if (it == g_zero.end()) {
    if (g_zero.size() >= kMaxZeroPools) g_zero.clear();
    it = g_zero.emplace(key, ZeroPool{}).first;
  }
  ZeroPool& p = it->second;
  if (!p.buf.defined() || p.used + words > kZeroPoolWords) {
    p.buf = at::detail::empty_cuda({kZeroPoolWords}, at::kInt, at::Device(at::kCUDA, stream.device_index()), std::nullopt);
    C10_CUDA_CHECK(cudaMemsetAsync(p.buf.data_ptr(), 0, kZeroPoolWords * 4, stream));
    p.used = 0;
  }
  const ZeroedWords out{p.buf, static_cast<uint32_t*>(p.buf.data_ptr()) + p.used};
  p.used += words;
  return out;
}

// Mapped pinned words into which a build reports its counts; returned to the free list after each build, so there are as
// many as builds have ever run at the same time.
struct HostWords {
  volatile uint32_t* host = nullptr;
  uint32_t* dev = nullptr;
  uint32_t seq = 0;
};
std::mutex g_words_mu;
std::vector<HostWords> g_words_free;
int64_t g_words_made = 0;
constexpr int kHostWords = 16;  // per slot: FGB_HOST_WORDS, and a line of its own
static_assert(FGB_HOST_WORDS <= kHostWords);

// What a kernel has told the host.
struct Told {
  uint32_t count, status;
};

// A slot for the length of one build.  It goes back when the build has reported, and also when the call ends before:
// at once if nothing that writes to it can have been queued, after the stream's work otherwise (and not at all where the
// stream cannot be waited for).
class HostSlot {
 public:
  HostSlot() = default;
  HostSlot(HostSlot&& o) noexcept { std::swap(w_, o.w_), std::swap(stream_, o.stream_), std::swap(queued_, o.queued_); }
  HostSlot(const HostSlot&) = delete;
  HostSlot& operator=(const HostSlot&) = delete;
  ~HostSlot() {
    if (w_.host == nullptr) return;
    if (queued_ && cudaStreamSynchronize(stream_) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    give_back();
  }
  // for the next call into the library, whose stream is `stream`
  void take(cudaStream_t stream, uint32_t** dev, uint32_t* seq) {
    std::lock_guard<std::mutex> lock(g_words_mu);
    if (g_words_free.empty()) {
      void *host = nullptr, *mapped = nullptr;
      constexpr int kSlots = 16;
      C10_CUDA_CHECK(cudaHostAlloc(&host, kSlots * kHostWords * 4, cudaHostAllocMapped | cudaHostAllocPortable));
      C10_CUDA_CHECK(cudaHostGetDevicePointer(&mapped, host, 0));
      memset(host, 0, kSlots * kHostWords * 4);
      for (int i = 0; i < kSlots; ++i)
        g_words_free.push_back({static_cast<volatile uint32_t*>(host) + i * kHostWords, static_cast<uint32_t*>(mapped) + i * kHostWords, 0});
      g_words_made += kSlots;
    }
    w_ = g_words_free.back();
    g_words_free.pop_back();
    stream_ = stream, queued_ = false;
    *dev = w_.dev, *seq = ++w_.seq;
  }
  // the library is about to queue the kernels that write to the slot
  void queued() { queued_ = true; }
  // Waits until the stream's work has stored the sequence number; the GIL is released meanwhile.
  Told take_back() {
    std::exception_ptr failed;
    Py_BEGIN_ALLOW_THREADS;
    try {
      wait();
    } catch (...) {
      failed = std::current_exception();
    }
    Py_END_ALLOW_THREADS;
    if (failed) std::rethrow_exception(failed);
    const Told r{w_.host[FGB_HOST_COUNT], w_.host[FGB_HOST_STATUS]};
    give_back();
    return r;
  }

 private:
  void wait() const {
    for (uint64_t i = 1; w_.host[FGB_HOST_SEQ] != w_.seq; ++i) {
#if defined(__x86_64__)
      __builtin_ia32_pause();
#endif
      if ((i & 0xFFFu) == 0) {
        const cudaError_t e = cudaStreamQuery(stream_);
        if (e == cudaErrorNotReady) continue;
        C10_CUDA_CHECK(e);
        if (w_.host[FGB_HOST_SEQ] != w_.seq) throw std::runtime_error("flexgemm_b200: the neighbour-map build ended without its pair count");
      }
    }
    std::atomic_thread_fence(std::memory_order_acquire);
  }
  void give_back() {
    std::lock_guard<std::mutex> lock(g_words_mu);
    g_words_free.push_back(w_);
    w_ = HostWords{};
  }
  HostWords w_;
  cudaStream_t stream_ = nullptr;
  bool queued_ = false;
};

// ------------------------------------------------------------------ tensors
Tensor new_tensor(at::IntArrayRef size, at::ScalarType dtype, at::Device dev) { return at::detail::empty_cuda(size, dtype, dev, std::nullopt); }
c10::DataPtr scratch(int64_t bytes) { return c10::cuda::CUDACachingAllocator::get()->allocate(static_cast<size_t>(bytes > 0 ? bytes : 1)); }
const void* ptr(const Tensor& t) { return t.defined() && t.numel() > 0 ? t.const_data_ptr() : nullptr; }
template <typename T>
const T* cptr(const Tensor& t) { return static_cast<const T*>(ptr(t)); }

int dtype_code(at::ScalarType t, bool tf32) {  // -1: not a feature dtype
  switch (t) {
    case at::kHalf: return FGB_F16;
    case at::kBFloat16: return FGB_BF16;
    case at::kFloat: return tf32 ? FGB_F32_TF32 : FGB_F32_IEEE;
    default: return -1;
  }
}

// rows of a [rows, width] matrix cut or zero-padded to `width_out` elements, rows from rows_in on zero
Tensor resize_rows(const Tensor& t, int64_t rows_in, int64_t width, at::IntArrayRef out_size, int64_t rows_out, int64_t width_out,
                   cudaStream_t s) {
  Tensor out = new_tensor(out_size, t.scalar_type(), t.device());
  const int64_t eb = t.element_size();
  check(api.fgb_resize_rows(ptr(t), out.numel() > 0 ? out.data_ptr() : nullptr, rows_in, rows_out, width * eb, width_out * eb, s), "fgb_resize_rows");
  return out;
}
int64_t round_up(int64_t c, int64_t m) { return (c + m - 1) / m * m; }

// ------------------------------------------------------------------ the passes
struct Maps {  // a neighbour map with its row order, tile masks and schedule
  Tensor nbr, sorted_idx, masks, order;
};
struct Pairs {
  Tensor vs_i, vs_o, seg, block_offsets;
};

// Channels of a pass as the kernels take them (rows of whole 16-byte pieces), and the padded copies where they differ.
struct Channels {
  int64_t ci, co, ci_p, co_p;
  Channels(int64_t ci_, int64_t co_, int64_t eb) : ci(ci_), co(co_), ci_p(round_up(ci_, 16 / eb)), co_p(round_up(co_, 16 / eb)) {}
  bool exact() const { return ci == ci_p && co == co_p; }
};
Tensor pad_channels(const Tensor& t, int64_t c, int64_t c_p, cudaStream_t s) {
  return c == c_p ? t : resize_rows(t, t.size(0), c, {t.size(0), c_p}, t.size(0), c_p, s);
}
Tensor pad_weight(const Tensor& w, const Channels& ch, int64_t V, cudaStream_t s) {
  if (ch.exact()) return w;
  return resize_rows(w, ch.co * V, ch.ci, {ch.co_p, V, ch.ci_p}, ch.co_p * V, ch.ci_p, s);
}

// weight: [Co, ..., Ci] with V = product of the extents between
Tensor run_fprop(const Tensor& feats, const Tensor& weight, const Tensor& bias, const Maps& m, int64_t V, int dtype) {
  const auto stream = c10::cuda::getCurrentCUDAStream(feats.device().index());
  DeviceState& ds = device_state(feats.device().index());
  poll(ds, stream);
  const Channels ch(feats.size(1), weight.size(0), feats.element_size());
  const Tensor x = pad_channels(feats, ch.ci, ch.ci_p, stream);
  const Tensor w = pad_weight(weight, ch, V, stream);
  const Tensor b = !bias.defined() || ch.co == ch.co_p ? bias : resize_rows(bias, 1, ch.co, {ch.co_p}, 1, ch.co_p, stream);
  const int64_t n = m.nbr.size(0);
  Tensor out = new_tensor({n, ch.co_p}, feats.scalar_type(), feats.device());
  fgb_conv_call c{};
  c.x = ptr(x), c.weight = ptr(w), c.bias = b.defined() ? ptr(b) : nullptr;
  c.neighbor_map = cptr<uint32_t>(m.nbr), c.sorted_idx = cptr<int64_t>(m.sorted_idx), c.tile_masks = cptr<uint32_t>(m.masks);
  c.block_order = cptr<uint32_t>(m.order);
  c.out = n > 0 ? out.data_ptr() : nullptr;
  c.n = n, c.n_src = feats.size(0);
  c.ci = static_cast<int32_t>(ch.ci_p), c.co = static_cast<int32_t>(ch.co_p), c.v = static_cast<int32_t>(V), c.dtype = dtype;
  c.workspace_bytes = check_bytes(api.fgb_conv_call_workspace_bytes(&c, 0), "fgb_conv_call_workspace_bytes");
  const c10::DataPtr ws = scratch(c.workspace_bytes);
  c.workspace = ws.get();
  const ZeroedWords counter = zeroed_words(stream, 1);
  c.counters = counter.words;
  c.status = static_cast<int32_t*>(ds.status.data_ptr());
  check(api.fgb_conv_call_fprop(&c, stream), "fgb_conv_call_fprop");
  return ch.co == ch.co_p ? out : resize_rows(out, n, ch.co_p, {n, ch.co}, n, ch.co, stream);
}

Tensor run_dgrad(const Tensor& grad_out, const Tensor& weight, const Maps& m, int64_t V, int64_t ci, int dtype, bool mirror) {
  const auto stream = c10::cuda::getCurrentCUDAStream(grad_out.device().index());
  DeviceState& ds = device_state(grad_out.device().index());
  const Channels ch(ci, grad_out.size(1), grad_out.element_size());
  const Tensor g = pad_channels(grad_out, ch.co, ch.co_p, stream);
  const Tensor w = pad_weight(weight, ch, V, stream);
  const int64_t n = m.nbr.size(0);
  Tensor out = new_tensor({n, ch.ci_p}, grad_out.scalar_type(), grad_out.device());
  fgb_conv_call c{};
  c.x = ptr(g), c.weight = ptr(w);
  c.neighbor_map = cptr<uint32_t>(m.nbr), c.sorted_idx = cptr<int64_t>(m.sorted_idx), c.tile_masks = cptr<uint32_t>(m.masks);
  c.block_order = cptr<uint32_t>(m.order);
  c.out = n > 0 ? out.data_ptr() : nullptr;
  c.n = n, c.n_src = grad_out.size(0);
  c.ci = static_cast<int32_t>(ch.ci_p), c.co = static_cast<int32_t>(ch.co_p), c.v = static_cast<int32_t>(V), c.dtype = dtype;
  c.mirror = mirror ? 1 : 0;
  c.workspace_bytes = check_bytes(api.fgb_conv_call_workspace_bytes(&c, 1), "fgb_conv_call_workspace_bytes");
  const c10::DataPtr ws = scratch(c.workspace_bytes);
  c.workspace = ws.get();
  const ZeroedWords counter = zeroed_words(stream, 1);
  c.counters = counter.words;
  c.status = static_cast<int32_t*>(ds.status.data_ptr());
  check(api.fgb_conv_call_dgrad(&c, stream), "fgb_conv_call_dgrad");
  return ch.ci == ch.ci_p ? out : resize_rows(out, n, ch.ci_p, {n, ch.ci}, n, ch.ci, stream);
}

// weight gradient in `weight_size`, and the bias gradient where it is wanted
std::pair<Tensor, Tensor> run_wgrad(const Tensor& grad_out, const Tensor& feats, const Pairs& p, at::IntArrayRef weight_size, int64_t V,
                                    int dtype, bool want_bias) {
  const auto stream = c10::cuda::getCurrentCUDAStream(feats.device().index());
  DeviceState& ds = device_state(feats.device().index());
  const Channels ch(feats.size(1), grad_out.size(1), feats.element_size());
  const Tensor g = pad_channels(grad_out, ch.co, ch.co_p, stream);
  const Tensor x = pad_channels(feats, ch.ci, ch.ci_p, stream);
  Tensor gw = ch.exact() ? new_tensor(weight_size, feats.scalar_type(), feats.device())
                         : new_tensor({ch.co_p, V, ch.ci_p}, feats.scalar_type(), feats.device());
  Tensor gb = want_bias ? new_tensor({ch.co_p}, feats.scalar_type(), feats.device()) : Tensor();
  fgb_wgrad_call c{};
  c.grad_out = ptr(g), c.feats = ptr(x);
  c.valid_signal_i = cptr<uint32_t>(p.vs_i), c.valid_signal_o = cptr<uint32_t>(p.vs_o), c.valid_signal_seg = cptr<uint32_t>(p.seg);
  c.block_offsets = p.block_offsets.defined() ? cptr<uint32_t>(p.block_offsets) : nullptr;
  c.grad_weight = gw.data_ptr(), c.grad_bias = want_bias ? gb.data_ptr() : nullptr;
  c.n_out = grad_out.size(0), c.n_in = feats.size(0), c.n_pairs = p.vs_i.size(0);
  c.ci = static_cast<int32_t>(ch.ci_p), c.co = static_cast<int32_t>(ch.co_p), c.v = static_cast<int32_t>(V), c.dtype = dtype;
  c.workspace_bytes = check_bytes(api.fgb_wgrad_call_workspace_bytes(&c), "fgb_wgrad_call_workspace_bytes");
  const c10::DataPtr ws = scratch(c.workspace_bytes);
  c.workspace = ws.get();
  c.status = static_cast<int32_t*>(ds.status.data_ptr());
  check(api.fgb_wgrad_call_run(&c, stream), "fgb_wgrad_call_run");
  if (!ch.exact()) gw = resize_rows(gw, ch.co * V, ch.ci_p, weight_size, ch.co * V, ch.ci, stream);
  if (want_bias && ch.co != ch.co_p) gb = resize_rows(gb, 1, ch.co_p, {ch.co}, 1, ch.co, stream);
  return {gw, gb};
}

Tensor run_bias_grad(const Tensor& grad_out, int dtype) {
  const auto stream = c10::cuda::getCurrentCUDAStream(grad_out.device().index());
  const int64_t co = grad_out.size(1);
  Tensor gb = new_tensor({co}, grad_out.scalar_type(), grad_out.device());
  const int64_t bytes = check_bytes(api.fgb_bias_grad_workspace_bytes(static_cast<int>(co)), "fgb_bias_grad_workspace_bytes");
  const c10::DataPtr ws = scratch(bytes);
  check(api.fgb_subm_conv_bias_grad(ptr(grad_out), gb.data_ptr(), nullptr, grad_out.size(0), static_cast<int>(co), dtype, ws.get(), bytes, stream),
        "fgb_subm_conv_bias_grad");
  return gb;
}

struct Grads {
  Tensor feats, weight, bias;
};
Grads run_backward(const Tensor& grad_output, const Tensor& feats, const Tensor& weight, const Maps& bwd, const Pairs& pairs, bool mirror,
                   int64_t V, int dtype, bool need_x, bool need_w, bool need_b) {
  c10::cuda::CUDAGuard guard(feats.device());
  const auto stream = c10::cuda::getCurrentCUDAStream(feats.device().index());
  poll(device_state(feats.device().index()), stream);
  const Tensor g = grad_output.contiguous();
  Grads r;
  if (need_x) r.feats = run_dgrad(g, weight, bwd, V, feats.size(1), dtype, mirror);
  if (need_w) std::tie(r.weight, r.bias) = run_wgrad(g, feats, pairs, weight.sizes(), V, dtype, need_b);
  else if (need_b) r.bias = run_bias_grad(g, dtype);
  return r;
}

// ------------------------------------------------------------------ Python objects
PyObject *s_neighbor_map, *s_gray_code, *s_sorted_idx, *s_tile_masks, *s_block_order, *s_vs_i, *s_vs_o, *s_seg, *s_block_offsets, *s_build_status;
PyObject *s_neighbor_map_bwd, *s_sorted_idx_bwd, *s_tile_masks_bwd, *s_block_order_bwd, *s_ensure_bwd, *s_m_tile_masks, *s_m_block_order,
    *s_m_tile_masks_bwd, *s_m_block_order_bwd, *s_tile_rows, *s_gray_code_bwd;
PyObject* s_empty_tuple;

struct PyError {};  // a Python exception is set

Tensor tensor_arg(PyObject* o) { return o != Py_None && THPVariable_Check(o) ? THPVariable_Unpack(o) : Tensor(); }

// attribute of a cache as a tensor; undefined when it is missing or None
Tensor cache_tensor(PyObject* cache, PyObject* name) {
  PyObject* v = PyObject_GetAttr(cache, name);
  if (v == nullptr) {
    if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw PyError{};
    PyErr_Clear();
    return Tensor();
  }
  Tensor t = tensor_arg(v);
  Py_DECREF(v);
  return t;
}
// the same, made by the cache's own method (tile rows as argument) when it is not there yet
Tensor cache_tensor_or(PyObject* cache, PyObject* name, PyObject* method) {
  Tensor t = cache_tensor(cache, name);
  if (t.defined()) return t;
  PyObject* v = PyObject_CallMethodObjArgs(cache, method, s_tile_rows, nullptr);
  if (v == nullptr) throw PyError{};
  t = tensor_arg(v);
  Py_DECREF(v);
  return t;
}
void set_tensor(PyObject* cache, PyObject* name, const Tensor& t) {
  PyObject* v = THPVariable_Wrap(t);
  const int rc = v != nullptr ? PyObject_SetAttr(cache, name, v) : -1;
  Py_XDECREF(v);
  if (rc != 0) throw PyError{};
}

Maps fwd_maps(PyObject* cache) {
  Maps m;
  m.nbr = cache_tensor(cache, s_neighbor_map);
  m.sorted_idx = cache_tensor(cache, s_sorted_idx);
  if (!m.nbr.defined() || !m.sorted_idx.defined()) return Maps{};
  m.masks = cache_tensor_or(cache, s_tile_masks, s_m_tile_masks);
  m.order = cache_tensor_or(cache, s_block_order, s_m_block_order);
  return m;
}
Maps bwd_maps(PyObject* cache) {
  Maps m;
  m.nbr = cache_tensor(cache, s_neighbor_map_bwd);
  if (!m.nbr.defined()) return Maps{};
  PyObject* r = PyObject_CallMethodObjArgs(cache, s_ensure_bwd, nullptr);
  if (r == nullptr) throw PyError{};
  Py_DECREF(r);
  m.sorted_idx = cache_tensor(cache, s_sorted_idx_bwd);
  m.masks = cache_tensor_or(cache, s_tile_masks_bwd, s_m_tile_masks_bwd);
  m.order = cache_tensor_or(cache, s_block_order_bwd, s_m_block_order_bwd);
  return m;
}
Pairs pairs_of(PyObject* cache) {
  Pairs p;
  p.vs_i = cache_tensor(cache, s_vs_i);
  if (!p.vs_i.defined()) return p;
  p.vs_o = cache_tensor(cache, s_vs_o);
  p.seg = cache_tensor(cache, s_seg);
  p.block_offsets = cache_tensor(cache, s_block_offsets);
  return p;
}

// k integers of a sequence; false when it is none
bool int_args(PyObject* seq, int k, int64_t* out) {
  PyObject* f = PySequence_Fast(seq, "");
  if (f == nullptr) {
    PyErr_Clear();
    return false;
  }
  bool ok = PySequence_Fast_GET_SIZE(f) == k;
  for (int i = 0; ok && i < k; ++i) {
    out[i] = PyLong_AsLongLong(PySequence_Fast_GET_ITEM(f, i));
    if (out[i] == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      ok = false;
    }
  }
  Py_DECREF(f);
  return ok;
}

// 32-bit keys while a (N, C, W, H, D) grid has fewer than 2^32 cells, else 64-bit; 0 where those cannot tell its cells
// apart either (utils.hashmap_key_bits, which raises for such a grid)
int key_bits_of(const int64_t* shape) {
  unsigned __int128 cells = 1;
  for (int i : {0, 2, 3, 4}) {
    if (shape[i] <= 0) return 32;  // refused by the call
    cells *= static_cast<uint64_t>(shape[i]);
    if (cells >> 64 != 0) return 0;
  }
  return cells >> 32 != 0 ? 64 : 32;
}

// ------------------------------------------------------------------ autograd
// The byte that flexgemm_b200.kernels.config keeps equal to its allow_tf32: a backward pass reads the setting when it runs,
// in a thread that does not hold the GIL (taking it cost a small layer's backward pass a microsecond and a half).
const volatile char* g_allow_tf32 = nullptr;

struct ConvBackward : public torch::autograd::Node {
  torch::autograd::SavedVariable feats_, weight_;
  Maps bwd;
  Pairs pairs;
  bool mirror = true;
  int64_t V = 0;

  std::string name() const override { return mirror ? "SubMConv3dBackward" : "SparseConv3dBackward"; }
  void release_variables() override {
    feats_.reset_data();
    weight_.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(3);
    if (!grads[0].defined()) return out;
    const Tensor feats = feats_.unpack(), weight = weight_.unpack();
    const bool need_x = task_should_compute_output(0), need_w = task_should_compute_output(1), need_b = task_should_compute_output(2);
    if ((need_w && !pairs.vs_i.defined()) || (need_x && !bwd.nbr.defined()))
      throw torch::AttributeError(std::string("the neighbor cache was built for inference: it has no ") +
                                  (need_w ? "valid_signal_i" : "neighbor_map_bwd"));
    const int dtype = dtype_code(feats.scalar_type(), *g_allow_tf32 != 0);
    at::AutoDispatchBelowADInplaceOrView below;
    Grads g = run_backward(grads[0], feats, weight, bwd, pairs, mirror, V, dtype, need_x, need_w, need_b);
    out[0] = std::move(g.feats), out[1] = std::move(g.weight), out[2] = std::move(g.bias);
    return out;
  }
};

// Whether an input carries a forward-mode tangent.  There is no forward-mode derivative: the Python functions refuse
// such inputs, and the fast way, which looks at requires_grad, would drop the tangent.
bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(/*level=*/0).defined(); }

// the checks of the fast way
bool conv_args_ok(const Tensor& feats, const Tensor& weight, const Tensor& bias, PyObject* bias_obj, int64_t* V, int dtype) {
  if (!feats.defined() || !weight.defined() || dtype < 0) return false;
  if (has_tangent(feats) || has_tangent(weight) || has_tangent(bias)) return false;
  if (!feats.is_cuda() || feats.dim() != 2 || feats.size(0) == 0 || feats.size(1) == 0 || !feats.is_contiguous()) return false;
  if (weight.device() != feats.device() || weight.scalar_type() != feats.scalar_type() || weight.dim() != 5 || !weight.is_contiguous() ||
      weight.size(0) == 0 || weight.size(4) != feats.size(1))
    return false;
  *V = weight.size(1) * weight.size(2) * weight.size(3);
  if (*V < 1 || *V > 32) return false;
  if (bias_obj != Py_None &&
      (!bias.defined() || bias.device() != feats.device() || bias.scalar_type() != feats.scalar_type() || bias.dim() != 1 ||
       bias.size(0) != weight.size(0) || !bias.is_contiguous()))
    return false;
  return true;
}

// ------------------------------------------------------------------ submanifold cache
struct CacheBuild {
  Tensor nbr, gray, sorted_idx, masks, order, block_offsets, meta;
  HostSlot slot;
  int64_t n = 0;
  int V = 0;
  bool train = false;
};

// queues the build; with `train` the pair lists follow in finish_cache
CacheBuild start_cache(const Tensor& coords, const int64_t* shape, const int64_t* ks, const int64_t* dil, double ratio, bool train) {
  const auto stream = c10::cuda::getCurrentCUDAStream(coords.device().index());
  DeviceState& ds = device_state(coords.device().index());
  const at::Device dev = coords.device();
  CacheBuild b;
  const int64_t n = b.n = coords.size(0);
  const int V = b.V = static_cast<int>(ks[0] * ks[1] * ks[2]);
  b.train = train;
  const int64_t tiles = (n + 127) / 128, nblk = (n + 255) / 256;
  b.nbr = new_tensor({n, V}, at::kUInt32, dev);
  b.gray = new_tensor({n}, at::kInt, dev);
  b.sorted_idx = new_tensor({n}, at::kLong, dev);
  b.masks = new_tensor({tiles}, at::kUInt32, dev);
  b.order = new_tensor({std::max<int64_t>((tiles + 1) / 2, 1)}, at::kUInt32, dev);
  b.block_offsets = new_tensor({std::max<int64_t>(V * nblk, 1)}, at::kUInt32, dev);
  b.meta = new_tensor({V + 3}, at::kUInt32, dev);
  fgb_map_call c{};
  c.coords = cptr<int32_t>(coords);
  c.n = n;
  c.b = static_cast<int32_t>(shape[0]), c.w = static_cast<int32_t>(shape[2]), c.h = static_cast<int32_t>(shape[3]), c.d = static_cast<int32_t>(shape[4]);
  for (int i = 0; i < 3; ++i) c.k[i] = static_cast<int32_t>(ks[i]), c.dil[i] = static_cast<int32_t>(dil[i]);
  c.key_bits = key_bits_of(shape);
  c.slots = std::max<int64_t>({static_cast<int64_t>(ratio * static_cast<double>(n)), n, 1});
  c.scratch_bytes = check_bytes(api.fgb_subm_cache_scratch_bytes(&c), "fgb_subm_cache_scratch_bytes");
  const c10::DataPtr mem = scratch(c.scratch_bytes);
  c.scratch = mem.get();
  c.neighbor_map = static_cast<uint32_t*>(b.nbr.data_ptr());
  c.gray_code = static_cast<int32_t*>(b.gray.data_ptr());
  c.sorted_idx = static_cast<int64_t*>(b.sorted_idx.data_ptr());
  c.tile_masks = static_cast<uint32_t*>(b.masks.data_ptr());
  c.block_order = static_cast<uint32_t*>(b.order.data_ptr());
  c.block_offsets = static_cast<uint32_t*>(b.block_offsets.data_ptr());
  c.meta = static_cast<uint32_t*>(b.meta.data_ptr());
  if (train && n > 0) {
    b.slot.take(stream, &c.host_words, &c.host_seq);
  }
  c.status = static_cast<int32_t*>(ds.status.data_ptr());
  b.slot.queued();
  check(api.fgb_subm_cache_build(&c, stream), "fgb_subm_cache_build");
  return b;
}

// waits for the pair count and queues the pair lists; the GIL is released while it waits
Pairs finish_cache(CacheBuild& b) {
  const auto stream = c10::cuda::getCurrentCUDAStream(b.nbr.device().index());
  int64_t pairs = 0;
  if (b.n > 0) {
    const Told got = b.slot.take_back();
    pairs = got.count;
    if (got.status != 0u) throw_soft_error(static_cast<int>(got.status));
  }
  Pairs p;
  p.vs_i = new_tensor({pairs}, at::kUInt32, b.nbr.device());
  p.vs_o = new_tensor({pairs}, at::kUInt32, b.nbr.device());
  p.seg = b.meta.narrow(0, 0, b.V + 1);
  p.block_offsets = b.block_offsets;
  const uint32_t* meta = cptr<uint32_t>(b.meta);
  if (pairs > 0) {
    check(api.fgb_pp_valid_signal(cptr<uint32_t>(b.nbr), cptr<int32_t>(b.gray), b.n, b.V, cptr<uint32_t>(b.block_offsets), meta,
                                  static_cast<uint32_t*>(p.vs_i.data_ptr()), static_cast<uint32_t*>(p.vs_o.data_ptr()), meta + b.V + 1, stream),
          "fgb_pp_valid_signal");
  }
  return p;
}

PyObject* new_cache(PyObject* cls) {
  PyObject* cache = PyObject_Call(cls, s_empty_tuple, nullptr);
  if (cache == nullptr) throw PyError{};
  return cache;
}
void fill_cache(PyObject* cache, const CacheBuild& b, const Pairs* p) {
  set_tensor(cache, s_neighbor_map, b.nbr);
  set_tensor(cache, s_gray_code, b.gray);
  set_tensor(cache, s_sorted_idx, b.sorted_idx);
  set_tensor(cache, s_tile_masks, b.masks);
  set_tensor(cache, s_block_order, b.order);
  if (p != nullptr) {
    set_tensor(cache, s_seg, p->seg);
    set_tensor(cache, s_vs_i, p->vs_i);
    set_tensor(cache, s_vs_o, p->vs_o);
    // not part of the reference's cache: where each 256-row block starts in every offset's pair list, which lets wgrad
    // walk all lists in row bands that share L2
    set_tensor(cache, s_block_offsets, b.block_offsets);
  } else {
    // inference cache: nothing needs the host, so nothing waits; an overflowing table would show in this word
    set_tensor(cache, s_build_status, b.meta.narrow(0, b.V + 2, 1));
  }
}

bool coords_ok(const Tensor& coords, const int64_t* ks) {
  return coords.defined() && coords.is_cuda() && coords.scalar_type() == at::kInt && coords.dim() == 2 && coords.size(1) == 4 &&
         coords.is_contiguous() && ks[0] % 2 == 1 && ks[1] % 2 == 1 && ks[2] % 2 == 1 && ks[0] > 0 && ks[1] > 0 && ks[2] > 0 &&
         ks[0] * ks[1] * ks[2] <= 32;
}

// the exception in flight as a Python exception
void raise_python() {
  try {
    throw;
  } catch (const PyError&) {
  } catch (const c10::ValueError& e) {
    PyErr_SetString(PyExc_ValueError, e.what_without_backtrace());
  } catch (const c10::OutOfMemoryError& e) {
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* type = torch != nullptr ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
    if (type != nullptr) PyErr_SetString(type, e.what_without_backtrace());
    Py_XDECREF(type);
    Py_XDECREF(torch);
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
}

#define FGB_TRY try {
#define FGB_END                                   \
  }                                               \
  catch (...) {                                   \
    raise_python();                               \
    return nullptr;                               \
  }

// (cache_cls, coords, shape, kernel_size, dilation, ratio, train) -> cache or None
PyObject* py_subm_cache(PyObject*, PyObject* const* a, Py_ssize_t n) {
  FGB_TRY
  TORCH_CHECK(n == 7, "subm_cache takes 7 arguments");
  const Tensor coords = tensor_arg(a[1]);
  int64_t shape[5], ks[3], dil[3];
  if (!int_args(a[2], 5, shape) || !int_args(a[3], 3, ks) || !int_args(a[4], 3, dil) || !coords_ok(coords, ks) ||
      key_bits_of(shape) == 0)
    Py_RETURN_NONE;
  const double ratio = PyFloat_AsDouble(a[5]);
  if (ratio == -1.0 && PyErr_Occurred()) return nullptr;
  const bool train = PyObject_IsTrue(a[6]) == 1;
  c10::cuda::CUDAGuard guard(coords.device());
  at::AutoDispatchBelowADInplaceOrView below;
  CacheBuild b = start_cache(coords, shape, ks, dil, ratio, train);
  Pairs p;
  if (train) p = finish_cache(b);
  PyObject* cache = new_cache(a[0]);
  try {
    fill_cache(cache, b, train ? &p : nullptr);
  } catch (...) {
    Py_DECREF(cache);
    throw;
  }
  return cache;
  FGB_END
}

// Output of a convolution over `m`, with its autograd node where a gradient is wanted
Tensor conv_autograd(const Tensor& feats, const Tensor& weight, const Tensor& bias, const Maps& m, const Maps& bwd, const Pairs& pairs,
                     bool mirror, int64_t V, Tensor out) {
  if (!torch::autograd::compute_requires_grad(feats, weight, bias)) return out;
  std::shared_ptr<ConvBackward> node(new ConvBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(feats, weight, bias));
  node->feats_ = torch::autograd::SavedVariable(feats, false);
  node->weight_ = torch::autograd::SavedVariable(weight, false);
  node->bwd = bwd;
  node->pairs = pairs;
  node->mirror = mirror;
  node->V = V;
  torch::autograd::set_history(out, node);
  return out;
}

PyObject* pair_of(const Tensor& out, PyObject* cache /* stolen */) {
  PyObject* o = THPVariable_Wrap(out);
  PyObject* t = o != nullptr ? PyTuple_New(2) : nullptr;
  if (t == nullptr) {
    Py_XDECREF(o);
    Py_DECREF(cache);
    return nullptr;
  }
  PyTuple_SET_ITEM(t, 0, o);
  PyTuple_SET_ITEM(t, 1, cache);
  return t;
}

// (cache_cls, feats, coords, shape, weight, bias, cache, dilation, ratio, tf32) -> (out, cache) or None
PyObject* py_subm_conv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  FGB_TRY
  TORCH_CHECK(n == 10, "subm_conv takes 10 arguments");
  const Tensor feats = tensor_arg(a[1]), weight = tensor_arg(a[4]), bias = tensor_arg(a[5]);
  const bool tf32 = PyObject_IsTrue(a[9]) == 1;
  const int dtype = feats.defined() ? dtype_code(feats.scalar_type(), tf32) : -1;
  int64_t V = 0;
  if (!conv_args_ok(feats, weight, bias, a[5], &V, dtype)) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(feats.device());
  PyObject* cache = a[6];
  Tensor out;
  Maps m;
  Pairs pairs;
  if (cache != Py_None) {
    m = fwd_maps(cache);
    if (!m.nbr.defined() || m.nbr.device() != feats.device() || m.nbr.dim() != 2 || m.nbr.size(0) != feats.size(0) || m.nbr.size(1) != V)
      Py_RETURN_NONE;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      out = run_fprop(feats, weight, bias, m, V, dtype);
    }
    if (weight.requires_grad()) pairs = pairs_of(cache);
    Py_INCREF(cache);
  } else {
    const Tensor coords = tensor_arg(a[2]);
    int64_t shape[5], ks[3] = {weight.size(1), weight.size(2), weight.size(3)}, dil[3];
    if (!int_args(a[3], 5, shape) || !int_args(a[7], 3, dil) || !coords_ok(coords, ks) || coords.device() != feats.device() ||
        coords.size(0) != feats.size(0) || key_bits_of(shape) == 0)
      Py_RETURN_NONE;
    const double ratio = PyFloat_AsDouble(a[8]);
    if (ratio == -1.0 && PyErr_Occurred()) return nullptr;
    const bool train = feats.requires_grad() || weight.requires_grad() || (bias.defined() && bias.requires_grad());
    at::AutoDispatchBelowADInplaceOrView below;
    CacheBuild b = start_cache(coords, shape, ks, dil, ratio, train);
    m = Maps{b.nbr, b.sorted_idx, b.masks, b.order};
    // the convolution does not need the pair lists: it is queued before the host waits for their length
    out = run_fprop(feats, weight, bias, m, V, dtype);
    if (train) pairs = finish_cache(b);
    cache = new_cache(a[0]);
    try {
      fill_cache(cache, b, train ? &pairs : nullptr);
    } catch (...) {
      Py_DECREF(cache);
      throw;
    }
  }
  return pair_of(conv_autograd(feats, weight, bias, m, m, pairs, true, V, std::move(out)), cache);
  FGB_END
}

// (feats, weight, bias, cache, tf32, sparse) -> out or None: one convolution on an existing cache; sparse: the cache of
// the generic convolution, with a map of its own for the backward direction
PyObject* py_conv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  FGB_TRY
  TORCH_CHECK(n == 6, "conv takes 6 arguments");
  const Tensor feats = tensor_arg(a[0]), weight = tensor_arg(a[1]), bias = tensor_arg(a[2]);
  const int dtype = feats.defined() ? dtype_code(feats.scalar_type(), PyObject_IsTrue(a[4]) == 1) : -1;
  const bool sparse = PyObject_IsTrue(a[5]) == 1;
  int64_t V = 0;
  if (!conv_args_ok(feats, weight, bias, a[2], &V, dtype)) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(feats.device());
  const Maps m = fwd_maps(a[3]);
  if (!m.nbr.defined() || m.nbr.device() != feats.device() || m.nbr.dim() != 2 || m.nbr.size(1) != V || m.nbr.size(0) == 0) Py_RETURN_NONE;
  if (!sparse && m.nbr.size(0) != feats.size(0)) Py_RETURN_NONE;
  Tensor out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    out = run_fprop(feats, weight, bias, m, V, dtype);
  }
  Maps bwd = m;
  if (sparse) bwd = feats.requires_grad() && at::GradMode::is_enabled() ? bwd_maps(a[3]) : Maps{};
  Pairs pairs;
  if (weight.requires_grad()) pairs = pairs_of(a[3]);
  return THPVariable_Wrap(conv_autograd(feats, weight, bias, m, bwd, pairs, !sparse, V, std::move(out)));
  FGB_END
}

// (grad_output, feats, weight, cache, tf32, sparse, need_x, need_w, need_b) -> (grad_feats, grad_weight, grad_bias) or None
PyObject* py_conv_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  FGB_TRY
  TORCH_CHECK(n == 9, "conv_backward takes 9 arguments");
  const Tensor g = tensor_arg(a[0]), feats = tensor_arg(a[1]), weight = tensor_arg(a[2]);
  const int dtype = feats.defined() ? dtype_code(feats.scalar_type(), PyObject_IsTrue(a[4]) == 1) : -1;
  const bool sparse = PyObject_IsTrue(a[5]) == 1;
  const bool need_x = PyObject_IsTrue(a[6]) == 1, need_w = PyObject_IsTrue(a[7]) == 1, need_b = PyObject_IsTrue(a[8]) == 1;
  int64_t V = 0;
  if (!conv_args_ok(feats, weight, Tensor(), Py_None, &V, dtype) || !g.defined() || g.scalar_type() != feats.scalar_type() || g.dim() != 2 ||
      g.device() != feats.device() || g.size(1) != weight.size(0) || g.size(0) == 0)
    Py_RETURN_NONE;
  const Maps bwd = !need_x ? Maps{} : sparse ? bwd_maps(a[3]) : fwd_maps(a[3]);
  const Pairs pairs = need_w ? pairs_of(a[3]) : Pairs{};
  if ((need_x && (!bwd.nbr.defined() || bwd.nbr.size(0) != feats.size(0))) || (need_w && !pairs.vs_i.defined())) Py_RETURN_NONE;
  Grads r;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    r = run_backward(g, feats, weight, bwd, pairs, !sparse, V, dtype, need_x, need_w, need_b);
  }
  PyObject* t = PyTuple_New(3);
  if (t == nullptr) return nullptr;
  const Tensor* parts[3] = {&r.feats, &r.weight, &r.bias};
  for (int i = 0; i < 3; ++i) {
    PyObject* v = parts[i]->defined() ? THPVariable_Wrap(*parts[i]) : (Py_INCREF(Py_None), Py_None);
    if (v == nullptr) {
      Py_DECREF(t);
      return nullptr;
    }
    PyTuple_SET_ITEM(t, i, v);
  }
  return t;
  FGB_END
}

// ------------------------------------------------------------------ strided convolution
struct StridedBuild {
  fgb_strided_call c{};
  c10::DataPtr grid;
  Tensor out_coords, nbr, nbr_bwd, gray, gray_bwd, sorted_idx, sorted_bwd, masks, masks_bwd, order, order_bwd, block_offsets, meta;
  HostSlot slot;
  int V = 0;
};

// marks and counts the output voxels; false where the bit grid does not serve the case (or there are none)
bool strided_coords(StridedBuild& b, const Tensor& coords, const int64_t* shape, const int64_t* ks, const int64_t* st, const int64_t* pad,
                    const int64_t* dil, bool coords_only) {
  const auto stream = c10::cuda::getCurrentCUDAStream(coords.device().index());
  fgb_strided_call& c = b.c;
  c.coords = cptr<int32_t>(coords);
  c.n = coords.size(0);
  c.b = static_cast<int32_t>(shape[0]), c.w = static_cast<int32_t>(shape[2]), c.h = static_cast<int32_t>(shape[3]), c.d = static_cast<int32_t>(shape[4]);
  for (int i = 0; i < 3; ++i) {
    c.k[i] = static_cast<int32_t>(ks[i]), c.s[i] = static_cast<int32_t>(st[i]);
    c.p[i] = static_cast<int32_t>(pad[i]), c.dil[i] = static_cast<int32_t>(dil[i]);
  }
  b.V = static_cast<int>(ks[0] * ks[1] * ks[2]);
  const int64_t bytes = api.fgb_strided_grid_bytes(&c);
  if (bytes <= 0) return false;
  b.grid = scratch(bytes);
  c.grid_mem = b.grid.get(), c.grid_bytes = bytes;
  HostSlot slot;
  slot.take(stream, &c.host_words, &c.host_seq);
  slot.queued();
  check(api.fgb_strided_mark(&c, stream), "fgb_strided_mark");
  const Told got = slot.take_back();
  if (got.status != 0u) return false;  // rows of a batch beyond the shape's: the bits have no place for them
  c.n_out = got.count;
  c.host_words = nullptr;
  b.out_coords = new_tensor({c.n_out, 4}, at::kInt, coords.device());
  if (c.n_out == 0) return coords_only;
  c.out_coords = static_cast<int32_t*>(b.out_coords.data_ptr());
  if (coords_only) {
    check(api.fgb_strided_build(&c, stream), "fgb_strided_build");
  }
  return true;
}

void strided_maps(StridedBuild& b, at::Device dev, bool train) {
  const auto stream = c10::cuda::getCurrentCUDAStream(dev.index());
  fgb_strided_call& c = b.c;
  const int64_t n = c.n, m = c.n_out, V = b.V;
  auto tiles = [](int64_t rows) { return (rows + 127) / 128; };
  auto make = [&](Tensor& t, at::IntArrayRef size, at::ScalarType dt) {
    t = new_tensor(size, dt, dev);
    return t.data_ptr();
  };
  c.neighbor_map = static_cast<uint32_t*>(make(b.nbr, {m, V}, at::kUInt32));
  c.gray_code = static_cast<int32_t*>(make(b.gray, {m}, at::kInt));
  c.sorted_idx = static_cast<int64_t*>(make(b.sorted_idx, {m}, at::kLong));
  c.tile_masks = static_cast<uint32_t*>(make(b.masks, {tiles(m)}, at::kUInt32));
  c.block_order = static_cast<uint32_t*>(make(b.order, {(tiles(m) + 1) / 2}, at::kUInt32));
  c.block_offsets = static_cast<uint32_t*>(make(b.block_offsets, {V * ((m + 255) / 256)}, at::kUInt32));
  c.meta = static_cast<uint32_t*>(make(b.meta, {V + 1}, at::kUInt32));
  if (train) {
    c.neighbor_map_bwd = static_cast<uint32_t*>(make(b.nbr_bwd, {n, V}, at::kUInt32));
    c.gray_code_bwd = static_cast<int32_t*>(make(b.gray_bwd, {n}, at::kInt));
    c.sorted_idx_bwd = static_cast<int64_t*>(make(b.sorted_bwd, {n}, at::kLong));
    c.tile_masks_bwd = static_cast<uint32_t*>(make(b.masks_bwd, {tiles(n)}, at::kUInt32));
    c.block_order_bwd = static_cast<uint32_t*>(make(b.order_bwd, {(tiles(n) + 1) / 2}, at::kUInt32));
    b.slot.take(stream, &c.host_words, &c.host_seq);
  }
  c.scratch_bytes = check_bytes(api.fgb_strided_build_bytes(&c), "fgb_strided_build_bytes");
  const c10::DataPtr mem = scratch(c.scratch_bytes);
  c.scratch = mem.get();
  c.status = static_cast<int32_t*>(device_state(dev.index()).status.data_ptr());
  b.slot.queued();
  check(api.fgb_strided_build(&c, stream), "fgb_strided_build");
}

Pairs strided_pairs(StridedBuild& b) {
  const auto stream = c10::cuda::getCurrentCUDAStream(b.nbr.device().index());
  const int64_t pairs = b.slot.take_back().count;
  Pairs p;
  p.vs_i = new_tensor({pairs}, at::kUInt32, b.nbr.device());
  p.vs_o = new_tensor({pairs}, at::kUInt32, b.nbr.device());
  p.seg = b.meta;
  p.block_offsets = b.block_offsets;
  if (pairs > 0) {
    check(api.fgb_pp_valid_signal(cptr<uint32_t>(b.nbr), cptr<int32_t>(b.gray), b.c.n_out, b.V, cptr<uint32_t>(b.block_offsets), cptr<uint32_t>(b.meta),
                                  static_cast<uint32_t*>(p.vs_i.data_ptr()), static_cast<uint32_t*>(p.vs_o.data_ptr()), nullptr, stream),
          "fgb_pp_valid_signal");
  }
  return p;
}

bool geometry_args(PyObject* stride, PyObject* padding, PyObject* dilation, int64_t* st, int64_t* pad, int64_t* dil) {
  if (!int_args(stride, 3, st) || !int_args(padding, 3, pad) || !int_args(dilation, 3, dil)) return false;
  for (int i = 0; i < 3; ++i)
    if (st[i] < 1 || pad[i] < 0 || dil[i] < 1) return false;
  return true;
}
bool rows_ok(const Tensor& coords) {
  const int64_t one[3] = {1, 1, 1};
  return coords_ok(coords, one) && coords.size(0) > 0;
}

// (coords, shape, kernel_size, stride, padding, dilation) -> output coordinates in flat-index order, or None
PyObject* py_strided_coords(PyObject*, PyObject* const* a, Py_ssize_t n) {
  FGB_TRY
  TORCH_CHECK(n == 6, "strided_coords takes 6 arguments");
  const Tensor coords = tensor_arg(a[0]);
  int64_t shape[5], ks[3], st[3], pad[3], dil[3];
  if (!rows_ok(coords) || !int_args(a[1], 5, shape) || !int_args(a[2], 3, ks) || !geometry_args(a[3], a[4], a[5], st, pad, dil)) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(coords.device());
  at::AutoDispatchBelowADInplaceOrView below;
  StridedBuild b;
  if (!strided_coords(b, coords, shape, ks, st, pad, dil, true)) Py_RETURN_NONE;
  return THPVariable_Wrap(b.out_coords);
  FGB_END
}

// (cache_cls, feats, coords, shape, weight, bias, stride, padding, dilation, tf32) -> (out, out_coords, cache) or None
PyObject* py_strided_conv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  FGB_TRY
  TORCH_CHECK(n == 10, "strided_conv takes 10 arguments");
  const Tensor feats = tensor_arg(a[1]), coords = tensor_arg(a[2]), weight = tensor_arg(a[4]), bias = tensor_arg(a[5]);
  const int dtype = feats.defined() ? dtype_code(feats.scalar_type(), PyObject_IsTrue(a[9]) == 1) : -1;
  int64_t V = 0, shape[5], st[3], pad[3], dil[3];
  if (!conv_args_ok(feats, weight, bias, a[5], &V, dtype) || !rows_ok(coords) || coords.device() != feats.device() ||
      coords.size(0) != feats.size(0) || !int_args(a[3], 5, shape) || !geometry_args(a[6], a[7], a[8], st, pad, dil) ||
      key_bits_of(shape) == 0)
    Py_RETURN_NONE;
  const int64_t ks[3] = {weight.size(1), weight.size(2), weight.size(3)};
  c10::cuda::CUDAGuard guard(feats.device());
  StridedBuild b;
  Tensor out;
  Pairs pairs;
  Maps m, bwd;
  const bool train = feats.requires_grad() || weight.requires_grad() || (bias.defined() && bias.requires_grad());
  {
    at::AutoDispatchBelowADInplaceOrView below;
    if (!strided_coords(b, coords, shape, ks, st, pad, dil, false)) Py_RETURN_NONE;
    strided_maps(b, feats.device(), train);
    m = Maps{b.nbr, b.sorted_idx, b.masks, b.order};
    if (train) bwd = Maps{b.nbr_bwd, b.sorted_bwd, b.masks_bwd, b.order_bwd};
    out = run_fprop(feats, weight, bias, m, V, dtype);
    if (train) pairs = strided_pairs(b);
  }
  PyObject* cache = new_cache(a[0]);
  PyObject* t = nullptr;
  try {
    set_tensor(cache, s_neighbor_map, b.nbr);
    set_tensor(cache, s_gray_code, b.gray);
    set_tensor(cache, s_sorted_idx, b.sorted_idx);
    set_tensor(cache, s_tile_masks, b.masks);
    set_tensor(cache, s_block_order, b.order);
    if (train) {
      set_tensor(cache, s_neighbor_map_bwd, b.nbr_bwd);
      set_tensor(cache, s_gray_code_bwd, b.gray_bwd);
      set_tensor(cache, s_sorted_idx_bwd, b.sorted_bwd);
      set_tensor(cache, s_tile_masks_bwd, b.masks_bwd);
      set_tensor(cache, s_block_order_bwd, b.order_bwd);
      set_tensor(cache, s_seg, pairs.seg);
      set_tensor(cache, s_vs_i, pairs.vs_i);
      set_tensor(cache, s_vs_o, pairs.vs_o);
      set_tensor(cache, s_block_offsets, b.block_offsets);
    } else if (PyObject_SetAttr(cache, s_neighbor_map_bwd, Py_None) != 0) {
      throw PyError{};
    }
    out = conv_autograd(feats, weight, bias, m, bwd, pairs, false, V, std::move(out));
    PyObject* o = THPVariable_Wrap(out);
    PyObject* oc = o != nullptr ? THPVariable_Wrap(b.out_coords) : nullptr;
    t = oc != nullptr ? PyTuple_New(3) : nullptr;
    if (t == nullptr) {
      Py_XDECREF(o);
      Py_XDECREF(oc);
      throw PyError{};
    }
    PyTuple_SET_ITEM(t, 0, o);
    PyTuple_SET_ITEM(t, 1, oc);
    PyTuple_SET_ITEM(t, 2, cache);
  } catch (...) {
    Py_DECREF(cache);
    throw;
  }
  return t;
  FGB_END
}

// ------------------------------------------------------------------ grid sample
Tensor run_sample_grad(const Tensor& grad_out /* [..., C] */, const Tensor& indices, const Tensor& weight, int64_t n, int64_t V) {
  c10::cuda::CUDAGuard guard(grad_out.device());
  const auto stream = c10::cuda::getCurrentCUDAStream(grad_out.device().index());
  const int64_t C = grad_out.size(-1), M = C > 0 ? grad_out.numel() / C : 0;
  Tensor out = new_tensor({n, C}, grad_out.scalar_type(), grad_out.device());
  const int dtype = dtype_code(grad_out.scalar_type(), false);
  const int64_t bytes = check_bytes(api.fgb_indice_weighted_sum_grad_full_bytes(M, n, static_cast<int>(C), static_cast<int>(V), dtype),
                                    "fgb_indice_weighted_sum_grad_full_bytes");
  const c10::DataPtr ws = scratch(bytes);
  check(api.fgb_indice_weighted_sum_grad(ptr(grad_out), cptr<uint32_t>(indices), weight.defined() ? cptr<float>(weight) : nullptr,
                                         n > 0 ? out.data_ptr() : nullptr, M, n, static_cast<int>(C), static_cast<int>(V),
                                         dtype, ws.get(), bytes, stream),
        "fgb_indice_weighted_sum_grad");
  return out;
}

struct GridSampleBackward : public torch::autograd::Node {
  torch::autograd::SavedVariable indices_, weight_;
  int64_t n = 0, V = 1;
  std::string name() const override { return "GridSample3dBackward"; }
  void release_variables() override {
    indices_.reset_data();
    weight_.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (!grads[0].defined() || !task_should_compute_output(0)) return out;
    const Tensor indices = indices_.unpack(), weight = weight_.unpack();
    at::AutoDispatchBelowADInplaceOrView below;
    out[0] = run_sample_grad(grads[0].contiguous(), indices, weight, n, V);
    return out;
  }
};

// (feats, coords, shape, grid, trilinear, ratio) -> [B, L, C] or None
PyObject* py_grid_sample(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  FGB_TRY
  TORCH_CHECK(n_args == 6, "grid_sample takes 6 arguments");
  const Tensor feats = tensor_arg(a[0]), coords = tensor_arg(a[1]);
  Tensor grid = tensor_arg(a[3]);
  const bool trilinear = PyObject_IsTrue(a[4]) == 1;
  int64_t shape[5];
  const int64_t one[3] = {1, 1, 1};
  if (!feats.defined() || !feats.is_cuda() || feats.dim() != 2 || !feats.is_contiguous() || feats.size(0) == 0 || feats.size(1) == 0 ||
      feats.size(1) % 4 != 0 || dtype_code(feats.scalar_type(), false) < 0 || !coords_ok(coords, one) || coords.device() != feats.device() ||
      coords.size(0) != feats.size(0) || !grid.defined() || grid.device() != feats.device() || grid.dim() != 3 || grid.size(2) != 3 ||
      grid.scalar_type() != at::kFloat || !grid.is_contiguous() || grid.numel() == 0 || !int_args(a[2], 5, shape) ||
      (reinterpret_cast<uintptr_t>(feats.const_data_ptr()) & 15) != 0 || has_tangent(feats) || has_tangent(grid))
    Py_RETURN_NONE;
  // query points that want a gradient get none, but a backward pass from the output has to go through
  if (torch::autograd::compute_requires_grad(grid)) Py_RETURN_NONE;
  const double ratio = PyFloat_AsDouble(a[5]);
  if (ratio == -1.0 && PyErr_Occurred()) return nullptr;
  c10::cuda::CUDAGuard guard(feats.device());
  const auto stream = c10::cuda::getCurrentCUDAStream(feats.device().index());
  const bool want_grad = torch::autograd::compute_requires_grad(feats);
  const int64_t n = feats.size(0), C = feats.size(1), B = grid.size(0), L = grid.size(1), V = trilinear ? 8 : 1;
  const int64_t slots = std::max<int64_t>({static_cast<int64_t>(ratio * static_cast<double>(n)), n, 1});
  const int key_bits = key_bits_of(shape);
  if (key_bits == 0) Py_RETURN_NONE;
  Tensor out, indices, weight;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    out = new_tensor({B, L, C}, feats.scalar_type(), feats.device());
    if (want_grad) {
      indices = new_tensor({B * L, V}, at::kUInt32, feats.device());
      if (trilinear) weight = new_tensor({B * L, V}, at::kFloat, feats.device());
    }
    const c10::DataPtr table = scratch(check_bytes(api.fgb_hash_table_bytes(slots, key_bits), "fgb_hash_table_bytes"));
    // the table has a slot for every row, so it cannot run full: no status word to read back
    check(api.fgb_grid_sample_fused(cptr<int32_t>(coords), n, ptr(feats), cptr<float>(grid), B, L, static_cast<int>(shape[2]), static_cast<int>(shape[3]),
                                    static_cast<int>(shape[4]), static_cast<int>(C), dtype_code(feats.scalar_type(), false), trilinear ? 1 : 0,
                                    table.get(), slots, key_bits, nullptr, out.data_ptr(),
                                    want_grad ? static_cast<uint32_t*>(indices.data_ptr()) : nullptr,
                                    want_grad && trilinear ? static_cast<float*>(weight.data_ptr()) : nullptr, stream),
          "fgb_grid_sample_fused");
  }
  if (want_grad) {
    std::shared_ptr<GridSampleBackward> node(new GridSampleBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(feats));
    node->indices_ = torch::autograd::SavedVariable(indices, false);
    node->weight_ = torch::autograd::SavedVariable(weight, false);
    node->n = n, node->V = V;
    torch::autograd::set_history(out, node);
  }
  return THPVariable_Wrap(out);
  FGB_END
}

// (grad_out [M, C], indices [M, V], weight or None, n) -> [n, C]
PyObject* py_sample_grad(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  FGB_TRY
  TORCH_CHECK(n_args == 4, "sample_grad takes 4 arguments");
  const Tensor g = tensor_arg(a[0]), indices = tensor_arg(a[1]);
  at::AutoDispatchBelowADInplaceOrView below;
  return THPVariable_Wrap(run_sample_grad(g, indices, tensor_arg(a[2]), PyLong_AsLongLong(a[3]), indices.size(1)));
  FGB_END
}

PyObject* py_status_word(PyObject*, PyObject* index) {
  FGB_TRY
  return THPVariable_Wrap(device_state(static_cast<c10::DeviceIndex>(PyLong_AsLong(index))).status);
  FGB_END
}
PyObject* py_poll(PyObject*, PyObject* index) {
  FGB_TRY
  const auto d = static_cast<c10::DeviceIndex>(PyLong_AsLong(index));
  c10::cuda::CUDAGuard guard(d);
  poll(device_state(d), c10::cuda::getCurrentCUDAStream(d));
  Py_RETURN_NONE;
  FGB_END
}
// forgets what the mirror holds (the caller has synchronised and cleared the word)
PyObject* py_clear_mirror(PyObject*, PyObject* index) {
  FGB_TRY
  *device_state(static_cast<c10::DeviceIndex>(PyLong_AsLong(index))).mirror.load() = 0;
  Py_RETURN_NONE;
  FGB_END
}
// (slots made, slots free)
PyObject* py_host_slots(PyObject*, PyObject*) {
  std::lock_guard<std::mutex> lock(g_words_mu);
  return Py_BuildValue("Ln", static_cast<long long>(g_words_made), static_cast<Py_ssize_t>(g_words_free.size()));
}

// (handle, address): the CUDA library's dlopen handle, the byte of allow_tf32
PyObject* py_init(PyObject*, PyObject* const* a, Py_ssize_t n) {
  FGB_TRY
  TORCH_CHECK(n == 2, "init takes 2 arguments");
  void* lib = PyLong_AsVoidPtr(a[0]);
  if (lib == nullptr) return nullptr;
  g_allow_tf32 = static_cast<const char*>(PyLong_AsVoidPtr(a[1]));
  if (g_allow_tf32 == nullptr) return nullptr;
#define X(f)                                                    \
  api.f = reinterpret_cast<decltype(api.f)>(dlsym(lib, #f));    \
  TORCH_CHECK(api.f != nullptr, "the CUDA library lacks " #f);
  FGB_TORCH_API(X)
#undef X
  Py_RETURN_NONE;
  FGB_END
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(f)), METH_FASTCALL
PyMethodDef methods[] = {
    {"init", FAST(py_init), "bind the CUDA library (its dlopen handle) and the settings"},
    {"subm_cache", FAST(py_subm_cache), "neighbour cache of a submanifold conv"},
    {"subm_conv", FAST(py_subm_conv), "submanifold conv"},
    {"conv", FAST(py_conv), "convolution on an existing cache"},
    {"conv_backward", FAST(py_conv_backward), "gradients of a convolution"},
    {"strided_coords", FAST(py_strided_coords), "output coordinates of a strided conv"},
    {"strided_conv", FAST(py_strided_conv), "strided conv"},
    {"grid_sample", FAST(py_grid_sample), "sparse grid sample"},
    {"sample_grad", FAST(py_sample_grad), "gradient of a weighted gather"},
    {"status_word", py_status_word, METH_O, "device status word"},
    {"poll", py_poll, METH_O, "raise a soft error that the device has reported"},
    {"clear_mirror", py_clear_mirror, METH_O, "forget the host copy of the status word"},
    {"host_slots", py_host_slots, METH_NOARGS, "slots through which builds report: (made, free)"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fgb_torch", "torch host code of flexgemm_b200", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fgb_torch(void) {
  s_neighbor_map = PyUnicode_InternFromString("neighbor_map");
  s_gray_code = PyUnicode_InternFromString("gray_code");
  s_sorted_idx = PyUnicode_InternFromString("sorted_idx");
  s_tile_masks = PyUnicode_InternFromString("tile_masks_128");
  s_block_order = PyUnicode_InternFromString("block_order_128");
  s_vs_i = PyUnicode_InternFromString("valid_signal_i");
  s_vs_o = PyUnicode_InternFromString("valid_signal_o");
  s_seg = PyUnicode_InternFromString("valid_signal_seg");
  s_block_offsets = PyUnicode_InternFromString("pair_block_offsets");
  s_build_status = PyUnicode_InternFromString("build_status");
  s_neighbor_map_bwd = PyUnicode_InternFromString("neighbor_map_bwd");
  s_sorted_idx_bwd = PyUnicode_InternFromString("sorted_idx_bwd");
  s_tile_masks_bwd = PyUnicode_InternFromString("tile_masks_bwd_128");
  s_block_order_bwd = PyUnicode_InternFromString("block_order_bwd_128");
  s_gray_code_bwd = PyUnicode_InternFromString("gray_code_bwd");
  s_ensure_bwd = PyUnicode_InternFromString("_ensure_bwd_order");
  s_m_tile_masks = PyUnicode_InternFromString("tile_masks");
  s_m_block_order = PyUnicode_InternFromString("block_order");
  s_m_tile_masks_bwd = PyUnicode_InternFromString("tile_masks_bwd");
  s_m_block_order_bwd = PyUnicode_InternFromString("block_order_bwd");
  s_tile_rows = PyLong_FromLong(128);
  s_empty_tuple = PyTuple_New(0);
  return PyModule_Create(&module);
}
