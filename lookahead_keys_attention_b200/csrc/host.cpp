// Host side of the operators: everything between a Python call and the C ABI's launches, natively.
//
// A small call of this framework (a decode step, a short training step) spends its time on the host: building tensor
// descriptors through ctypes, Python autograd functions and chains of small torch operations took 60 to 120 us per
// call on the token path and 800 us for the smallest training step, against 10 to 150 us of kernels.  This module does
// the same work in C++: descriptors, scratch, the autograd node, the choice of the passes around the kernels, and for
// the plain `Castle` module the projections around the core as well.  It holds no kernels; the C ABI of
// libcastle_b200.so is bound by address (`bind`).
//
// Operators and their semantics: ops.py and castle.py.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/grad_mode.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/PyInterpreter.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <ATen/autocast_mode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <array>
#include <limits>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <vector>

#include "../../include/castle_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

struct AssertError : std::runtime_error { using std::runtime_error::runtime_error; };   // raised as AssertionError

// ------------------------------------------------------------------------------------------------ the C ABI, by address
struct Api {
  decltype(&castle_last_error) last_error;
  decltype(&castle_fwd_workspace_bytes) fwd_workspace_bytes;
  decltype(&castle_fwd) fwd;
  decltype(&castle_fwd_prefill) fwd_prefill;
  decltype(&castle_rmsnorm_fwd) rmsnorm_fwd;
  decltype(&castle_rmsnorm_bwd_workspace_bytes) rmsnorm_bwd_workspace_bytes;
  decltype(&castle_rmsnorm_bwd) rmsnorm_bwd;
  decltype(&castle_bwd_workspace_bytes) bwd_workspace_bytes;
  decltype(&castle_bwd) bwd;
  decltype(&castle_transform) transform;
  decltype(&castle_amax_scale) amax_scale;
  decltype(&castle_decode_workspace_bytes) decode_workspace_bytes;
  decltype(&castle_decode_step_fused) decode_step_fused;
  decltype(&castle_token_linear_fits) token_linear_fits;
  decltype(&castle_token_linear) token_linear;
  decltype(&castle_linear) linear;
  decltype(&castle_token_layer_fits) token_layer_fits;
  decltype(&castle_token_layer_workspace_bytes) token_layer_workspace_bytes;
  decltype(&castle_token_layer) token_layer;
} api{};

void check(int rc, const char* what) {
  if (rc != 0)
    throw std::runtime_error(std::string(what) + " failed (rc=" + std::to_string(rc) + "): " + api.last_error());
}

void need(bool ok, const char* message) {
  if (!ok) throw std::runtime_error(message);
}

// ------------------------------------------------------------------------------------------------ device state kept between calls
// Scratch per (device, stream): kernels of one stream run in order, so its calls can share a buffer; two streams must
// not.  Grown on demand, given back by release_workspaces().  `words` are zeroed counters that every kernel using them
// leaves zeroed.  The containers are never destroyed (the CUDA context may be gone before static destructors run).
//
// Calls of several host threads on one stream (the autograd engine's among them) must not mix: what a call's launches
// hand on through the scratch would be overwritten by a launch of another call in between.  A StreamUse is the stream's
// turn: it holds the stream's lock from before the first launch that touches the scratch until after the last.  Nobody
// waits for it (or for state_mutex) holding the interpreter lock, which a holder may need.
//
// What is captured into a CUDA graph gets scratch and words of its own (a fill of the words is a node of the graph): a
// replay runs when it likes, beside eager work and other graphs that were captured on the same stream.
struct StreamState {
  std::recursive_mutex mutex;
  Tensor scratch, words;
  unsigned long long capture = 0;   // the capture that scratch and words belong to, 0 = none
};
std::mutex state_mutex;   // of the maps alone
auto& stream_states = *new std::map<std::pair<int, void*>, std::shared_ptr<StreamState>>();
auto& status_words = *new std::map<int, Tensor>();

constexpr int64_t kAmaxWords = 4;   // words [0, 4): castle_amax_scale; then the decode step's counters

class StreamUse {
 public:
  explicit StreamUse(const c10::cuda::CUDAStream& s) : device(s.device_index()) {
    {
      std::lock_guard<std::mutex> lock(state_mutex);
      auto& e = stream_states[{(int)device, (void*)s.stream()}];
      if (!e) e = std::make_shared<StreamState>();
      state = e;
    }
    turn = std::unique_lock<std::recursive_mutex>(state->mutex);
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long capture = 0;
    if (cudaStreamGetCaptureInfo(s.stream(), &status, &capture) != cudaSuccess) (void)cudaGetLastError();   // (the launch will say why)
    if (status != cudaStreamCaptureStatusActive) capture = 0;
    if (capture != state->capture) {
      state->scratch = state->words = Tensor();
      state->capture = capture;
    }
  }
  Tensor scratch(size_t bytes) {
    Tensor& t = state->scratch;
    if (!t.defined() || (size_t)t.numel() < bytes) {
      t = Tensor();   // give the old buffer back before asking for the larger one
      t = at::empty({(int64_t)std::max<size_t>(bytes, (size_t)1 << 20)}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, device));
    }
    return t;
  }
  Tensor zero_words(int64_t count) {
    Tensor& t = state->words;
    if (!t.defined() || t.numel() < kAmaxWords + count)
      t = at::zeros({kAmaxWords + std::max<int64_t>(count, 1020)}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
    return t;
  }

 private:
  c10::DeviceIndex device;
  std::shared_ptr<StreamState> state;   // (release_workspaces() may drop it from the map meanwhile)
  std::unique_lock<std::recursive_mutex> turn;
};

// One word per device for all streams and graphs, so it is cleared outside of both: a fill on the caller's stream could
// run after another stream's kernel has set a bit, and captured into a graph it would clear the word at each replay.
Tensor status_word(int device) {
  std::lock_guard<std::mutex> lock(state_mutex);
  Tensor& t = status_words[device];
  if (!t.defined()) {
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
    const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);   // of another stream's capture
    void* p = nullptr;
    cudaStream_t side = nullptr;
    C10_CUDA_CHECK(cudaMalloc(&p, sizeof(int32_t)));
    C10_CUDA_CHECK(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
    C10_CUDA_CHECK(cudaMemsetAsync(p, 0, sizeof(int32_t), side));
    C10_CUDA_CHECK(cudaStreamSynchronize(side));
    C10_CUDA_CHECK(cudaStreamDestroy(side));
    const c10::InferenceMode normal(false);   // check_status() clears it in any mode
    t = at::from_blob(p, {1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));   // never given back
  }
  return t;
}

// ------------------------------------------------------------------------------------------------ descriptors
int dtype_code(at::ScalarType t) {
  return t == at::kBFloat16 ? CASTLE_BF16 : t == at::kHalf ? CASTLE_F16 : t == at::kFloat ? CASTLE_F32 : -1;
}

castle_tensor_t desc(const Tensor& t) {   // (B, H, N, d), last dimension contiguous
  return {t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)};
}

// The ABI's rules: 16-byte base and strides, the last dimension contiguous, and no dimension that repeats one element's
// row (stride 0, as expand() leaves it), which the kernels' tensor maps cannot express.  And the memory holds the tensor's values,
// which a lazy negation's (an imaginary part of a conjugate) does not; a copy has them.
bool aligned(const Tensor& t) {
  if (t.is_neg()) return false;
  if ((t.stride(-1) != 1 && t.size(-1) != 1) || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0) return false;
  for (int64_t i = 0; i + 1 < t.dim(); ++i)
    if (t.stride(i) * t.element_size() % 16 != 0 || (t.stride(i) == 0 && t.size(i) > 1)) return false;
  return true;
}
Tensor aligned_view(const Tensor& t) { return aligned(t) ? t : t.clone(at::MemoryFormat::Contiguous); }

// Slot i of a packed (B, N, 6, H, d) tensor as a (B, H, N, d) descriptor.
castle_tensor_t packed_desc(const Tensor& p, int i) {
  return {static_cast<char*>(p.data_ptr()) + i * p.stride(2) * p.element_size(), p.stride(0), p.stride(3), p.stride(1)};
}

// Contiguous at a 16-byte boundary (contiguous() leaves a view at an odd offset as it is).
Tensor aligned_contiguous(const Tensor& t) {
  return !t.is_neg() && t.is_contiguous() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 ? t : t.clone(at::MemoryFormat::Contiguous);
}

castle_tensor_t rect(castle_tensor_t t, int64_t es, int64_t b, int64_t h) {
  t.ptr = static_cast<char*>(t.ptr) + (b * t.stride_b + h * t.stride_h) * es;
  return t;
}

Tensor empty_bnhd(int64_t B, int64_t H, int64_t N, int64_t d, const at::TensorOptions& o) {
  // a (B, H, N, d) tensor laid out (B, N, H, d): merging the heads afterwards is a free reshape
  return at::empty_strided({B, H, N, d}, {N * H * d, d, H * d, 1}, o);
}

// ------------------------------------------------------------------------------------------------ parallel pass
struct Rotary {
  Tensor freqs;
  int64_t position0 = 0;
  bool on() const { return freqs.defined(); }
  castle_rotary_t desc(bool inverse) const {
    return {freqs.data_ptr(), dtype_code(freqs.scalar_type()), inverse ? 1 : 0, position0};
  }
  // The kernels read dim_head / 2 values at the frequencies' address: a buffer that was left on the CPU or replaced is
  // brought to where and how they expect it, as the element-wise form does, or refused.
  void fit(const at::Device& dev, int64_t dim_head) {
    if (!on()) return;
    const int64_t count = freqs.numel();
    if (count != 1 && (2 * count != dim_head || freqs.size(-1) != count))
      throw std::runtime_error("castle: rotary frequencies must be (dim_head / 2) = " + std::to_string(dim_head / 2) + " values, or one");
    const bool type_ok = dtype_code(freqs.scalar_type()) >= 0;
    if (freqs.device() == dev && freqs.is_contiguous() && type_ok && 2 * count == dim_head) return;
    at::NoGradGuard no_grad;
    freqs = freqs.to(dev, type_ok ? freqs.scalar_type() : at::kFloat).reshape({count}).expand({dim_head / 2}).contiguous();
  }
};
constexpr int kPackedOrder[6] = {3, 4, 5, 0, 1, 2};   // between the operator's order qc, kc, vc, qu, ku, vu and the packed one, both ways
constexpr uint32_t kRotated = 0x1f;   // of qu, ku, vu, qc, kc, vc all but vc

struct Options {
  double scale = 1;
  bool return_U = false, need_grad = false;
  int64_t limit = 0;           // bytes of scratch per launch
  int64_t long_seq = 0;        // from this length on bf16 callers are computed with fp16 operands
  Rotary rotary;
  std::vector<Tensor> caches;  // four (B, H, N, d) views (U, qu, kc, vc) to fill, or empty
};

// The kernels' inputs: six (B, H, N, dp) descriptors in the order qu, ku, vu, qc, kc, vc and what keeps them alive.
struct Inputs {
  castle_tensor_t t[6];
  std::vector<Tensor> keep;   // one packed tensor, or six
};

struct Problem {
  int64_t B, H, N, d, dp;
  at::ScalarType dtype, cdtype;   // the caller's and the operands'
};

castle_problem_t c_problem(const Problem& p, double scale, at::ScalarType t, int64_t d) {
  return {(int32_t)p.B, (int32_t)p.H, (int32_t)p.N, (int32_t)d, dtype_code(t), (float)scale};
}

Problem make_problem(at::IntArrayRef bhnd, at::ScalarType dtype, int64_t long_seq) {
  Problem p{bhnd[0], bhnd[1], bhnd[2], bhnd[3], 0, dtype, dtype};
  if (p.d > 128 || p.d % 8 || p.d < 1)
    throw std::runtime_error("castle_attention: dim_head " + std::to_string(p.d) + " not supported (multiples of 8 up to 128)");
  need(dtype_code(dtype) >= 0, "castle_attention: tensors must be bf16, fp16 or fp32");
  p.dp = p.d <= 64 ? 64 : 128;
  if (!(dtype == at::kHalf || (dtype == at::kBFloat16 && p.N < long_seq))) p.cdtype = at::kHalf;
  return p;
}

// Rectangles of the (batch, head) grid that each need at most `limit` bytes of scratch: whole batch rows, or head
// ranges of one row, so that per-pair buffers of a rectangle stay contiguous; as few as that takes, all about the same size.
template <typename F>
void for_chunks(int64_t B, int64_t H, int64_t per_pair, int64_t limit, F&& f) {
  need(B > 0 && H > 0, "castle_attention: empty problem");
  const int64_t pairs = limit / std::max<int64_t>(per_pair, 1);
  if (pairs < 1)
    throw std::runtime_error("castle_attention: one (batch, head) pair needs " + std::to_string(per_pair) +
                             " bytes of forward scratch, more than the " + std::to_string(limit) +
                             "-byte bound (sequence too long for this build)");
  auto size = [](int64_t total, int64_t most) { const int64_t n = (total + most - 1) / most; return (total + n - 1) / n; };
  if (pairs >= H) {
    const int64_t s = size(B, std::min(B, pairs / H));
    for (int64_t b = 0; b < B; b += s) f(b, std::min(B, b + s), (int64_t)0, H);
  } else {
    const int64_t s = size(H, pairs);
    for (int64_t b = 0; b < B; ++b)
      for (int64_t h = 0; h < H; h += s) f(b, b + 1, h, std::min(H, h + s));
  }
}

struct Result {
  Tensor out;             // (B, H, N, d), the caller's type
  Tensor U;
  Inputs in;
  Tensor out16, lse, w_state;
};

Result run_forward(const Problem& p, Inputs in, const Options& o, const at::Device& dev) {
  const c10::cuda::CUDAGuard guard(dev);
  const auto stream = c10::cuda::getCurrentCUDAStream(dev.index());
  const auto f32 = at::TensorOptions().dtype(at::kFloat).device(dev);
  const auto ct = f32.dtype(p.cdtype), st = f32.dtype(p.dtype);
  Result r;
  // The forward kernels fill the caches from their operand tiles where those are the caller's values.
  const bool caches = !o.caches.empty();
  const bool kernel_fill = caches && p.dtype == p.cdtype && p.d == p.dp;
  if (p.dtype != p.cdtype || p.d != p.dp || o.rotary.on() || (caches && !kernel_fill)) {
    Tensor packed = at::empty({p.B, p.N, 6, p.H, p.dp}, ct);
    castle_tensor_t dst[6], copies[6] = {};
    for (int i = 0; i < 6; ++i) dst[i] = packed_desc(packed, i);
    if (caches && !kernel_fill) {
      copies[0] = desc(o.caches[1]); copies[4] = desc(o.caches[2]); copies[5] = desc(o.caches[3]);
    }
    const castle_problem_t cp = c_problem(p, o.scale, p.dtype, p.d);
    castle_rotary_t rot{};
    if (o.rotary.on()) rot = o.rotary.desc(false);
    check(api.transform(&cp, 6, in.t, dst, dtype_code(p.cdtype), (int32_t)p.dp, copies, o.rotary.on() ? &rot : nullptr, kRotated,
                        nullptr, stream.stream()), "castle_transform");
    for (int i = 0; i < 6; ++i) in.t[i] = dst[i];
    in.keep = {packed};
  }
  r.out16 = empty_bnhd(p.B, p.H, p.N, p.dp, ct);
  r.lse = at::empty({p.B, p.H, p.N}, f32);
  Tensor u;   // what the kernel writes U to
  if (caches && p.d == p.dp) u = o.caches[0];
  else if (o.return_U || caches) u = at::empty({p.B, p.H, p.N, p.dp}, st);
  if (o.need_grad) r.w_state = at::empty({p.B, p.H, p.N, p.dp}, f32);
  const Tensor status = status_word(dev.index());
  castle_problem_t one = c_problem(p, o.scale, p.cdtype, p.dp);
  one.batch = one.heads = 1;
  const int64_t per_pair = std::max<int64_t>((int64_t)api.fwd_workspace_bytes(&one), 1);
  int64_t most = 0;
  for_chunks(p.B, p.H, per_pair, o.limit, [&](int64_t b0, int64_t b1, int64_t h0, int64_t h1) { most = std::max(most, (b1 - b0) * (h1 - h0)); });
  StreamUse use(stream);
  const Tensor ws = use.scratch((size_t)(most * per_pair));
  const castle_tensor_t out_d = desc(r.out16);
  for_chunks(p.B, p.H, per_pair, o.limit, [&](int64_t b0, int64_t b1, int64_t h0, int64_t h1) {
    castle_problem_t cp = one;
    cp.batch = (int32_t)(b1 - b0);
    cp.heads = (int32_t)(h1 - h0);
    castle_tensor_t t[6];
    for (int i = 0; i < 6; ++i) t[i] = rect(in.t[i], 2, b0, h0);
    const castle_tensor_t od = rect(out_d, 2, b0, h0);
    const int64_t pair0 = b0 * p.H + h0;
    float* lse = r.lse.data_ptr<float>() + pair0 * p.N;
    float* w = o.need_grad ? r.w_state.data_ptr<float>() + pair0 * p.N * p.dp : nullptr;
    castle_tensor_t ud{};
    if (u.defined()) ud = rect(desc(u), u.element_size(), b0, h0);
    if (kernel_fill) {
      castle_tensor_t c[3];
      for (int i = 0; i < 3; ++i) c[i] = rect(desc(o.caches[1 + i]), 2, b0, h0);
      check(api.fwd_prefill(&cp, &t[3], &t[4], &t[5], &t[0], &t[1], &t[2], &od, lse, &ud, &c[0], &c[1], &c[2], w, ws.data_ptr(),
                            ws.numel(), status.data_ptr<int32_t>(), stream.stream()), "castle_fwd_prefill");
    } else {
      check(api.fwd(&cp, &t[3], &t[4], &t[5], &t[0], &t[1], &t[2], &od, lse, u.defined() ? &ud : nullptr, dtype_code(p.dtype), w,
                    ws.data_ptr(), ws.numel(), status.data_ptr<int32_t>(), stream.stream()), "castle_fwd");
    }
  });
  r.out = r.out16;
  if (p.dtype != p.cdtype || p.d != p.dp) {
    r.out = empty_bnhd(p.B, p.H, p.N, p.d, st);
    const castle_problem_t cp = c_problem(p, o.scale, p.cdtype, p.dp);
    const castle_tensor_t dst = desc(r.out);
    check(api.transform(&cp, 1, &out_d, &dst, dtype_code(p.dtype), (int32_t)p.d, nullptr, nullptr, 0, nullptr, stream.stream()),
          "castle_transform");
  }
  if (caches && p.d != p.dp) o.caches[0].copy_(u.narrow(3, 0, p.d));
  if (o.return_U) r.U = caches ? o.caches[0].narrow(3, 0, p.d) : u.narrow(3, 0, p.d);
  r.in = std::move(in);
  return r;
}

// The six input gradients as one packed (B, N, 6, H, d) tensor in the caller's type.
Tensor run_backward(const Problem& p, const castle_tensor_t* in, const Tensor& out16, const Tensor& lse, const Tensor& w_state,
                    Tensor grad, const Options& o) {
  const at::Device dev = out16.device();
  const c10::cuda::CUDAGuard guard(dev);
  const auto stream = c10::cuda::getCurrentCUDAStream(dev.index());
  const auto ct = at::TensorOptions().dtype(p.cdtype).device(dev);
  StreamUse use(stream);
  Tensor factor;   // [s, 1 / s]
  if (p.dtype != p.cdtype) {
    // fp16 operands for a caller with a wider exponent range: bring the upstream gradient to a fixed magnitude with a
    // power of two (exact; every gradient is linear in it) and undo it on the results, so that neither small gradients
    // underflow nor large ones overflow in fp16.  Everything stays on the device.
    if (!grad.is_non_overlapping_and_dense() || !aligned(grad)) grad = grad.clone(at::MemoryFormat::Contiguous);
    factor = at::empty({2}, ct.dtype(at::kFloat));
    const Tensor words = use.zero_words(0);
    check(api.amax_scale(dtype_code(p.dtype), grad.data_ptr(), grad.numel(), reinterpret_cast<uint32_t*>(words.data_ptr()),
                         factor.data_ptr<float>(), stream.stream()), "castle_amax_scale");
  }
  if (p.dtype != p.cdtype || p.d != p.dp) {
    grad = aligned_view(grad);
    Tensor g16 = empty_bnhd(p.B, p.H, p.N, p.dp, ct);
    const castle_problem_t cp = c_problem(p, o.scale, p.dtype, p.d);
    const castle_tensor_t src = desc(grad), dst = desc(g16);
    check(api.transform(&cp, 1, &src, &dst, dtype_code(p.cdtype), (int32_t)p.dp, nullptr, nullptr, 0,
                        factor.defined() ? factor.data_ptr<float>() : nullptr, stream.stream()), "castle_transform");
    grad = g16;
  }
  grad = aligned_view(grad);
  Tensor packed = at::empty({p.B, p.N, 6, p.H, p.dp}, ct);
  castle_tensor_t g[6];
  for (int i = 0; i < 6; ++i) g[i] = packed_desc(packed, i);
  const castle_problem_t cp = c_problem(p, o.scale, p.cdtype, p.dp);
  int64_t bytes = (int64_t)api.bwd_workspace_bytes(&cp);
  if (p.dp == 128 && bytes > o.limit) {
    // the tile hand-over scratch of the dim_head-128 kernels may be smaller than asked for: the (batch, head) pairs
    // then run in smaller chunks, down to one pair at a time
    const int64_t nblk = (p.N + 127) / 128, pair = nblk * (nblk + 1) / 2 * 3 * 32768;
    const int64_t asked = std::min<int64_t>(p.B * p.H, std::max<int64_t>(1, ((int64_t)8 << 30) / pair));
    bytes = std::max(bytes - (asked - 1) * pair, o.limit);
  }
  const Tensor ws = use.scratch((size_t)bytes);
  const castle_tensor_t od = desc(out16), gd = desc(grad);
  check(api.bwd(&cp, &in[3], &in[4], &in[5], &in[0], &in[1], &in[2], &od, &gd, lse.data_ptr<float>(), w_state.data_ptr<float>(),
                &g[3], &g[4], &g[5], &g[0], &g[1], &g[2], ws.data_ptr(), ws.numel(), status_word(dev.index()).data_ptr<int32_t>(),
                stream.stream()), "castle_bwd");
  if (p.dtype == p.cdtype && p.d == p.dp && !o.rotary.on()) return packed;
  Tensor result = at::empty({p.B, p.N, 6, p.H, p.d}, ct.dtype(p.dtype));
  castle_tensor_t dst[6];
  for (int i = 0; i < 6; ++i) dst[i] = packed_desc(result, i);
  castle_rotary_t rot{};
  if (o.rotary.on()) rot = o.rotary.desc(true);
  check(api.transform(&cp, 6, g, dst, dtype_code(p.dtype), (int32_t)p.d, nullptr, o.rotary.on() ? &rot : nullptr, kRotated,
                      factor.defined() ? factor.data_ptr<float>() + 1 : nullptr, stream.stream()), "castle_transform");
  return result;
}

// A tensor that went through saved-tensor hooks: whatever they gave back must be the tensor that was saved, since the
// kernels get its address.  Its strides may be others (save_on_cpu gives contiguous ones).
Tensor restored(const Tensor& t, at::IntArrayRef sizes, at::ScalarType dtype, const at::Device& dev) {
  if (!t.defined() || t.sizes() != sizes || t.scalar_type() != dtype || t.device() != dev || t.layout() != at::kStrided)
    throw std::runtime_error("castle_attention: a saved tensor came back from its hooks with another shape, type or device");
  return t;
}
Tensor restored_contiguous(const Tensor& t, at::IntArrayRef sizes, at::ScalarType dtype, const at::Device& dev) {
  restored(t, sizes, dtype, dev);
  return aligned_contiguous(t);
}

// What the core's backward needs of its forward.  Unpacking may run a user's hooks (checkpointing runs the whole forward
// again there), so it comes before anything that changes the thread's dispatch or gradient mode.
struct SavedCore {
  Problem p;
  Options o;
  std::vector<SavedVariable> inputs;   // one packed tensor, or six
  SavedVariable out16, lse, w_state, freqs;
  bool out_is_output = false;

  struct Unpacked { std::vector<Tensor> inputs; Tensor out16, lse, w_state, freqs; };

  // After set_history() of the node's output; `output`: out16 is that output.
  void save(const Problem& problem, const Options& options, const Result& r, bool output) {
    p = problem;
    o = options;
    o.caches.clear();
    freqs = SavedVariable(o.rotary.freqs, false);
    for (const auto& t : r.in.keep) inputs.emplace_back(t, false);
    out_is_output = output;
    out16 = SavedVariable(r.out16, output);
    lse = SavedVariable(r.lse, false);
    w_state = SavedVariable(r.w_state, false);
  }
  void reset() {
    for (auto& v : inputs) v.reset_data();
    out16.reset_data(); lse.reset_data(); w_state.reset_data(); freqs.reset_data();
  }
  Unpacked unpack(const std::shared_ptr<Node>& self) const {
    Unpacked u;
    for (const auto& v : inputs) u.inputs.push_back(v.unpack());
    u.out16 = out_is_output ? out16.unpack(self) : out16.unpack();
    u.lse = lse.unpack(); u.w_state = w_state.unpack(); u.freqs = freqs.unpack();
    return u;
  }
  Tensor backward(const Unpacked& u, const Tensor& grad) const {
    const at::Device dev = grad.device();
    const std::array<int64_t, 4> grad_sizes{p.B, p.H, p.N, p.d};
    need(grad.sizes() == at::IntArrayRef(grad_sizes) && grad.scalar_type() == p.dtype, "castle_attention: the gradient's shape or type is not the output's");
    const std::vector<int64_t> bhnd{p.B, p.H, p.N, p.dp};
    Options now = o;
    if (o.rotary.on()) now.rotary.freqs = restored_contiguous(u.freqs, o.rotary.freqs.sizes(), o.rotary.freqs.scalar_type(), dev);
    castle_tensor_t in[6];
    std::vector<Tensor> keep;
    for (const auto& t : u.inputs) {
      if (u.inputs.size() == 1) keep.push_back(aligned_view(restored(t, {p.B, p.N, 6, p.H, p.dp}, p.cdtype, dev)));
      else keep.push_back(aligned_view(restored(t, bhnd, p.cdtype, dev)));
    }
    for (int i = 0; i < 6; ++i) in[i] = keep.size() == 1 ? packed_desc(keep[0], i) : desc(keep[i]);
    return run_backward(p, in, aligned_view(restored(u.out16, bhnd, p.cdtype, dev)), restored_contiguous(u.lse, {p.B, p.H, p.N}, at::kFloat, dev),
                        restored_contiguous(u.w_state, bhnd, at::kFloat, dev), grad, now);
  }
};

// Gradient node of both operators: one packed input, or six in the operator's order qc, kc, vc, qu, ku, vu.
struct CastleBackward : public Node {
  SavedCore core;
  bool packed = false;

  std::string name() const override { return "CastleAttentionBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    core.reset();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list result(packed ? 1 : 6);
    if (grads.empty() || !grads[0].defined()) return result;
    const SavedCore::Unpacked saved = core.unpack(shared_from_this());
    at::NoGradGuard no_grad;
    Tensor g = core.backward(saved, grads[0]);
    if (packed) {
      result[0] = std::move(g);
    } else {
      for (int i = 0; i < 6; ++i) result[i] = g.select(2, kPackedOrder[i]).permute({0, 2, 1, 3});
    }
    return result;
  }
};

// Whether forward-mode differentiation goes through the tensor, which the kernels would drop.
bool has_tangent(const Tensor& t) {
  const torch::autograd::AutogradMeta* m = t.defined() ? torch::autograd::impl::get_autograd_meta(t) : nullptr;
  return m && m->fw_grad_ && t._fw_grad(/*level=*/0).defined();
}

// Forward with its gradient node; `vars` are the differentiable inputs (one packed, or six in operator order).
Result attention(const Problem& p, Inputs in, Options o, const std::vector<Tensor>& vars) {
  bool any = false;
  for (const auto& v : vars) {
    any |= v.requires_grad();
    TORCH_CHECK_NOT_IMPLEMENTED(!has_tangent(v), "castle_attention: forward-mode differentiation is not implemented");
  }
  o.need_grad = any && at::GradMode::is_enabled();
  const at::Device dev = vars[0].device();
  Result r;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    r = run_forward(p, std::move(in), o, dev);
  }
  if (!o.need_grad) return r;
  auto node = std::shared_ptr<CastleBackward>(new CastleBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(vars));
  node->packed = vars.size() == 1;
  torch::autograd::set_history(r.out, node);
  node->core.save(p, o, r, r.out.is_same(r.out16));
  return r;
}

Result attention_six(const Tensor* v /* qc, kc, vc, qu, ku, vu */, const Options& o) {
  for (int i = 0; i < 6; ++i) {
    need(v[i].is_cuda(), "castle_attention: expected CUDA tensors; this package has no CPU path");
    need(v[i].dim() == 4 && v[i].sizes() == v[0].sizes() && v[i].device() == v[0].device(),
         "castle_attention: six (B, H, N, d) tensors of one shape and device expected");
  }
  const Problem p = make_problem(v[0].sizes(), v[0].scalar_type(), o.long_seq);
  Inputs in;
  {
    at::NoGradGuard no_grad;
    for (int i = 0; i < 6; ++i) {
      Tensor t = v[kPackedOrder[i]];
      if (t.scalar_type() != p.dtype) t = t.to(p.dtype);
      t = aligned_view(t);
      in.t[i] = desc(t);
      in.keep.push_back(t);
    }
  }
  return attention(p, std::move(in), o, std::vector<Tensor>(v, v + 6));
}

Result attention_packed(const Tensor& packed, Options o) {   // (B, N, 6, H, d), order qu, ku, vu, qc, kc, vc
  need(packed.is_cuda(), "castle_attention: expected CUDA tensors; this package has no CPU path");
  need(packed.dim() == 5 && packed.size(2) == 6, "castle_attention_packed: a (B, N, 6, H, d) tensor expected");
  const int64_t B = packed.size(0), N = packed.size(1), H = packed.size(3), d = packed.size(4);
  const Problem p = make_problem({B, H, N, d}, packed.scalar_type(), o.long_seq);
  o.rotary.fit(packed.device(), d);
  Tensor t;
  {
    at::NoGradGuard no_grad;
    t = aligned_view(packed);
  }
  Inputs in;
  for (int i = 0; i < 6; ++i) in.t[i] = packed_desc(t, i);
  in.keep = {t};
  return attention(p, std::move(in), o, {packed});
}

// ------------------------------------------------------------------------------------------------ decode step
void check_caches(const Tensor* caches, int64_t B, int64_t H, int64_t d, at::ScalarType dtype, const at::Device& dev) {
  const int64_t cap = caches[0].size(2);
  for (int i = 0; i < 4; ++i) {
    const Tensor& c = caches[i];
    if (!(c.scalar_type() == dtype && c.dim() == 4 && c.size(0) == B && c.size(1) == H && c.size(2) == cap && c.size(3) == d &&
          c.stride(3) == 1))
      throw AssertError("castle_decode_step: the caches must be (B, H, capacity, d) buffers of the token's type");
    need(c.device() == dev, "castle_decode_step: the caches must be on the token's device");
  }
}

// `news` in the operator's order qc, kc, vc, qu, ku, vu; `caches` U, qu, kc, vc; `out` contiguous (B, H, 1, d).
void launch_decode(const castle_problem_t& cp, const castle_tensor_t* news, const Tensor* caches, void* out, int64_t t, const Rotary& rotary,
                   bool overlap, void* ws, size_t ws_bytes, const c10::cuda::CUDAStream& stream, StreamUse& use) {
  const Tensor words = use.zero_words((int64_t)cp.batch * cp.heads), status = status_word(stream.device_index());
  castle_tensor_t c[4];
  for (int i = 0; i < 4; ++i) c[i] = desc(caches[i]);
  const castle_tensor_t od{out, (int64_t)cp.heads * cp.dim_head, cp.dim_head, cp.dim_head};
  castle_rotary_t rot{};
  if (rotary.on()) rot = rotary.desc(false);
  check(api.decode_step_fused(&cp, (int32_t)t, (int32_t)caches[0].size(2), &news[0], &news[1], &news[2], &news[3], &news[4], &news[5],
                              &c[0], &c[1], &c[2], &c[3], &od, rotary.on() ? &rot : nullptr,
                              reinterpret_cast<uint32_t*>(words.data_ptr()) + kAmaxWords, overlap, ws, ws_bytes, status.data_ptr<int32_t>(),
                              stream.stream()), "castle_decode_step");
}

Tensor decode_core(const castle_tensor_t* news, const Tensor* caches, int64_t B, int64_t H, int64_t d, at::ScalarType dtype,
                   int64_t t, double scale, Rotary rotary, const at::Device& dev) {
  const c10::cuda::CUDAGuard guard(dev);
  rotary.fit(dev, d);
  const auto stream = c10::cuda::getCurrentCUDAStream(dev.index());
  check_caches(caches, B, H, d, dtype, dev);
  Tensor out = at::empty({B, H, 1, d}, caches[0].options());
  const castle_problem_t cp{(int32_t)B, (int32_t)H, 1, (int32_t)d, dtype_code(dtype), (float)scale};
  StreamUse use(stream);
  const Tensor ws = use.scratch(api.decode_workspace_bytes(&cp, (int32_t)t));
  launch_decode(cp, news, caches, out.data_ptr(), t, rotary, false, ws.data_ptr(), ws.numel(), stream, use);
  return out;
}

Tensor decode_step(const Tensor* news, const Tensor* caches, int64_t t, double scale) {
  need(news[0].is_cuda(), "castle_decode_step: expected CUDA tensors; this package has no CPU path");
  if (news[0].dim() != 4 || news[0].size(2) != 1) throw AssertError("castle_decode_step: (B, H, 1, d) tensors expected");
  const auto dtype = news[0].scalar_type();
  if (dtype_code(dtype) < 0) throw std::runtime_error("castle_decode_step: dtype " + std::string(at::toString(dtype)) + " not supported");
  at::NoGradGuard no_grad;
  Tensor keep[6];
  castle_tensor_t nd[6];
  for (int i = 0; i < 6; ++i) {
    need(news[i].scalar_type() == dtype && news[i].sizes() == news[0].sizes() && news[i].device() == news[0].device(),
         "castle_decode_step: the new rows must have one shape, type and device");
    keep[i] = aligned_view(news[i]);
    nd[i] = desc(keep[i]);
  }
  return decode_core(nd, caches, news[0].size(0), news[0].size(1), news[0].size(3), dtype, t, scale, Rotary{}, news[0].device());
}

// ------------------------------------------------------------------------------------------------ the plain module
struct Layer {
  Tensor norm, to_qkv, combine;   // norm may be undefined
  std::optional<double> eps;
  int64_t heads = 0, dim_head = 0;
};

// Whether the layer can run natively around the core, too: plain CUDA tensors of one type, and nothing that changes what a
// linear call means (autocast, a dispatch mode, forward-mode differentiation).
bool plain_layer(const Tensor& x, const Layer& l) {
  auto plain = [&](const Tensor& t) {
    return t.is_cuda() && t.scalar_type() == x.scalar_type() && t.is_contiguous() && t.layout() == at::kStrided && t.device() == x.device() &&
           reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && !t.is_neg() && !t.unsafeGetTensorImpl()->is_python_dispatch() && !has_tangent(t);
  };
  const int64_t inner = l.heads * l.dim_head;
  return x.dim() == 3 && x.is_cuda() && x.numel() > 0 && x.layout() == at::kStrided && !x.is_neg() && !x.unsafeGetTensorImpl()->is_python_dispatch() && !has_tangent(x) &&
         dtype_code(x.scalar_type()) >= 0 && x.size(2) % 8 == 0 && plain(l.to_qkv) && plain(l.combine) &&
         (!l.norm.defined() || (plain(l.norm) && l.norm.dim() == 1 && l.norm.size(0) == x.size(2))) && l.to_qkv.dim() == 2 &&
         l.to_qkv.size(0) == 6 * inner && l.to_qkv.size(1) == x.size(2) && l.combine.dim() == 2 && l.combine.size(1) == inner &&
         !at::autocast::is_autocast_enabled(at::kCUDA) && !c10::impl::dispatch_mode_enabled();
}

float norm_eps(const Layer& l) { return (float)l.eps.value_or(std::numeric_limits<float>::epsilon()); }   // torch's default for every type

// Whether a product of a call over `rows` positions is the framework's own launch (csrc/linear.cu).  A library product costs the
// host 8 to 10 us, an own one 4, and such calls are bound by the host; on the GPU the library is 1 to 2 us faster in 16 bits
// (us, own / library: 197 x 512 -> 3072 4.9 / 3.4, 512 x 512 -> 3072 9.1 / 4.3, 2048 x 512 -> 3072 14.7 / 8.3) and slower in
// fp32 but where the tiles are many (512 x 128 -> 768 8.6 / 6.2, 512 x 768 -> 128 10.2 / 14.4, its weight's gradient 7.0 / 10.3,
// 197 x 512 -> 3072 33.6 / 25.4).  From some 1024 positions on the GPU is the bound.  A graph's replay costs the host nothing, so a
// capture takes the library's products; the two add in different orders, so a replay and an eager call differ by fp32 rounding of the
// sums (and a 16-bit result now and then by its last place).  A loop whose host runs ahead of the GPU pays the 1 to 2 us.
bool small_product(int64_t rows, int64_t m, int64_t n, int64_t k, at::ScalarType t) {
  const bool f32 = t == at::kFloat;
  if (rows > 1024 || 2 * m * n * k > (f32 ? 128000000LL : 1000000000LL)) return false;
  return dtype_code(t) >= 0 && std::min(n, k) >= 64;
}
// layout 0: a @ b^T; 1: a @ b; 2: a^T @ b, for two-dimensional a and b
Tensor product(int layout, const Tensor& a, const Tensor& b, int64_t rows) {
  const int64_t k = layout == 2 ? a.size(0) : a.size(1), m = layout == 2 ? a.size(1) : a.size(0), n = layout == 0 ? b.size(0) : b.size(1);
  const int64_t unit = 16 / a.element_size();
  // a tensor without memory of its own (a batched gradient's wrapper) and a dispatch mode that counts or replaces the products: the library's path
  auto fits = [&](const Tensor& t) { return !at::isTensorSubclassLike(t) && t.stride(1) == 1 && t.stride(0) >= t.size(1) && aligned(t); };
  // what does not match (in k, type or device) is the library's to refuse
  const bool match = b.scalar_type() == a.scalar_type() && b.device() == a.device() && b.size(layout == 0 ? 1 : 0) == k;
  if (match && small_product(rows, m, n, k, a.scalar_type()) && n % unit == 0 && (layout == 2 ? m : k) % unit == 0 && fits(a) && fits(b)) {
    const auto stream = c10::cuda::getCurrentCUDAStream(a.device().index());
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream.stream(), &capture) != cudaSuccess) (void)cudaGetLastError();
    if (capture == cudaStreamCaptureStatusNone) {
      const Tensor c = at::empty({m, n}, a.options().requires_grad(false)), status = status_word(a.device().index());
      check(api.linear(dtype_code(a.scalar_type()), layout, (int32_t)m, (int32_t)n, (int32_t)k, a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0),
                       c.data_ptr(), n, status.data_ptr<int32_t>(), stream.stream()), "castle_linear");
      return c;
    }
  }
  return layout == 0 ? at::mm(a, b.t()) : layout == 1 ? at::mm(a, b) : at::mm(a.t(), b);
}

// Gradient node of a whole layer.  Autograd over the single operations (norm, two linear layers, the views between them
// and the core) cost 250 us of host time per training step where the kernels of a small one take 120.
struct LayerBackward : public Node {
  int64_t dim = 0;
  bool has_norm = false, separate_h = false, separate_merged = false;
  at::ScalarType dtype = at::kFloat;
  std::vector<int64_t> x_sizes;
  // Like autograd over the single operations would, each kept only where a gradient that was asked for needs it, and
  // nothing is kept beside them: a hook (checkpointing, save_on_cpu) sees all of it.
  SavedCore core;
  SavedVariable x, to_qkv, combine, norm, rstd;
  SavedVariable h;        // the projection's input, unless that is x
  SavedVariable merged;   // the output projection's input, unless that is the core's output

  std::string name() const override { return "CastleLayerBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    core.reset();
    for (SavedVariable* v : {&x, &to_qkv, &combine, &norm, &rstd, &h, &merged}) v->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list result(has_norm ? 4 : 3);
    if (grads.empty() || !grads[0].defined()) return result;
    const bool need_x = task_should_compute_output(0), need_qkv = task_should_compute_output(1), need_combine = task_should_compute_output(2),
               need_norm = has_norm && task_should_compute_output(3);
    const bool need_core = need_x || need_qkv || need_norm, need_out = need_combine && !separate_merged;
    const Problem& p = core.p;
    const int64_t rows = p.B * p.N, inner = p.H * p.d;
    const at::Device dev = grads[0].device();
    SavedCore::Unpacked saved;   // (unpacking raises on a second backward)
    if (need_core) saved = core.unpack(shared_from_this());
    else if (need_out) saved.out16 = core.out16.unpack();
    const Tensor wc = need_core ? restored(combine.unpack(), {grads[0].size(-1), inner}, dtype, dev) : Tensor(),
                 wq = need_x || need_norm ? restored(to_qkv.unpack(), {6 * inner, dim}, dtype, dev) : Tensor(),
                 xs = (need_qkv && !separate_h) || (has_norm && (need_x || need_norm)) ? restored(x.unpack(), x_sizes, dtype, dev) : Tensor(),
                 hs = need_qkv && separate_h ? restored(h.unpack(), {rows, dim}, dtype, dev) : Tensor(),
                 ms = need_combine && separate_merged ? restored(merged.unpack(), {rows, inner}, dtype, dev) : Tensor(),
                 ws_norm = has_norm && (need_x || need_norm) ? norm.unpack() : Tensor(),
                 rs_norm = has_norm && (need_x || need_norm) ? rstd.unpack() : Tensor();
    at::AutoDispatchBelowADInplaceOrView below;
    // A backward called under autocast: the products keep the layer's type, in which the kernels behind them read their results.
    const c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    const c10::cuda::CUDAGuard guard(dev);
    const auto stream = c10::cuda::getCurrentCUDAStream(dev.index());
    const Tensor g = grads[0].reshape({rows, grads[0].size(-1)});
    if (need_combine)
      result[2] = product(2, g, separate_merged ? ms : restored(saved.out16, {p.B, p.H, p.N, p.dp}, p.cdtype, dev).permute({0, 2, 1, 3}).reshape({rows, inner}), rows);
    if (!need_core) return result;
    const Tensor dcore = product(1, g, wc, rows).view({p.B, p.N, p.H, p.d}).permute({0, 2, 1, 3});
    const Tensor dqkv = core.backward(saved, dcore).view({rows, 6 * inner});
    if (need_qkv) result[1] = product(2, dqkv, separate_h ? hs : xs.reshape({rows, dim}), rows);
    if (!(need_x || need_norm)) return result;
    Tensor dh = product(1, dqkv, wq, rows);
    if (!has_norm) {
      result[0] = dh.view(x_sizes);
      return result;
    }
    const Tensor xc = aligned_contiguous(xs), wn = restored_contiguous(ws_norm, {dim}, dtype, dev),
                 rs = restored_contiguous(rs_norm, {rows}, at::kFloat, dev);
    if (need_x) result[0] = at::empty(x_sizes, dh.options());
    if (need_norm) result[3] = at::empty({dim}, dh.options());
    const size_t bytes = api.rmsnorm_bwd_workspace_bytes(rows, (int32_t)dim);
    StreamUse use(stream);
    const Tensor ws = use.scratch(bytes);
    check(api.rmsnorm_bwd(dtype_code(dtype), rows, (int32_t)dim, dh.data_ptr(), xc.data_ptr(), wn.data_ptr(), rs.data_ptr<float>(),
                          need_x ? result[0].data_ptr() : nullptr, need_norm ? result[3].data_ptr() : nullptr, ws.data_ptr(), ws.numel(),
                          stream.stream()), "castle_rmsnorm_bwd");
    return result;
  }
};

// Norm, projection, core and output projection, for plain_layer().
Tensor layer_native(const Tensor& x, const Layer& l, Options o) {
  const bool grad = at::GradMode::is_enabled(), has_norm = l.norm.defined();
  const bool need_x = grad && x.requires_grad(), need_qkv = grad && l.to_qkv.requires_grad(), need_combine = grad && l.combine.requires_grad(),
             need_norm = grad && has_norm && l.norm.requires_grad();
  o.need_grad = need_x || need_qkv || need_norm;
  const int64_t B = x.size(0), N = x.size(1), dim = x.size(2), rows = B * N, inner = l.heads * l.dim_head;
  const Problem p = make_problem({B, l.heads, N, l.dim_head}, x.scalar_type(), o.long_seq);
  o.rotary.fit(x.device(), l.dim_head);
  Tensor out, h, rstd, merged;
  Result r;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    const c10::cuda::CUDAGuard guard(x.device());
    const auto stream = c10::cuda::getCurrentCUDAStream(x.device().index());
    h = x.contiguous().view({rows, dim});
    if (has_norm) {
      const Tensor src = aligned_contiguous(h);
      h = at::empty({rows, dim}, x.options().requires_grad(false));
      if (o.need_grad) rstd = at::empty({rows}, x.options().dtype(at::kFloat).requires_grad(false));
      check(api.rmsnorm_fwd(dtype_code(p.dtype), rows, (int32_t)dim, src.data_ptr(), l.norm.data_ptr(), norm_eps(l), h.data_ptr(),
                            o.need_grad ? rstd.data_ptr<float>() : nullptr, stream.stream()), "castle_rmsnorm_fwd");
    }
    const Tensor packed = product(0, h, l.to_qkv, rows).view({B, N, 6, l.heads, l.dim_head});
    Inputs in;
    for (int i = 0; i < 6; ++i) in.t[i] = packed_desc(packed, i);
    in.keep = {packed};
    r = run_forward(p, std::move(in), o, x.device());
    merged = r.out.permute({0, 2, 1, 3}).view({rows, inner});
    out = product(0, merged, l.combine, rows).view({B, N, l.combine.size(0)});
  }
  if (!(o.need_grad || need_combine)) return out;
  auto node = std::shared_ptr<LayerBackward>(new LayerBackward(), torch::autograd::deleteNode);
  std::vector<Tensor> vars{x, l.to_qkv, l.combine};
  if (has_norm) vars.push_back(l.norm);
  node->set_next_edges(torch::autograd::collect_next_edges(vars));
  node->dim = dim;
  node->has_norm = has_norm;
  node->dtype = p.dtype;
  node->x_sizes = x.sizes().vec();
  torch::autograd::set_history(out, node);
  auto keep = [](const Tensor& t) { return SavedVariable(t, false); };
  if (o.need_grad) {
    node->core.save(p, o, r, false);
    node->combine = keep(l.combine);
  } else {
    node->core.p = p;
  }
  node->separate_merged = need_combine && !(o.need_grad && r.out.is_same(r.out16));
  if (node->separate_merged) node->merged = keep(merged);
  node->separate_h = need_qkv && (has_norm || !x.is_contiguous());
  if (node->separate_h) node->h = keep(h);
  if ((need_qkv && !node->separate_h) || (has_norm && (need_x || need_norm))) node->x = keep(x);
  if (need_x || need_norm) node->to_qkv = keep(l.to_qkv);
  if (has_norm && (need_x || need_norm)) {
    node->norm = keep(l.norm);
    node->rstd = keep(rstd);
  }
  return out;
}

Tensor project(const Tensor& x, const Layer& l) {   // (B, N, 6, H, d)
  Tensor h = l.norm.defined() ? at::rms_norm(x, {x.size(-1)}, l.norm, l.eps) : x;
  return at::linear(h, l.to_qkv).view({x.size(0), x.size(1), 6, l.heads, l.dim_head});
}

Tensor layer_forward(const Tensor& x, const Layer& l, const Options& o) {
  if (plain_layer(x, l)) return layer_native(x, l, o);
  const Tensor out = attention_packed(project(x, l), o).out;
  return at::linear(out.permute({0, 2, 1, 3}).reshape({x.size(0), x.size(1), l.heads * l.dim_head}), l.combine);
}

// One token from its packed projection (B, 1, 6, H, d): the core's output, (B, 1, H * d).
Tensor decode_packed(const Tensor& packed, const Tensor* caches, int64_t t, double scale, const Rotary& rotary) {
  need(packed.is_cuda(), "castle_decode_step: expected CUDA tensors; this package has no CPU path");
  const int64_t B = packed.size(0), H = packed.size(3), d = packed.size(4);
  need(dtype_code(packed.scalar_type()) >= 0, "castle_decode_step: bf16, fp16 or fp32 expected");
  at::NoGradGuard no_grad;
  castle_tensor_t nd[6];
  for (int i = 0; i < 6; ++i) nd[i] = packed_desc(packed, kPackedOrder[i]);
  return decode_core(nd, caches, B, H, d, packed.scalar_type(), t, scale, rotary, packed.device()).view({B, 1, H * d});
}

// Whether one projection of a token is the framework's own launch.  It is the faster one on the host (3 us against 8 for a
// library call, with the norm in it); on the GPU the library wins in 16 bits where the weights are large for the rows (own /
// library in us, weights from memory: 8 x 512 -> 3072 4.2 / 4.0, 8 x 1024 -> 6144 6.1 / 5.2, 8 x 1408 -> 8448 9.3 / 6.6,
// 2 x 1408 -> 8448 8.6 / 7.0, 2 x 2176 -> 13056 14.6 / 11.8, 1 x 2176 -> 13056 12.2 / 12.0).  In fp32, where every row count
// takes the FMA kernel, the library is the slower one on both sides of the bound (3 x 512 -> 3072 5.9 / 7.0, 8 x 512 -> 3072
// 7.2 / 14.7, 8 x 1024 -> 6144 12.8 / 27.2), but at one row (512 -> 3072 4.5 / 4.1).
bool own_projection(int dtype, int64_t rows, int64_t k, int64_t n, int64_t es) {
  return rows <= 8 && k * n * es <= (rows == 1 ? 64 << 20 : rows == 2 ? 16 << 20 : 8 << 20) &&
         api.token_linear_fits(dtype, (int32_t)rows, (int32_t)k);
}

// Whether the layer's whole token is one launch (csrc/token_layer.cu).
bool whole_token_layer(const castle_problem_t& p, const Tensor* caches, int64_t t, int64_t dim, int64_t out_features, int64_t es) {
  for (int i = 0; i < 4; ++i)
    if (!aligned(caches[i]) || caches[i].stride(2) != p.dim_head) return false;
  return api.token_layer_fits(&p, (int32_t)t, (int32_t)dim, (int32_t)out_features);
}

// Norm, projection, step and output projection of one token, with what passes between them in the stream's scratch: on
// the host the allocations would cost as much as the launches.
Tensor token_layer(const Tensor& x, const Layer& l, const Tensor* caches, int64_t t, double scale, Rotary rotary) {
  const at::Device dev = x.device();
  const c10::cuda::CUDAGuard guard(dev);
  rotary.fit(dev, l.dim_head);
  at::AutoDispatchBelowADInplaceOrView below;
  const auto stream = c10::cuda::getCurrentCUDAStream(dev.index());
  const auto dtype = x.scalar_type();
  const int64_t B = x.size(0), dim = x.size(2), H = l.heads, d = l.dim_head, inner = H * d, es = x.element_size();
  check_caches(caches, B, H, d, dtype, dev);
  const castle_problem_t cp{(int32_t)B, (int32_t)H, 1, (int32_t)d, dtype_code(dtype), (float)scale};
  const Tensor xs = x.stride(2) == 1 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0 && x.stride(0) * es % 16 == 0 ? x : aligned_contiguous(x);
  if (whole_token_layer(cp, caches, t, dim, l.combine.size(0), es)) {
    const int64_t N = l.combine.size(0);
    castle_tensor_t c[4];
    for (int i = 0; i < 4; ++i) c[i] = desc(caches[i]);
    castle_rotary_t rot{};
    if (rotary.on()) rot = rotary.desc(false);
    Tensor y = at::empty({B, 1, N}, x.options().requires_grad(false));
    StreamUse use(stream);
    const Tensor words = use.zero_words(8 * B), ws = use.scratch(api.token_layer_workspace_bytes(&cp, (int32_t)N)), status = status_word(dev.index());
    check(api.token_layer(&cp, (int32_t)t, (int32_t)caches[0].size(2), (int32_t)dim, (int32_t)N, xs.data_ptr(), xs.stride(0),
                          l.norm.defined() ? l.norm.data_ptr() : nullptr, norm_eps(l), l.to_qkv.data_ptr(), l.combine.data_ptr(), &c[0], &c[1],
                          &c[2], &c[3], rotary.on() ? &rot : nullptr, y.data_ptr(), reinterpret_cast<uint32_t*>(words.data_ptr()) + kAmaxWords,
                          1, ws.data_ptr(), ws.numel(), status.data_ptr<int32_t>(), stream.stream()), "castle_token_layer");
    return y;
  }
  const int64_t row = (B * inner * es + 255) / 256 * 256;
  const size_t part = (api.decode_workspace_bytes(&cp, (int32_t)t) + 255) / 256 * 256;
  StreamUse use(stream);
  const Tensor ws = use.scratch(part + 7 * row);
  char* packed = static_cast<char*>(ws.data_ptr()) + part;
  char* core = packed + 6 * row;
  Tensor keep;
  // The step and the last projection are launched ahead (see the C ABI's `overlap`).  The buffers they fetch early must be
  // in place before the first of the three launches: the words and the status word may launch a fill on first use.
  const bool overlap = own_projection(cp.dtype, B, dim, 6 * inner, es);
  use.zero_words(B * H);
  status_word(dev.index());
  if (overlap) {
    check(api.token_linear(cp.dtype, (int32_t)B, (int32_t)dim, (int32_t)(6 * inner), xs.data_ptr(), xs.stride(0),
                           l.norm.defined() ? l.norm.data_ptr() : nullptr, norm_eps(l), l.to_qkv.data_ptr(), packed, 0, stream.stream()),
          "castle_token_linear");
  } else {
    Tensor h = aligned_contiguous(xs).view({B, dim});
    if (l.norm.defined()) {
      const Tensor src = h;
      h = at::empty({B, dim}, x.options().requires_grad(false));
      check(api.rmsnorm_fwd(cp.dtype, B, (int32_t)dim, src.data_ptr(), l.norm.data_ptr(), norm_eps(l), h.data_ptr(), nullptr, stream.stream()),
            "castle_rmsnorm_fwd");
    }
    keep = at::mm(h, l.to_qkv.t());
    packed = static_cast<char*>(keep.data_ptr());
  }
  castle_tensor_t news[6];
  for (int i = 0; i < 6; ++i) news[i] = {packed + kPackedOrder[i] * inner * es, 6 * inner, d, 6 * inner};
  if (own_projection(cp.dtype, B, inner, l.combine.size(0), es)) {
    launch_decode(cp, news, caches, core, t, rotary, overlap, ws.data_ptr(), part, stream, use);
    Tensor y = at::empty({B, 1, l.combine.size(0)}, x.options().requires_grad(false));
    check(api.token_linear(cp.dtype, (int32_t)B, (int32_t)inner, (int32_t)l.combine.size(0), core, inner, nullptr, 0.f,
                           l.combine.data_ptr(), y.data_ptr(), 1, stream.stream()), "castle_token_linear");
    return y;
  }
  const Tensor o = at::empty({B, inner}, x.options().requires_grad(false));
  launch_decode(cp, news, caches, o.data_ptr(), t, rotary, overlap, ws.data_ptr(), part, stream, use);
  return at::mm(o, l.combine.t()).view({B, 1, l.combine.size(0)});
}

Tensor layer_decode(const Tensor& x, const Layer& l, const Tensor* caches, int64_t t, double scale, const Rotary& rotary) {
  // no gradient flows through the cached step, so only the last projection could need a graph
  if (plain_layer(x, l) && x.size(1) == 1 && !(at::GradMode::is_enabled() && l.combine.requires_grad()))
    return token_layer(x, l, caches, t, scale, rotary);
  return at::linear(decode_packed(project(x, l), caches, t, scale, rotary), l.combine);
}

// ------------------------------------------------------------------------------------------------ Python
template <typename F>
PyObject* guarded(F&& f) {   // C++ exceptions become Python ones; `f` runs without the interpreter lock where it says so
  try {
    return f();
  } catch (const AssertError& e) {
    PyErr_SetString(PyExc_AssertionError, e.what());
  } catch (const std::exception&) {   // as torch's own bindings do: a Python exception of a hook, OutOfMemoryError and so on
    torch::translate_exception_to_python(std::current_exception());
  }
  return nullptr;
}
struct Unlocked {   // releases the interpreter lock for its lifetime
  PyThreadState* s = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(s); }
};

const Tensor& arg_tensor(PyObject* o) {
  if (!THPVariable_Check(o)) throw std::runtime_error("castle: a tensor expected");
  return THPVariable_Unpack(o);
}
Tensor arg_optional(PyObject* o) { return o == Py_None ? Tensor() : arg_tensor(o); }
int64_t arg_int(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); throw std::runtime_error("castle: an integer expected"); }
  return v;
}
double arg_float(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); throw std::runtime_error("castle: a number expected"); }
  return v;
}
std::vector<Tensor> arg_caches(PyObject* o) {
  std::vector<Tensor> v;
  if (o == Py_None) return v;
  PyObject* fast = PySequence_Fast(o, "castle: four cache tensors expected");
  if (!fast) { PyErr_Clear(); throw std::runtime_error("castle: four cache tensors expected"); }
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(fast); ++i) {
    PyObject* item = PySequence_Fast_GET_ITEM(fast, i);
    if (!THPVariable_Check(item)) { Py_DECREF(fast); throw std::runtime_error("castle: four cache tensors expected"); }
    v.push_back(THPVariable_Unpack(item));
  }
  Py_DECREF(fast);
  if (v.size() != 4) throw std::runtime_error("castle: four cache tensors expected");
  return v;
}
void arg_count(Py_ssize_t n, Py_ssize_t want) {
  if (n != want) throw std::runtime_error("castle: wrong number of arguments");
}

// The operators' rule for caches: the kernels store their 16-bit operand tiles.
void check_cache_out(const Options& o, at::IntArrayRef bhnd, at::ScalarType dtype, const at::Device& dev) {
  if (o.caches.empty()) return;
  const bool fills = (dtype == at::kHalf || (dtype == at::kBFloat16 && bhnd[2] < o.long_seq)) && (bhnd[3] == 64 || bhnd[3] == 128);
  need(o.return_U && fills, "castle_attention: cache_out needs return_U, a 16-bit dtype and dim_head 64 or 128");
  for (const auto& c : o.caches)
    need(c.sizes() == bhnd && c.scalar_type() == dtype && c.stride(3) == 1 && c.device() == dev,
         "castle_attention: cache_out tensors must be (B, H, N, d) views in the input dtype, on the inputs' device");
}

// t[:, :, :rows] without the dispatcher (a token makes four of these; caches are no part of any graph).
Tensor first_rows(const Tensor& t, int64_t rows) {
  if (t.dim() != 4 || rows < 0 || rows > t.size(2) || t.requires_grad()) return t.narrow(2, 0, rows);
  Tensor v = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(t.storage()), t.key_set(), t.dtype());
  c10::TensorImpl* impl = v.unsafeGetTensorImpl();
  impl->set_storage_offset(t.storage_offset());
  impl->set_sizes_and_strides(std::array<int64_t, 4>{t.size(0), t.size(1), rows, t.size(3)}, t.strides());
  return v;
}

PyObject* wrap_result(Result r, bool with_U) {
  PyObject* out = THPVariable_Wrap(r.out);
  if (!with_U || !out) return out;
  PyObject* u = THPVariable_Wrap(r.U);
  if (!u) { Py_DECREF(out); return nullptr; }
  PyObject* t = PyTuple_Pack(2, out, u);
  Py_DECREF(out);
  Py_DECREF(u);
  return t;
}

// attention(qc, kc, vc, qu, ku, vu, scale, return_U, cache_out, limit, long_seq)
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    arg_count(n, 11);
    Tensor v[6];
    for (int i = 0; i < 6; ++i) v[i] = arg_tensor(a[i]);
    Options o;
    o.scale = arg_float(a[6]);
    o.return_U = PyObject_IsTrue(a[7]) == 1;
    o.caches = arg_caches(a[8]);
    o.limit = arg_int(a[9]);
    o.long_seq = arg_int(a[10]);
    Result r;
    {
      Unlocked u;
      if (v[0].dim() == 4) check_cache_out(o, v[0].sizes(), v[0].scalar_type(), v[0].device());
      r = attention_six(v, o);
    }
    return wrap_result(std::move(r), o.return_U);
  });
}

// attention_packed(packed, scale, return_U, cache_out, limit, long_seq, rotary freqs or None, strict): `strict` = the
// operator's rule for cache_out; the module's own caches may have any type and width
PyObject* py_attention_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    arg_count(n, 8);
    const Tensor packed = arg_tensor(a[0]);
    Options o;
    o.scale = arg_float(a[1]);
    o.return_U = PyObject_IsTrue(a[2]) == 1;
    o.caches = arg_caches(a[3]);
    o.limit = arg_int(a[4]);
    o.long_seq = arg_int(a[5]);
    o.rotary.freqs = arg_optional(a[6]);
    const bool strict = PyObject_IsTrue(a[7]) == 1;
    Result r;
    {
      Unlocked u;
      if (strict && packed.dim() == 5)
        check_cache_out(o, {packed.size(0), packed.size(3), packed.size(1), packed.size(4)}, packed.scalar_type(), packed.device());
      r = attention_packed(packed, o);
    }
    return wrap_result(std::move(r), o.return_U);
  });
}

// decode_step(qc, kc, vc, qu, ku, vu, U, qu_cache, kc_cache, vc_cache, cache_len, scale)
PyObject* py_decode_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    arg_count(n, 12);
    Tensor v[10], out;
    for (int i = 0; i < 10; ++i) v[i] = arg_tensor(a[i]);
    const int64_t t = arg_int(a[10]);
    const double scale = arg_float(a[11]);
    {
      Unlocked u;
      out = decode_step(v, v + 6, t, scale);
    }
    return THPVariable_Wrap(out);
  });
}

Layer arg_layer(PyObject* const* a) {   // norm weight or None, eps or None, to_all_qkv weight, combine_heads weight, heads, dim_head
  Layer l;
  l.norm = arg_optional(a[0]);
  if (a[1] != Py_None) l.eps = arg_float(a[1]);
  l.to_qkv = arg_tensor(a[2]);
  l.combine = arg_tensor(a[3]);
  l.heads = arg_int(a[4]);
  l.dim_head = arg_int(a[5]);
  return l;
}

// Whether something records torch operations or may replace torch functions, so that the layer's have to be called from
// Python: jit tracing, a tensor class of its own, or a torch function mode (but a default device).
PyObject* device_context = nullptr;   // torch's class of the modes that set one
bool watched(PyObject* const* a) {   // (x, <layer: 6>, ...)
  if (torch::jit::tracer::isTracing()) return true;
  for (int i : {0, 1, 3, 4})
    if (a[i] != Py_None && !THPVariable_CheckExact(a[i])) return true;
  for (int64_t i = 0; i < at::impl::PythonTorchFunctionTLS::stack_len(); ++i)
    if (reinterpret_cast<PyObject*>(Py_TYPE(at::impl::PythonTorchFunctionTLS::get_stack_at(i)->ptr(getPyInterpreter()))) != device_context) return true;
  return false;
}

// layer_forward(x, <layer: 6>, scale, rotary freqs or None, caches or None, limit, long_seq); None where it is watched()
PyObject* py_layer_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arg_count(n, 12);
    if (watched(a)) Py_RETURN_NONE;
    const Tensor x = arg_tensor(a[0]);
    const Layer l = arg_layer(a + 1);
    Options o;
    o.scale = arg_float(a[7]);
    o.rotary.freqs = arg_optional(a[8]);
    o.caches = arg_caches(a[9]);
    o.limit = arg_int(a[10]);
    o.long_seq = arg_int(a[11]);
    Tensor out;
    {
      Unlocked u;
      out = layer_forward(x, l, o);
    }
    return THPVariable_Wrap(out);
  });
}

// layer_decode(x, <layer: 6>, scale, rotary freqs or None, caches, cache_len); None where it is watched()
PyObject* py_layer_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arg_count(n, 11);
    if (watched(a)) Py_RETURN_NONE;
    const Tensor x = arg_tensor(a[0]);
    const Layer l = arg_layer(a + 1);
    const double scale = arg_float(a[7]);
    Rotary rotary;
    rotary.freqs = arg_optional(a[8]);
    const std::vector<Tensor> caches = arg_caches(a[9]);
    if (caches.size() != 4) throw std::runtime_error("castle: four cache tensors expected");
    const int64_t t = rotary.position0 = arg_int(a[10]);
    Tensor out;
    {
      Unlocked u;
      out = layer_decode(x, l, caches.data(), t, scale, rotary);
    }
    return THPVariable_Wrap(out);
  });
}

// decode_packed(packed, scale, rotary freqs or None, caches, cache_len)
PyObject* py_decode_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    arg_count(n, 5);
    const Tensor packed = arg_tensor(a[0]);
    const double scale = arg_float(a[1]);
    Rotary rotary;
    rotary.freqs = arg_optional(a[2]);
    const std::vector<Tensor> caches = arg_caches(a[3]);
    if (caches.size() != 4) throw std::runtime_error("castle: four cache tensors expected");
    const int64_t t = rotary.position0 = arg_int(a[4]);
    Tensor out;
    {
      Unlocked u;
      out = decode_packed(packed, caches.data(), t, scale, rotary);
    }
    return THPVariable_Wrap(out);
  });
}

// forward_chunks(B, H, bytes per pair, limit): the rectangles of a forward's launches as (b0, b1, h0, h1)
PyObject* py_forward_chunks(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arg_count(n, 4);
    std::vector<std::array<int64_t, 4>> r;
    for_chunks(arg_int(a[0]), arg_int(a[1]), arg_int(a[2]), arg_int(a[3]),
               [&](int64_t b0, int64_t b1, int64_t h0, int64_t h1) { r.push_back({b0, b1, h0, h1}); });
    PyObject* list = PyList_New((Py_ssize_t)r.size());
    for (size_t i = 0; i < r.size(); ++i)
      PyList_SET_ITEM(list, (Py_ssize_t)i, Py_BuildValue("(LLLL)", (long long)r[i][0], (long long)r[i][1], (long long)r[i][2], (long long)r[i][3]));
    return list;
  });
}

// first_rows(buffers, n): the buffers' [:, :, :n] views as a tuple
PyObject* py_first_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arg_count(n, 2);
    const std::vector<Tensor> bufs = arg_caches(a[0]);
    const int64_t rows = arg_int(a[1]);
    PyObject* t = PyTuple_New((Py_ssize_t)bufs.size());
    for (size_t i = 0; i < bufs.size(); ++i) PyTuple_SET_ITEM(t, (Py_ssize_t)i, THPVariable_Wrap(first_rows(bufs[i], rows)));
    return t;
  });
}

// new_caches(like, B, H, capacity, d): four buffers of like's type and device (one by one from Python they cost 8 us of a prompt)
PyObject* py_new_caches(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arg_count(n, 5);
    const at::TensorOptions o = arg_tensor(a[0]).options().requires_grad(false).memory_format(c10::nullopt);
    const std::array<int64_t, 4> sizes{arg_int(a[1]), arg_int(a[2]), arg_int(a[3]), arg_int(a[4])};
    PyObject* list = PyList_New(4);
    for (Py_ssize_t i = 0; list && i < 4; ++i) {
      PyObject* t = nullptr;
      try {
        t = THPVariable_Wrap(at::empty(sizes, o));
      } catch (...) {
        Py_DECREF(list);
        throw;
      }
      PyList_SET_ITEM(list, i, t);
    }
    return list;
  });
}

PyObject* py_status_word(PyObject*, PyObject* device) {
  return guarded([&] {
    const int64_t index = arg_int(device);
    Tensor t;
    {
      Unlocked u;
      t = status_word((int)index);
    }
    return THPVariable_Wrap(t);
  });
}
PyObject* py_status_devices(PyObject*, PyObject*) {
  std::vector<int> devices;
  {
    Unlocked u;
    std::lock_guard<std::mutex> lock(state_mutex);
    for (const auto& kv : status_words) devices.push_back(kv.first);
  }
  PyObject* list = PyList_New(0);
  for (int d : devices) {
    PyObject* i = PyLong_FromLong(d);
    PyList_Append(list, i);
    Py_DECREF(i);
  }
  return list;
}
PyObject* py_release_workspaces(PyObject*, PyObject*) {
  std::map<std::pair<int, void*>, std::shared_ptr<StreamState>> old;
  {
    Unlocked u;
    std::lock_guard<std::mutex> lock(state_mutex);
    old.swap(stream_states);
  }
  Py_RETURN_NONE;
}

// bind({name: address}): the C ABI's entry points
PyObject* py_bind(PyObject*, PyObject* d) {
  return guarded([&]() -> PyObject* {
    auto get = [&](const char* name) {
      PyObject* v = PyDict_GetItemString(d, name);
      if (!v) throw std::runtime_error(std::string("castle: no address for ") + name);
      return PyLong_AsVoidPtr(v);
    };
#define CASTLE_BIND(f) api.f = reinterpret_cast<decltype(api.f)>(get("castle_" #f))
    CASTLE_BIND(last_error); CASTLE_BIND(fwd_workspace_bytes); CASTLE_BIND(fwd); CASTLE_BIND(fwd_prefill);
    CASTLE_BIND(rmsnorm_fwd); CASTLE_BIND(rmsnorm_bwd_workspace_bytes); CASTLE_BIND(rmsnorm_bwd); CASTLE_BIND(bwd_workspace_bytes); CASTLE_BIND(bwd); CASTLE_BIND(transform); CASTLE_BIND(amax_scale);
    CASTLE_BIND(decode_workspace_bytes); CASTLE_BIND(decode_step_fused); CASTLE_BIND(token_linear_fits); CASTLE_BIND(token_linear);
    CASTLE_BIND(linear); CASTLE_BIND(token_layer_fits); CASTLE_BIND(token_layer_workspace_bytes); CASTLE_BIND(token_layer);
#undef CASTLE_BIND
    PyObject* module = PyImport_ImportModule("torch.utils._device");
    Py_XDECREF(device_context);
    device_context = module ? PyObject_GetAttrString(module, "DeviceContext") : nullptr;
    Py_XDECREF(module);
    if (!device_context) return nullptr;
    Py_RETURN_NONE;
  });
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL
PyMethodDef methods[] = {{"bind", py_bind, METH_O, nullptr},
                         {"attention", FAST(py_attention), nullptr},
                         {"attention_packed", FAST(py_attention_packed), nullptr},
                         {"decode_step", FAST(py_decode_step), nullptr},
                         {"layer_forward", FAST(py_layer_forward), nullptr},
                         {"layer_decode", FAST(py_layer_decode), nullptr},
                         {"decode_packed", FAST(py_decode_packed), nullptr},
                         {"forward_chunks", FAST(py_forward_chunks), nullptr},
                         {"first_rows", FAST(py_first_rows), nullptr},
                         {"new_caches", FAST(py_new_caches), nullptr},
                         {"status_word", py_status_word, METH_O, nullptr},
                         {"status_devices", py_status_devices, METH_NOARGS, nullptr},
                         {"release_workspaces", py_release_workspaces, METH_NOARGS, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "Native host path of the operators.", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module_def); }
