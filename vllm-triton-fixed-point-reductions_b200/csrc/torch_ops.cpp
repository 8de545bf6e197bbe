// torch operators over the C ABI: argument checks, output allocation, launch policy and the call,
// without entering the Python interpreter.  A decode step is some forty of these calls, each a
// kernel of 5-50 us; the same steps in Python took 20-30 us per call, longer than the kernels.
//
// `fxpr::*` are the public operators (schemas in fxpr_vllm/_lib.py, CUDA key only, so CPU tensors
// get the dispatcher's NotImplementedError); `fxpr_b200::*` serve the decoder's fused steps.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/Exception.h>
#include <torch/library.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>
#include <vector>

#include "../../include/fxpr_b200.h"
#include "host_policy.h"

namespace {

using at::Tensor;
using std::optional;

// ------------------------------------------------------------------ configuration
// The process-wide knobs come from the environment through fxpr_vllm.config, which pushes them
// here when it loads them; an operator that runs first asks Python for them once.
struct Config {
  std::atomic<int> loaded{0};
  std::atomic<int> frac_bits{16}, gemm_k_tile{0}, gemm_split_k{0};
};
Config g_config;
std::atomic<void (*)()> g_config_loader{nullptr};

const Config& config() {
  if (!g_config.loaded.load(std::memory_order_acquire)) {
    if (auto load = g_config_loader.load()) load();
  }
  return g_config;
}

// Per-thread overrides of the kernel selection (fxpr_vllm._lib.overrides, static_weights).
struct Overrides {
  int gemm_k_tile = -1, gemm_split_k = -1;    // -1: not set
  int gemm_flags = 0, attn_flags = 0;
  bool gemm_portable = false, attn_portable = false, gemm_partials = false;
  Tensor last_partials;
};
thread_local Overrides t_ovr;

// ------------------------------------------------------------------ per-device state
constexpr int kMaxDevices = 64;
struct DeviceState {
  std::mutex mu;
  std::atomic<int32_t*> status_ptr{nullptr};
  std::atomic<int> sms{0};
  Tensor status;                       // int32 the kernels set when a bounded wait gives up
  // Zero-initialised split-K scratch, grown on demand: one buffer for each of the streams that used one last,
  // and one for all graphs.
  struct StreamScratch { cudaStream_t stream; Tensor buffer; };
  std::vector<StreamScratch> scratch;  // most recent use last, at most kScratchStreams
  Tensor graph_scratch;
  std::vector<Tensor> retired;         // replaced graph scratch: graphs captured with it stay valid
};
constexpr size_t kScratchStreams = 16;
// never destroyed: the tensors must not outlive the CUDA context at process exit
DeviceState* const g_dev = new DeviceState[kMaxDevices];

DeviceState& device_state(int dev) {
  TORCH_CHECK(dev >= 0 && dev < kMaxDevices, "fxpr: device index ", dev, " out of range");
  return g_dev[dev];
}

int num_sms(int dev) {
  DeviceState& d = device_state(dev);
  int n = d.sms.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    d.sms.store(n > 0 ? n : 148);
    n = d.sms.load();
  }
  return n;
}

int32_t* status_ptr(int dev) {
  DeviceState& d = device_state(dev);
  int32_t* p = d.status_ptr.load(std::memory_order_acquire);
  if (!p) {
    std::lock_guard<std::mutex> lock(d.mu);
    if (!d.status.defined()) d.status = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, dev));
    p = d.status.data_ptr<int32_t>();
    d.status_ptr.store(p, std::memory_order_release);
  }
  return p;
}

bool capturing() {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(c10::cuda::getCurrentCUDAStream(), &st) == cudaSuccess &&
         st != cudaStreamCaptureStatusNone;
}

// The kernels re-zero the counters they used, so one buffer serves call after call -- of ONE stream: calls that
// overlap would take each other's partial sums and arrivals, so every stream has its own.  A stream's buffer is
// allocated, cleared and used on that stream alone, so the allocator's own ordering makes dropping it safe, and the
// stream not used for longest gives its buffer back.  Graphs share one further buffer, which outlives them
// (graphs that run at the same time must not both split); growing it during a capture would allocate and
// zero-fill inside the graph, so that is refused.
Tensor gemm_scratch(int dev, int64_t bytes) {
  DeviceState& d = device_state(dev);
  const auto cleared = [&] {
    return at::zeros({std::max<int64_t>(bytes, 1 << 20)}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, dev));
  };
  std::lock_guard<std::mutex> lock(d.mu);
  const int64_t for_graphs = d.graph_scratch.defined() ? d.graph_scratch.numel() : 0;
  if (capturing()) {
    TORCH_CHECK(for_graphs >= std::max<int64_t>(bytes, 1), "gemm_fxp: split-K scratch of ", bytes,
                " bytes needed during CUDA-graph capture but only ", for_graphs,
                " are allocated; run the shape once (or warmup_gemm) before capturing");
    return d.graph_scratch;
  }
  if (for_graphs < std::max<int64_t>(bytes, 1)) {
    if (d.graph_scratch.defined()) d.retired.push_back(d.graph_scratch);
    d.graph_scratch = cleared();
  }
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  auto& v = d.scratch;
  auto it = std::find_if(v.begin(), v.end(), [&](const auto& s) { return s.stream == stream; });
  if (it == v.end()) {
    if (v.size() == kScratchStreams) v.erase(v.begin());
    v.push_back({stream, cleared()});
  } else {
    if (it->buffer.numel() < bytes) it->buffer = cleared();
    std::rotate(it, it + 1, v.end());
  }
  return v.back().buffer;
}

// ------------------------------------------------------------------ small helpers
int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return FXPR_F16;
    case at::kBFloat16: return FXPR_BF16;
    case at::kFloat: return FXPR_F32;
    case at::kDouble: return FXPR_F64;
    default: return -1;
  }
}
bool is_io(at::ScalarType t) { return t == at::kFloat || t == at::kHalf || t == at::kBFloat16; }
int int_bits_of(at::ScalarType t) { return t == at::kShort ? 16 : t == at::kInt ? 32 : t == at::kLong ? 64 : 0; }
at::ScalarType int_type(int64_t bits) { return bits == 16 ? at::kShort : bits == 32 ? at::kInt : at::kLong; }

void check_int_bits(int64_t n) { TORCH_CHECK_VALUE(n == 16 || n == 32 || n == 64, "int_bits must be 16/32/64, got ", n); }
void check_frac_bits(int64_t n) { TORCH_CHECK_VALUE(n == 8 || n == 16 || n == 32, "fxp_frac_bits must be 8/16/32, got ", n); }

// A C status as the exception type the same class of error raises everywhere in the package.
void check_status(int st, const char* what) {
  if (st == FXPR_OK) return;
  const char* detail = st == FXPR_ERR_CUDA ? fxpr_last_error() : "";
  const std::string text = std::string(what) + ": " + fxpr_status_string(st) + (detail[0] ? std::string(" [") + detail + "]" : "");
  if (st == FXPR_ERR_BAD_ARG) TORCH_CHECK_VALUE(false, text);
  if (st == FXPR_ERR_UNSUPPORTED) TORCH_CHECK_TYPE(false, text);
  TORCH_CHECK(false, text);
}

Tensor empty_on(at::IntArrayRef sizes, at::ScalarType t, const Tensor& like) {
  return at::detail::empty_cuda(sizes, t, like.device(), std::nullopt);
}
const void* ptr(const optional<Tensor>& t) { return t.has_value() && t->defined() ? t->data_ptr() : nullptr; }

// Device guard and stream of a call.
struct On {
  c10::cuda::CUDAGuard guard;
  int dev;
  explicit On(const Tensor& t) : guard(t.device()), dev(t.device().index()) {}
  void* stream() const { return c10::cuda::getCurrentCUDAStream(dev).stream(); }
};

// ------------------------------------------------------------------ casts
Tensor float_to_fixed(const Tensor& x, int64_t int_bits, int64_t frac_bits) {
  check_int_bits(int_bits);
  check_frac_bits(frac_bits);
  const auto t = x.scalar_type();
  TORCH_CHECK_TYPE(t == at::kHalf || t == at::kFloat || t == at::kDouble, "float_to_fixed: unsupported input dtype ", t,
                   "; expected float16, float32 or float64");
  On on(x);
  const Tensor xc = x.contiguous();
  Tensor y = empty_on(xc.sizes(), int_type(int_bits), xc);
  if (xc.numel())
    check_status(fxpr_float_to_fixed(xc.data_ptr(), dtype_code(t), y.data_ptr(), (int)int_bits, (int)frac_bits, xc.numel(),
                                     on.stream()), "float_to_fixed");
  return y;
}

Tensor fixed_to_float(const Tensor& x, int64_t float_bits, int64_t frac_bits) {
  TORCH_CHECK_VALUE(float_bits == 16 || float_bits == 32 || float_bits == 64, "float_bits must be 16/32/64, got ", float_bits);
  check_frac_bits(frac_bits);
  const int bits = int_bits_of(x.scalar_type());
  TORCH_CHECK_TYPE(bits, "fixed_to_float: unsupported input dtype ", x.scalar_type(), "; expected int16, int32 or int64");
  On on(x);
  const Tensor xc = x.contiguous();
  Tensor y = empty_on(xc.sizes(), float_bits == 16 ? at::kHalf : float_bits == 32 ? at::kFloat : at::kDouble, xc);
  if (xc.numel())
    check_status(fxpr_fixed_to_float(xc.data_ptr(), bits, y.data_ptr(), (int)float_bits, (int)frac_bits, xc.numel(),
                                     on.stream()), "fixed_to_float");
  return y;
}

// ------------------------------------------------------------------ norms
Tensor rms_norm_launch(const Tensor& x, const Tensor& w, const Tensor* residual, double eps) {
  TORCH_CHECK(x.is_cuda() && w.is_cuda(), "rms_norm: x and w must be CUDA");
  TORCH_CHECK_TYPE(is_io(x.scalar_type()), "rms_norm: unsupported input dtype ", x.scalar_type());
  TORCH_CHECK_TYPE(w.scalar_type() == x.scalar_type(), "rms_norm: weight dtype must match input dtype");
  if (residual) {
    TORCH_CHECK(residual->is_cuda(), "rms_norm: residual must be CUDA");
    TORCH_CHECK_TYPE(residual->scalar_type() == x.scalar_type(), "rms_norm: residual dtype must match input dtype");
    TORCH_CHECK_VALUE(residual->sizes() == x.sizes(), "rms_norm: residual shape must match x");
  }
  On on(x);
  const int64_t hidden = x.size(-1);
  const Tensor xc = x.contiguous();
  Tensor y = empty_on(xc.sizes(), xc.scalar_type(), xc);
  const int64_t rows = hidden ? xc.numel() / hidden : 0;
  if (rows == 0) return y;
  Tensor rc;
  if (residual) rc = residual->contiguous();
  const Tensor wc = w.contiguous();
  check_status(fxpr_rms_norm(xc.data_ptr(), residual ? rc.data_ptr() : nullptr, wc.data_ptr(), y.data_ptr(),
                             dtype_code(xc.scalar_type()), rows, hidden, (float)eps, config().frac_bits, on.stream()), "rms_norm");
  if (residual && rc.data_ptr() != residual->data_ptr()) residual->copy_(rc);
  return y;
}

Tensor rms_norm_fxp(const Tensor& x, const Tensor& w, double eps) { return rms_norm_launch(x, w, nullptr, eps); }

Tensor rms_norm_fxp_residual(const Tensor& x, const Tensor& residual, const Tensor& w, double eps) {
  return rms_norm_launch(x, w, &residual, eps);
}

Tensor gemm_fxp_epilogue_any(const Tensor& c_int, const optional<Tensor>& bias, at::ScalarType out_dtype, int64_t frac_bits) {
  const int bits = int_bits_of(c_int.scalar_type());
  TORCH_CHECK_TYPE(bits, "gemm_fxp_epilogue: c_int must be an integer tensor, got ", c_int.scalar_type());
  TORCH_CHECK_TYPE(is_io(out_dtype), "gemm_fxp_epilogue: unsupported output dtype ", out_dtype);
  TORCH_CHECK_VALUE(c_int.dim() == 2, "gemm_fxp_epilogue: c_int must be [M, N]");
  On on(c_int);
  const Tensor cc = c_int.contiguous();
  const int64_t M = cc.size(0), N = cc.size(1);
  Tensor c = empty_on({M, N}, out_dtype, cc);
  if (M == 0 || N == 0) return c;
  optional<Tensor> b = bias;
  if (b.has_value() && b->defined() && b->scalar_type() != out_dtype) b = b->to(out_dtype);
  check_status(fxpr_gemm_epilogue_from_int(cc.data_ptr(), bits, ptr(b), c.data_ptr(), dtype_code(out_dtype), M, N, N,
                                           (int)frac_bits, on.stream()), "gemm_fxp_epilogue");
  return c;
}

Tensor gemm_fxp_epilogue(const Tensor& c_int, const optional<Tensor>& bias, at::ScalarType out_dtype, int64_t frac_bits) {
  check_frac_bits(frac_bits);
  return gemm_fxp_epilogue_any(c_int, bias, out_dtype, frac_bits);
}

// Integer accumulators of a row-parallel GEMM (after the cross-rank integer sum) -> GEMM epilogue +
// residual add + RMSNorm in one kernel; same bits as the separate ones.
Tensor rms_norm_fxp_from_int(const Tensor& acc, const Tensor& residual, const Tensor& w, const optional<Tensor>& bias,
                             double eps, int64_t gemm_frac_bits) {
  const int bits = int_bits_of(acc.scalar_type());
  const auto t = residual.scalar_type();
  TORCH_CHECK_TYPE(bits, "rms_norm_fxp_from_int: acc must be an integer tensor, got ", acc.scalar_type());
  TORCH_CHECK(acc.is_cuda() && residual.is_cuda() && w.is_cuda(), "rms_norm_fxp_from_int: tensors must be CUDA");
  TORCH_CHECK_TYPE(is_io(t) && w.scalar_type() == t, "rms_norm_fxp_from_int: residual and weight must share one io dtype");
  TORCH_CHECK_VALUE(acc.sizes() == residual.sizes() && acc.is_contiguous() && residual.is_contiguous(),
                    "rms_norm_fxp_from_int: acc and residual must be contiguous and of one shape");
  On on(acc);
  const int64_t hidden = residual.size(-1), rows = hidden ? residual.numel() / hidden : 0;
  if (rows == 0) return empty_on(residual.sizes(), t, residual);
  if (hidden * 4 > 64 * 1024) {                       // a row that the fused kernel cannot park in shared memory
    const Tensor x = gemm_fxp_epilogue_any(acc.view({rows, hidden}), bias, t, gemm_frac_bits);
    return rms_norm_launch(x.view(residual.sizes()), w, &residual, eps);
  }
  Tensor y = empty_on(residual.sizes(), t, residual);
  optional<Tensor> b;
  if (bias.has_value() && bias->defined()) b = bias->to(t).contiguous();
  const Tensor wc = w.contiguous();
  check_status(fxpr_rms_norm_from_int(acc.data_ptr(), bits, ptr(b), residual.data_ptr(), wc.data_ptr(), y.data_ptr(),
                                      dtype_code(t), rows, hidden, (float)eps, (int)gemm_frac_bits, config().frac_bits,
                                      on.stream()), "rms_norm_fxp_from_int");
  return y;
}

// ------------------------------------------------------------------ log-softmax
Tensor log_softmax_fxp(const Tensor& x, int64_t frac_bits) {
  check_frac_bits(frac_bits);
  TORCH_CHECK_TYPE(is_io(x.scalar_type()), "log_softmax_fxp: unsupported input dtype ", x.scalar_type());
  On on(x);
  const Tensor xc = x.contiguous();
  const int64_t cols = xc.dim() ? xc.size(-1) : 1;
  Tensor y = empty_on(xc.sizes(), at::kFloat, xc);
  if (xc.numel())
    check_status(fxpr_log_softmax(xc.data_ptr(), dtype_code(xc.scalar_type()), y.data_ptr<float>(), xc.numel() / cols, cols,
                                  (int)frac_bits, on.stream()), "log_softmax_fxp");
  return y;
}

// ------------------------------------------------------------------ GEMM
struct GemmWants {
  bool c = true, c_int = false, silu_pairs = false, argmax = false;
  int64_t n_offset = 0;
};
struct GemmOut {
  Tensor c, c_int, keys;
  bool unsupported = false;             // the fused form does not take this shape: nothing was launched
};

GemmOut gemm_common(const Tensor& a, const Tensor& b, const optional<Tensor>& bias_in, int64_t int_bits, int64_t frac_bits,
                    const GemmWants& want, const Tensor* out_int = nullptr) {
  TORCH_CHECK_VALUE(a.dim() == 2 && b.dim() == 2, "gemm_fxp: a and b must be matrices");
  const auto t = a.scalar_type();
  const int64_t M = a.size(0), K = a.size(1), N = b.size(1);
  On on(a);
  GemmOut r;
  if (want.c) r.c = empty_on({M, want.silu_pairs ? N / 2 : N}, t, a);
  if (out_int) {
    TORCH_CHECK_VALUE(out_int->dim() == 2 && out_int->size(0) == M && out_int->size(1) == N &&
                          out_int->scalar_type() == int_type(int_bits) && out_int->is_contiguous() &&
                          out_int->device() == a.device(),
                      "gemm_fxp_int_into: out must be a contiguous [M, N] tensor of the accumulator type");
    r.c_int = *out_int;
  } else if (want.c_int) {
    r.c_int = empty_on({M, N}, int_type(int_bits), a);
  }
  if (want.argmax) r.keys = (M == 0 || N == 0) ? at::zeros({M}, a.options().dtype(at::kLong)) : empty_on({M}, at::kLong, a);
  if (M == 0 || N == 0) return r;
  TORCH_CHECK_TYPE(is_io(t) && b.scalar_type() == t, "gemm_fxp: unsupported dtypes ", t, " x ", b.scalar_type());
  TORCH_CHECK(b.is_cuda(), "gemm_fxp: tensors must be CUDA");
  TORCH_CHECK_VALUE(b.size(0) >= K, "gemm_fxp: b has ", b.size(0), " rows, a has ", K, " columns");

  const Overrides& o = t_ovr;
  const Config& cfg = config();
  int k_tile = o.gemm_k_tile >= 0 ? o.gemm_k_tile : cfg.gemm_k_tile.load();
  if (k_tile <= 0) k_tile = fxpr::default_k_tile(t == at::kFloat);
  const int64_t k_tiles = fxpr::ceil_div(K, k_tile);
  int flags = (o.gemm_portable ? FXPR_GEMM_FORCE_PORTABLE : 0) | o.gemm_flags | (want.silu_pairs ? FXPR_GEMM_SILU_MUL : 0);
  optional<Tensor> bias = bias_in;
  if (bias.has_value() && bias->defined() && bias->scalar_type() != t) bias = bias->to(t);

  if (want.argmax) {
    const int st = fxpr_gemm_argmax(a.data_ptr(), b.data_ptr(), ptr(bias), r.c.data_ptr(), (uint64_t*)r.keys.data_ptr(),
                                    want.n_offset, dtype_code(t), M, N, K, a.stride(0), a.stride(1), b.stride(0), b.stride(1),
                                    N, (int)int_bits, (int)frac_bits, k_tile, flags, status_ptr(on.dev), on.stream());
    if (st == FXPR_ERR_UNSUPPORTED) { r.unsupported = true; return r; }
    check_status(st, "gemm_fxp_argmax");
    return r;
  }

  int split = o.gemm_split_k >= 0 ? o.gemm_split_k : cfg.gemm_split_k.load();
  if (split <= 0)
    split = fxpr::pick_gemm_split_k(M, N, K, k_tile, (int)int_bits, num_sms(on.dev), fxpr::wide_kernels((int)frac_bits, flags));
  split = (int)std::max<int64_t>(1, std::min<int64_t>(split, std::max<int64_t>(1, k_tiles)));
  Tensor partials, scratch;
  if (o.gemm_partials && split == 1) {
    partials = at::zeros({k_tiles, M, N}, a.options().dtype(at::kFloat));
    t_ovr.last_partials = partials;
  }
  const auto call = [&](int64_t scratch_bytes) {
    return fxpr_gemm(a.data_ptr(), b.data_ptr(), ptr(bias), r.c.defined() ? r.c.data_ptr() : nullptr,
                     r.c_int.defined() ? r.c_int.data_ptr() : nullptr, dtype_code(t), M, N, K, a.stride(0), a.stride(1),
                     b.stride(0), b.stride(1), r.c.defined() ? r.c.stride(0) : N, (int)int_bits, (int)frac_bits, k_tile,
                     split, flags, scratch.defined() ? scratch.data_ptr() : nullptr, scratch_bytes,
                     partials.defined() && partials.numel() ? partials.data_ptr<float>() : nullptr, status_ptr(on.dev),
                     on.stream());
  };
  // Most splits are merged without scratch, and the library says, before it does anything, where they are not.
  int st = call(0);
  if (st == FXPR_ERR_SCRATCH) {
    const int64_t bytes = fxpr_gemm_scratch_bytes(M, N, (int)int_bits, split);
    scratch = gemm_scratch(on.dev, bytes);
    st = call(bytes);
  }
  if (want.silu_pairs && st == FXPR_ERR_UNSUPPORTED) { r.unsupported = true; return r; }
  check_status(st, "gemm_fxp");
  return r;
}

Tensor gemm_any(const Tensor& a, const Tensor& b, const optional<Tensor>& bias, int64_t int_bits, int64_t frac_bits) {
  return gemm_common(a, b, bias, int_bits, frac_bits, GemmWants{}).c;
}

Tensor gemm_fxp(const Tensor& a, const Tensor& b, const optional<Tensor>& bias, int64_t int_bits, int64_t frac_bits) {
  check_int_bits(int_bits);
  check_frac_bits(frac_bits);
  return gemm_any(a, b, bias, int_bits, frac_bits);
}

Tensor gemm_fxp_int(const Tensor& a, const Tensor& b, int64_t int_bits, int64_t frac_bits) {
  check_int_bits(int_bits);
  check_frac_bits(frac_bits);
  GemmWants w;
  w.c = false;
  w.c_int = true;
  return gemm_common(a, b, std::nullopt, int_bits, frac_bits, w).c_int;
}

void gemm_fxp_int_into(const Tensor& a, const Tensor& b, const Tensor& out, int64_t int_bits, int64_t frac_bits) {
  GemmWants w;
  w.c = false;
  gemm_common(a, b, std::nullopt, int_bits, frac_bits, w, &out);
}

// ------------------------------------------------------------------ decoder-layer steps
Tensor silu_mul(const Tensor& gate_up, bool pairs) {
  TORCH_CHECK_TYPE(is_io(gate_up.scalar_type()) && gate_up.dim() == 2 && gate_up.size(1) % 2 == 0,
                   "silu_mul: [rows, 2f] tensor of an io dtype expected");
  On on(gate_up);
  const Tensor g = gate_up.contiguous();
  const int64_t rows = g.size(0), f = g.size(1) / 2;
  Tensor out = empty_on({rows, f}, g.scalar_type(), g);
  if (rows && f) {
    auto fn = pairs ? fxpr_silu_mul_pairs : fxpr_silu_mul;
    check_status(fn(g.data_ptr(), dtype_code(g.scalar_type()), out.data_ptr(), rows, f, on.stream()), "silu_mul");
  }
  return out;
}

// At most 64 rows: the decode-shape GEMM combines the column pairs in its epilogue; otherwise the
// GEMM and the element-wise kernel run one after the other.  Same bits.
Tensor gemm_silu_mul(const Tensor& a, const Tensor& b_pairs, int64_t int_bits, int64_t frac_bits) {
  TORCH_CHECK_VALUE(b_pairs.dim() == 2 && b_pairs.size(1) % 2 == 0, "gemm_silu_mul: the weight needs an even number of columns");
  if (a.size(0) <= 64) {
    GemmWants w;
    w.silu_pairs = true;
    GemmOut r = gemm_common(a, b_pairs, std::nullopt, int_bits, frac_bits, w);
    if (!r.unsupported) return r.c;
  }
  return silu_mul(gemm_any(a, b_pairs, std::nullopt, int_bits, frac_bits), true);
}

// (logits, keys), or (logits, empty) when the fused kernel does not take the shape and the caller
// has to form the keys from the logits.
std::tuple<Tensor, Tensor> gemm_argmax(const Tensor& a, const Tensor& b, const optional<Tensor>& bias, int64_t int_bits,
                                       int64_t frac_bits, int64_t n_offset) {
  const auto t = a.scalar_type();
  if (a.size(0) <= 64 && (t == at::kHalf || t == at::kBFloat16) && b.scalar_type() == t) {
    GemmWants w;
    w.argmax = true;
    w.n_offset = n_offset;
    GemmOut r = gemm_common(a, b, bias, int_bits, frac_bits, w);
    if (!r.unsupported) return {r.c, r.keys};
  }
  return {gemm_any(a, b, bias, int_bits, frac_bits), at::empty({0}, a.options().dtype(at::kLong))};
}

// Split qkv [T, (q_heads + 2 kv_heads) * d], rotate Q and K, return Q [T, q_heads, d] and write K, V
// into the paged cache (num_blocks, 2, page, kv_heads, d).
Tensor rope_kv_write(const Tensor& qkv, const Tensor& cos, const Tensor& sin, const Tensor& positions, const Tensor& seq_ids,
                     const Tensor& block_table, const Tensor& kv_cache, int64_t q_heads, int64_t kv_heads) {
  TORCH_CHECK_VALUE(qkv.dim() == 2 && kv_cache.dim() == 5, "rope_kv_write: qkv [T, cols], kv_cache of five dimensions");
  On on(qkv);
  const int64_t T = qkv.size(0), d = kv_cache.size(-1);
  Tensor q = empty_on({T, q_heads, d}, qkv.scalar_type(), qkv);
  if (T == 0) return q;
  TORCH_CHECK_TYPE(qkv.is_contiguous() && cos.scalar_type() == at::kFloat && sin.scalar_type() == at::kFloat &&
                       positions.scalar_type() == at::kLong && seq_ids.scalar_type() == at::kLong &&
                       block_table.scalar_type() == at::kInt && kv_cache.scalar_type() == qkv.scalar_type(),
                   "rope_kv_write: contiguous qkv, fp32 tables, int64 positions / ids, int32 block table");
  check_status(fxpr_rope_kv_write(qkv.data_ptr(), dtype_code(qkv.scalar_type()), cos.data_ptr<float>(), sin.data_ptr<float>(),
                                  positions.data_ptr<int64_t>(), seq_ids.data_ptr<int64_t>(), block_table.data_ptr<int32_t>(),
                                  block_table.stride(0), q.data_ptr(), kv_cache.data_ptr(), T, (int)q_heads, (int)kv_heads, (int)d,
                                  (int)kv_cache.size(2), kv_cache.stride(0), kv_cache.stride(1), kv_cache.stride(2),
                                  kv_cache.stride(3), on.stream()), "rope_kv_write");
  return q;
}

// ------------------------------------------------------------------ attention
void unified_attention_fxp(const Tensor& q, const Tensor& kv, const Tensor& o, const Tensor& query_start_loc,
                           const Tensor& seq_lens, const Tensor& block_table_in, int64_t max_query_len,
                           const optional<Tensor>& alibi_slopes, bool is_causal, optional<double> softmax_scale,
                           int64_t int_bits, int64_t frac_bits, double logit_softcap, int64_t window_size,
                           int64_t num_kv_splits) {
  check_int_bits(int_bits);
  check_frac_bits(frac_bits);
  TORCH_CHECK(q.is_cuda() && kv.is_cuda() && o.is_cuda(), "unified_attention_fxp: tensors must be CUDA");
  const auto t = q.scalar_type();
  TORCH_CHECK_TYPE(is_io(t), "unified_attention_fxp: unsupported q dtype ", t);
  TORCH_CHECK_VALUE(kv.dim() == 5 && kv.size(1) == 2, "kv_cache must be (num_blocks, 2, page_size, num_kv_heads, head_dim)");
  TORCH_CHECK_TYPE(kv.scalar_type() == t && o.scalar_type() == t, "kv_cache and o must share dtype with q");
  TORCH_CHECK_TYPE(query_start_loc.scalar_type() == at::kInt, "query_start_loc must be int32");
  TORCH_CHECK_TYPE(seq_lens.scalar_type() == at::kInt, "seq_lens must be int32");
  TORCH_CHECK_TYPE(block_table_in.scalar_type() == at::kInt, "block_table must be int32");
  TORCH_CHECK_VALUE(num_kv_splits >= 0, "num_kv_splits must be >= 0, got ", num_kv_splits);
  const bool has_alibi = alibi_slopes.has_value() && alibi_slopes->defined() && alibi_slopes->numel() > 0;
  TORCH_CHECK_TYPE(!has_alibi || alibi_slopes->scalar_type() == at::kFloat, "alibi_slopes must be float32");
  TORCH_CHECK_VALUE(q.dim() == 3 && o.dim() == 3, "q and o must be [tokens, heads, head_dim]");

  const int64_t tokens = q.size(0), num_heads = q.size(1), head_dim = q.size(2);
  const int64_t page = kv.size(2), num_kv_heads = kv.size(3), num_requests = seq_lens.size(0);
  TORCH_CHECK_VALUE(num_kv_heads > 0 && num_heads % num_kv_heads == 0, "num_heads must be divisible by num_kv_heads");
  if (num_requests == 0 || tokens == 0) return;
  TORCH_CHECK_VALUE(q.stride(2) == 1 && o.stride(2) == 1 && kv.stride(4) == 1,
                    "unified_attention_fxp: head_dim must be the unit-stride dimension");
  On on(q);
  const double ss = softmax_scale.has_value() ? *softmax_scale : 1.0 / std::sqrt((double)head_dim);
  const bool table2d = block_table_in.dim() == 2;
  const int64_t max_keys = std::max<int64_t>(1, (table2d ? block_table_in.size(1) : 0) * page);
  const char* k_base = (const char*)kv.data_ptr();
  const char* v_base = k_base + kv.stride(1) * kv.element_size();
  const bool tc = !t_ovr.attn_portable && !(t_ovr.attn_flags & FXPR_ATTN_FORCE_PORTABLE) &&
                  fxpr::attention_tensor_core_route({t == at::kHalf || t == at::kBFloat16, head_dim, page, num_heads, num_kv_heads,
                                                     num_requests, q.stride(0), q.stride(1), kv.stride(0), kv.stride(2),
                                                     kv.stride(3), q.data_ptr(), k_base, v_base});
  int64_t splits;
  if (tc) {
    splits = fxpr::pick_attention_ranks(num_kv_splits, num_requests, max_query_len, num_heads, num_kv_heads, max_keys,
                                        num_sms(on.dev));
  } else {
    const int64_t block_m = max_query_len <= 1 ? 16 : 32, block_n = t == at::kFloat ? 32 : 64;
    const int64_t q_blocks = std::max<int64_t>(1, fxpr::ceil_div(std::max<int64_t>(1, max_query_len), block_m));
    splits = fxpr::pick_attention_splits(num_kv_splits, num_requests, q_blocks, num_heads, fxpr::ceil_div(max_keys, block_n),
                                         num_sms(on.dev));
  }
  Tensor scratch;
  int64_t scratch_bytes = 0;
  if (splits > 1 && !tc) {
    // only the CUDA-core route keeps per-split maxima, integer totals and arrival counters in
    // scratch; the tensor-core kernels merge their splits inside a thread-block cluster
    scratch_bytes = fxpr_attention_scratch_bytes(tokens, (int)num_heads, (int)head_dim, (int)int_bits, (int)splits);
    scratch = empty_on({scratch_bytes}, at::kByte, q);
  }
  Tensor alibi;
  if (has_alibi) alibi = alibi_slopes->contiguous();
  const int flags = (is_causal ? FXPR_ATTN_CAUSAL : 0) | (t_ovr.attn_portable ? FXPR_ATTN_FORCE_PORTABLE : 0) | t_ovr.attn_flags;
  const Tensor qsl = query_start_loc.contiguous(), sl = seq_lens.contiguous();
  const Tensor bt = table2d && block_table_in.stride(1) != 1 ? block_table_in.contiguous() : block_table_in;
  check_status(
      fxpr_attention(q.data_ptr(), k_base, v_base, o.data_ptr(), qsl.data_ptr<int32_t>(),
                     sl.data_ptr<int32_t>(), bt.data_ptr<int32_t>(), has_alibi ? alibi.data_ptr<float>() : nullptr, dtype_code(t),
                     tokens, (int)num_requests, (int)num_heads, (int)num_kv_heads, (int)head_dim, (int)page, q.stride(0),
                     q.stride(1), o.stride(0), o.stride(1), kv.stride(0), kv.stride(2), kv.stride(3), table2d ? bt.stride(0) : 0,
                     (int)max_query_len, flags, ss, logit_softcap, (int)window_size, (int)int_bits, (int)frac_bits, (int)splits,
                     scratch.defined() ? scratch.data_ptr() : nullptr, scratch_bytes, status_ptr(on.dev), on.stream()),
      "unified_attention_fxp");
}

Tensor status_word(int64_t dev) {
  status_ptr((int)dev);
  return g_dev[dev].status;
}

std::vector<Tensor> status_words() {
  std::vector<Tensor> v;
  for (int i = 0; i < kMaxDevices; ++i) {
    DeviceState& d = g_dev[i];
    std::lock_guard<std::mutex> lock(d.mu);
    if (d.status.defined()) v.push_back(d.status);
  }
  return v;
}

Tensor last_partials() { return t_ovr.last_partials.defined() ? t_ovr.last_partials : at::empty({0}); }

}  // namespace

TORCH_LIBRARY_IMPL(fxpr, CUDA, m) {
  m.impl("float_to_fixed", float_to_fixed);
  m.impl("fixed_to_float", fixed_to_float);
  m.impl("rms_norm_fxp", rms_norm_fxp);
  m.impl("rms_norm_fxp_residual", rms_norm_fxp_residual);
  m.impl("rms_norm_fxp_from_int", rms_norm_fxp_from_int);
  m.impl("log_softmax_fxp", log_softmax_fxp);
  m.impl("gemm_fxp", gemm_fxp);
  m.impl("gemm_fxp_int", gemm_fxp_int);
  m.impl("gemm_fxp_epilogue", gemm_fxp_epilogue);
  m.impl("unified_attention_fxp", unified_attention_fxp);
}

TORCH_LIBRARY(fxpr_b200, m) {
  m.def("gemm_fxp_int_into(Tensor a, Tensor b, Tensor(a!) out, int int_bits, int frac_bits) -> ()");
  m.def("gemm_silu_mul(Tensor a, Tensor b_pairs, int int_bits, int frac_bits) -> Tensor");
  m.def("gemm_argmax(Tensor a, Tensor b, Tensor? bias, int int_bits, int frac_bits, int n_offset) -> (Tensor, Tensor)");
  m.def("silu_mul(Tensor gate_up, bool pairs) -> Tensor");
  m.def("rope_kv_write(Tensor qkv, Tensor cos, Tensor sin, Tensor positions, Tensor seq_ids, Tensor block_table, "
        "Tensor(a!) kv_cache, int q_heads, int kv_heads) -> Tensor");
  m.def("status_word(int device) -> Tensor", status_word);
  m.def("status_words() -> Tensor[]", status_words);
  m.def("gemm_scratch(int device, int nbytes) -> Tensor", [](int64_t dev, int64_t n) { return gemm_scratch((int)dev, n); });
  m.def("last_partials() -> Tensor", last_partials);
}

TORCH_LIBRARY_IMPL(fxpr_b200, CUDA, m) {
  m.impl("gemm_fxp_int_into", gemm_fxp_int_into);
  m.impl("gemm_silu_mul", gemm_silu_mul);
  m.impl("gemm_argmax", gemm_argmax);
  m.impl("silu_mul", silu_mul);
  m.impl("rope_kv_write", rope_kv_write);
}

// Plain C hooks for fxpr_vllm._native (ctypes: cheaper than an operator call).
extern "C" __attribute__((visibility("default"))) void fxpr_torch_set_overrides(int k_tile, int split_k, int gemm_portable, int attn_portable, int partials,
                                         int gemm_flags, int attn_flags) {
  Overrides& o = t_ovr;
  o.gemm_k_tile = k_tile;
  o.gemm_split_k = split_k;
  o.gemm_portable = gemm_portable;
  o.attn_portable = attn_portable;
  o.gemm_partials = partials;
  o.gemm_flags = gemm_flags;
  o.attn_flags = attn_flags;
  if (!partials) o.last_partials.reset();
}
extern "C" __attribute__((visibility("default"))) void fxpr_torch_set_config(int loaded, int frac_bits, int gemm_k_tile, int gemm_split_k) {
  g_config.frac_bits = frac_bits;
  g_config.gemm_k_tile = gemm_k_tile;
  g_config.gemm_split_k = gemm_split_k;
  g_config.loaded.store(loaded, std::memory_order_release);
}
extern "C" __attribute__((visibility("default"))) void fxpr_torch_set_config_loader(void (*load)()) { g_config_loader = load; }
