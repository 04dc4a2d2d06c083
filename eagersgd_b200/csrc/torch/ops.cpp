// Autograd operators over the sm_100a kernels, in C++.
//
// The kernels themselves are plain launchers in libesgd_cuda.so.  What surrounds a launch -- shape checks, output
// allocation, autograd bookkeeping, the choice of a kernel -- used to run in Python and cost 60 to 150 us per operator and
// direction, several times what the GPU needs for a CIFAR layer or a single image; here it costs a few microseconds, and
// the backward half runs on the autograd thread without the interpreter lock.
//
// GradSinks: while a training step of this package is active, the backward of an operator adds its parameter gradients
// straight to fp32 accumulators of the optimizer's flat buckets and tells the bucket so, instead of handing autograd a
// bf16 tensor that is cast, added to a zeroed .grad and cast again: three small kernels and a Python hook fewer per tensor.
#include <torch/extension.h>
#include "../cuda/bn_grad.h"
#include <ATen/SavedTensorHooks.h>
#include <torch/csrc/autograd/anomaly_mode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <atomic>
#include <mutex>
#include <shared_mutex>
#include <unordered_map>

extern "C" {
int esgd_sm_count();
int esgd_gemm_wgrad_splits(int64_t pixels, int64_t cout, int64_t cin, int sms);
int esgd_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int a_mn, int b_mn,
                   int out_mode, const float* scale, const void* bias, int relu, int splits, float* col_sum, float* col_sqsum,
                   const void* residual, int ldr, int* error_flag, void* stream);
int esgd_conv2d_fwd(const void* x, const void* w, void* y, int N, int H, int W, int Cin, int Cout, int R, int S, int stride,
                    int pad, const float* scale, const float* bias, const void* residual, int relu, float* col_sum,
                    float* col_sqsum, int* error_flag, void* stream);
int esgd_gemm_bn_dgrad(const void* dy, const void* w, void* dx, int M, int N, int K, const void* residual, const esgd_bn_grad* bn,
                       int* error_flag, void* stream);
int esgd_conv2d_dgrad(const void* dy, const void* w, void* dx, int N, int H, int W, int Cin, int Cout, int R, int S, int stride,
                      int pad, const void* residual, const esgd_bn_grad* bn, int* error_flag, void* stream);
int esgd_conv2d_wgrad(const void* x, const void* dy, float* dw, int N, int H, int W, int Cin, int Cout, int R, int S,
                      int stride, int pad, int* error_flag, void* stream);
int esgd_conv2d_wgrad_halo(const void* x, const void* dy, float* dw, int N, int H, int W, int Cin, int Cout, int R, int S,
                           int pad, int* error_flag, void* stream);
int esgd_conv_narrow_fwd(const void* x, const void* w, void* y, int N, int H, int W, int Cin, int Cout, int stride, const float* scale,
                         const float* shift, const void* residual, int relu, float* sum, float* sqsum, void* stream);
int esgd_conv_narrow_dgrad(const void* dy, const void* w, void* dx, int N, int H, int W, int Cin, int Cout, const void* residual,
                           const esgd_bn_grad* bn, void* stream);
int esgd_conv_narrow_bn_fwd(const void* by, void* z, void* mask, const float* bsum, const float* bsqsum, const float* gamma, const float* beta,
                            float* running_mean, float* running_var, float* aux, int relu, float momentum, float eps, const void* w,
                            void* y, int N, int H, int W, int C, float* sum, float* sqsum, void* stream);
int esgd_conv_narrow_bwd(const void* x, const void* w, const void* dz, const void* y, const float* aux, const float* gamma, const float* dbeta,
                         const float* dgamma, float* acc_dgamma, float* acc_dbeta, void* dx, float* dw, int N, int H, int W, int C,
                         const void* residual, const esgd_bn_grad* bn, void* stream);
int esgd_conv_narrow_wgrad(const void* x, const void* dy, float* dw, int N, int H, int W, int Cin, int Cout, int stride, void* stream);
int esgd_im2col_small_c(const void* x, void* col, int N, int H, int W, int C, int R, int S, int stride, int pad, int seg,
                        int Kpad, void* stream);
int esgd_stem_fwd(const void* x, const void* w2d, void* y, void* keep, int N, int H, int W, int C, int Cout, int R, int S, int stride, int pad,
                  int kpad, const float* scale, const float* shift, int relu, float* sum, float* sqsum, int* error_flag, void* stream);
int esgd_stem_wgrad(const void* x, const void* dy, float* col, int N, int H, int W, int C, int Cout, int R, int S, int stride, int pad, int kpad,
                    int* error_flag, void* stream);
int esgd_stem_pack(const void* w, void* out, int Cout, int R, int sc, int seg, int Kpad, void* stream);
int esgd_stem_unpack(const float* col, void* dw, float* acc, int Cout, int R, int sc, int seg, int Kpad, void* stream);
int esgd_subsample2_fwd(const void* x, void* y, int N, int H, int W, int C, void* stream);
int esgd_subsample2_bwd(const void* dy, void* dx, int N, int H, int W, int C, void* stream);
int esgd_bn_stats(const void* y, int64_t M, int C, float* sum, float* sqsum, void* stream);
int esgd_bn_fwd(const void* y, const void* residual, void* z, void* mask, const float* sum, const float* sqsum, const float* gamma,
                const float* beta, float* running_mean, float* running_var, float* aux, int64_t M, int C, int relu, float momentum,
                float eps, void* stream);
int esgd_bn_coefficients(const void* layers, int n, float eps, void* stream);
int esgd_bn_bwd_reduce(const void* dz, const void* mask, const void* y, const float* aux, int64_t M, int C, int mode, float* dbeta,
                       float* dgamma, void* stream);
int esgd_bn_bwd_apply(const void* dz, const void* mask, const void* y, const float* aux, const float* gamma, const float* dbeta,
                      const float* dgamma, void* dy, void* dres, int64_t M, int C, int mode, int last_first, float* acc_dgamma, float* acc_dbeta,
                      void* stream);
int esgd_softmax_ce(const void* logits, int is_bf16, const int64_t* labels, int batch, int classes, int ld, float grad_scale,
                    float* loss_sum, float* per_sample, void* dlogits, void* stream);
int esgd_maxpool3x3s2_fwd(const void* x, void* y, void* idx, int N, int H, int W, int C, void* stream);
int esgd_maxpool3x3s2_bwd(const void* idx, const void* dy, void* dx, int N, int H, int W, int C, void* stream);
int esgd_avgpool_fwd(const void* x, void* y, int N, int HW, int C, void* stream);
int esgd_avgpool_bwd(const void* dy, void* dx, int N, int HW, int C, void* stream);
int esgd_lstm_persistent_ok(int B, int H, int backward);
int esgd_lstm_persistent_fwd(const void* xproj, const void* w_hh, const float* bias, float* c, void* y, void* gates,
                             int T, int B, int H, int* error_flag, void* stream);
int esgd_lstm_persistent_bwd(const void* gates, const float* c, const void* dy, const void* w_hh, void* dG, float* db,
                             int T, int B, int H, int* error_flag, void* stream);
int esgd_lstm_seq_fwd(const void* xproj, const void* w_hh, const float* bias, float* c, void* y, void* gates, float* hprojT, int T,
                      int B, int H, int* error_flag, void* stream);
int esgd_lstm_seq_bwd(const void* gates, const float* c, const void* dy, const void* w_hh, void* dG, float* dc, float* dh_recT, int T,
                      int B, int H, int* error_flag, void* stream);
int esgd_cast_colsum(const float* dy, int64_t ld, int M, int N, int np, void* out, float* colsum, void* stream);
}

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
constexpr auto kCL = at::MemoryFormat::ChannelsLast;
constexpr float kBnEps = 1e-5f;

void ck(int rc, const char* what) { TORCH_CHECK(rc == 0, what, " failed with code ", rc); }
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
float* fptr(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
// The kernels load 16 bytes at a time and TMA starts on 16 bytes: a tensor that begins elsewhere (a view into a larger one) is
// copied.
Tensor aligned(Tensor t) { return ((uintptr_t)t.data_ptr() & 15) ? t.clone() : t; }
Tensor nhwc(const Tensor& t) { return aligned(t.contiguous(kCL)); }
Tensor dense(const Tensor& t) { return aligned(t.contiguous()); }
Tensor empty_nhwc(int64_t n, int64_t c, int64_t h, int64_t w, const Tensor& like) {
  return at::empty({n, c, h, w}, like.options(), kCL);
}

// ---------------------------------------------------------------- operands
// The kernels take bare pointers: what an operator is handed is compared here, before anything is allocated or launched.  The
// checks read sizes that are in the tensors anyway and cost nanoseconds.
void check_operand(const char* op, const char* name, const Tensor& t, const Tensor& x, at::ScalarType type) {
  TORCH_CHECK(t.scalar_type() == type, op, ": ", name, " is ", t.scalar_type(), ", not ", type);
  TORCH_CHECK(t.device() == x.device(), op, ": ", name, " is on ", t.device(), ", the input on ", x.device());
}
void check_vector(const char* op, const char* name, const Tensor& t, const Tensor& x, int64_t numel) {
  TORCH_CHECK(t.numel() == numel && t.is_contiguous(), op, ": ", name, " has to hold ", numel, " elements in a row, not ", t.sizes());
  check_operand(op, name, t, x, at::kFloat);
}
void check_conv(const Tensor& x, const Tensor& w, int64_t stride, int64_t pad, bool stem) {
  TORCH_CHECK(x.dim() == 4 && w.dim() == 4, "conv2d: takes a 4-D input and filter, not ", x.sizes(), " and ", w.sizes());
  TORCH_CHECK(x.size(1) == w.size(1), "conv2d: the filter ", w.sizes(), " does not have the ", x.size(1), " channels of the input");
  TORCH_CHECK(x.size(2) + 2 * pad >= w.size(2) && x.size(3) + 2 * pad >= w.size(3), "conv2d: the filter ", w.sizes(),
              " is larger than the padded input ", x.sizes());
  check_operand("conv2d", "the input", x, x, at::kBFloat16);
  check_operand("conv2d", "the filter", w, x, stem && w.is_floating_point() ? w.scalar_type() : at::kBFloat16);
}

// ---------------------------------------------------------------- per-device error word of the tensor-core kernels
Tensor error_flag(int64_t device) {
  static std::mutex m;
  static Tensor flags[64];
  TORCH_CHECK(device >= 0 && device < 64);
  std::lock_guard<std::mutex> g(m);
  if (!flags[device].defined())
    flags[device] = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, (c10::DeviceIndex)device));
  return flags[device];
}
int* flag_ptr(const Tensor& t) {
  static std::atomic<int*> cached[64];
  const int d = t.get_device();
  int* p = cached[d].load(std::memory_order_acquire);
  if (p == nullptr) {
    p = error_flag(d).data_ptr<int>();
    cached[d].store(p, std::memory_order_release);
  }
  return p;
}

// ---------------------------------------------------------------- zeroed scratch of a training step
// One fp32 buffer cleared by a single memset at the start of a step, from which the operators take their zero-initialised
// scratch (statistics and reduction accumulators).  A slice must not outlive the step.
class ZeroArena {
 public:
  void begin(at::Device device, int64_t numel);
  void end();
  Tensor take(at::IntArrayRef shape) {
    std::lock_guard<std::mutex> g(m_);
    const int64_t n = c10::multiply_integers(shape), n_al = (n + 63) / 64 * 64;    // 256-byte aligned slices
    if (off_ + n_al > cap_) return Tensor();
    if (!buf_.defined()) buf_ = at::zeros({cap_}, at::TensorOptions().dtype(at::kFloat).device(device_));
    Tensor out = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(buf_.storage()), buf_.key_set(), buf_.dtype());
    out.unsafeGetTensorImpl()->set_storage_offset(off_);           // a view without a trip through the dispatcher
    out.unsafeGetTensorImpl()->set_sizes_contiguous(shape);
    off_ += n_al;
    dirty_ = std::max(dirty_, off_);
    return out;
  }

 private:
  std::mutex m_;
  Tensor buf_;
  int64_t off_ = 0, dirty_ = 0, cap_ = 0;
  at::Device device_ = at::Device(at::kCPU);
};
std::atomic<ZeroArena*> g_arena[65];        // the active arena of the CPU (0) and of every GPU (1 + index)
std::atomic<ZeroArena*>& arena_slot(at::Device d) { return g_arena[d.is_cuda() ? 1 + d.index() : 0]; }

void ZeroArena::begin(at::Device device, int64_t numel) {
  if (device.is_cuda() && !device.has_index()) device = at::Device(at::kCUDA, c10::cuda::current_device());
  std::lock_guard<std::mutex> g(m_);
  if (buf_.defined() && (buf_.device() != device || buf_.numel() < numel)) { buf_ = Tensor(); dirty_ = 0; }
  device_ = device;
  if (buf_.defined() && dirty_ > 0) buf_.narrow(0, 0, dirty_).zero_();             // what earlier steps used
  off_ = 0;
  cap_ = numel;
  arena_slot(device).store(this, std::memory_order_release);
}
void ZeroArena::end() {
  ZeroArena* me = this;
  arena_slot(device_).compare_exchange_strong(me, nullptr);
}

Tensor zeros_f32(at::IntArrayRef shape, at::Device device) {
  if (ZeroArena* a = arena_slot(device).load(std::memory_order_acquire)) {
    Tensor t = a->take(shape);
    if (t.defined()) return t;
  }
  return at::zeros(shape, at::TensorOptions().dtype(at::kFloat).device(device));
}

// ---------------------------------------------------------------- gradient sinks
class GradSinks;
struct SinkEntry : torch::CustomClassHolder {
  float* acc = nullptr;          // fp32 accumulator, in the parameter's own memory order (OHWI for channels_last filters)
  int bucket = 0;
  c10::weak_intrusive_ptr<at::TensorImpl, at::UndefinedTensorImpl> param;
  // of the step that is under way:
  int uses = 0;                  // forward uses whose backward has not run yet
  bool used = false;             // an operator writes the accumulator
  bool recomputed = false;       // used inside a backward pass (checkpointing): there may be another such use to come
  bool hooked = false;           // autograd has written .grad
  bool counted = false;          // taken off its bucket's count
  explicit SinkEntry(const Tensor& p) : param(p.getIntrusivePtr()) {}
  // Autograd may still add to .grad: the parameter is in a graph, too, and its accumulation has not run.  Looked up without a
  // reference of our own, which costs 0.8 us a parameter (a tensor that Python knows); in a step its owner keeps it.
  bool awaited() const {
    if (recomputed) return true;
    if (hooked || !used || param.expired()) return false;
    const auto* meta = static_cast<const torch::autograd::AutogradMeta*>(param._unsafe_get_target()->autograd_meta());
    return meta != nullptr && !meta->grad_accumulator_.expired();
  }
  std::atomic<GradSinks*> owner{nullptr};
};
using Sink = c10::intrusive_ptr<SinkEntry>;

std::shared_mutex g_sink_mutex;
std::unordered_map<at::TensorImpl*, Sink> g_sinks;

class GradSinks {
 public:
  GradSinks(std::vector<int> params_per_bucket, py::function on_bucket)
      : total_(std::move(params_per_bucket)), pending_(total_), written_(total_.size(), 0), complete_(total_.size(), 0),
        in_bucket_(total_.size()), on_bucket_(std::move(on_bucket)) {}
  ~GradSinks() {
    close();
    if (side_) {
      cudaEventDestroy(forked_);
      cudaEventDestroy(joined_);
    }
  }
  void close() {
    std::unique_lock<std::shared_mutex> g(g_sink_mutex);
    for (auto& kv : mine_) {
      kv.second->owner.store(nullptr);
      const auto it = g_sinks.find(kv.first);
      if (it != g_sinks.end() && it->second == kv.second) g_sinks.erase(it);       // unless a later one has taken it over
    }
    mine_.clear();
    for (auto& b : in_bucket_) b.clear();
  }
  void add(const Tensor& param, const Tensor& acc, int bucket) {
    TORCH_CHECK(acc.scalar_type() == at::kFloat && acc.numel() == param.numel());
    auto e = c10::make_intrusive<SinkEntry>(param);
    e->acc = acc.data_ptr<float>();
    e->bucket = bucket;
    e->owner.store(this);
    std::unique_lock<std::shared_mutex> g(g_sink_mutex);
    g_sinks[param.unsafeGetTensorImpl()] = e;
    mine_[param.unsafeGetTensorImpl()] = e;
    in_bucket_.at(bucket).push_back(e.get());
  }
  void begin_step() {
    pending_ = total_;
    std::fill(complete_.begin(), complete_.end(), 0);
    for (auto& kv : mine_) {
      SinkEntry& e = *kv.second;
      e.uses = 0;
      e.used = e.recomputed = e.hooked = e.counted = false;
    }
  }
  void set_active(bool on) {
    if (!on) join();
    active_.store(on);
  }
  // Weight gradients go to a stream of their own: nothing waits for them before the bucket is complete, and neither they nor
  // the chain of the other gradients fills the GPU all of the time.  Outside a capture the events cost the host 3 us, so only
  // where the GPU has more to do than that for the layer: from a GFLOP on.  Milliseconds of an uncaptured step without /
  // with the side stream: ResNet-44 on 32 x 32 images, batch 100 (0.47 GFLOP a layer) 2.87 / 2.94, 128 (0.60) 2.65 / 2.74, 150
  // (0.71) 2.85 / 2.92, 200 (0.94) 2.93 / 2.74, 256 (1.21) 3.17 / 2.94, 400 (1.89) 3.85 / 3.41; ResNet-50 on 128 x 128
  // images, batch 16 (1.21, and 0.54 for 1x1 filters) 3.36 / 3.42, batch 64 3.64 / 3.43.  The operands are kept until the
  // streams have met again.
  c10::cuda::CUDAStream fork(const Tensor& a, const Tensor& b, double flops) {
    const auto main = c10::cuda::getCurrentCUDAStream(a.get_device());
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(main.stream(), &status) != cudaSuccess || status == cudaStreamCaptureStatusInvalidated ||
        (status == cudaStreamCaptureStatusNone && flops < 1e9))
      return main;
    if (!side_) {
      side_ = c10::cuda::getStreamFromPool(false, a.get_device());
      C10_CUDA_CHECK(cudaEventCreateWithFlags(&forked_, cudaEventDisableTiming));
      C10_CUDA_CHECK(cudaEventCreateWithFlags(&joined_, cudaEventDisableTiming));
    }
    C10_CUDA_CHECK(cudaEventRecord(forked_, main.stream()));
    C10_CUDA_CHECK(cudaStreamWaitEvent(side_->stream(), forked_, 0));
    held_.push_back(a);
    held_.push_back(b);
    return *side_;
  }
  void join() {
    if (held_.empty()) return;
    C10_CUDA_CHECK(cudaEventRecord(joined_, side_->stream()));
    C10_CUDA_CHECK(cudaStreamWaitEvent(c10::cuda::getCurrentCUDAStream(side_->device_index()).stream(), joined_, 0));
    held_.clear();
  }
  bool active() const { return active_.load(); }
  bool used(const Tensor& param) const {
    auto it = mine_.find(param.unsafeGetTensorImpl());
    return it != mine_.end() && it->second->used;
  }
  bool written(int bucket) const { return written_[bucket] != 0; }
  void clear_written() { std::fill(written_.begin(), written_.end(), 0); }
  void mark_written(int bucket) { written_[bucket] = 1; }
  // A parameter's gradient is complete once its operators' backward passes have run and, where autograd writes it as well,
  // that has happened, too; it is counted once whichever comes last.
  void sink_ready(SinkEntry& e) {
    if (!e.counted) {
      e.counted = true;
      --pending_[e.bucket];
    }
    settle(e.bucket);
  }
  void hooked(const Tensor& param) {
    auto it = mine_.find(param.unsafeGetTensorImpl());
    if (it == mine_.end()) return;
    it->second->hooked = true;
    if (it->second->uses == 0) sink_ready(*it->second);
  }

 private:
  // Announces a bucket whose every gradient is there; one with a parameter that may still get more goes with the step.
  void settle(int bucket) {
    if (pending_[bucket] > 0 || complete_[bucket]) return;
    for (const SinkEntry* e : in_bucket_[bucket])
      if (e->awaited()) return;
    complete_[bucket] = 1;
    join();
    py::gil_scoped_acquire gil;
    on_bucket_(bucket);
  }
  std::vector<int> total_, pending_, written_, complete_;
  std::vector<std::vector<const SinkEntry*>> in_bucket_;
  std::atomic<bool> active_{false};
  py::function on_bucket_;
  c10::optional<c10::cuda::CUDAStream> side_;
  cudaEvent_t forked_ = nullptr, joined_ = nullptr;
  std::vector<Tensor> held_;
  std::unordered_map<at::TensorImpl*, Sink> mine_;
};

// The sink of a parameter in a step that is under way, or null.
Sink find_sink(const Tensor& p) {
  if (!p.defined() || !p.requires_grad() || !p.is_leaf() || !at::GradMode::is_enabled()) return Sink();
  std::shared_lock<std::shared_mutex> g(g_sink_mutex);
  if (g_sinks.empty()) return Sink();
  auto it = g_sinks.find(p.unsafeGetTensorImpl());
  if (it == g_sinks.end()) return Sink();
  GradSinks* o = it->second->owner.load();
  return o != nullptr && o->active() ? it->second : Sink();
}
// Called in an operator's forward for a parameter that its backward will write.
void sink_use(const Sink& s) {
  if (!s) return;
  ++s->uses;
  s->used = true;
  if (torch::autograd::get_current_graph_task_id() != -1) s->recomputed = true;
}
// The parameter as the operator's autograd input: detached when a sink takes its gradient, so that autograd neither
// expects one nor calls the parameter's hooks.
Tensor graph_input(const Tensor& p, const Sink& s) { return s ? p.detach() : p; }
// The same without the detached view's microsecond: the tensor as an argument that autograd does not look at, and none where
// it would.
struct Held {
  Tensor t;
};
c10::optional<Tensor> graph_only(const Tensor& p, const Sink& s) { return s ? c10::nullopt : c10::optional<Tensor>(p); }
// What then keeps the operator in the graph when nothing else requires a gradient (the first layer of a network).
c10::optional<Tensor> anchor_for(const Tensor& x, bool any_sink) {
  if (!any_sink || x.requires_grad()) return c10::nullopt;
  static std::mutex m;
  static Tensor anchors[64];
  const int d = x.get_device();
  std::lock_guard<std::mutex> g(m);
  if (!anchors[d].defined()) anchors[d] = at::empty({0}, x.options().dtype(at::kFloat)).set_requires_grad(true);
  return anchors[d];
}
// Called in its backward once the kernel that writes the accumulator has been launched.
void sink_done(const Sink& s) {
  GradSinks* o = s->owner.load();
  if (o == nullptr || s->uses <= 0) return;
  o->mark_written(s->bucket);
  if (--s->uses == 0) o->sink_ready(*s);
}
void save_sink(AutogradContext* ctx, const char* key, const Sink& s) {
  if (s) ctx->saved_data[key] = c10::IValue::make_capsule(s);
}
Sink load_sink(AutogradContext* ctx, const char* key) {
  auto it = ctx->saved_data.find(key);
  if (it == ctx->saved_data.end()) return Sink();
  Sink s = c10::static_intrusive_pointer_cast<SinkEntry>(it->second.toCapsule());
  return s->owner.load() != nullptr ? s : Sink();
}

// ---------------------------------------------------------------- GEMM
int gemm(const void* a, const void* b, void* c, int64_t m, int64_t n, int64_t k, int64_t lda, int64_t ldb, int64_t ldc,
         bool a_mn, bool b_mn, int mode, int splits, float* cs, float* cq, const void* res, int64_t ldr, const Tensor& like,
         const void* bias = nullptr, int flags = 0, const float* scale = nullptr) {
  return esgd_gemm_bf16(a, b, c, (int)m, (int)n, (int)k, (int)lda, (int)ldb, (int)ldc, a_mn, b_mn, mode, scale, bias, flags, splits, cs,
                        cq, res, (int)ldr, flag_ptr(like), stream_of(like));
}

// Split-K factor of a weight-gradient GEMM (K = pixels).  Looked for among a hundred of them: a thread remembers its sizes.
int wgrad_splits(int64_t pixels, int64_t cout, int64_t cin, int64_t sms) {
  struct Known {
    int64_t pixels = 0, cout = 0, cin = 0, sms = 0;
    int splits = 0;
  };
  static thread_local Known known[64];
  Known& k = known[(pixels * 31 + cout * 7 + cin) / 8 % 64];
  if (k.splits == 0 || k.pixels != pixels || k.cout != cout || k.cin != cin || k.sms != sms)
    k = Known{pixels, cout, cin, sms, esgd_gemm_wgrad_splits(pixels, cout, cin, (int)sms)};
  return k.splits;
}

// ---------------------------------------------------------------- convolutions
enum ConvKind : int64_t { kOneByOne = 0, kGeneral = 1, kStem = 2 };

constexpr int kNotTaken = -100;      // a kernel's answer to a shape outside its range: the next one takes it

struct StemGeometry {
  int64_t seg, kpad;
  StemGeometry(int64_t c, int64_t r, int64_t s) {
    seg = (s * c + 7) / 8 * 8;                        // one filter row, padded to 16 bytes
    kpad = (r * seg + 63) / 64 * 64;
    while (kpad % seg) kpad += 64;
  }
};

// A batch norm whose output a convolution reads: the convolution's data gradient then leaves the gradient with the ReLU's
// mask applied and the two sums over it (bn_grad.h), and the batch norm's backward has one pass to do instead of two.
//
// Only inside a training step of this package (parameters with sinks), and only where nobody can tell a gradient whose masked
// elements are already zero: no hooks on the tensor, no gradient captured on the way.  The sums count when the very tensor
// that the data gradient wrote arrives, untouched; a sum with another consumer's gradient is another tensor, and goes
// through the mask and the reduction again.
struct BnRecord : torch::CustomClassHolder {
  Tensor y, mask, aux;
  std::weak_ptr<torch::autograd::Node> node;
  Tensor dz, sums;               // left by the data gradient
  uint32_t version = 0;

  bool observed() const {
    const auto n = node.lock();
    if (!n || !n->tensor_pre_hooks().empty() || !n->pre_hooks().empty() || !n->retains_grad_hooks().empty()) return true;
    const auto* captures = torch::autograd::get_current_graph_task_exec_info();
    return captures != nullptr && !captures->empty();
  }
  void fill(esgd_bn_grad* g, const Tensor& dx) {
    const int64_t c = dx.size(1);
    sums = zeros_f32({2, c}, dx.device());
    *g = esgd_bn_grad{y.data_ptr(), mask.defined() ? mask.data_ptr() : nullptr, fptr(aux), fptr(sums)};
  }
  void written(const Tensor& dx) {
    dz = dx;
    version = dx._version();
  }
};
using BnRef = c10::intrusive_ptr<BnRecord>;
BnRef bn_behind(const Tensor& x);     // the record of the batch norm that produced x, or null

// A convolution and the batch norm that is its output's only reader, inside a residual block: what the one's node leaves for the
// other's, so that a narrow layer's backward pass is one launch.  The batch norm hands on its own gradient dz in the place of
// dy, which the convolution's backward then makes from it on the way into shared memory; between the two nodes nobody looks.
struct LayerLink : torch::CustomClassHolder {
  std::weak_ptr<torch::autograd::Node> conv, norm;
  bool pending = false;                  // the rest is there: dz stands for dy
  Tensor dz, y, aux, gamma, sums;
  Sink gs, bs;
  uint32_t version = 0;

  bool observed() const {
    const auto c = conv.lock(), n = norm.lock();
    if (!c || !n || !c->tensor_pre_hooks().empty() || !c->pre_hooks().empty() || !c->retains_grad_hooks().empty() ||
        !n->post_hooks().empty() || torch::autograd::AnomalyMode::is_enabled()) return true;
    const auto* captures = torch::autograd::get_current_graph_task_exec_info();
    return captures != nullptr && !captures->empty();
  }
  void release() {
    pending = false;
    dz = y = aux = gamma = sums = Tensor();
    gs = bs = Sink();
  }
};
using Link = c10::intrusive_ptr<LayerLink>;

// A batch norm (without a residual) whose launch is left to the convolution that reads its output.
struct PendingNorm {
  Tensor y, z, mask, stats, gamma, beta, mean, var, aux;
  bool relu = false;
  float momentum = 0.0f;
  void launch(void* stream) const {
    const int64_t c = y.size(1);
    ck(esgd_bn_fwd(y.data_ptr(), nullptr, z.data_ptr(), mask.defined() ? mask.data_ptr() : nullptr, fptr(stats), fptr(stats) + c, fptr(gamma),
                   fptr(beta), fptr(mean), fptr(var), fptr(aux), y.numel() / c, c, relu, momentum, kBnEps, stream), "bn_fwd");
  }
};

// The windows of NHWC x as a matrix, one row per output pixel.
Tensor stem_columns(const Tensor& x, int64_t r, int64_t s, int64_t stride, int64_t pad) {
  const int64_t n = x.size(0), c = x.size(1), h = x.size(2), w = x.size(3);
  const StemGeometry g(c, r, s);
  Tensor col = at::empty({n * ((h + 2 * pad - r) / stride + 1) * ((w + 2 * pad - s) / stride + 1), g.kpad}, x.options());
  ck(esgd_im2col_small_c(x.data_ptr(), col.data_ptr(), n, h, w, c, r, s, stride, pad, g.seg, g.kpad, stream_of(x)), "im2col");
  return col;
}

// What a convolution's epilogue does to the product: statistics of it (training), or the affine map of an inference batch
// norm, a residual and a ReLU.
struct ConvEpilogue {
  float *sum = nullptr, *sqsum = nullptr;
  const float *scale = nullptr, *shift = nullptr;
  const void* residual = nullptr;
  bool relu = false;
  bool train = false;            // a backward pass may follow
};

// Launches the convolution of NHWC x with w into y; `kept` and `filters` are what a backward pass needs of the two.
// norm: x is its output and still to be computed.
void launch_conv(int64_t kind, const Tensor& x, const Tensor& w, const Tensor& y, int64_t stride, int64_t pad, const ConvEpilogue& e,
                 Tensor* kept, Tensor* filters, const PendingNorm* norm = nullptr) {
  const int64_t n = x.size(0), cin = x.size(1), h = x.size(2), wd = x.size(3), cout = w.size(0), r = w.size(2), s = w.size(3);
  const int64_t ho = y.size(2), wo = y.size(3);
  void* st = stream_of(x);
  if (norm != nullptr) {
    // 64 channels: rows of more than 32 pixels take two launches (rows in shared memory and these, us: 40 x 40, four images 9.5 and 8.5;
    // 56 x 56, one 9.1 and 8.3, two 10.0 and 8.3; 32 x 32, eight 8.2 and 9.2)
    if ((cin < 64 || wd <= 32) && kind == kGeneral && r == 3 && s == 3 && pad == 1 && stride == 1 && cin == cout && e.scale == nullptr && e.residual == nullptr && !e.relu) {
      *filters = nhwc(w);
      *kept = x;
      const int rc = esgd_conv_narrow_bn_fwd(norm->y.data_ptr(), x.data_ptr(), norm->mask.defined() ? norm->mask.data_ptr() : nullptr,
                                             fptr(norm->stats), fptr(norm->stats) + cin, fptr(norm->gamma), fptr(norm->beta), fptr(norm->mean),
                                             fptr(norm->var), fptr(norm->aux), norm->relu, norm->momentum, kBnEps, filters->data_ptr(),
                                             y.data_ptr(), n, h, wd, cin, e.sum, e.sqsum, st);
      if (rc == 0) return;
      if (rc != kNotTaken) ck(rc, "batch norm and conv2d");
    }
    norm->launch(st);
  }
  if (kind == kOneByOne) {
    *filters = dense(w);                            // [Cout, Cin]: a 1x1 filter has one memory order
    *kept = x;
    if (stride == 2 && !e.train) {                  // nothing reads the subsampled input again: its pixels are picked by the loads
      const int rc = esgd_conv2d_fwd(x.data_ptr(), filters->data_ptr(), y.data_ptr(), n, h, wd, cin, cout, 1, 1, 2, 0, e.scale, e.shift,
                                     e.residual, e.relu, e.sum, e.sqsum, flag_ptr(x), st);
      if (rc >= 0) {                                // negative: refused, nothing launched
        ck(rc, "1x1 convolution");
        return;
      }
    }
    if (stride == 2) {
      *kept = empty_nhwc(n, cin, ho, wo, x);
      ck(esgd_subsample2_fwd(x.data_ptr(), kept->data_ptr(), n, h, wd, cin, st), "subsample");
    }
    ck(gemm(kept->data_ptr(), filters->data_ptr(), y.data_ptr(), n * ho * wo, cout, cin, cin, cin, cout, false, false, 0, 1, e.sum,
            e.sqsum, e.residual, cout, x, e.shift, e.relu, e.scale), "1x1 convolution");
  } else if (kind == kGeneral) {
    *filters = nhwc(w);                             // [Cout][R][S][Cin] in memory
    *kept = x;
    int rc = kNotTaken;
    if (r == 3 && s == 3 && pad == 1)
      rc = esgd_conv_narrow_fwd(x.data_ptr(), filters->data_ptr(), y.data_ptr(), n, h, wd, cin, cout, stride, e.scale, e.shift,
                                e.residual, e.relu, e.sum, e.sqsum, st);
    if (rc == kNotTaken)
      rc = esgd_conv2d_fwd(x.data_ptr(), filters->data_ptr(), y.data_ptr(), n, h, wd, cin, cout, r, s, stride, pad, e.scale, e.shift,
                           e.residual, e.relu, e.sum, e.sqsum, flag_ptr(x), st);
    ck(rc, "conv2d");
  } else {
    *filters = nhwc(w.to(at::kBFloat16));           // packed anyway: any floating type
    const StemGeometry g(cin, r, s);
    Tensor w2d = at::empty({cout, g.kpad}, x.options());
    ck(esgd_stem_pack(filters->data_ptr(), w2d.data_ptr(), cout, r, s * cin, g.seg, g.kpad, st), "stem filters");
    if (e.residual == nullptr) {
      // the backward pass has a copy of the images: the caller may refill their buffer before it
      Tensor images = e.train ? empty_nhwc(n, cin, h, wd, x) : Tensor();
      const int rc = esgd_stem_fwd(x.data_ptr(), w2d.data_ptr(), y.data_ptr(), e.train ? images.data_ptr() : nullptr, n, h, wd, cin, cout, r, s,
                                   stride, pad, g.kpad, e.scale, e.shift, e.relu, e.sum, e.sqsum, flag_ptr(x), st);
      if (rc != kNotTaken) {
        ck(rc, "stem convolution");
        *kept = images;
        return;
      }
    }
    *kept = stem_columns(x, r, s, stride, pad);
    ck(gemm(kept->data_ptr(), w2d.data_ptr(), y.data_ptr(), n * ho * wo, cout, g.kpad, g.kpad, g.kpad, cout, false, false, 0, 1, e.sum,
            e.sqsum, e.residual, cout, x, e.shift, e.relu, e.scale), "stem convolution");
  }
}

// y = x (*) w, and on request the per-channel sum / sum of squares of y and the input itself.
//
// With `tap` the input is returned as a last output.  A residual block takes its shortcut from that output instead of
// from x itself: backward then receives the shortcut's gradient together with dy and adds it in the epilogue of the
// data-gradient GEMM, instead of autograd summing the two branches of x with a separate pass over the tensor.
struct ConvFn : public Function<ConvFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x_in, const c10::optional<Tensor>& w_in, int64_t kind,
                               int64_t stride, int64_t pad, bool want_stats, bool tap, const Sink& sink,
                               const c10::optional<Tensor>& anchor, const BnRef& bn, const Held& w_held, const Held& into, const Link& link,
                               const PendingNorm* norm) {
    const Tensor& w = w_in.has_value() ? *w_in : w_held.t;
    c10::cuda::CUDAGuard guard(x_in.device());
    Tensor x = nhwc(x_in);
    const int64_t n = x.size(0), cin = x.size(1), h = x.size(2), wd = x.size(3);
    const int64_t cout = w.size(0), r = w.size(2), s = w.size(3);
    const int64_t ho = (h + 2 * pad - r) / stride + 1, wo = (wd + 2 * pad - s) / stride + 1;
    Tensor stats = into.t;                            // given: not an output of the graph's
    ConvEpilogue e;
    e.train = true;
    if (want_stats) stats = zeros_f32({2, cout}, x.device());
    if (stats.defined()) {
      e.sum = fptr(stats);
      e.sqsum = e.sum + cout;
    }
    Tensor y = empty_nhwc(n, cout, ho, wo, x);
    Tensor saved_x, wk;
    launch_conv(kind, x, w, y, stride, pad, e, &saved_x, &wk, norm);
    ctx->save_for_backward({saved_x, wk});
    ctx->saved_data["cfg"] = std::vector<int64_t>{kind, stride, pad, n, cin, h, wd, want_stats, tap};
    save_sink(ctx, "w", sink);
    if (bn) ctx->saved_data["bn"] = c10::IValue::make_capsule(bn);
    if (link) ctx->saved_data["link"] = c10::IValue::make_capsule(link);
    ctx->set_materialize_grads(false);                // an unused tap must not cost a tensor of zeros
    variable_list out{y};
    if (want_stats) {
      ctx->mark_non_differentiable({stats});
      out.push_back(stats);
    }
    if (tap) out.push_back(x_in.view_as(x_in));
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto cfg = ctx->saved_data["cfg"].toIntVector();
    const int64_t kind = cfg[0], stride = cfg[1], pad = cfg[2], n = cfg[3], cin = cfg[4], h = cfg[5], wd = cfg[6];
    const bool want_stats = cfg[7], tap = cfg[8];
    variable_list none(14);
    Tensor d_tap = tap ? grads[want_stats ? 2 : 1] : Tensor();   // gradient that reached the input through the shortcut
    Sink sink = load_sink(ctx, "w");
    if (!grads[0].defined()) {
      none[0] = d_tap;
      return none;
    }
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    const int64_t cout = w.size(0), r = w.size(2), s = w.size(3);
    c10::cuda::CUDAGuard guard(x.device());
    Tensor dy = nhwc(grads[0]);
    const int64_t ho = dy.size(2), wo = dy.size(3), m = n * ho * wo;
    void* st = stream_of(x);
    Tensor dx, dw;
    const bool need_dx = ctx->needs_input_grad(0), need_dw = sink || ctx->needs_input_grad(1);
    BnRef bn;
    if (const auto it = ctx->saved_data.find("bn"); sink && it != ctx->saved_data.end()) {
      bn = c10::static_intrusive_pointer_cast<BnRecord>(it->second.toCapsule());
      if (!bn->y.defined() || bn->observed()) bn = BnRef();
    }
    esgd_bn_grad bg;
    if (const auto it = ctx->saved_data.find("link"); it != ctx->saved_data.end()) {
      const Link link = c10::static_intrusive_pointer_cast<LayerLink>(it->second.toCapsule());
      if (link->pending) {
        TORCH_CHECK(link->dz.is_same(grads[0]) && link->version == grads[0]._version(), "conv2d: somebody came between a layer and its batch norm");
        const Tensor sums = link->sums, lz = link->dz, ly = link->y, laux = link->aux, lgamma = link->gamma;
        const Sink gs = link->gs, bs = link->bs;
        link->release();
        int rc = kNotTaken;
        if (need_dx && sink) {
          Tensor res;
          if (d_tap.defined()) res = nhwc(d_tap.to(at::kBFloat16));
          dx = empty_nhwc(n, cin, h, wd, x);
          if (bn) bn->fill(&bg, dx);
          rc = esgd_conv_narrow_bwd(x.data_ptr(), w.data_ptr(), lz.data_ptr(), ly.data_ptr(), fptr(laux), fptr(lgamma), fptr(sums),
                                    fptr(sums) + cout, gs->acc, bs->acc, dx.data_ptr(), sink->acc, n, h, wd, cin,
                                    res.defined() ? res.data_ptr() : nullptr, bn ? &bg : nullptr, st);
          if (rc == 0 && bn) bn->written(dx);
        }
        if (rc == kNotTaken) {             // then as the batch norm would have done it
          dy = empty_nhwc(n, cout, ho, wo, x);
          ck(esgd_bn_bwd_apply(lz.data_ptr(), nullptr, ly.data_ptr(), fptr(laux), fptr(lgamma), fptr(sums), fptr(sums) + cout, dy.data_ptr(),
                               nullptr, m, cout, 0, 1, gs->acc, bs->acc, st), "bn_bwd_apply");
        } else {
          ck(rc, "backward pass of a layer");
        }
        sink_done(gs);
        sink_done(bs);
        if (rc == 0) {
          sink_done(sink);
          none[0] = dx;
          return none;
        }
      }
    }
    // The weight gradient goes first: what the data gradient leaves (and the batch norm's pass behind it reads) is then the
    // newest in L2.
    if (need_dw) {
      c10::cuda::OptionalCUDAStreamGuard forked;
      if (GradSinks* owner = sink && kind != kStem ? sink->owner.load() : nullptr) forked.reset_stream(owner->fork(dy, x, 2.0 * m * cin * cout * r * s));
      void* st = stream_of(x);
      if (kind == kOneByOne) {
        Tensor dw32;
        if (!sink) dw32 = zeros_f32({cout, cin}, x.device());
        ck(gemm(dy.data_ptr(), x.data_ptr(), sink ? sink->acc : fptr(dw32), cout, cin, m, cout, cin, cin, true, true, 2,
                wgrad_splits(m, cout, cin, esgd_sm_count()), nullptr, nullptr, nullptr, 0, x), "1x1 convolution weight gradient");
        if (!sink) dw = dw32.to(w.scalar_type()).view(w.sizes());
      } else if (kind == kGeneral) {
        Tensor dw32;
        if (!sink) dw32 = zeros_f32({cout, r, s, cin}, x.device());
        float* acc = sink ? sink->acc : fptr(dw32);
        int rc = kNotTaken;
        if (r == 3 && s == 3 && pad == 1)
          rc = esgd_conv_narrow_wgrad(x.data_ptr(), dy.data_ptr(), acc, n, h, wd, cin, cout, stride, st);
        if (rc == kNotTaken && stride == 1)      // shared input boxes, taps as shifted views
          rc = esgd_conv2d_wgrad_halo(x.data_ptr(), dy.data_ptr(), acc, n, h, wd, cin, cout, r, s, pad, flag_ptr(x), st);
        if (rc == kNotTaken)
          rc = esgd_conv2d_wgrad(x.data_ptr(), dy.data_ptr(), acc, n, h, wd, cin, cout, r, s, stride, pad, flag_ptr(x), st);
        ck(rc, "conv2d weight gradient");
        if (!sink) dw = dw32.to(w.scalar_type()).permute({0, 3, 1, 2});
      } else {
        const StemGeometry g(cin, r, s);
        Tensor col = zeros_f32({cout, g.kpad}, x.device());
        // the forward pass left the images where its kernel took them, else their columns
        ck(x.dim() == 4 ? esgd_stem_wgrad(x.data_ptr(), dy.data_ptr(), fptr(col), n, h, wd, cin, cout, r, s, stride, pad, g.kpad, flag_ptr(x), st)
                        : gemm(dy.data_ptr(), x.data_ptr(), fptr(col), cout, g.kpad, m, cout, g.kpad, g.kpad, true, true, 2, esgd_sm_count(),
                               nullptr, nullptr, nullptr, 0, x),
           "stem weight gradient");
        if (!sink) dw = at::empty(w.sizes(), w.options(), kCL);
        ck(esgd_stem_unpack(fptr(col), sink ? nullptr : dw.data_ptr(), sink ? sink->acc : nullptr, cout, r, s * cin, g.seg, g.kpad,
                            st), "stem filter gradient");
      }
    }
    if (need_dx && kind == kOneByOne) {
      Tensor res;
      if (d_tap.defined()) res = nhwc(d_tap.to(at::kBFloat16));
      dx = empty_nhwc(n, cin, ho, wo, x);
      int rc = kNotTaken;
      if (bn) {
        bn->fill(&bg, dx);
        rc = esgd_gemm_bn_dgrad(dy.data_ptr(), w.data_ptr(), dx.data_ptr(), m, cin, cout, res.defined() ? res.data_ptr() : nullptr, &bg,
                                flag_ptr(x), st);
        if (rc == 0) bn->written(dx);
      }
      if (rc == kNotTaken)
        rc = gemm(dy.data_ptr(), w.data_ptr(), dx.data_ptr(), m, cin, cout, cout, cin, cin, false, true, 0, 1, nullptr, nullptr,
                  res.defined() ? res.data_ptr() : nullptr, cin, x);
      ck(rc, "1x1 convolution data gradient");
      if (stride == 2) {
        Tensor full = empty_nhwc(n, cin, h, wd, x);
        ck(esgd_subsample2_bwd(dx.data_ptr(), full.data_ptr(), n, h, wd, cin, st), "subsample backward");
        dx = full;
      }
    } else if (need_dx && kind == kGeneral) {
      const bool square = r == s && pad <= r - 1;
      dx = empty_nhwc(n, cin, h, wd, x);
      if (square && stride == 1) {
        Tensor res;
        if (d_tap.defined()) res = nhwc(d_tap.to(at::kBFloat16));
        const void* rp = res.defined() ? res.data_ptr() : nullptr;
        if (bn) bn->fill(&bg, dx);
        auto launch = [&](const esgd_bn_grad* g) {
          int rc = kNotTaken;
          if (r == 3 && pad == 1)
            rc = esgd_conv_narrow_dgrad(dy.data_ptr(), w.data_ptr(), dx.data_ptr(), n, h, wd, cin, cout, rp, g, st);
          if (rc == kNotTaken)
            rc = esgd_conv2d_dgrad(dy.data_ptr(), w.data_ptr(), dx.data_ptr(), n, h, wd, cin, cout, r, s, 1, pad, rp, g, flag_ptr(x), st);
          return rc;
        };
        int rc = launch(bn ? &bg : nullptr);
        if (bn && rc == 0) bn->written(dx);
        if (bn && rc == kNotTaken) rc = launch(nullptr);
        ck(rc, "conv2d data gradient");
        d_tap = Tensor();
      } else if (stride == 2 && r == 3 && s == 3 && pad == 1 && h % 2 == 0 && wd % 2 == 0) {
        ck(esgd_conv2d_dgrad(dy.data_ptr(), w.data_ptr(), dx.data_ptr(), n, h, wd, cin, cout, 3, 3, 2, 1, nullptr, nullptr, flag_ptr(x), st),
           "strided conv2d data gradient");
      } else if (square) {
        // Any other stride / size: the gradient is spread out with (stride - 1) zeros between its pixels (plus the rows and
        // columns at the far edge that no window reached) and then goes through the stride-1 form above.
        const int64_t eh = (h + 2 * pad - r) % stride, ew = (wd + 2 * pad - s) % stride;
        Tensor spread = at::zeros({n, cout, (ho - 1) * stride + 1 + eh, (wo - 1) * stride + 1 + ew}, dy.options()).contiguous(kCL);
        spread.slice(2, 0, (ho - 1) * stride + 1, stride).slice(3, 0, (wo - 1) * stride + 1, stride).copy_(dy);
        ck(esgd_conv2d_dgrad(spread.data_ptr(), w.data_ptr(), dx.data_ptr(), n, h, wd, cin, cout, r, s, 1, pad, nullptr, nullptr, flag_ptr(x),
                             st), "conv2d data gradient");
      } else {
        dx = std::get<0>(at::convolution_backward(dy, x, w, c10::nullopt, {stride, stride}, {pad, pad}, {1, 1}, false, {0, 0}, 1,
                                                  {true, false, false}));
      }
      if (d_tap.defined()) dx = dx + d_tap;
    } else if (need_dx) {
      dx = d_tap;
    }
    if (need_dw && sink) sink_done(sink);
    none[0] = dx;
    none[1] = dw;
    return none;
  }
};

// Which kernel takes a convolution; -1: none, the shape is not this package's.
int64_t conv_kind_of(int64_t c, const Tensor& w, int64_t stride, int64_t pad, bool narrow, bool x_grad) {
  const int64_t k0 = w.size(0), r = w.size(2), s = w.size(3);
  if (stride < 1 || pad < 0) return -1;
  if (r == 1 && s == 1 && pad == 0 && stride <= 2 && c % 8 == 0 && k0 % 8 == 0) return kOneByOne;
  if (r > 1 && c <= 4 && k0 % 8 == 0 && !x_grad) return kStem;
  if (r > 1 && c % 8 == 0 && k0 % 8 == 0 && stride <= 2 && (narrow || c % 64 == 0)) return kGeneral;
  return -1;
}

int64_t conv_kind(const Tensor& x, const Tensor& w, int64_t stride, int64_t pad, bool narrow) {
  return conv_kind_of(x.size(1), w, stride, pad, narrow, x.requires_grad());
}

struct ConvOut {
  Tensor y, stats, tapped;       // stats, tapped: on request
};
ConvOut conv_train(int64_t kind, const Tensor& x, const Tensor& w, int64_t stride, int64_t pad, bool want_stats, bool tap,
                   const Tensor& into = Tensor(), const Link& link = Link(), const PendingNorm* norm = nullptr) {
  check_conv(x, w, stride, pad, kind == kStem);
  const int64_t r = w.size(2), s = w.size(3);
  // the stride-1 data gradients add the shortcut's gradient in their epilogue: elsewhere the tap is the input itself
  const bool fuse_tap = tap && (kind == kOneByOne || (kind == kGeneral && r == s && pad <= r - 1)) && stride == 1 && x.requires_grad() && at::GradMode::is_enabled();
  Sink sink = find_sink(w);
  sink_use(sink);
  variable_list out = ConvFn::apply(x, graph_only(w, sink), kind, stride, pad, want_stats, fuse_tap, sink, anchor_for(x, (bool)sink),
                                    sink && stride == 1 ? bn_behind(x) : BnRef(), Held{w}, Held{into}, link, norm);
  if (link) link->conv = out[0].grad_fn();
  return {out[0], want_stats ? out[1] : Tensor(), !tap ? Tensor() : (fuse_tap ? out.back() : x)};
}

// Returns (y, stats | None, tapped input | None), or None when the shape is not this package's.
py::object conv2d(const Tensor& x, const Tensor& w, int64_t stride, int64_t pad, bool want_stats, bool tap, bool narrow) {
  const int64_t kind = conv_kind(x, w, stride, pad, narrow);
  if (kind < 0) return py::none();
  const ConvOut o = conv_train(kind, x, w, stride, pad, want_stats, tap);
  return py::make_tuple(o.y, want_stats ? py::cast(o.stats) : py::none(), tap ? py::cast(o.tapped) : py::none());
}

// Inference: act(batch_norm(conv(x)) + residual) in one kernel.  coef [2][Cout] fp32: scale and shift (BnCoefficients), or
// None for a bare convolution.  No autograd; None when the shape is not this package's.
Tensor conv_eval(int64_t kind, const Tensor& x_in, const Tensor& w, int64_t stride, int64_t pad, const c10::optional<Tensor>& coef,
                 const c10::optional<Tensor>& residual, bool relu) {
  check_conv(x_in, w, stride, pad, kind == kStem);
  if (coef.has_value()) check_vector("conv2d", "the coefficients", *coef, x_in, 2 * w.size(0));
  const int64_t ho = (x_in.size(2) + 2 * pad - w.size(2)) / stride + 1, wo = (x_in.size(3) + 2 * pad - w.size(3)) / stride + 1;
  if (residual.has_value()) {
    TORCH_CHECK(residual->sizes() == at::IntArrayRef({x_in.size(0), w.size(0), ho, wo}), "conv2d: the residual ", residual->sizes(),
                " is not of the output's size");
    check_operand("conv2d", "the residual", *residual, x_in, at::kBFloat16);
  }
  c10::cuda::CUDAGuard guard(x_in.device());
  Tensor x = nhwc(x_in), res = residual.has_value() ? nhwc(*residual) : Tensor(), kept, filters;
  const int64_t cout = w.size(0);
  Tensor y = empty_nhwc(x.size(0), cout, ho, wo, x);
  ConvEpilogue e;
  if (coef.has_value()) {
    e.scale = fptr(*coef);
    e.shift = e.scale + cout;
  }
  if (res.defined()) e.residual = res.data_ptr();
  e.relu = relu;
  launch_conv(kind, x, w, y, stride, pad, e, &kept, &filters);
  return y;
}
py::object conv_bn_eval(const Tensor& x, const Tensor& w, int64_t stride, int64_t pad, const c10::optional<Tensor>& coef,
                        const c10::optional<Tensor>& residual, bool relu, bool narrow) {
  const int64_t kind = conv_kind(x, w, stride, pad, narrow);
  if (kind < 0 || w.scalar_type() != at::kBFloat16) return py::none();
  return py::cast(conv_eval(kind, x, w, stride, pad, coef, residual, relu));
}

// A residual block in inference: layers (filter, stride, padding, coefficients), each with a ReLU, the last one after the
// shortcut (through proj, which has none, or straight).  None when a layer is not this package's.
py::object residual_block_eval(const Tensor& x, const std::vector<py::tuple>& layers, const c10::optional<py::tuple>& proj, bool narrow) {
  struct Layer {
    Tensor w, coef;
    int64_t stride, pad, kind;
  };
  std::vector<Layer> ls;
  ls.reserve(layers.size() + 1);
  auto add = [&](const py::tuple& t) {
    Layer l{t[0].cast<Tensor>(), t[3].cast<Tensor>(), t[1].cast<int64_t>(), t[2].cast<int64_t>(), 0};
    l.kind = l.w.scalar_type() != at::kBFloat16 ? -1 : conv_kind_of(l.w.size(1), l.w, l.stride, l.pad, narrow, true);
    ls.push_back(l);
    return l.kind >= 0;
  };
  for (const auto& t : layers)
    if (!add(t)) return py::none();
  if (proj.has_value() && !add(*proj)) return py::none();
  if (x.size(1) != ls[0].w.size(1)) return py::none();
  Tensor y = x;
  {
    py::gil_scoped_release nogil;
    const size_t n = layers.size();
    Tensor shortcut = x;
    if (proj.has_value()) shortcut = conv_eval(ls[n].kind, x, ls[n].w, ls[n].stride, ls[n].pad, ls[n].coef, c10::nullopt, false);
    for (size_t i = 0; i < n; ++i)
      y = conv_eval(ls[i].kind, y, ls[i].w, ls[i].stride, ls[i].pad, ls[i].coef,
                    i + 1 == n ? c10::optional<Tensor>(shortcut) : c10::nullopt, true);
  }
  return py::cast(y);
}

// The affine maps of a network's batch norms, computed from their parameters and running statistics by one launch per
// forward pass.  The table of pointers lives on the device and is rebuilt when a tensor has moved.
class BnCoefficients {
 public:
  // layers: gamma, beta, mean, var; no result unless they are fp32, on the GPU and of one length a layer.
  std::vector<Tensor> compute(const std::vector<std::array<Tensor, 4>>& layers) {
    std::lock_guard<std::mutex> g(m_);
    for (const auto& l : layers)
      for (const auto& t : l)
        if (!t.defined() || !t.is_cuda() || t.scalar_type() != at::kFloat || !t.is_contiguous() || t.numel() != l[0].numel() ||
            t.device() != layers[0][0].device())
          return {};
    c10::cuda::CUDAGuard guard(layers.at(0)[0].device());
    std::vector<int64_t> key;
    key.reserve(layers.size() * 6);
    for (const auto& l : layers) {
      for (const auto& t : l) key.push_back((int64_t)t.data_ptr<float>());
      key.push_back(0);
      key.push_back(l[0].numel());
    }
    if (key != key_) {
      key_ = key;
      int64_t total = 0;
      for (const auto& l : layers) total += 2 * l[0].numel();
      const auto opt = layers[0][0].options().requires_grad(false);
      Tensor buf = at::empty({total}, opt);
      out_.clear();
      int64_t off = 0;
      for (size_t i = 0; i < layers.size(); ++i) {
        const int64_t c = layers[i][0].numel();
        out_.push_back(buf.narrow(0, off, 2 * c));
        key[6 * i + 4] = (int64_t)out_.back().data_ptr<float>();
        off += 2 * c;
      }
      table_ = at::tensor(key, at::kLong).to(buf.device());
    }
    ck(esgd_bn_coefficients(table_.data_ptr(), (int)layers.size(), kBnEps, stream_of(table_)), "batch-norm coefficients");
    return out_;
  }

 private:
  std::mutex m_;
  std::vector<int64_t> key_;
  std::vector<Tensor> out_;
  Tensor table_;
};

// The layers that a fused inference pass stands in for.  Whether calling them one by one would still do the same is asked in
// every pass (a layer may have been exchanged, parametrized or hooked since), and of 141 modules in a ResNet-56: 22 us here
// against 130 in Python, where a small CIFAR network's whole pass takes 270.
class EvalLayers {
 public:
  // modules: (module, the type whose forward the pass stands for; None for a container, whose forward nobody calls).  children:
  // what the lists were made from, the network's own `_modules`.
  EvalLayers(py::dict children, const std::vector<std::pair<py::object, py::object>>& modules, py::list convs, py::list norms)
      : norms(std::move(norms)), convs_(std::move(convs)) {
    root_.children = snapshot(children.ptr());
    root_.module = std::move(children);
    for (const auto& m : modules) {
      Entry e{m.first, m.second, {}};
      py::object d = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(m.first.ptr(), nullptr));
      e.children = snapshot(d ? PyDict_GetItem(d.ptr(), name().modules) : nullptr);
      entries_.push_back(std::move(e));
    }
  }
  // Every module is of its type, in evaluation mode, without hooks or a forward of its own, and where it was.
  bool unchanged() const {
    const Names& n = name();
    if (!same_children(root_.module.ptr(), root_.children)) return false;
    for (const Entry& e : entries_) {
      const bool called = !e.type.is_none();
      if (called && (PyObject*)Py_TYPE(e.module.ptr()) != e.type.ptr()) return false;
      const py::object d = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(e.module.ptr(), nullptr));
      if (!d || !same_children(PyDict_GetItem(d.ptr(), n.modules), e.children)) { PyErr_Clear(); return false; }
      if (!called) continue;
      if (PyDict_GetItem(d.ptr(), n.training) != Py_False || PyDict_GetItem(d.ptr(), n.forward) != nullptr) return false;
      for (PyObject* h : n.hooks) {
        PyObject* hooks = PyDict_GetItem(d.ptr(), h);
        if (hooks == nullptr || !PyDict_Check(hooks) || PyDict_Size(hooks) != 0) return false;
      }
    }
    for (const auto& c : convs_)
      if (!tensor(c.ptr(), n.parameters, n.weight).defined()) return false;
    return true;
  }
  // The affine maps of the norms, or none: layers have changed, or a tensor is not what the kernels take.  The table is the
  // network's and not these layers': a captured pass reads it for as long as it is replayed.
  c10::optional<std::vector<Tensor>> coefficients(BnCoefficients& table) const {
    if (!unchanged()) return c10::nullopt;
    const Names& n = name();
    std::vector<std::array<Tensor, 4>> layers;
    layers.reserve(norms.size());
    for (const auto& m : norms) {
      layers.push_back({tensor(m.ptr(), n.parameters, n.weight), tensor(m.ptr(), n.parameters, n.bias), tensor(m.ptr(), n.buffers, n.mean),
                        tensor(m.ptr(), n.buffers, n.var)});
    }
    std::vector<Tensor> out;
    if (!layers.empty() && (out = table.compute(layers)).empty()) return c10::nullopt;
    return out;
  }
  const py::list norms;

 private:
  struct Entry {
    py::object module, type;
    std::vector<py::object> children;
  };
  struct Names {
    PyObject *modules, *training, *forward, *parameters, *buffers, *weight, *bias, *mean, *var;
    std::array<PyObject*, 4> hooks;
  };
  static const Names& name() {
    static const Names n = [] {
      auto s = [](const char* t) { return PyUnicode_InternFromString(t); };
      return Names{s("_modules"), s("training"), s("forward"), s("_parameters"), s("_buffers"), s("weight"), s("bias"), s("running_mean"),
                   s("running_var"), {s("_forward_hooks"), s("_forward_pre_hooks"), s("_backward_hooks"), s("_backward_pre_hooks")}};
    }();
    return n;
  }
  static std::vector<py::object> snapshot(PyObject* dict) {
    std::vector<py::object> out;
    PyObject *k, *v;
    for (Py_ssize_t i = 0; dict != nullptr && PyDict_Check(dict) && PyDict_Next(dict, &i, &k, &v);) out.push_back(py::reinterpret_borrow<py::object>(v));
    return out;
  }
  static bool same_children(PyObject* dict, const std::vector<py::object>& want) {
    if (dict == nullptr || !PyDict_Check(dict) || (size_t)PyDict_Size(dict) != want.size()) return false;
    PyObject *k, *v;
    size_t j = 0;
    for (Py_ssize_t i = 0; PyDict_Next(dict, &i, &k, &v);)
      if (want[j++].ptr() != v) return false;
    return true;
  }
  // A parameter or buffer where a module keeps it; undefined when there is none.
  static Tensor tensor(PyObject* module, PyObject* where, PyObject* key) {
    const py::object d = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(module, nullptr));
    if (!d) PyErr_Clear();
    PyObject* dict = d ? PyDict_GetItem(d.ptr(), where) : nullptr;
    PyObject* t = dict != nullptr && PyDict_Check(dict) ? PyDict_GetItem(dict, key) : nullptr;
    return t != nullptr && THPVariable_Check(t) ? THPVariable_Unpack(t) : Tensor();
  }
  Entry root_;
  std::vector<Entry> entries_;
  py::list convs_;
};

// ---------------------------------------------------------------- dense layer: fp32 logits out of bf16 operands
struct LinearFn : public Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_in, const Tensor& w_in, const c10::optional<Tensor>& b_in,
                        const Sink& ws, const Sink& bs, const c10::optional<Tensor>& anchor) {
    const Tensor b = b_in.has_value() ? *b_in : Tensor();
    c10::cuda::CUDAGuard guard(x_in.device());
    Tensor x = dense(x_in), w = dense(w_in);
    const int64_t m = x.size(0), k = x.size(1), n = w.size(0), np = (n + 7) / 8 * 8;
    Tensor y = at::empty({m, np}, x.options().dtype(at::kFloat));
    Tensor bias = b.defined() ? b.contiguous() : Tensor();
    if (bias.defined() && (bias.scalar_type() != at::kBFloat16 || ((uintptr_t)bias.data_ptr() & 7))) bias = bias.to(at::kFloat).clone();
    ck(gemm(x.data_ptr(), w.data_ptr(), y.data_ptr(), m, n, k, k, k, np, false, false, 1, 1, nullptr, nullptr, nullptr, 0, x,
            bias.defined() ? bias.data_ptr() : nullptr, bias.defined() && bias.scalar_type() == at::kBFloat16 ? 2 : 0), "dense layer");
    ctx->save_for_backward({x, w});
    ctx->saved_data["bias"] = b.defined() ? (int64_t)b.scalar_type() : (int64_t)-1;
    save_sink(ctx, "w", ws);
    save_sink(ctx, "b", bs);
    return n == np ? y : y.narrow(1, 0, n);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t m = x.size(0), k = x.size(1), n = w.size(0), np = (n + 7) / 8 * 8;
    Sink ws = load_sink(ctx, "w"), bs = load_sink(ctx, "b");
    Tensor dy = grads[0];
    if (dy.scalar_type() != at::kFloat) dy = dy.to(at::kFloat);
    if (dy.stride(1) != 1 || (dy.stride(0) < n && m > 1)) dy = dy.contiguous();
    const int64_t bias_type = ctx->saved_data["bias"].toInt();
    const bool need_b = bs || (bias_type >= 0 && ctx->needs_input_grad(2));
    Tensor db32;
    if (need_b && !bs) db32 = zeros_f32({n}, x.device());
    Tensor dy16 = at::empty({m, np}, x.options());
    ck(esgd_cast_colsum(dy.data_ptr<float>(), dy.stride(0), m, n, np, dy16.data_ptr(), !need_b ? nullptr : (bs ? bs->acc : fptr(db32)),
                        stream_of(x)), "dense layer gradient");
    Tensor dx, dw, db;
    if (ctx->needs_input_grad(0)) {
      dx = at::empty({m, k}, x.options());
      ck(gemm(dy16.data_ptr(), w.data_ptr(), dx.data_ptr(), m, k, n, np, k, k, false, true, 0, 1, nullptr, nullptr, nullptr, 0, x),
         "dense layer data gradient");
    }
    if (ws || ctx->needs_input_grad(1)) {
      if (!ws) dw = at::empty({n, k}, w.options());
      ck(gemm(dy16.data_ptr(), x.data_ptr(), ws ? (void*)ws->acc : dw.data_ptr(), n, k, m, np, k, k, true, true, ws ? 2 : 0, 1, nullptr,
              nullptr, nullptr, 0, x), "dense layer weight gradient");
      if (ws) sink_done(ws);
    }
    if (need_b) {
      if (bs) sink_done(bs);
      else db = db32.to((at::ScalarType)bias_type, false, true);
    }
    return {dx, dw, db, Tensor(), Tensor(), Tensor()};
  }
};

// None when the shape is not this package's.
py::object linear(const Tensor& x, const Tensor& w, const c10::optional<Tensor>& b) {
  if (x.size(1) % 8 || w.scalar_type() != at::kBFloat16) return py::none();
  TORCH_CHECK(x.dim() == 2 && w.dim() == 2, "linear: takes a 2-D input and weight, not ", x.sizes(), " and ", w.sizes());
  TORCH_CHECK(x.size(1) == w.size(1), "linear: the weight ", w.sizes(), " does not have the ", x.size(1), " columns of the input");
  check_operand("linear", "the input", x, x, at::kBFloat16);
  check_operand("linear", "the weight", w, x, at::kBFloat16);
  if (b.has_value()) {
    TORCH_CHECK(b->numel() == w.size(0), "linear: the bias ", b->sizes(), " does not have the ", w.size(0), " outputs of the weight");
    check_operand("linear", "the bias", *b, x, b->scalar_type());
  }
  Tensor bias = b.has_value() ? *b : Tensor();
  Sink ws = find_sink(w), bs = find_sink(bias);
  sink_use(ws);
  sink_use(bs);
  c10::optional<Tensor> bias_in;
  if (bias.defined()) bias_in = graph_input(bias, bs);
  return py::cast(LinearFn::apply(x, graph_input(w, ws), bias_in, ws, bs, anchor_for(x, ws || bs)));
}

// ---------------------------------------------------------------- batch norm (+ residual) (+ ReLU)
struct BnActFn : public Function<BnActFn> {
  using Opt = c10::optional<Tensor>;
  static Tensor forward(AutogradContext* ctx, const Tensor& y_in, const Opt& gamma_in, const Opt& beta_in, const Opt& res_in,
                        const Held& rm_in, const Held& rv_in, double momentum, bool relu, const Held& stats_in, const Sink& gs,
                        const Sink& bs, const Opt& anchor, const Held& gamma_held, const Held& beta_held, const Link& link, PendingNorm* later) {
    const Tensor &gamma = gamma_in.has_value() ? *gamma_in : gamma_held.t, &beta = beta_in.has_value() ? *beta_in : beta_held.t;
    c10::cuda::CUDAGuard guard(y_in.device());
    Tensor y = nhwc(y_in), res = res_in.has_value() ? nhwc(*res_in) : Tensor(), stats = stats_in.t, rm = rm_in.t, rv = rv_in.t;
    const int64_t n = y.size(0), c = y.size(1), m = n * y.size(2) * y.size(3);
    void* st = stream_of(y);
    if (!stats.defined()) {
      stats = zeros_f32({2, c}, y.device());
      ck(esgd_bn_stats(y.data_ptr(), m, c, fptr(stats), fptr(stats) + c, st), "bn_stats");
    }
    Tensor aux = at::empty({4, c}, gamma.options());       // mean, invstd, scale, shift
    Tensor z = empty_nhwc(n, c, y.size(2), y.size(3), y);
    // ReLU mask of the backward pass: a bit per element where a residual was added, else recomputed from y
    // (a bit as well where a convolution's data gradient may have to apply it)
    const int64_t mode = !relu ? 0 : (res.defined() || (gs && bs) ? 1 : 2);
    Tensor mask;
    if (mode == 1) mask = at::empty({m, c / 8}, y.options().dtype(at::kByte));
    if (later != nullptr) {
      *later = PendingNorm{y, z, mask, stats, gamma, beta, rm, rv, aux, relu, (float)momentum};
    } else {
      ck(esgd_bn_fwd(y.data_ptr(), res.defined() ? res.data_ptr() : nullptr, z.data_ptr(), mode == 1 ? mask.data_ptr() : nullptr,
                     fptr(stats), fptr(stats) + c, fptr(gamma), fptr(beta), fptr(rm), fptr(rv), fptr(aux), m, c, relu, (float)momentum,
                     kBnEps, st), "bn_fwd");
    }
    ctx->save_for_backward({y, mask, gamma, aux});
    ctx->saved_data["mode"] = mode;
    ctx->saved_data["res"] = res.defined();
    save_sink(ctx, "g", gs);
    save_sink(ctx, "b", bs);
    // Saved-tensor hooks (checkpointing, offloading) are there to let go of activations: no record then, which would keep them.
    if (gs && bs && !at::SavedTensorDefaultHooks::get_hooks().has_value()) {
      auto rec = c10::make_intrusive<BnRecord>();
      rec->y = y;
      rec->mask = mask;
      rec->aux = aux;
      ctx->saved_data["rec"] = c10::IValue::make_capsule(rec);
      if (link) ctx->saved_data["link"] = c10::IValue::make_capsule(link);
    }
    return z;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &y = saved[0], &mask = saved[1], &gamma = saved[2], &aux = saved[3];
    c10::cuda::CUDAGuard guard(y.device());
    int64_t mode = ctx->saved_data["mode"].toInt();
    const int64_t c = y.size(1), m = y.numel() / c;
    const bool has_res = ctx->saved_data["res"].toBool();
    Sink gs = load_sink(ctx, "g"), bs = load_sink(ctx, "b");
    Tensor dz = nhwc(grads[0]);
    void* st = stream_of(y);
    const void* mp = mask.defined() ? mask.data_ptr() : nullptr;
    Tensor red, dres;
    BnRef rec;
    if (const auto it = ctx->saved_data.find("rec"); it != ctx->saved_data.end())
      rec = c10::static_intrusive_pointer_cast<BnRecord>(it->second.toCapsule());
    const bool fused = gs && bs && rec && rec->dz.defined() && rec->dz.is_same(dz) && rec->version == dz._version();
    if (fused) {
      red = rec->sums;             // dz is masked, its sums are there, and it is the shortcut's gradient as it stands
      mode = 0;
      if (has_res) dres = dz;
    } else {
      // dbeta, dgamma; handed to autograd unless both go to sinks, so then not from the step's scratch
      red = gs && bs ? zeros_f32({2, c}, y.device()) : at::zeros({2, c}, aux.options());
      ck(esgd_bn_bwd_reduce(dz.data_ptr(), mp, y.data_ptr(), fptr(aux), m, c, (int)mode, fptr(red), fptr(red) + c, st), "bn_bwd_reduce");
    }
    if (rec) {
      rec->y = rec->mask = rec->dz = rec->sums = Tensor();
    }
    variable_list out(16);
    if (const auto it = ctx->saved_data.find("link"); it != ctx->saved_data.end()) {
      const Link link = c10::static_intrusive_pointer_cast<LayerLink>(it->second.toCapsule());
      link->release();                     // of an earlier pass that broke off before the convolution's backward
      if (fused && !link->observed()) {    // the convolution's backward, which comes next, does it on the way
        link->dz = dz;
        link->version = dz._version();
        link->y = y;
        link->aux = aux;
        link->gamma = gamma;
        link->sums = red;
        link->gs = gs;
        link->bs = bs;
        link->pending = true;
        out[0] = dz;
        out[3] = dres;
        return out;
      }
    }
    float* rd = fptr(red);
    Tensor dy = empty_nhwc(y.size(0), c, y.size(2), y.size(3), y);
    const bool write_res = has_res && !dres.defined();
    if (write_res) dres = empty_nhwc(y.size(0), c, y.size(2), y.size(3), y);
    ck(esgd_bn_bwd_apply(dz.data_ptr(), mp, y.data_ptr(), fptr(aux), fptr(gamma), rd, rd + c, dy.data_ptr(),
                         write_res ? dres.data_ptr() : nullptr, m, c, (int)mode, fused, gs ? gs->acc : nullptr, bs ? bs->acc : nullptr, st),
       "bn_bwd_apply");
    Tensor dgamma, dbeta;
    if (gs) sink_done(gs);
    else dgamma = red.select(0, 1);
    if (bs) sink_done(bs);
    else dbeta = red.select(0, 0);
    out[0] = dy; out[1] = dgamma; out[2] = dbeta; out[3] = dres;
    return out;
  }
};

Tensor bn_train(const Tensor& y, const Tensor& gamma, const Tensor& beta, const c10::optional<Tensor>& res,
              const c10::optional<Tensor>& rm, const c10::optional<Tensor>& rv, double momentum, bool relu,
              const c10::optional<Tensor>& stats, const Link& link, PendingNorm* later) {
  TORCH_CHECK(y.dim() == 4, "bn_act: takes a 4-D input, not ", y.sizes());
  const int64_t c = y.size(1);
  check_operand("bn_act", "the input", y, y, at::kBFloat16);
  check_vector("bn_act", "gamma", gamma, y, c);
  check_vector("bn_act", "beta", beta, y, c);
  if (rm.has_value()) check_vector("bn_act", "the running mean", *rm, y, c);
  if (rv.has_value()) check_vector("bn_act", "the running variance", *rv, y, c);
  if (stats.has_value() && stats->defined()) check_vector("bn_act", "the statistics", *stats, y, 2 * c);
  if (res.has_value()) {
    TORCH_CHECK(res->sizes() == y.sizes(), "bn_act: the residual ", res->sizes(), " is not of the input's size ", y.sizes());
    check_operand("bn_act", "the residual", *res, y, at::kBFloat16);
  }
  Sink gs = find_sink(gamma), bs = find_sink(beta);
  sink_use(gs);
  sink_use(bs);
  auto held = [](const c10::optional<Tensor>& o) { return Held{o.has_value() ? *o : Tensor()}; };
  Tensor z = BnActFn::apply(y, graph_only(gamma, gs), graph_only(beta, bs), res, held(rm), held(rv), momentum, relu, held(stats), gs,
                            bs, anchor_for(y, gs || bs), Held{gamma}, Held{beta}, link, later);
  if (gs && bs) {
    auto* node = static_cast<torch::autograd::CppNode<BnActFn>*>(z.grad_fn().get());
    const auto it = node->ctx_.saved_data.find("rec");
    if (it != node->ctx_.saved_data.end()) c10::static_intrusive_pointer_cast<BnRecord>(it->second.toCapsule())->node = z.grad_fn();
    if (link) link->norm = z.grad_fn();
  }
  return z;
}
Tensor bn_act(const Tensor& y, const Tensor& gamma, const Tensor& beta, const c10::optional<Tensor>& res,
              const c10::optional<Tensor>& rm, const c10::optional<Tensor>& rv, double momentum, bool relu,
              const c10::optional<Tensor>& stats) {
  return bn_train(y, gamma, beta, res, rm, rv, momentum, relu, stats, Link(), nullptr);
}

// A residual block in training (convolution, batch norm and ReLU in a row, the last batch norm adding the shortcut): what the
// two operators above do layer by layer, in one call from Python, which spent 9 us a layer between them.  A layer is (filter,
// stride, padding, gamma, beta, running mean, running variance, momentum); proj: the shortcut's, or None.  None when a layer
// is not this package's.
struct BlockLayer {
  Tensor w, gamma, beta;
  int64_t stride, pad, kind;
  c10::optional<Tensor> mean, var;
  double momentum;
  BlockLayer(const py::tuple& t, const Tensor& x, bool narrow)
      : w(t[0].cast<Tensor>()), gamma(t[3].cast<Tensor>()), beta(t[4].cast<Tensor>()), stride(t[1].cast<int64_t>()),
        pad(t[2].cast<int64_t>()), mean(t[5].cast<c10::optional<Tensor>>()), var(t[6].cast<c10::optional<Tensor>>()),
        momentum(t[7].cast<double>()) {
    kind = w.size(2) > 1 && w.size(1) <= 4 ? -1 : conv_kind_of(w.size(1), w, stride, pad, narrow, true);
    if (w.scalar_type() != at::kBFloat16 || gamma.scalar_type() != at::kFloat || w.size(0) % 8) kind = -1;
  }
  Tensor stats;                  // of the convolution's output, for the batch norm behind it
  Link link;                     // ... where one launch may do the backward pass of both
  bool rows() const { return kind == kGeneral && w.size(2) == 3 && w.size(3) == 3 && stride == 1 && pad == 1 && w.size(0) == w.size(1); }
  // later: the batch norm that x is still to come from
  ConvOut conv(const Tensor& x, bool tap, const PendingNorm* later = nullptr) {
    stats = zeros_f32({2, w.size(0)}, x.device());
    if (rows() && (w.size(0) == 16 || w.size(0) == 32) && at::GradMode::is_enabled()) link = c10::make_intrusive<LayerLink>();
    return conv_train(kind, x, w, stride, pad, false, tap, stats, link, later);
  }
  Tensor norm(const ConvOut& o, bool relu, const c10::optional<Tensor>& res, PendingNorm* later = nullptr) const {
    return bn_train(o.y, gamma, beta, res, mean, var, momentum, relu, stats, link, later);
  }
};
py::object residual_block(const Tensor& x, const std::vector<py::tuple>& layers, const c10::optional<py::tuple>& proj, bool narrow) {
  std::vector<BlockLayer> ls;
  ls.reserve(layers.size() + 1);
  for (const auto& t : layers) ls.emplace_back(t, x, narrow);
  if (proj.has_value()) ls.emplace_back(*proj, x, narrow);
  for (const auto& l : ls)
    if (l.kind < 0) return py::none();
  if (x.size(1) != ls[0].w.size(1)) return py::none();
  Tensor out;
  {
    py::gil_scoped_release nogil;
    const size_t n = layers.size();
    ConvOut c = ls[0].conv(x, true);
    c10::optional<Tensor> shortcut = c.tapped;
    if (proj.has_value()) {
      shortcut = ls[n].norm(ls[n].conv(c.tapped, false), false, c10::nullopt);
    }
    // A batch norm between two convolutions is left to the second where the kernels for rows in shared memory may take it (up to 64
    // channels); not when somebody packs what is saved for the backward pass, which would then not be there yet.
    const bool may_wait = !at::SavedTensorDefaultHooks::get_hooks().has_value();
    PendingNorm later;
    bool waiting = false;
    for (size_t i = 0; i < n; ++i) {
      if (i > 0) c = ls[i].conv(out, false, waiting ? &later : nullptr);
      waiting = may_wait && i + 1 < n && ls[i + 1].rows() && ls[i + 1].w.size(0) <= 64;
      out = ls[i].norm(c, true, i + 1 == n ? shortcut : c10::nullopt, waiting ? &later : nullptr);
    }
  }
  return py::cast(out);
}

BnRef bn_behind(const Tensor& x) {
  auto* node = dynamic_cast<torch::autograd::CppNode<BnActFn>*>(x.grad_fn().get());
  if (node == nullptr || !x.is_contiguous(kCL)) return BnRef();
  const auto it = node->ctx_.saved_data.find("rec");
  if (it == node->ctx_.saved_data.end()) return BnRef();
  return c10::static_intrusive_pointer_cast<BnRecord>(it->second.toCapsule());
}

// ---------------------------------------------------------------- softmax cross-entropy
struct SoftmaxCEFn : public Function<SoftmaxCEFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits_in, const Tensor& labels) {
    c10::cuda::CUDAGuard guard(logits_in.device());
    // rows padded to a multiple of eight (the dense layer's) are read as they are, and the gradient is laid out alike; a column
    // slice of something wider is copied, or the gradient would be as wide
    const int64_t b = logits_in.size(0), c = logits_in.size(1), ld = logits_in.stride(0);
    Tensor logits = logits_in.stride(1) == 1 && ld >= c && ld < c + 8 ? logits_in : logits_in.contiguous();
    Tensor loss = at::zeros({}, logits.options().dtype(at::kFloat));
    Tensor d = at::empty_strided({b, c}, {logits.stride(0), 1}, logits.options());
    ck(esgd_softmax_ce(logits.data_ptr(), logits.scalar_type() == at::kBFloat16, labels.contiguous().data_ptr<int64_t>(), b, c,
                       logits.stride(0), 1.0f / (float)b, fptr(loss), nullptr, d.data_ptr(), stream_of(logits)), "softmax_ce");
    ctx->save_for_backward({d});
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) { return {ctx->get_saved_variables()[0] * grads[0], Tensor()}; }
};
Tensor softmax_ce(const Tensor& logits, const Tensor& labels) {
  TORCH_CHECK(logits.dim() == 2, "softmax_ce: takes 2-D logits, not ", logits.sizes());
  TORCH_CHECK(labels.numel() == logits.size(0), "softmax_ce: ", labels.numel(), " labels for ", logits.size(0), " rows");
  check_operand("softmax_ce", "the labels", labels, logits, at::kLong);
  return SoftmaxCEFn::apply(logits, labels);
}

// ---------------------------------------------------------------- pooling
struct MaxPoolFn : public Function<MaxPoolFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_in) {
    c10::cuda::CUDAGuard guard(x_in.device());
    Tensor x = nhwc(x_in);
    const int64_t n = x.size(0), c = x.size(1), h = x.size(2), w = x.size(3), oh = (h + 1) / 2, ow = (w + 1) / 2;
    Tensor y = empty_nhwc(n, c, oh, ow, x);
    Tensor idx;
    if (x_in.requires_grad()) idx = at::empty({n * oh * ow, c}, x.options().dtype(at::kByte));
    ck(esgd_maxpool3x3s2_fwd(x.data_ptr(), y.data_ptr(), idx.defined() ? idx.data_ptr() : nullptr, n, h, w, c, stream_of(x)), "maxpool");
    if (idx.defined()) ctx->save_for_backward({idx});
    ctx->saved_data["dims"] = std::vector<int64_t>{n, c, h, w};
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto d = ctx->saved_data["dims"].toIntVector();
    const Tensor idx = ctx->get_saved_variables()[0];
    Tensor dy = nhwc(grads[0]);
    c10::cuda::CUDAGuard guard(dy.device());
    Tensor dx = empty_nhwc(d[0], d[1], d[2], d[3], dy);
    ck(esgd_maxpool3x3s2_bwd(idx.data_ptr(), dy.data_ptr(), dx.data_ptr(), d[0], d[2], d[3], d[1], stream_of(dy)), "maxpool backward");
    return {dx};
  }
};
Tensor max_pool(const Tensor& x) { return MaxPoolFn::apply(x); }

struct AvgPoolFn : public Function<AvgPoolFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_in) {
    c10::cuda::CUDAGuard guard(x_in.device());
    Tensor x = nhwc(x_in);
    const int64_t n = x.size(0), c = x.size(1), h = x.size(2), w = x.size(3);
    Tensor y = at::empty({n, c}, x.options());
    ck(esgd_avgpool_fwd(x.data_ptr(), y.data_ptr(), n, h * w, c, stream_of(x)), "avgpool");
    ctx->saved_data["dims"] = std::vector<int64_t>{n, c, h, w};
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto d = ctx->saved_data["dims"].toIntVector();
    Tensor dy = dense(grads[0]);
    c10::cuda::CUDAGuard guard(dy.device());
    Tensor dx = empty_nhwc(d[0], d[1], d[2], d[3], dy);
    ck(esgd_avgpool_bwd(dy.data_ptr(), dx.data_ptr(), d[0], d[2] * d[3], d[1], stream_of(dy)), "avgpool backward");
    return {dx};
  }
};
Tensor avg_pool(const Tensor& x) { return AvgPoolFn::apply(x); }

// ---------------------------------------------------------------- LSTM layer
// x . W_ih^T of all steps is one GEMM; the recurrence is one persistent kernel per direction where the shape allows it
// (weights resident on the chip), else a native loop of split-K GEMMs and cell kernels; the weight and input gradients are
// single GEMMs over all steps.
struct LstmFn : public Function<LstmFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_in, const Tensor& w_ih_in, const Tensor& w_hh_in, const Tensor& bias,
                        const Sink& s_ih, const Sink& s_hh, const Sink& s_b, const c10::optional<Tensor>& anchor) {
    c10::cuda::CUDAGuard guard(x_in.device());
    Tensor x = dense(x_in), w_ih = dense(w_ih_in), w_hh = dense(w_hh_in);
    const int64_t t = x.size(0), b = x.size(1), in = x.size(2), h = w_hh.size(1);
    void* st = stream_of(x);
    const auto f32 = x.options().dtype(at::kFloat);
    Tensor xproj = at::empty({t * b, 4 * h}, x.options());
    ck(gemm(x.data_ptr(), w_ih.data_ptr(), xproj.data_ptr(), t * b, 4 * h, in, in, in, 4 * h, false, false, 0, 1, nullptr, nullptr,
            nullptr, 0, x), "lstm input projection");
    Tensor y = at::empty({t, b, h}, x.options()), c = at::empty({t, b, h}, f32), gates = at::empty({t, b, 4 * h}, x.options());
    if (esgd_lstm_persistent_ok((int)b, (int)h, 0)) {
      ck(esgd_lstm_persistent_fwd(xproj.data_ptr(), w_hh.data_ptr(), fptr(bias), fptr(c), y.data_ptr(), gates.data_ptr(),
                                  t, b, h, flag_ptr(x), st), "lstm forward recurrence");
    } else {
      Tensor hproj = at::empty({4 * h, b}, f32);
      ck(esgd_lstm_seq_fwd(xproj.data_ptr(), w_hh.data_ptr(), fptr(bias), fptr(c), y.data_ptr(), gates.data_ptr(), fptr(hproj), t, b, h,
                           flag_ptr(x), st), "lstm forward recurrence");
    }
    ctx->save_for_backward({x, w_ih, w_hh, y, c, gates});
    save_sink(ctx, "ih", s_ih);
    save_sink(ctx, "hh", s_hh);
    save_sink(ctx, "b", s_b);
    return y;
  }

  // dw [m][n] = a^T b over `rows`, added to the sink's accumulator or returned in the weights' type.  The tiles of these
  // gradients fill the GPU by themselves unless the layer is small: only then is the reduction split.
  static Tensor weight_grad(const Sink& sink, const Tensor& a, const void* ap, const Tensor& w, const void* bp, int64_t rows, int64_t m,
                            int64_t n) {
    const int64_t bn = n <= 64 ? 64 : (n <= 128 ? 128 : 256), tiles = ((m + 127) / 128) * ((n + bn - 1) / bn);
    const int64_t splits = std::max<int64_t>(1, std::min<int64_t>(esgd_sm_count() / tiles, rows / 512));
    Tensor dw;
    if (sink || splits > 1) {
      if (!sink) dw = at::zeros({m, n}, w.options().dtype(at::kFloat));
      ck(gemm(ap, bp, sink ? sink->acc : fptr(dw), m, n, rows, m, n, n, true, true, 2, (int)splits, nullptr, nullptr, nullptr, 0, a),
         "lstm weight gradient");
      return sink ? Tensor() : dw.to(w.scalar_type());
    }
    dw = at::empty({m, n}, w.options());
    ck(gemm(ap, bp, dw.data_ptr(), m, n, rows, m, n, n, true, true, 0, 1, nullptr, nullptr, nullptr, 0, a), "lstm weight gradient");
    return dw;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w_ih = saved[1], &w_hh = saved[2], &y = saved[3], &c = saved[4], &gates = saved[5];
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t t = x.size(0), b = x.size(1), in = x.size(2), h = w_hh.size(1);
    Sink s_ih = load_sink(ctx, "ih"), s_hh = load_sink(ctx, "hh"), s_b = load_sink(ctx, "b");
    const auto f32 = x.options().dtype(at::kFloat);
    void* st = stream_of(x);
    Tensor dy = dense(grads[0]);
    Tensor dG = at::empty({t * b, 4 * h}, x.options());
    Tensor dx, dw_ih, dw_hh, db;
    const bool need_b = s_b || ctx->needs_input_grad(3);
    if (esgd_lstm_persistent_ok((int)b, (int)h, 1)) {
      if (need_b && !s_b) db = at::zeros({4 * h}, f32);
      ck(esgd_lstm_persistent_bwd(gates.data_ptr(), fptr(c), dy.data_ptr(), w_hh.data_ptr(), dG.data_ptr(),
                                  !need_b ? nullptr : (s_b ? s_b->acc : fptr(db)), t, b, h, flag_ptr(x), st),
         "lstm backward recurrence");
    } else {
      Tensor dc = at::empty({b, h}, f32), dh = at::empty({h, b}, f32);
      ck(esgd_lstm_seq_bwd(gates.data_ptr(), fptr(c), dy.data_ptr(), w_hh.data_ptr(), dG.data_ptr(), fptr(dc), fptr(dh), t, b, h,
                           flag_ptr(x), st), "lstm backward recurrence");
      if (need_b) {
        db = dG.sum(0, false, at::kFloat);
        if (s_b) {
          at::from_blob(s_b->acc, {4 * h}, f32).add_(db);
          db = Tensor();
        }
      }
    }
    if (need_b && s_b) sink_done(s_b);
    if (ctx->needs_input_grad(0)) {
      dx = at::empty({t, b, in}, x.options());
      ck(gemm(dG.data_ptr(), w_ih.data_ptr(), dx.data_ptr(), t * b, in, 4 * h, 4 * h, in, in, false, true, 0, 1, nullptr, nullptr,
              nullptr, 0, x), "lstm input gradient");
    }
    if (s_ih || ctx->needs_input_grad(1)) {
      dw_ih = weight_grad(s_ih, x, dG.data_ptr(), w_ih, x.data_ptr(), t * b, 4 * h, in);
      if (s_ih) sink_done(s_ih);
    }
    if (s_hh || ctx->needs_input_grad(2)) {
      if (t > 1)
        dw_hh = weight_grad(s_hh, x, (const char*)dG.data_ptr() + b * 4 * h * 2, w_hh, y.data_ptr(), (t - 1) * b, 4 * h, h);
      else if (!s_hh)
        dw_hh = at::zeros_like(w_hh);
      if (s_hh) sink_done(s_hh);
    }
    variable_list out(8);
    out[0] = dx; out[1] = dw_ih; out[2] = dw_hh; out[3] = db;
    return out;
  }
};

// x [T, B, I] bf16, weights [4H, I] / [4H, H] bf16, bias [4H] fp32 -> h [T, B, H]; T, B, I, H multiples of 8 except T.
Tensor lstm_layer(const Tensor& x, const Tensor& w_ih, const Tensor& w_hh, const Tensor& bias) {
  TORCH_CHECK(x.dim() == 3 && w_ih.dim() == 2 && w_hh.dim() == 2, "lstm_layer: takes a 3-D input and 2-D weights, not ", x.sizes(), ", ",
              w_ih.sizes(), " and ", w_hh.sizes());
  const int64_t h = w_hh.size(1);
  TORCH_CHECK(w_hh.size(0) == 4 * h && w_ih.size(0) == 4 * h && w_ih.size(1) == x.size(2), "lstm_layer: weights ", w_ih.sizes(), " and ",
              w_hh.sizes(), " for an input of ", x.sizes());
  TORCH_CHECK(x.size(1) % 8 == 0 && x.size(2) % 8 == 0 && h % 8 == 0, "lstm_layer: takes multiples of 8");
  check_operand("lstm_layer", "the input", x, x, at::kBFloat16);
  check_operand("lstm_layer", "the input weight", w_ih, x, at::kBFloat16);
  check_operand("lstm_layer", "the recurrent weight", w_hh, x, at::kBFloat16);
  check_vector("lstm_layer", "the bias", bias, x, 4 * h);
  Sink s_ih = find_sink(w_ih), s_hh = find_sink(w_hh), s_b = find_sink(bias);
  sink_use(s_ih);
  sink_use(s_hh);
  sink_use(s_b);
  return LstmFn::apply(x, graph_input(w_ih, s_ih), graph_input(w_hh, s_hh), graph_input(bias, s_b), s_ih, s_hh, s_b,
                       anchor_for(x, s_ih || s_hh || s_b));
}

}  // namespace

PYBIND11_MODULE(_esgd_torch, m) {
  m.doc() = "autograd operators over the sm_100a kernels of eagersgd_b200";
  m.def("error_flag", &error_flag);
  m.def("zeros_f32", [](std::vector<int64_t> shape, at::Device d) { return zeros_f32(shape, d); });
  m.def("wgrad_splits", &wgrad_splits, py::arg("pixels"), py::arg("cout"), py::arg("cin"), py::arg("sms") = 148);
  m.def("conv2d", &conv2d);
  m.def("conv_bn_eval", &conv_bn_eval);
  py::class_<BnCoefficients, std::shared_ptr<BnCoefficients>>(m, "BnCoefficients").def(py::init<>()).def("compute", &BnCoefficients::compute);
  py::class_<EvalLayers, std::shared_ptr<EvalLayers>>(m, "EvalLayers")
      .def(py::init<py::dict, const std::vector<std::pair<py::object, py::object>>&, py::list, py::list>())
      .def("unchanged", &EvalLayers::unchanged)
      .def("coefficients", &EvalLayers::coefficients)
      .def_readonly("norms", &EvalLayers::norms);
  m.def("linear", &linear);
  m.def("bn_act", &bn_act);
  m.def("residual_block", &residual_block);
  m.def("residual_block_eval", &residual_block_eval);
  m.def("softmax_ce", &softmax_ce);
  m.def("lstm_layer", &lstm_layer);
  m.def("max_pool", &max_pool);
  m.def("avg_pool", &avg_pool);
  py::class_<ZeroArena, std::shared_ptr<ZeroArena>>(m, "ZeroArena")
      .def(py::init<>())
      .def("begin", &ZeroArena::begin)
      .def("end", &ZeroArena::end);
  py::class_<GradSinks, std::shared_ptr<GradSinks>>(m, "GradSinks")
      .def(py::init<std::vector<int>, py::function>())
      .def("add", &GradSinks::add)
      .def("begin_step", &GradSinks::begin_step)
      .def("clear_written", &GradSinks::clear_written)
      .def("set_active", &GradSinks::set_active)
      .def("active", &GradSinks::active)
      .def("used", &GradSinks::used)
      .def("written", &GradSinks::written)
      .def("hooked", &GradSinks::hooked)
      .def("close", &GradSinks::close);
}
