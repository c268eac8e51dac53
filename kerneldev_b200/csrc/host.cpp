// Host path of the operator as a torch extension: argument checks, the plan cache, allocations, the autograd
// node and the calls into libkd_attention.so, without a Python frame between flash_attention() and the launches.
//
// A forward or backward of a small problem is a few microseconds of kernels; the same path written in Python
// (ctypes structures, an autograd.Function whose backward takes the interpreter lock on the engine's thread) cost
// 65 us per forward and 185 us per backward whatever the size. The C ABI stays the boundary to the kernels: this
// file holds no device code and gets the library's entry points as addresses (bind), so that a test can bind
// another build of the library.
#include <torch/extension.h>

#include <ATen/TracerMode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <atomic>
#include <chrono>
#include <deque>
#include <list>
#include <memory>
#include <mutex>
#include <unordered_map>

#include "../../include/kd_attention.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

// Whether at::empty would do more than allocate: a dispatch mode or a function transform of the caller's sees this thread's operators, or
// torch fills new memory (deterministic algorithms).
bool allocations_are_seen() {
  const auto& context = at::globalContext();
  return !(c10::impl::tls_local_dispatch_key_set().included_ - c10::default_included_set).empty() ||
         (context.deterministicAlgorithms() && context.deterministicFillUninitializedMemory());
}

// Uninitialised device tensors from torch's CUDA allocator, where nothing sees them without the trip through the dispatcher, which is
// most of what at::empty costs: a forward allocates two and a backward five (0.4 us each: a forward's host time without its launch 5.0 -> 4.3 us).
Tensor empty_on(at::IntArrayRef sizes, at::ScalarType type, at::Device device) {
  if (allocations_are_seen()) return at::empty(sizes, at::TensorOptions().dtype(type).device(device));
  return Tensor(at::detail::empty_cuda(sizes, type, device, std::nullopt));
}
// in the memory order of a dense tensor, as at::empty_like
Tensor empty_like_of(const Tensor& like, at::ScalarType type) {
  if (!like.is_non_overlapping_and_dense() || allocations_are_seen()) return at::empty_like(like, like.options().dtype(type));
  return Tensor(at::detail::empty_strided_cuda(like.sizes(), like.strides(), type, like.device()));
}

// ---- the library -----------------------------------------------------------------------------------------------

struct Library {
  decltype(&kd_plan_layout_get) plan_layout_get = nullptr;
  decltype(&kd_classify) classify = nullptr;
  decltype(&kd_attn_fwd) attn_fwd = nullptr;
  decltype(&kd_attn_bwd) attn_bwd = nullptr;
  decltype(&kd_attn_bwd_hadamard) attn_bwd_hadamard = nullptr;
  decltype(&kd_attn_fwd_f32) attn_fwd_f32 = nullptr;
  decltype(&kd_attn_bwd_f32) attn_bwd_f32 = nullptr;
  decltype(&kd_hadamard) hadamard = nullptr;
  decltype(&kd_metadata_from_tokens) metadata_from_tokens = nullptr;
  decltype(&kd_cocktail_index) cocktail_index = nullptr;
  decltype(&kd_cocktail_scores) cocktail_scores = nullptr;
  decltype(&kd_cocktail_grad) cocktail_grad = nullptr;
  decltype(&kd_cast) cast = nullptr;
  decltype(&kd_last_error) last_error = nullptr;
};
Library lib;

template <typename F>
void take(F& slot, const py::dict& addresses, const char* name) {
  slot = reinterpret_cast<F>(addresses[name].cast<uintptr_t>());
}

void bind(const py::dict& a) {
  take(lib.plan_layout_get, a, "kd_plan_layout_get");
  take(lib.classify, a, "kd_classify");
  take(lib.attn_fwd, a, "kd_attn_fwd");
  take(lib.attn_bwd, a, "kd_attn_bwd");
  take(lib.attn_bwd_hadamard, a, "kd_attn_bwd_hadamard");
  take(lib.attn_fwd_f32, a, "kd_attn_fwd_f32");
  take(lib.attn_bwd_f32, a, "kd_attn_bwd_f32");
  take(lib.hadamard, a, "kd_hadamard");
  take(lib.metadata_from_tokens, a, "kd_metadata_from_tokens");
  take(lib.cocktail_index, a, "kd_cocktail_index");
  take(lib.cocktail_scores, a, "kd_cocktail_scores");
  take(lib.cocktail_grad, a, "kd_cocktail_grad");
  take(lib.cast, a, "kd_cast");
  take(lib.last_error, a, "kd_last_error");
}

// an entry point rejected its arguments or a CUDA call failed: _capi.KdError in Python, from the autograd engine's threads too
struct LibraryError : torch::PyTorchError {
  using torch::PyTorchError::PyTorchError;
  PyObject* python_type() override { return py::module_::import("kerneldev_b200._capi").attr("KdError").ptr(); }
};

void check(int rc) {
  if (rc != 0) throw LibraryError("libkd_attention: error " + std::to_string(rc) + ": " + lib.last_error());
}

#define KD_VALUE(cond, ...) TORCH_CHECK_VALUE(cond, __VA_ARGS__)

// ---- plans -----------------------------------------------------------------------------------------------------

constexpr uint32_t kStatusTimeout = KD_STATUS_TIMEOUT, kStatusSpanRange = KD_STATUS_SPAN_RANGE;

// Status mirrors of the plans: words of pinned blocks of 1024 (pinning is a slow, device-wide call). A word belongs to one plan
// as long as that lives. Words that come back go to the end of the queue: a kernel of a plan that is gone may still report.
class StatusWords {
 public:
  using Word = std::pair<Tensor, int>;   // the block and the word's index in it
  Word take() {
    std::lock_guard<std::mutex> lock(m_);
    if (free_.empty()) {
      const Tensor block = at::zeros({kBlock}, at::TensorOptions().dtype(at::kInt)).pin_memory();
      for (int i = 0; i < kBlock; ++i) free_.emplace_back(block, i);
    }
    Word w = std::move(free_.front());
    free_.pop_front();
    w.first.data_ptr<int32_t>()[w.second] = 0;
    return w;
  }
  void give_back(Word w) {
    std::lock_guard<std::mutex> lock(m_);
    free_.push_back(std::move(w));
  }

 private:
  static constexpr int kBlock = 1024;
  std::mutex m_;
  std::deque<Word> free_;
};
StatusWords& status_words() {
  static StatusWords* w = new StatusWords;   // never destroyed: plans outlive the statics of this file
  return *w;
}

bool check_every_launch() {
  const char* e = std::getenv("KD_CHECK_STATUS");
  return e != nullptr && e[0] == '1' && e[1] == 0;
}

// Whether a stream is being captured, and into which graph.
struct Capture {
  bool active;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  explicit Capture(cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    active = cudaStreamGetCaptureInfo_v2(stream, &status, &id, &graph) != cudaSuccess || status != cudaStreamCaptureStatusNone;
    if (status != cudaStreamCaptureStatusActive) graph = nullptr;
  }
};

struct Plan {
  int64_t B, T;
  at::Device device;
  kd_plan_layout layout;
  Tensor buf;
  struct Mirror {                  // the status word's copy in host memory
    StatusWords::Word word = status_words().take();
    volatile uint32_t* const at = reinterpret_cast<volatile uint32_t*>(word.first.data_ptr<int32_t>() + word.second);
    ~Mirror() { status_words().give_back(std::move(word)); }
  };
  std::shared_ptr<Mirror> mirror = std::make_shared<Mirror>();   // (the cache looks at those of plans that it has dropped)
  volatile uint32_t* host_word = mirror->at;
  // the status word and its mirror as tensors: views cost more than a launch, and only reports and tests want them
  Tensor status_dev() const { return buf.narrow(0, static_cast<int64_t>(layout.off_status), 4).view(at::kInt); }
  Tensor status_host() const { return mirror->word.first.narrow(0, mirror->word.second, 1); }
  // Memory of the caller's metadata, then of its converted copies, alive as long as the plan is cached. (Not the tensors: with a Python object one
  // counts as held by somebody for good.)
  std::vector<c10::Storage> keep;
  size_t asked_with = 0;      // of `keep`: the caller's
  at::cuda::CUDAStream built_on;
  at::cuda::CUDAEvent built;
  std::atomic<cudaStream_t> used_on{reinterpret_cast<cudaStream_t>(-1)};   // the stream of the plan's last eager launch

  std::atomic<unsigned long long> held_by{0};   // the last capture whose graph has been given this plan to hold

  // kd_attn_params.plan_ready for a launch. A captured launch says nothing about the stream it was captured from.
  bool ready_on(cudaStream_t stream, const Capture& capture) const { return !capture.active && used_on.load() == stream; }
  void launched_on(cudaStream_t stream, const Capture& capture) {
    if (!capture.active && used_on.load() != stream) used_on.store(stream);
  }

  Plan(int64_t B_, int64_t T_, at::Device dev, const OptTensor& in_span, const OptTensor& span_id, const OptTensor& is_prefix,
       const OptTensor& lens, bool causal, bool rules)
      : B(B_), T(T_), device(dev), built_on(at::cuda::getCurrentCUDAStream(dev.index())) {
    check(lib.plan_layout_get(static_cast<int32_t>(B), static_cast<int32_t>(T), &layout));
    // the caching allocator returns 512-byte aligned blocks, which covers the 256 the ABI asks for
    buf = empty_on({static_cast<int64_t>(layout.total)}, at::kByte, dev);
    for (const OptTensor* t : {&in_span, &span_id, &is_prefix, &lens})
      if (t->has_value() && (*t)->has_storage()) keep.push_back((*t)->storage());
    asked_with = keep.size();
    kd_meta meta{};
    meta.B = layout.B;
    meta.T = layout.T;
    meta.in_span = static_cast<const uint8_t*>(per_token(in_span, at::kBool, "in_span", &meta.in_span_stride_b));
    meta.span_id = static_cast<const int64_t*>(per_token(span_id, at::kLong, "span_id", &meta.span_id_stride_b));
    meta.is_prefix = static_cast<const uint8_t*>(per_token(is_prefix, at::kBool, "is_prefix", &meta.is_prefix_stride_b));
    if (lens.has_value()) {
      KD_VALUE(lens->scalar_type() == at::kInt && lens->dim() == 1 && lens->size(0) == B, "lens must be an int32 tensor of shape (B,)");
      KD_VALUE(lens->device() == device, "lens must live on ", device);
      Tensor l = lens->contiguous();
      keep.push_back(l.storage());
      meta.lens = l.data_ptr<int32_t>();
    }
    meta.causal = causal;
    meta.rules = rules;
    meta.status_mirror = const_cast<uint32_t*>(host_word);
    c10::cuda::CUDAGuard guard(dev);
    check(lib.classify(&meta, buf.data_ptr(), built_on.stream()));
    for (const c10::Storage& s : keep)   // the plan may go before the classifier has run: memory of other streams waits for it
      c10::cuda::CUDACachingAllocator::recordStream(s.data_ptr(), built_on);
    built.record(built_on);
    if (check_every_launch()) check_status();
  }

  const void* per_token(const OptTensor& o, at::ScalarType dtype, const char* name, int64_t* stride_b) {
    if (!o.has_value()) return nullptr;
    Tensor t = *o;
    KD_VALUE(t.dim() == 2 && t.size(0) == B && t.size(1) == T, name, " must have shape (B, T) = (", B, ", ", T, "), got ", t.sizes());
    KD_VALUE(t.device() == device, name, " must live on ", device);
    if (dtype == at::kBool) KD_VALUE(t.scalar_type() == at::kBool, name, " must be a torch.bool tensor (the rule negates it logically)");
    if (t.scalar_type() != dtype) t = t.to(dtype);
    if (t.stride(1) != 1) t = t.contiguous();
    keep.push_back(t.storage());
    *stride_b = t.stride(0);
    return t.data_ptr();
  }

  // Whether nobody else holds the memory of one of the tensors this plan was asked for with: its cache key names that memory, so that no
  // call can ask for it again.
  bool orphaned() const {
    for (size_t i = 0; i < asked_with; ++i) {
      size_t mine = 0;
      for (const c10::Storage& s : keep) mine += s.is_alias_of(keep[i]);
      if (keep[i].use_count() <= mine) return true;
    }
    return false;
  }

  // Orders the current stream after the classifier when the plan was built on another one.
  void use_on_current_stream() {
    auto cur = at::cuda::getCurrentCUDAStream(device.index());
    if (cur == built_on) return;
    built.block(cur);
    buf.record_stream(cur);
  }

  // Raises if a finished launch has reported a status to the host mirror. Never synchronises.
  void poll() {
    const uint32_t s = *host_word;
    if (s != 0) report(s);
  }

  // Synchronises the current stream, reads the device status word and raises if it is set.
  void check_status() {
    const uint32_t s = static_cast<uint32_t>(status_dev().item<int32_t>());
    if (s != 0) report(s);
  }

  [[noreturn]] void report(uint32_t s) {
    // both copies are cleared, so that one event is reported once and later launches start clean
    status_dev().zero_();
    *host_word = 0;
    raise_status(s);
  }

  [[noreturn]] static void raise_status(uint32_t s) {
    TORCH_CHECK_VALUE((s & kStatusSpanRange) == 0, "span_id values must fit in 24 signed bits (|span_id| < 2**23)");
    char hex[16], site[16];
    snprintf(hex, sizeof hex, "0x%08x", s);
    snprintf(site, sizeof site, "0x%x", s & 0xFFFFu);
    TORCH_CHECK((s & kStatusTimeout) == 0, "a device-side wait timed out (status ", hex, ", wait site ", site,
                "); the results of that launch are invalid");
    TORCH_CHECK(false, "device status ", hex);
  }

  void after_launch() {
    if (check_every_launch()) check_status();
  }
};
using PlanPtr = std::shared_ptr<Plan>;

// Plans that graphs have let go of. The driver runs a graph's destructors on a thread of its own, where no CUDA call may be made, and a plan
// that goes frees memory and an event: the next look-up of a plan does.
class LetGo {
 public:
  void add(PlanPtr plan) {
    std::lock_guard<std::mutex> lock(m_);
    plans_.push_back(std::move(plan));
    any_.store(true);
  }
  void clear() {
    if (!any_.load()) return;
    std::vector<PlanPtr> gone;   // destroyed after the lock is released
    std::lock_guard<std::mutex> lock(m_);
    gone.swap(plans_);
    any_.store(false);
  }

 private:
  std::mutex m_;
  std::vector<PlanPtr> plans_;
  std::atomic<bool> any_{false};
};
LetGo& let_go() {
  static LetGo* l = new LetGo;   // never destroyed: graphs outlive the statics of this file
  return *l;
}

// A captured launch has the plan's address and nothing else, and the cache may drop the plan: the graph keeps it, as do the graphs made from it.
void hold_for_graph(const PlanPtr& plan, const Capture& capture) {
  if (capture.graph == nullptr || plan->held_by.load() == capture.id) return;
  auto held = std::make_unique<PlanPtr>(plan);
  cudaUserObject_t object;
  C10_CUDA_CHECK(cudaUserObjectCreate(&object, held.get(), [](void* p) {
    std::unique_ptr<PlanPtr> h(static_cast<PlanPtr*>(p));
    let_go().add(std::move(*h));
  }, 1, cudaUserObjectNoDestructorSync));
  held.release();
  const cudaError_t e = cudaGraphRetainUserObject(capture.graph, object, 1, cudaGraphUserObjectMove);
  if (e != cudaSuccess) cudaUserObjectRelease(object, 1);
  C10_CUDA_CHECK(e);
  plan->held_by.store(capture.id);
}

// The cache key: identity, version and geometry of the metadata tensors (the plan keeps their memory alive, so an address
// cannot be reused while its plan is cached) and the flags of the mask.
struct PlanKey {
  struct Slot {
    const void* ptr = nullptr;
    uint32_t version = 0;
    int64_t s0 = 0, s1 = 0, st0 = 0, st1 = 0;
    int32_t dtype = -1, dim = 0;
    bool operator==(const Slot& o) const {
      return ptr == o.ptr && version == o.version && s0 == o.s0 && s1 == o.s1 && st0 == o.st0 && st1 == o.st1 && dtype == o.dtype && dim == o.dim;
    }
  };
  int64_t B, T;
  int32_t device, flags;
  Slot slot[4];
  bool operator==(const PlanKey& o) const {
    return B == o.B && T == o.T && device == o.device && flags == o.flags && slot[0] == o.slot[0] && slot[1] == o.slot[1] &&
           slot[2] == o.slot[2] && slot[3] == o.slot[3];
  }
};
struct PlanKeyHash {
  size_t operator()(const PlanKey& k) const {
    size_t h = static_cast<size_t>(k.B * 1000003 + k.T) * 31 + static_cast<size_t>(k.device * 4 + k.flags);
    for (const auto& s : k.slot) h = (h ^ reinterpret_cast<uintptr_t>(s.ptr) ^ s.version) * 0x9E3779B97F4A7C15ull;
    return h;
  }
};

class PlanCache {
 public:
  // Plans kept: so many, and so many bytes of device memory with the newest (the visibility words of a plan are a bit for each pair of tokens, up to
  // 256 MB), but the newest always.
  static constexpr size_t kSize = 64, kBytes = size_t(512) << 20;
  PlanPtr find(const PlanKey& key) {
    std::lock_guard<std::mutex> lock(m_);
    auto it = map_.find(key);
    if (it == map_.end()) return nullptr;
    order_.splice(order_.end(), order_, it->second);
    return it->second->second;
  }
  // Raises if a launch of a plan that an earlier insertion has dropped, or this one drops, has reported a status.
  void insert(const PlanKey& key, PlanPtr plan) {
    std::vector<PlanPtr> evicted;   // destroyed after the lock is released
    if (const uint32_t s = add(key, std::move(plan), evicted)) Plan::raise_status(s);
  }
  std::vector<PlanPtr> values() {
    std::lock_guard<std::mutex> lock(m_);
    std::vector<PlanPtr> v;
    for (auto& e : order_) v.push_back(e.second);
    return v;
  }
  void clear() {
    std::list<std::pair<PlanKey, PlanPtr>> gone;
    std::lock_guard<std::mutex> lock(m_);
    map_.clear();
    gone.swap(order_);
    bytes_ = 0;
  }

 private:
  using Entries = std::list<std::pair<PlanKey, PlanPtr>>;
  uint32_t add(const PlanKey& key, PlanPtr plan, std::vector<PlanPtr>& evicted) {
    std::lock_guard<std::mutex> lock(m_);
    if (map_.count(key)) return 0;
    // Plans that no call can ask for any more go back to the allocator at once: a training step's plan has the memory of the last
    // one's, and not a new block until the cache is full (a first pass at 3 x 1357 tokens 175 us, 158 with this).
    for (auto it = order_.begin(); it != order_.end();) it = it->second->orphaned() ? drop(it, evicted) : std::next(it);
    bytes_ += plan->layout.total;
    order_.emplace_back(key, std::move(plan));
    map_[key] = std::prev(order_.end());
    while (order_.size() > kSize || (bytes_ > kBytes && order_.size() > 1)) drop(order_.begin(), evicted);
    // Their launches may still run, and no call looks at these plans any more: the last backward of a step would report to nobody.
    for (const PlanPtr& p : evicted) dropped_.push_back(p->mirror);
    while (dropped_.size() > kSize) dropped_.pop_front();
    for (auto it = dropped_.begin(); it != dropped_.end(); ++it) {
      volatile uint32_t* const word = (*it)->at;
      const uint32_t s = *word;
      if (s == 0) continue;
      *word = 0;
      dropped_.erase(it);
      return s;
    }
    return 0;
  }
  Entries::iterator drop(Entries::iterator it, std::vector<PlanPtr>& gone) {
    bytes_ -= it->second->layout.total;
    gone.push_back(std::move(it->second));
    map_.erase(it->first);
    return order_.erase(it);
  }
  std::mutex m_;
  size_t bytes_ = 0;   // of the plans in the cache
  Entries order_;   // least recently used first
  std::deque<std::shared_ptr<Plan::Mirror>> dropped_;   // status words of the last kSize plans that left for others
  std::unordered_map<PlanKey, Entries::iterator, PlanKeyHash> map_;
};
PlanCache& cache() {
  static PlanCache* c = new PlanCache;   // never destroyed: at exit the CUDA context may be gone before it
  return *c;
}

bool fill_slot(PlanKey::Slot& s, const OptTensor& t) {
  if (!t.has_value()) return true;
  if (t->is_inference()) return false;   // no version counter: a rewrite could not be told from the original
  s.ptr = t->data_ptr();
  s.version = static_cast<uint32_t>(t->_version());
  s.dim = static_cast<int32_t>(t->dim());
  s.dtype = static_cast<int32_t>(t->scalar_type());
  if (s.dim > 0) { s.s0 = t->size(0); s.st0 = t->stride(0); }
  if (s.dim > 1) { s.s1 = t->size(1); s.st1 = t->stride(1); }
  return true;
}

PlanPtr get_plan(int64_t B, int64_t T, at::Device device, const OptTensor& in_span, const OptTensor& span_id,
                 const OptTensor& is_prefix, const OptTensor& lens, bool causal, bool rules) {
  if (!device.has_index()) device = at::Device(device.type(), at::cuda::current_device());
  let_go().clear();
  PlanKey key{B, T, device.index(), (causal ? 1 : 0) | (rules ? 2 : 0), {}};
  const bool keyed = fill_slot(key.slot[0], in_span) && fill_slot(key.slot[1], span_id) && fill_slot(key.slot[2], is_prefix) &&
                     fill_slot(key.slot[3], lens);
  if (keyed) {
    if (PlanPtr p = cache().find(key)) {
      p->use_on_current_stream();
      p->poll();
      return p;
    }
  }
  auto p = std::make_shared<Plan>(B, T, device, in_span, span_id, is_prefix, lens, causal, rules);
  if (keyed) cache().insert(key, p);
  return p;
}

// ---- kernel calls ----------------------------------------------------------------------------------------------

int dtype_code(at::ScalarType t) { return t == at::kHalf ? KD_F16 : t == at::kBFloat16 ? KD_BF16 : KD_F32; }

kd_tensor desc(const Tensor& t) { return kd_tensor{t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)}; }

// rows of 16-byte pieces: unit stride along D, pointer and strides multiples of 16 bytes
bool aligned(const Tensor& t) {
  const int64_t es = t.element_size();
  bool ok = t.stride(3) == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  for (int i = 0; i < 3; ++i) ok = ok && (t.stride(i) * es) % 16 == 0;
  return ok;
}
// ... which TMA can describe: positive strides
bool tma_ready(const Tensor& t) { return aligned(t) && t.stride(0) > 0 && t.stride(1) > 0 && t.stride(2) > 0; }

// t itself when TMA can describe it, else one contiguous copy
Tensor usable(const Tensor& t) { return tma_ready(t) ? t : t.contiguous(); }

Tensor empty_out(const Tensor& like, bool like_input, at::ScalarType type) {
  // empty_like keeps the strides of a dense tensor, e.g. (B,T,H,D) memory seen as (B,H,T,D)
  return like_input ? empty_like_of(like, type) : empty_on(like.sizes(), type, like.device());
}
Tensor empty_out(const Tensor& like, bool like_input) { return empty_out(like, like_input, like.scalar_type()); }

kd_attn_params params(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Plan& plan,
                      double sm_scale) {
  kd_attn_params p{};
  p.B = static_cast<int32_t>(q.size(0));
  p.H = static_cast<int32_t>(q.size(1));
  p.T = static_cast<int32_t>(q.size(2));
  p.D = static_cast<int32_t>(q.size(3));
  p.dtype = dtype_code(q.scalar_type());
  p.sm_scale = static_cast<float>(sm_scale);
  p.q = desc(q);
  p.k = desc(k);
  p.v = desc(v);
  if (o.defined()) p.o = desc(o);
  p.lse = lse.defined() ? lse.data_ptr<float>() : nullptr;
  p.plan = plan.buf.data_ptr();
  return p;
}

// `o32`: receives O as float32 (of a float32 call); the 16-bit O is undefined then unless it is wanted.
std::tuple<Tensor, Tensor> forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const PlanPtr& plan, double sm_scale,
                                   bool like_input, bool want_lse = true, Tensor* o32 = nullptr, bool want_o16 = true) {
  const Tensor q = usable(q_), k = usable(k_), v = usable(v_);
  Tensor o, lse;
  if (want_o16) o = empty_out(q, like_input);
  kd_attn_f32 f{};
  if (o32 != nullptr) {
    *o32 = empty_out(q, like_input, at::kFloat);
    f.o = desc(*o32);
  }
  if (want_lse) lse = empty_on({q.size(0), q.size(1), q.size(2)}, at::kFloat, q.device());
  kd_attn_params p = params(q, k, v, o, lse, *plan, sm_scale);
  plan->poll();
  c10::cuda::CUDAGuard guard(q.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  const Capture capture(stream);
  hold_for_graph(plan, capture);
  p.plan_ready = plan->ready_on(stream, capture) ? 1 : 0;
  check(o32 != nullptr ? lib.attn_fwd_f32(&p, &f, stream) : lib.attn_fwd(&p, stream));
  plan->launched_on(stream, capture);
  plan->after_launch();
  return {o, lse};
}

// f32: of a float32 call; dO may be float32, and dQ, dK and dV are.
// signs: q and k are transforms with these, and dQ and dK are wanted of what they were made from (not deterministic).
// `phases` selects a part of the backward (kd_attn_params.bwd_phases); defined tensors among dq .. dq_acc are reused.
std::tuple<Tensor, Tensor, Tensor> backward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& o, const Tensor& lse,
                                            const Tensor& d_o_, const PlanPtr& plan, double sm_scale, int phases, Tensor dq, Tensor dk,
                                            Tensor dv, Tensor delta, Tensor dq_acc, bool like_input, bool deterministic, bool f32 = false,
                                            const float* signs = nullptr) {
  const Tensor q = usable(q_), k = usable(k_), v = usable(v_);
  kd_attn_f32 f{};
  Tensor d_o;
  const bool rounds = f32 && d_o_.scalar_type() == at::kFloat && aligned(d_o_);
  if (rounds) d_o = empty_like_of(d_o_, at::kHalf);
  if (rounds && tma_ready(d_o)) {
    f.d_o = desc(d_o_);   // the delta kernel fills d_o
  } else {
    d_o = usable(f32 ? d_o_.to(at::kHalf) : d_o_);
  }
  if (!dq.defined()) {
    const auto type = f32 ? at::kFloat : q.scalar_type();
    dq = empty_out(q, like_input, type);
    dk = empty_out(k, like_input, type);
    dv = empty_out(v, like_input, type);
  }
  if (!delta.defined()) delta = empty_on({q.size(0), q.size(1), q.size(2)}, at::kFloat, q.device());
  const bool fused = !deterministic;
  // rows as wide as the kernel's tile (kd_workspace_bytes_fused)
  if (fused && !f32 && !dq_acc.defined()) dq_acc = empty_on({q.size(0), q.size(1), q.size(2), q.size(3) <= 64 ? 64 : 128}, at::kFloat, q.device());
  kd_attn_params p = params(q, k, v, o, lse, *plan, sm_scale);
  p.d_o = desc(d_o);
  (f32 ? f.dq : p.dq) = desc(dq);
  (f32 ? f.dk : p.dk) = desc(dk);
  (f32 ? f.dv : p.dv) = desc(dv);
  p.delta = delta.data_ptr<float>();
  p.bwd_phases = phases;
  if (fused) {
    p.bwd_mode = KD_BWD_FUSED;
    if (!f32) p.dq_acc = dq_acc.data_ptr<float>();
  }
  plan->poll();
  c10::cuda::CUDAGuard guard(q.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  const Capture capture(stream);
  hold_for_graph(plan, capture);
  p.plan_ready = plan->ready_on(stream, capture) ? 1 : 0;
  check(f32 ? lib.attn_bwd_f32(&p, &f, stream) : signs != nullptr ? lib.attn_bwd_hadamard(&p, signs, stream) : lib.attn_bwd(&p, stream));
  plan->after_launch();
  return {dq, dk, dv};
}

// float32 <-> float16 copies of up to three tensors of one shape, in the memory order of the originals, by one kernel.
// Tensors whose strides it cannot address go through the library's conversion.
std::array<Tensor, KD_CAST_MAX> cast(std::initializer_list<Tensor> in, at::ScalarType to) {
  std::array<Tensor, KD_CAST_MAX> out;
  kd_tensor src[KD_CAST_MAX], dst[KD_CAST_MAX];
  int n = 0, slot = 0;
  const Tensor& first = *in.begin();
  for (const Tensor& x : in) {
    Tensor y = empty_like_of(x, to);
    if (x.numel() > 0 && x.scalar_type() != to && aligned(x) && aligned(y)) {
      src[n] = desc(x);
      dst[n++] = desc(y);
    } else {
      y = x.to(to);
    }
    out[slot++] = y;
  }
  if (n > 0) {
    c10::cuda::CUDAGuard guard(first.device());
    check(lib.cast(src, dst, n, static_cast<int32_t>(first.size(0)), static_cast<int32_t>(first.size(1)), static_cast<int32_t>(first.size(2)),
                   static_cast<int32_t>(first.size(3)), to == at::kFloat ? 1 : 0, at::cuda::getCurrentCUDAStream()));
  }
  return out;
}

Tensor hadamard(const Tensor& x_, const OptTensor& signs, bool inverse) {
  const Tensor x = usable(x_);
  Tensor y = empty_on(x.sizes(), x.scalar_type(), x.device());
  const kd_tensor xs = desc(x), ys = desc(y);
  c10::cuda::CUDAGuard guard(x.device());
  check(lib.hadamard(&xs, &ys, static_cast<int32_t>(x.size(0)), static_cast<int32_t>(x.size(1)), static_cast<int32_t>(x.size(2)),
                     static_cast<int32_t>(x.size(3)), dtype_code(x.scalar_type()), signs.has_value() ? signs->data_ptr<float>() : nullptr,
                     inverse ? 1 : 0, at::cuda::getCurrentCUDAStream()));
  return y;
}

// ---- autograd --------------------------------------------------------------------------------------------------

struct Options {
  double sm_scale;
  bool like_input, deterministic;
};

// dQ, dK, dV of one flash_attention call. Saves the operands the kernels read: for float32 tensors their float16
// copies, with incoherent processing the transformed Q and K.
struct AttentionBackward : torch::autograd::Node {
  torch::autograd::SavedVariable q, k, v, o, lse;
  PlanPtr plan;
  Options opt;
  OptTensor signs;
  bool widen;   // float32 tensors: gradients go back as float32

  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    torch::autograd::variable_list out(3);
    Tensor tq, tk, tv, to, tlse;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      tq = q.unpack();
      tk = k.unpack();
      tv = v.unpack();
      to = o.unpack(shared_from_this());
      tlse = lse.unpack();
    }
    at::NoGradGuard no_grad;
    // a gradient that a later node left undefined counts as zeros, as for autograd.Function
    const bool direct = widen && !signs.has_value();   // the transform of dQ and dK works on 16-bit tensors
    Tensor d_o = grads[0].defined() ? grads[0] : at::zeros_like(to);
    // The engine brings a gradient like the output; a node that is called by hand may get any, which the kernels would read as what it is not.
    KD_VALUE(d_o.sizes() == to.sizes() && d_o.device() == to.device(), "the gradient of an output of shape ", to.sizes(), " on ", to.device(), " has shape ",
             d_o.sizes(), " on ", d_o.device());
    if (grads[0].defined()) d_o = d_o.to(widen ? at::kFloat : to.scalar_type());
    if (widen && !direct) d_o = cast({d_o}, at::kHalf)[0];
    const bool with_gradients = signs.has_value() && !opt.deterministic;
    auto [dq, dk, dv] = backward(tq, tk, tv, to, tlse, d_o, plan, opt.sm_scale, 0, {}, {}, {}, {}, {}, opt.like_input, opt.deterministic, direct,
                                 with_gradients ? signs->data_ptr<float>() : nullptr);
    if (signs.has_value() && !with_gradients) {
      // y = x diag(s) W / sqrt(D) with W symmetric, so dx = dy W / sqrt(D) diag(s)
      dq = hadamard(dq, signs, true);
      dk = hadamard(dk, signs, true);
    }
    if (widen && !direct) {
      auto wide = cast({dq, dk, dv}, at::kFloat);
      dq = wide[0];
      dk = wide[1];
      dv = wide[2];
    }
    out[0] = dq;
    out[1] = dk;
    out[2] = dv;
    return out;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    q.reset_data();
    k.reset_data();
    v.reset_data();
    o.reset_data();
    lse.reset_data();
  }
  std::string name() const override { return "FlashAttentionBackward"; }
};

// A trace would hold the allocation of the results and not the kernels that fill them.
void refuse_tracing(const char* name) {
  using c10::impl::TorchDispatchModeTLS;
  const bool recorded = TorchDispatchModeTLS::any_modes_set() && TorchDispatchModeTLS::get_mode(c10::impl::TorchDispatchModeKey::PROXY).has_value();
  TORCH_CHECK(!at::tracer::impl::is_dispatch_enabled() && !recorded, name, " cannot be traced: its kernels are not recorded");
}

// The nodes of this file have no formula for tangents: without this check they would be lost without a word.
template <typename... T>
void refuse_forward_ad(const char* name, const T&... inputs) {
  TORCH_CHECK_NOT_IMPLEMENTED(!(inputs._fw_grad(/*level=*/0).defined() || ...), name, " does not support forward mode AD");
}

void check_inputs(const Tensor& q, const Tensor& k, const Tensor& v) {
  KD_VALUE(q.dim() == 4, "q, k, v must be (batch, heads, time, head_dim)");
  KD_VALUE(q.sizes() == k.sizes() && q.sizes() == v.sizes(), "q, k, v must have the same shape, got ", q.sizes(), ", ", k.sizes(), ", ", v.sizes());
  TORCH_CHECK(q.is_cuda(), "flash_attention runs on CUDA sm_100 devices only; there is no CPU path");
  const auto t = q.scalar_type();
  KD_VALUE((t == at::kHalf || t == at::kBFloat16 || t == at::kFloat) && k.scalar_type() == t && v.scalar_type() == t,
           "q, k, v must share dtype float16, bfloat16 or float32");
  KD_VALUE(q.size(3) % 16 == 0 && q.size(3) >= 16 && q.size(3) <= 128, "head_dim ", q.size(3), " is not supported (a multiple of 16 from 16 to 128)");
  KD_VALUE(k.device() == q.device() && v.device() == q.device(), "q, k, v must be on the same device");
}

std::tuple<Tensor, Tensor> attention(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& lens, std::optional<double> sm_scale,
                                     bool causal, const OptTensor& in_span, const OptTensor& span_id, const OptTensor& is_prefix, bool rules,
                                     const OptTensor& signs, bool like_input, bool deterministic, bool return_lse) {
  check_inputs(q, k, v);
  refuse_forward_ad("flash_attention", q, k, v);
  refuse_tracing("flash_attention");
  const double scale = sm_scale.has_value() ? *sm_scale : 1.0 / std::sqrt(static_cast<double>(q.size(3)));
  KD_VALUE(scale > 0.0 && std::isfinite(scale), "sm_scale must be positive and finite");
  PlanPtr plan = get_plan(q.size(0), q.size(2), q.device(), in_span, span_id, is_prefix, lens, causal, rules);
  const bool track = at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
  const bool f32 = q.scalar_type() == at::kFloat;
  Tensor o, lse, q2, k2, v2, o16;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    if (f32) {
      auto half = cast({q, k, v}, at::kHalf);
      q2 = half[0];
      k2 = half[1];
      v2 = half[2];
    } else {
      q2 = q;
      k2 = k;
      v2 = v;
    }
    if (signs.has_value()) {
      q2 = hadamard(q2, signs, false);
      k2 = hadamard(k2, signs, false);
    }
    std::tie(o16, lse) = forward(q2, k2, v2, plan, scale, like_input, return_lse || track, f32 ? &o : nullptr, !f32 || track);
    if (!f32) o = o16;
  }
  if (track) {
    auto node = std::shared_ptr<AttentionBackward>(new AttentionBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
    node->plan = std::move(plan);
    node->opt = Options{scale, like_input, deterministic};
    node->signs = signs;
    node->widen = f32;
    torch::autograd::set_history(o, node);
    node->q = torch::autograd::SavedVariable(q2, false);
    node->k = torch::autograd::SavedVariable(k2, false);
    node->v = torch::autograd::SavedVariable(v2, false);
    node->o = torch::autograd::SavedVariable(o16, !f32);   // for float32 tensors o16 is a copy of its own, not the output
    node->lse = torch::autograd::SavedVariable(lse, false);
  }
  return {o, lse};
}

// ---- metadata --------------------------------------------------------------------------------------------------

std::tuple<Tensor, Tensor, Tensor> metadata_from_tokens(const Tensor& tokens_, int64_t tok_span, int64_t tok_es, int64_t tok_cls, int64_t tok_maskq) {
  const Tensor tokens = tokens_.stride(1) == 1 ? tokens_ : tokens_.contiguous();
  const int64_t B = tokens.size(0), T = tokens.size(1);
  Tensor in_span = empty_on({B, T}, at::kBool, tokens.device());
  Tensor span_id = empty_on({B, T}, at::kLong, tokens.device());
  Tensor is_prefix = empty_on({B, T}, at::kBool, tokens.device());
  c10::cuda::CUDAGuard guard(tokens.device());
  check(lib.metadata_from_tokens(tokens.data_ptr<int64_t>(), B > 1 ? tokens.stride(0) : std::max<int64_t>(T, 1), static_cast<int32_t>(B),
                                 static_cast<int32_t>(T), tok_span, tok_es, tok_cls, tok_maskq, static_cast<uint8_t*>(in_span.data_ptr()),
                                 span_id.data_ptr<int64_t>(), static_cast<uint8_t*>(is_prefix.data_ptr()), at::cuda::getCurrentCUDAStream()));
  return {in_span, span_id, is_prefix};
}

// ---- cocktail-party head ---------------------------------------------------------------------------------------

// the marker index of a batch as one int32 tensor: starts and ends (B,T each), their counts and the first [MASK] (B each)
int64_t index_words(int64_t B, int64_t T) { return 2 * B * T + 3 * B; }
void point_into_index(kd_cocktail& p, const Tensor& index) {
  const int64_t rows = static_cast<int64_t>(p.B) * p.T;
  const int32_t* words = index.data_ptr<int32_t>();
  p.starts = words;
  p.ends = words + rows;
  p.n_starts = words + 2 * rows;
  p.n_ends = p.n_starts + p.B;
  p.first_mask = p.n_ends + p.B;
}

// Gradient of the gradient. With h(x) the means and the [MASK]'s embedding of x, which are linear in x, gx is linear in ds and in
// h(x), and so is what comes back for a gradient v of gx: gx's own formula with h(v) for x, and for ds_j
// <h_ctx(x), h_j(v)> + <h_ctx(v), h_j(x)>.
struct CocktailDoubleBackward : torch::autograd::Node {
  torch::autograd::SavedVariable ds, h, index;
  kd_cocktail p{};   // shapes and type

  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    torch::autograd::variable_list out(2);
    if (!grads[0].defined()) return out;
    Tensor tds, th, ti;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      tds = ds.unpack();
      th = h.unpack();
      ti = index.unpack();
    }
    at::NoGradGuard no_grad;
    const Tensor v = grads[0].contiguous();
    tds = tds.contiguous();
    ti = ti.contiguous();
    Tensor unused = at::empty_like(tds), hv = at::empty({p.B, p.S + 1, p.C}, v.options().dtype(at::kFloat)), gx = at::empty_like(v);
    c10::cuda::CUDAGuard guard(v.device());
    const cudaStream_t stream = at::cuda::getCurrentCUDAStream();
    kd_cocktail q = p;
    point_into_index(q, ti);
    q.x = v.data_ptr();
    q.x_sb = v.stride(0);
    q.x_st = v.stride(1);
    q.scores = unused.data_ptr();
    q.h = hv.data_ptr<float>();
    check(lib.cocktail_scores(&q, stream));
    q.scores = tds.data_ptr();
    q.gx = gx.data_ptr();
    check(lib.cocktail_grad(&q, stream));
    auto dots = [&](const Tensor& ctx, const Tensor& means) {   // (B,S)
      return (ctx.narrow(1, p.S, 1) * means.narrow(1, 0, p.S)).sum(2);
    };
    out[0] = (dots(th, hv) + dots(hv, th)).to(tds.scalar_type());
    out[1] = gx;
    return out;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    ds.reset_data();
    h.reset_data();
    index.reset_data();
  }
  std::string name() const override { return "CocktailScoresDoubleBackward"; }
};

// gradient of cocktail_scores: one kernel that writes every row of grad_x
struct CocktailBackward : torch::autograd::Node {
  torch::autograd::SavedVariable h, index;
  kd_cocktail p{};   // shapes and type; the pointers are those of the unpacked tensors, which need not be the saved ones
  Tensor like;     // an empty tensor with x's options

  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    torch::autograd::variable_list out(1);
    Tensor th, ti;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      th = h.unpack();
      ti = index.unpack();
    }
    const bool again = at::GradMode::is_enabled() && p.S > 0 && p.T > 0 && p.C > 0;   // create_graph: gx is differentiated in its turn
    at::NoGradGuard no_grad;
    const Tensor ds = grads[0].defined() ? grads[0].contiguous() : at::zeros({p.B, p.S}, like.options());
    // without a span nothing reaches x, and there is no kernel to write the zeros
    Tensor gx = p.S == 0 ? at::zeros({p.B, p.T, p.C}, like.options()) : empty_on({p.B, p.T, p.C}, like.scalar_type(), like.device());
    kd_cocktail q = p;
    ti = ti.contiguous();
    th = th.contiguous();
    point_into_index(q, ti);
    q.scores = ds.data_ptr();
    q.h = th.data_ptr<float>();
    q.gx = gx.data_ptr();
    c10::cuda::CUDAGuard guard(gx.device());
    check(lib.cocktail_grad(&q, at::cuda::getCurrentCUDAStream()));
    if (again) {
      auto node = std::shared_ptr<CocktailDoubleBackward>(new CocktailDoubleBackward(), torch::autograd::deleteNode);
      node->set_next_edges({grads[0].defined() ? torch::autograd::impl::gradient_edge(grads[0]) : torch::autograd::Edge(), next_edge(0)});
      node->p = p;
      torch::autograd::set_history(gx, node);
      node->ds = torch::autograd::SavedVariable(ds, false);
      node->h = torch::autograd::SavedVariable(th, false);
      node->index = torch::autograd::SavedVariable(ti, false);
    }
    out[0] = gx;
    return out;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    h.reset_data();
    index.reset_data();
  }
  std::string name() const override { return "CocktailScoresBackward"; }
};

Tensor cocktail_scores(const Tensor& x_, const Tensor& tokens_, int64_t tok_span, int64_t tok_es, int64_t tok_mask) {
  KD_VALUE(tokens_.dim() == 2 && tokens_.scalar_type() == at::kLong, "tokens must be an int64 tensor of shape (batch, time)");
  TORCH_CHECK(tokens_.is_cuda(), "span_index runs on CUDA devices only; there is no CPU path");
  const auto t = x_.scalar_type();
  KD_VALUE(x_.dim() == 3 && (t == at::kHalf || t == at::kBFloat16 || t == at::kFloat), "x_embed must be (batch, time, dim) in float16, bfloat16 or float32");
  TORCH_CHECK(x_.is_cuda(), "span_means runs on CUDA devices only; there is no CPU path");
  // one row may have more embeddings than tokens: the rest belongs to no span
  KD_VALUE(x_.size(0) == tokens_.size(0) && (x_.size(1) == tokens_.size(1) || (x_.size(0) == 1 && x_.size(1) > tokens_.size(1))) &&
               x_.device() == tokens_.device(),
           "x_embed and tokens must have the same batch, time and device");
  refuse_forward_ad("cocktail_scores", x_);
  refuse_tracing("cocktail_scores");
  const int64_t B = x_.size(0), T = x_.size(1), C = x_.size(2);
  const bool track = at::GradMode::is_enabled() && x_.requires_grad();
  Tensor scores, h, index;
  kd_cocktail p{};
  {
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor tokens = tokens_.stride(1) == 1 ? tokens_ : tokens_.contiguous();
    const Tensor x = x_.stride(2) == 1 ? x_ : x_.contiguous();
    index = empty_on({index_words(B, T)}, at::kInt, tokens.device());
    p.B = static_cast<int32_t>(B);
    p.T = static_cast<int32_t>(T);
    p.C = static_cast<int32_t>(C);
    p.dtype = t == at::kFloat ? KD_F32 : dtype_code(t);
    point_into_index(p, index);
    auto out = [](const int32_t* words) { return const_cast<int32_t*>(words); };
    Tensor counts = at::empty({B}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    std::fill_n(counts.data_ptr<int32_t>(), B, -1);   // not there yet
    c10::cuda::CUDAGuard guard(x.device());
    auto stream = at::cuda::getCurrentCUDAStream();
    const int64_t n_tokens = tokens.size(1);
    check(lib.cocktail_index(tokens.data_ptr<int64_t>(), B > 1 ? tokens.stride(0) : std::max<int64_t>(n_tokens, 1), static_cast<int32_t>(B),
                             static_cast<int32_t>(n_tokens), tok_span, tok_es, tok_mask, out(p.starts), out(p.ends), out(p.n_starts), out(p.n_ends), out(p.first_mask),
                             counts.data_ptr<int32_t>(), stream));
    int32_t S = 0;   // the width of the scores has to be known here: the one wait for the device
    if (B > 0 && n_tokens > 0) {
      // The counts arrive while the kernel still writes the markers. A wait for the stream would add the rest of the kernel, its end and
      // the wake-up (16 x 4096 x 1024, forward and backward on an idle stream 72.2 -> 61 us). It follows only where they never come, or take
      // long because of work queued ahead: such a call gains nothing, and its thread has turned for 200 us where the wait turns as well.
      volatile int32_t* words = counts.data_ptr<int32_t>();
      const auto give_up = std::chrono::steady_clock::now() + std::chrono::microseconds(200);
      int64_t b = 0;
      for (; b < B; ++b) {
        while (words[b] < 0 && std::chrono::steady_clock::now() < give_up) {}
        if (words[b] < 0) break;
      }
      if (b < B) C10_CUDA_CHECK(cudaStreamSynchronize(stream));
      for (b = 0; b < B; ++b) S = std::max(S, static_cast<int32_t>(words[b]));
    }
    scores = C == 0 ? at::zeros({B, S}, x.options()) : empty_on({B, S}, x.scalar_type(), x.device());
    if (track) h = empty_on({B, S + 1, C}, at::kFloat, x.device());
    p.x = x.data_ptr();
    p.x_sb = x.stride(0);
    p.x_st = x.stride(1);
    p.S = S;
    p.scores = scores.data_ptr();
    p.h = track ? h.data_ptr<float>() : nullptr;
    check(lib.cocktail_scores(&p, stream));
  }
  if (track) {
    auto node = std::shared_ptr<CocktailBackward>(new CocktailBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x_));
    node->p.B = p.B;
    node->p.T = p.T;
    node->p.C = p.C;
    node->p.S = p.S;
    node->p.dtype = p.dtype;
    node->like = empty_on({0}, x_.scalar_type(), x_.device());
    torch::autograd::set_history(scores, node);
    node->h = torch::autograd::SavedVariable(h, false);
    node->index = torch::autograd::SavedVariable(index, false);
  }
  return scores;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.doc() = "host path of the attention operator";
  // torch's own translation (out of memory, Python errors raised in hooks, LibraryError), for this module's functions alone
  py::register_local_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const py::builtin_exception&) {
      throw;
    } catch (const std::exception&) {
      torch::translate_exception_to_python(std::current_exception());
    }
  });
  // Everything that allocates, launches or waits runs without the interpreter lock: a launch waits while the stream's queue is
  // full, and other threads go on meanwhile.
  using NoGil = py::call_guard<py::gil_scoped_release>;
  py::class_<Plan, PlanPtr>(m, "Plan")
      .def(py::init<int64_t, int64_t, at::Device, const OptTensor&, const OptTensor&, const OptTensor&, const OptTensor&, bool, bool>(), NoGil())
      .def_readonly("B", &Plan::B)
      .def_readonly("T", &Plan::T)
      .def_readonly("device", &Plan::device)
      .def_readonly("buf", &Plan::buf)
      .def_property_readonly("status_dev", &Plan::status_dev)
      .def_property_readonly("status_host", &Plan::status_host)
      .def("use_on_current_stream", &Plan::use_on_current_stream, NoGil());
  m.def("bind", &bind);
  m.def("get_plan", &get_plan, NoGil());
  m.def("cached_plans", [] { return cache().values(); });
  m.def("clear_plans", [] { cache().clear(); });
  m.def("forward", [](const Tensor& q, const Tensor& k, const Tensor& v, const PlanPtr& plan, double sm_scale, bool like_input) {
    return forward(q, k, v, plan, sm_scale, like_input);
  }, NoGil());
  m.def("backward", [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& d_o, const PlanPtr& plan,
                       double sm_scale, int phases, const std::vector<Tensor>& bufs, bool like_input, bool deterministic) {
    Tensor b[5];
    for (size_t i = 0; i < bufs.size() && i < 5; ++i) b[i] = bufs[i];
    return backward(q, k, v, o, lse, d_o, plan, sm_scale, phases, b[0], b[1], b[2], b[3], b[4], like_input, deterministic);
  }, NoGil());
  m.def("hadamard", &hadamard, NoGil());
  m.def("attention", &attention, NoGil());
  m.def("metadata_from_tokens", &metadata_from_tokens, NoGil());
  m.def("cocktail_scores", &cocktail_scores, NoGil());
}
