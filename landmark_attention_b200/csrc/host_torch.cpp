// Host layer between PyTorch and libb200lmk.so: argument checks, output allocation, autograd nodes and kernel calls of
// the public entry points in native code.
//
// Why it exists: the kernels of a short call take 5 - 50 us, and the same steps written in Python (ctypes conversions,
// Python autograd functions, torch.library wrappers) took 75 - 160 us of host time per call, so every small and
// medium call was host-bound (a 77-token prompt: 83 us a call in Python, 48 us here with the same kernels; the GPT layer's
// training step 416 -> 328 us).  Here a call is one Python -> C++ transition, and the backward pass runs in the autograd
// engine without the interpreter lock.
//
// The C ABI of include/b200lmk.h stays the only way into the kernels: its functions are looked up in the library that
// the Python side has loaded (init()), so an override of the library's location holds here as well.
#include <dlfcn.h>

#include <cmath>
#include <mutex>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>
#include <Python.h>

#include "../../include/b200lmk.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// ------------------------------------------------------------------------------------------------ library functions
#define LMK_FUNCS(X)                                                                                             \
  X(lmk_last_error) X(lmk_attn_fwd) X(lmk_attn_bwd_workspace) X(lmk_attn_bwd_strided) X(lmk_attn_mask_fwd)               \
  X(lmk_attn_mask_bwd_workspace) X(lmk_attn_mask_bwd_strided) X(lmk_grouped_softmax_fwd) X(lmk_grouped_softmax_bwd_typed)      \
  X(lmk_grouped_softmax_causal_fwd) X(lmk_grouped_softmax_causal_bwd_typed) X(lmk_rotary_apply) X(lmk_mask_is_regular)        \
  X(lmk_decode_supported) X(lmk_decode_attend) X(lmk_block_select) X(lmk_block_select_supported)                  \
  X(lmk_prefix_gather) X(lmk_prefix_gather_supported) X(lmk_prefix_pv) X(lmk_landmark_scores)                     \
  X(lmk_landmark_scores_workspace) X(lmk_topk_sorted) X(lmk_chunk_rotate) X(lmk_attn_fwd_lse)                     \
  X(lmk_selected_attend) X(lmk_gather_kv_to) X(lmk_cached_rows) X(lmk_cached_rows_supported)
struct Lib {
#define X(name) decltype(&::name) name = nullptr;
  LMK_FUNCS(X)
#undef X
} lib;

// ------------------------------------------------------------------------------------------------ errors
// AssertionError from any thread, with or without the interpreter lock (the backward pass runs without it)
[[noreturn]] void raise_assertion(const std::string& msg) {
  pybind11::gil_scoped_acquire gil;
  PyErr_SetString(PyExc_AssertionError, msg.c_str());
  python_error e;
  e.persist();
  throw e;
}
#define LMK_ASSERT(cond, msg) do { if (!(cond)) raise_assertion(msg); } while (0)

// status codes -> the exception classes the reference raises for the same mistake
void check(int rc, const char* what) {
  if (rc == LMK_OK) return;
  const std::string msg = lib.lmk_last_error();
  if (rc == LMK_ERR_INVALID) raise_assertion(std::string(what) + ": " + msg);
  if (rc == LMK_ERR_UNSUPPORTED) C10_THROW_ERROR(NotImplementedError, std::string(what) + ": " + msg);
  TORCH_CHECK(false, what, " failed (", rc, "): ", msg);
}

void require_cuda(const Tensor& t) {
  LMK_ASSERT(t.is_cuda(), "landmark_attention_b200 runs on CUDA tensors only (no CPU path)");
}

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return LMK_F32;
    case at::kHalf: return LMK_F16;
    case at::kBFloat16: return LMK_BF16;
    default: raise_assertion(std::string("unsupported dtype ") + c10::toString(t.scalar_type()));
  }
}

struct S3 {
  int64_t v[3];
  explicit S3(const Tensor& t) { auto st = t.strides(); v[0] = st[0]; v[1] = st[1]; v[2] = st[2]; }
};

Tensor last_dim_dense(const Tensor& t) { return t.stride(3) == 1 ? t : t.contiguous(); }
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
Tensor empty_like_dtype(at::IntArrayRef sizes, const Tensor& like) { return at::empty(sizes, like.options().requires_grad(false)); }
Tensor empty_f32(at::IntArrayRef sizes, const Tensor& like) {
  return at::empty(sizes, like.options().requires_grad(false).dtype(at::kFloat));
}
// dO as the kernels read it: q's type, dense features, rows of 16-byte vectors (a view of the output projection's gradient
// comes as [B, L, H, D] and is read in place)
Tensor grad_rows(const Tensor& g, const Tensor& q) {
  const Tensor t = g.scalar_type() == q.scalar_type() ? g : g.to(q.scalar_type());
  const int64_t vec = 16 / t.element_size(), D = t.size(3);
  const bool ok = t.stride(3) == 1 && t.stride(0) > 0 && t.stride(1) > 0 && t.stride(0) % vec == 0 && t.stride(1) % vec == 0 &&
                  t.stride(2) % vec == 0 && t.stride(2) >= D && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
  return ok ? t : t.clone(at::MemoryFormat::Contiguous);
}
// Whether a derivative through the call is asked for: backward, or forward (a tangent; the autograd nodes here refuse those, which
// the raw kernel calls would drop).
bool needs_grad(std::initializer_list<std::reference_wrapper<const Tensor>> ts) {
  const bool backward = at::GradMode::is_enabled(), forward = c10::AutogradState::get_tls_state().get_fw_grad_mode();
  for (const Tensor& t : ts)
    if ((backward && t.requires_grad()) || (forward && t._fw_grad(0).defined())) return true;
  return false;
}

// ------------------------------------------------------------------------------------------------ fused attention
// statistics [2, B*H, Lq]: the outer softmax's sum and maximum
Tensor attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, double scale, int64_t block, int64_t path, Tensor* stats) {
  const auto B = q.size(0), H = q.size(1), Lq = q.size(2), D = q.size(3), Lk = k.size(2);
  Tensor o = empty_like_dtype({B, H, Lq, D}, q);
  *stats = empty_f32({2, B * H, Lq}, q);
  float* l = stats->data_ptr<float>();
  check(lib.lmk_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), l, l + B * H * Lq, B, H, Lq, Lk, D,
                         S3(q).v, S3(k).v, S3(v).v, block, (float)scale, dtype_code(q), path, stream_of(q)),
        "lmk_attn_fwd");
  return o;
}

struct FusedLandmark : public torch::autograd::Function<FusedLandmark> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, double scale,
                        int64_t block, int64_t path) {
    at::AutoDispatchBelowADInplaceOrView below;
    Tensor stats, o = attn_fwd(q, k, v, scale, block, path, &stats);
    ctx->save_for_backward({q, k, v, o, stats});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["block"] = block;
    ctx->saved_data["path"] = path;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2], &o = saved[3], &stats = saved[4];
    const int64_t block = ctx->saved_data["block"].toInt(), path = ctx->saved_data["path"].toInt();
    const double scale = ctx->saved_data["scale"].toDouble();
    const auto B = q.size(0), H = q.size(1), Lq = q.size(2), D = q.size(3), Lk = k.size(2);
    c10::cuda::OptionalCUDAGuard guard(q.device());
    const Tensor dO = grad_rows(grads[0], q);
    Tensor dq = empty_like_dtype({B, H, Lq, D}, q), dk = empty_like_dtype({B, H, Lk, D}, q), dv = empty_like_dtype({B, H, Lk, D}, q);
    const int code = dtype_code(q);
    const size_t need = std::max<size_t>(lib.lmk_attn_bwd_workspace(B, H, Lq, Lk, D, block, code, path), 256);
    Tensor ws = at::empty({(int64_t)need}, q.options().requires_grad(false).dtype(at::kByte));
    const float* l = stats.data_ptr<float>();
    check(lib.lmk_attn_bwd_strided(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), dO.data_ptr(), l, l + B * H * Lq,
                           dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), ws.data_ptr(), need, B, H, Lq, Lk, D, S3(q).v,
                           S3(k).v, S3(v).v, S3(dO).v, block, (float)scale, code, path, stream_of(q)),
          "lmk_attn_bwd");
    return {dq, dk, dv, Tensor(), Tensor(), Tensor()};
  }
};

// What the tensor-core kernels read in place (16-bit types): an aligned base, positive batch and head strides, rows that do not
// overlap, all of them multiples of 16 bytes.  A copy of the rest costs a fraction of what the general kernels take, which also have no
// backward pass for sequences that end inside a block (B2 H8 D128 bf16, keys and values of one head broadcast: L1000 forward 973 us on
// the general kernels, 36 with copies; L1024 forward and backward 4206 / 83).
bool tma_rows(const Tensor& t) {
  return t.stride(0) > 0 && t.stride(1) > 0 && t.stride(2) >= t.size(3) && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 &&
         t.stride(2) % 8 == 0 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}

// The checks of FusedLandmarkAttention.forward (flash_landmark_attention.py:319-324), then the kernels.
Tensor fused_attention(const Tensor& q_, const Tensor& k_, const Tensor& v_, int64_t n_prefix, double scale, int64_t block,
                       int64_t path) {
  require_cuda(q_); require_cuda(k_); require_cuda(v_);
  LMK_ASSERT(q_.dim() == 4 && k_.dim() == 4 && v_.dim() == 4, "expected q, k, v of shape [B, H, L, D]");
  const auto d = q_.size(3);
  for (const Tensor* t : {&k_, &v_})
    LMK_ASSERT(t->size(0) == q_.size(0) && t->size(1) == q_.size(1) && t->size(2) == k_.size(2) && t->size(3) == d,
               "k and v must be [B, H, Lk, D] with q's batch, heads and head dim");
  LMK_ASSERT(d <= 128, "FlashAttention only support head dimensions up to 128");
  LMK_ASSERT(q_.scalar_type() == k_.scalar_type() && q_.scalar_type() == v_.scalar_type(), "All tensors must have the same type");
  LMK_ASSERT(k_.size(2) - q_.size(2) == n_prefix * block, "key history must be whole blocks");
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  Tensor q = last_dim_dense(q_), k = last_dim_dense(k_), v = last_dim_dense(v_);
  if (path == LMK_PATH_AUTO && scale > 0 && d % 8 == 0 && (q.scalar_type() == at::kHalf || q.scalar_type() == at::kBFloat16))
    for (Tensor* t : {&q, &k, &v})
      if (!tma_rows(*t)) *t = t->clone(at::MemoryFormat::Contiguous);      // part of the graph where a gradient is wanted
  if (!needs_grad({q, k, v})) {
    Tensor stats;
    return attn_fwd(q, k, v, scale, block, path, &stats);
  }
  return FusedLandmark::apply(q, k, v, scale, block, path);
}

// ------------------------------------------------------------------------------------------------ landmark mask check
// A word of mapped host memory that one kernel may write, and the event behind that kernel.  Words are handed from check to check
// through a list of idle ones (16 bytes of pinned memory each, as many as there were checks at one time): a word is idle again once
// its kernel has finished, whether or not anybody asked for the result.
class FlagWord {
 public:
  explicit FlagWord(int dev) : idle_(idle_of(dev)) {
    const std::lock_guard<std::mutex> lock(idle_.mutex);
    if (idle_.words.empty()) {
      C10_CUDA_CHECK(cudaHostAlloc(reinterpret_cast<void**>(&w_.word), 16, cudaHostAllocMapped | cudaHostAllocPortable));
      C10_CUDA_CHECK(cudaEventCreateWithFlags(&w_.event, cudaEventDisableTiming));
    } else {
      w_ = idle_.words.back();
      idle_.words.pop_back();
    }
    *w_.word = 0;
  }
  ~FlagWord() {
    // a check that was given up (an exception between its launch and its result): the kernel may still be queued
    if (queued_ && (!recorded_ || cudaEventSynchronize(w_.event) != cudaSuccess)) {
      (void)cudaGetLastError();
      return;                          // the kernel may still write it: no other check gets this word
    }
    const std::lock_guard<std::mutex> lock(idle_.mutex);
    idle_.words.push_back(w_);
  }
  FlagWord(const FlagWord&) = delete;
  FlagWord& operator=(const FlagWord&) = delete;

  int* word() const { return w_.word; }
  void launched(cudaStream_t stream) {             // behind the launch of the kernel that writes the word
    queued_ = true;
    C10_CUDA_CHECK(cudaEventRecord(w_.event, stream));
    recorded_ = true;
  }
  int wait() {
    if (queued_) C10_CUDA_CHECK(cudaEventSynchronize(w_.event));
    queued_ = false;
    return *static_cast<volatile int*>(w_.word);
  }

 private:
  struct Word { int* word = nullptr; cudaEvent_t event = nullptr; };
  struct Idle { std::mutex mutex; std::vector<Word> words; };
  static Idle& idle_of(int dev) {
    constexpr int kMax = 64;
    static Idle* idle = new Idle[kMax];            // not destroyed: a thread may end after the program's statics
    TORCH_CHECK(dev >= 0 && dev < kMax, "device index out of range");
    return idle[dev];
  }
  Idle& idle_;
  Word w_;
  bool queued_ = false, recorded_ = false;
};

// One kernel compares every flag with the regular pattern and writes its word; the host waits for that kernel alone, so what
// the caller enqueues between the constructor and failed() overlaps with it.
class RegularCheck {
 public:
  RegularCheck(const Tensor& is_mem, int64_t block) {
    Tensor m = is_mem.contiguous();
    if (!m.is_cuda()) {
      const Tensor want = at::arange(m.size(-1), m.options().dtype(at::kLong)).remainder(block).eq(block - 1);
      host_failed_ = !m.eq(want).all().item<bool>();
      return;
    }
    c10::cuda::OptionalCUDAGuard guard(m.device());
    if (m.element_size() != 1) m = m.eq(1).to(at::kByte).add_(m.ne(0).logical_and_(m.ne(1)), 2);     // 2: neither
    flag_.emplace(m.get_device());
    check(lib.lmk_mask_is_regular((const uint8_t*)m.data_ptr(), m.numel(), m.size(-1), block, flag_->word(), stream_of(m)),
          "lmk_mask_is_regular");
    flag_->launched((cudaStream_t)stream_of(m));
  }
  bool failed() { return flag_ ? flag_->wait() != 0 : host_failed_; }

 private:
  std::optional<FlagWord> flag_;
  bool host_failed_ = false;
};

// ------------------------------------------------------------------------------------------------ masked attention
Tensor flags_u8(const Tensor& is_mem) {
  const Tensor m = is_mem.scalar_type() == at::kByte || is_mem.scalar_type() == at::kBool ? is_mem : is_mem.to(at::kByte);
  return m.stride(-1) == 1 ? m : m.contiguous();
}

std::tuple<Tensor, Tensor, Tensor> masked_fwd_cuda(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& is_mem,
                                                   double scale, int64_t G) {
  require_cuda(q_); require_cuda(k_); require_cuda(v_); require_cuda(is_mem);
  const auto B = q_.size(0), H = q_.size(1), Lq = q_.size(2), D = q_.size(3), Lk = k_.size(2);
  for (const Tensor* t : {&k_, &v_})
    LMK_ASSERT(t->dim() == 4 && t->size(0) == B && t->size(1) == H && t->size(2) == Lk && t->size(3) == D, "k and v must be [B, H, Lk, D]");
  LMK_ASSERT(q_.scalar_type() == k_.scalar_type() && q_.scalar_type() == v_.scalar_type(), "All tensors must have the same type");
  LMK_ASSERT(is_mem.dim() == 2 && is_mem.size(0) == B && is_mem.size(1) == Lk, "is_mem must hold one flag per (batch row, key)");
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = last_dim_dense(q_), k = last_dim_dense(k_), v = last_dim_dense(v_), m = flags_u8(is_mem);
  Tensor o = empty_like_dtype({B, H, Lq, D}, q), R = empty_f32({B * H, Lq}, q), A = empty_f32({B * H, G, Lq}, q);
  check(lib.lmk_attn_mask_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), (const uint8_t*)m.data_ptr(), m.stride(0), o.data_ptr(),
                              R.data_ptr<float>(), A.data_ptr<float>(), B, H, Lq, Lk, D, S3(q).v, S3(k).v, S3(v).v, G,
                              (float)scale, dtype_code(q), stream_of(q)),
        "lmk_attn_mask_fwd");
  return {o, R, A};
}

std::tuple<Tensor, Tensor, Tensor> masked_bwd_cuda(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& is_mem,
                                                   const Tensor& o_, const Tensor& do_, const Tensor& R, const Tensor& A,
                                                   double scale, int64_t G) {
  const auto B = q_.size(0), H = q_.size(1), Lq = q_.size(2), D = q_.size(3), Lk = k_.size(2);
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = last_dim_dense(q_), k = last_dim_dense(k_), v = last_dim_dense(v_), m = flags_u8(is_mem), o = o_.contiguous();
  const Tensor dO = grad_rows(do_, q);
  Tensor dq = empty_like_dtype({B, H, Lq, D}, q), dk = empty_like_dtype({B, H, Lk, D}, q), dv = empty_like_dtype({B, H, Lk, D}, q);
  const size_t need = std::max<size_t>(lib.lmk_attn_mask_bwd_workspace(B, H, Lq, G), 256);
  Tensor ws = at::empty({(int64_t)need}, q.options().requires_grad(false).dtype(at::kByte));
  check(lib.lmk_attn_mask_bwd_strided(q.data_ptr(), k.data_ptr(), v.data_ptr(), (const uint8_t*)m.data_ptr(), m.stride(0), o.data_ptr(),
                              dO.data_ptr(), R.data_ptr<float>(), A.data_ptr<float>(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                              ws.data_ptr(), need, B, H, Lq, Lk, D, S3(q).v, S3(k).v, S3(v).v, S3(dO).v, G, (float)scale,
                              dtype_code(q), stream_of(q)),
        "lmk_attn_mask_bwd");
  return {dq, dk, dv};
}

using MaskedFwdSig = std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, double, int64_t);
using MaskedBwdSig = std::tuple<Tensor, Tensor, Tensor>(const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&,
                                                        const Tensor&, const Tensor&, const Tensor&, double, int64_t);
const c10::TypedOperatorHandle<MaskedFwdSig>& masked_fwd_op() {
  static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("lmk::masked_attention_fwd", "").typed<MaskedFwdSig>();
  return op;
}
const c10::TypedOperatorHandle<MaskedBwdSig>& masked_bwd_op() {
  static auto op = c10::Dispatcher::singleton().findSchemaOrThrow("lmk::masked_attention_bwd", "").typed<MaskedBwdSig>();
  return op;
}

struct MaskedLandmark : public torch::autograd::Function<MaskedLandmark> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& is_mem,
                               double scale, int64_t G) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [o, R, A] = masked_fwd_op().call(q, k, v, is_mem, scale, G);
    ctx->save_for_backward({q, k, v, is_mem, o, R, A});
    ctx->mark_non_differentiable({R, A});
    ctx->set_materialize_grads(false);             // no zero gradients for the statistics
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["groups"] = G;
    return {o, R, A};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    auto s = ctx->get_saved_variables();
    auto [dq, dk, dv] = masked_bwd_op().call(s[0], s[1], s[2], s[3], s[4], grads[0], s[5], s[6],
                                             ctx->saved_data["scale"].toDouble(), ctx->saved_data["groups"].toInt());
    return {dq, dk, dv, Tensor(), Tensor(), Tensor()};
  }
};

std::tuple<Tensor, Tensor, Tensor> masked_fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& is_mem,
                                                       double scale, int64_t G) {
  if (!needs_grad({q, k, v})) {
    at::AutoDispatchBelowADInplaceOrView below;
    return masked_fwd_op().call(q, k, v, is_mem, scale, G);
  }
  auto r = MaskedLandmark::apply(q, k, v, is_mem, scale, G);
  return {r[0], r[1], r[2]};
}

// ------------------------------------------------------------------------------------------------ rotary
std::tuple<Tensor, Tensor> rotary_launch(const Tensor& q_, const Tensor& k_, const Tensor& cos, const Tensor& sin, int64_t pos0,
                                         int64_t mode, bool inverse) {
  for (const Tensor* t : {&q_, &k_, &cos, &sin}) require_cuda(*t);
  const auto B = q_.size(0), H = q_.size(1), T = q_.size(2), D = q_.size(3);
  LMK_ASSERT(q_.sizes() == k_.sizes() && q_.scalar_type() == k_.scalar_type() && q_.scalar_type() == cos.scalar_type() &&
             q_.scalar_type() == sin.scalar_type(), "rotary: q, k and the tables must agree in shape and type");
  LMK_ASSERT(cos.is_contiguous() && sin.is_contiguous() && cos.size(1) == D, "rotary: tables must be dense [n_pos, D]");
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = last_dim_dense(q_), k = last_dim_dense(k_);
  Tensor qo = empty_like_dtype({B, H, T, D}, q), ko = empty_like_dtype({B, H, T, D}, q);
  check(lib.lmk_rotary_apply(q.data_ptr(), k.data_ptr(), S3(q).v, S3(k).v, cos.data_ptr(), sin.data_ptr(), cos.size(0), pos0,
                             mode, inverse, qo.data_ptr(), ko.data_ptr(), B, H, T, D, dtype_code(q), stream_of(q)),
        "lmk_rotary_apply");
  return {qo, ko};
}

struct RotaryPair : public torch::autograd::Function<RotaryPair> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin,
                               int64_t pos0, int64_t mode) {
    at::AutoDispatchBelowADInplaceOrView below;
    ctx->save_for_backward({cos, sin});
    ctx->saved_data["pos0"] = pos0;
    ctx->saved_data["mode"] = mode;
    auto [qo, ko] = rotary_launch(q, k, cos, sin, pos0, mode, false);
    return {qo, ko};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    if (!g[0].defined()) g[0] = at::zeros_like(g[1]);
    if (!g[1].defined()) g[1] = at::zeros_like(g[0]);
    auto [dq, dk] = rotary_launch(g[0], g[1], s[0], s[1], ctx->saved_data["pos0"].toInt(), ctx->saved_data["mode"].toInt(), true);
    return {dq, dk, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

std::tuple<Tensor, Tensor> rotary_apply(const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin, int64_t pos0,
                                        int64_t mode) {
  if (!needs_grad({q, k})) return rotary_launch(q, k, cos, sin, pos0, mode, false);
  auto r = RotaryPair::apply(q, k, cos, sin, pos0, mode);
  return {r[0], r[1]};
}

// ------------------------------------------------------------------------------------------------ grouped softmax
// byte mask with element strides of the [B, H, Lq, Lk] scores (0 where broadcast)
struct Mask {
  Tensor keep;
  const uint8_t* ptr = nullptr;
  int64_t st[4] = {0, 0, 0, 0};
  Mask(const Tensor& m, at::IntArrayRef shape) {
    if (!m.defined()) return;
    keep = m.scalar_type() == at::kBool ? m : m.ne(0);          // the kernels read bit 0 of every byte
    ptr = reinterpret_cast<const uint8_t*>(keep.data_ptr());
    const int64_t off = 4 - keep.dim();
    LMK_ASSERT(off >= 0, "mask has more than four dimensions");
    for (int64_t i = 0; i < keep.dim(); ++i) {
      const int64_t n = keep.size(i), want = shape[off + i];
      LMK_ASSERT(n == want || n == 1, "mask does not broadcast to the scores");
      st[off + i] = n == 1 ? 0 : keep.stride(i);
    }
  }
  const int64_t* strides() const { return ptr ? st : nullptr; }
};

struct GroupedSoftmax : public torch::autograd::Function<GroupedSoftmax> {
  static std::tuple<Tensor, Tensor> run(const Tensor& x, const Tensor& is_mem, const Tensor& last, const Tensor& hidden, bool guards,
                                        int64_t max_groups, int64_t max_mem_cnt) {
    const auto B = x.size(0), H = x.size(1), Lq = x.size(2), Lk = x.size(3);
    Tensor probs = empty_f32({B, H, Lq, Lk}, x), gp;
    if (max_mem_cnt) gp = empty_f32({B, H, Lq, max_mem_cnt}, x);
    Mask m(is_mem, x.sizes()), l(last, x.sizes()), h(hidden, x.sizes());
    check(lib.lmk_grouped_softmax_fwd(x.data_ptr(), S3(x).v, m.ptr, m.strides(), l.ptr, l.strides(), h.ptr, h.strides(),
                                      probs.data_ptr<float>(), max_mem_cnt ? gp.data_ptr<float>() : nullptr, max_mem_cnt, B, H,
                                      Lq, Lk, dtype_code(x), guards, max_groups, stream_of(x)),
          "lmk_grouped_softmax_fwd");
    return {probs, gp};
  }
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& is_mem, const Tensor& last,
                               const std::optional<Tensor>& hidden, bool guards, int64_t max_groups, int64_t max_mem_cnt) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [probs, gp] = run(x, is_mem, last, hidden.value_or(Tensor()), guards, max_groups, max_mem_cnt);
    if (hidden) ctx->save_for_backward({x, is_mem, last, *hidden});
    else ctx->save_for_backward({x, is_mem, last});
    ctx->saved_data["guards"] = guards;
    ctx->saved_data["groups"] = max_groups;
    if (!gp.defined()) return {probs};
    ctx->mark_non_differentiable({gp});
    return {probs, gp};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    const Tensor& x = s[0];
    const auto B = x.size(0), H = x.size(1), Lq = x.size(2), Lk = x.size(3);
    c10::cuda::OptionalCUDAGuard guard(x.device());
    Tensor gprobs = g[0].to(at::kFloat).contiguous(), gx = at::empty({B, H, Lq, Lk}, x.options());
    Mask m(s[1], x.sizes()), l(s[2], x.sizes()), h(s.size() > 3 ? s[3] : Tensor(), x.sizes());
    check(lib.lmk_grouped_softmax_bwd_typed(x.data_ptr(), S3(x).v, m.ptr, m.strides(), l.ptr, l.strides(), h.ptr, h.strides(),
                                      gprobs.data_ptr<float>(), gx.data_ptr(), B, H, Lq, Lk, dtype_code(x),
                                      ctx->saved_data["guards"].toBool(), ctx->saved_data["groups"].toInt(), stream_of(x)),
          "lmk_grouped_softmax_bwd");
    return {gx, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

std::tuple<Tensor, Tensor> grouped_softmax(const Tensor& x_, const Tensor& is_mem, const Tensor& last, const Tensor& hidden,
                                           bool guards, int64_t max_groups, int64_t max_mem_cnt) {
  require_cuda(x_); require_cuda(is_mem); require_cuda(last);
  if (hidden.defined()) require_cuda(hidden);
  TORCH_CHECK_VALUE(x_.dim() == 4, "expected scores of shape [B, H, Lq, Lk]");
  c10::cuda::OptionalCUDAGuard guard(x_.device());
  const Tensor x = last_dim_dense(x_);
  if (!needs_grad({x})) return GroupedSoftmax::run(x, is_mem, last, hidden, guards, max_groups, max_mem_cnt);
  auto r = GroupedSoftmax::apply(x, is_mem, last, hidden.defined() ? std::optional<Tensor>(hidden) : std::nullopt, guards,
                                 max_groups, max_mem_cnt);
  return {r[0], r.size() > 1 ? r[1] : Tensor()};
}

struct GroupedSoftmaxCausal : public torch::autograd::Function<GroupedSoftmaxCausal> {
  static Tensor run(const Tensor& x, const Tensor& flags, int64_t max_groups) {
    const auto B = x.size(0), H = x.size(1), Lq = x.size(2), Lk = x.size(3);
    Tensor probs = empty_f32({B, H, Lq, Lk}, x);
    check(lib.lmk_grouped_softmax_causal_fwd(x.data_ptr(), S3(x).v, (const uint8_t*)flags.data_ptr(), flags.stride(0),
                                             probs.data_ptr<float>(), B, H, Lq, Lk, dtype_code(x), max_groups, stream_of(x)),
          "lmk_grouped_softmax_causal_fwd");
    return probs;
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& flags, int64_t max_groups) {
    at::AutoDispatchBelowADInplaceOrView below;
    ctx->save_for_backward({x, flags});
    ctx->saved_data["groups"] = max_groups;
    return run(x, flags, max_groups);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    auto s = ctx->get_saved_variables();
    const Tensor &x = s[0], &flags = s[1];
    const auto B = x.size(0), H = x.size(1), Lq = x.size(2), Lk = x.size(3);
    c10::cuda::OptionalCUDAGuard guard(x.device());
    Tensor gprobs = g[0].to(at::kFloat).contiguous(), gx = at::empty({B, H, Lq, Lk}, x.options());
    check(lib.lmk_grouped_softmax_causal_bwd_typed(x.data_ptr(), S3(x).v, (const uint8_t*)flags.data_ptr(), flags.stride(0),
                                             gprobs.data_ptr<float>(), gx.data_ptr(), B, H, Lq, Lk, dtype_code(x),
                                             ctx->saved_data["groups"].toInt(), stream_of(x)),
          "lmk_grouped_softmax_causal_bwd");
    return {gx, Tensor(), Tensor()};
  }
};

Tensor grouped_softmax_causal(const Tensor& x_, const Tensor& is_mem_row, int64_t max_groups) {
  require_cuda(x_); require_cuda(is_mem_row);
  c10::cuda::OptionalCUDAGuard guard(x_.device());
  const Tensor x = last_dim_dense(x_);
  Tensor flags = is_mem_row.scalar_type() == at::kBool ? is_mem_row : is_mem_row.ne(0);
  if (flags.stride(-1) != 1) flags = flags.contiguous();
  if (!needs_grad({x})) return GroupedSoftmaxCausal::run(x, flags, max_groups);
  return GroupedSoftmaxCausal::apply(x, flags, max_groups);
}

// ------------------------------------------------------------------------------------------------ retrieval
// rows of 16-byte vectors: dense features, strides that are multiples of 8 elements, aligned base
Tensor vector_rows(const Tensor& t) {
  const bool ok = t.stride(3) == 1 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0 &&
                  (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
  return ok ? t : t.clone(at::MemoryFormat::Contiguous);
}

// Behind a cache of whole blocks the generation kernel takes up to this many tokens; more go the chunk's way, whose scores and local
// attention run on the tensor cores.  Measured on the device (us, generation kernel / chunk kernels, blocks of 64, top 4): 8 heads,
// 64 blocks, 8 tokens 18.6 / 32.6, 16 35.0 / 33.4, 32 67 / 35; 1024 blocks, 16 39.9 / 35.7; 32 heads, 64 blocks, 4 tokens
// 35.1 / 33.1, 16 129 / 37; 1024 blocks, 4 39.9 / 58.8, 8 77 / 60, 16 158 / 68.  The line is right for 8 heads; with 32 it lies at
// 4 to 8 tokens, and between there and 16 the chunk would be up to 3.4 times as fast.
constexpr int64_t kDecodeMaxWholeBlockTokens = 16;

// One layer of token generation behind `len` cached tokens (lmk_decode_attend): tokens that stay inside the unfinished
// block; undefined where the kernel does not take them, and where a gradient is asked for behind an unfinished block: the tensor
// formulation that runs there is differentiable through the unfinished block's keys and values and the new ones.  (Behind whole
// blocks the other route has no gradient either.)
Tensor decode_attend(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& kc, const Tensor& vc, int64_t len,
                     bool append, int64_t block, int64_t top_k, const Tensor& cos, const Tensor& sin) {
  const auto st = q_.scalar_type();
  if (block < 2 || top_k < 1 || len < block) return Tensor();
  const int64_t tail = len % block;
  if (tail && needs_grad({q_, k_, v_, kc, vc, cos, sin})) return Tensor();
  top_k = std::min(top_k, len / block);
  if (!q_.is_cuda() || (st != at::kHalf && st != at::kBFloat16) || q_.dim() != 4 || kc.dim() != 4) return Tensor();
  const auto B = q_.size(0), H = q_.size(1), T = q_.size(2), D = q_.size(3);
  for (const Tensor* t : {&k_, &v_, &kc, &vc, &cos, &sin})
    if (!t->is_cuda() || t->scalar_type() != st) return Tensor();
  auto cache_ok = [&](const Tensor& t) {
    return t.stride(3) == 1 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0 && t.size(0) == B &&
           t.size(1) == H && t.size(3) == D && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
  };
  auto table_ok = [&](const Tensor& t) {
    return t.is_contiguous() && t.dim() == 2 && t.size(1) == D && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
  };
  if (!cache_ok(kc) || !cache_ok(vc) || k_.sizes() != q_.sizes() || v_.sizes() != q_.sizes() || !table_ok(cos) ||
      !table_ok(sin) || B * H > 65535 || T + tail > block || (!tail && T > kDecodeMaxWholeBlockTokens) ||
      kc.size(2) < len + (append ? T : 0) || vc.size(2) < len + (append ? T : 0) ||
      !lib.lmk_decode_supported(D, block, top_k, len, T, dtype_code(q_)))
    return Tensor();
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = vector_rows(q_), k = vector_rows(k_), v = vector_rows(v_);
  Tensor out = empty_like_dtype({B, H, T, D}, q);
  check(lib.lmk_decode_attend(q.data_ptr(), k.data_ptr(), v.data_ptr(), S3(q).v, S3(k).v, S3(v).v, kc.data_ptr(), vc.data_ptr(),
                              S3(kc).v, S3(vc).v, len, append, block, top_k, cos.data_ptr(), sin.data_ptr(), cos.size(0),
                              out.data_ptr(), B, H, T, D, 1.0 / std::sqrt((double)D), dtype_code(q), stream_of(q)),
        "lmk_decode_attend");
  return out;
}

lmk_cache_desc block_desc(const Tensor& t, bool block_before_head, int64_t n, int64_t ring_start, int64_t block, int64_t top_k) {
  lmk_cache_desc d{};
  d.stride_b = t.stride(0);
  d.stride_h = t.stride(block_before_head ? 3 : 1);
  d.stride_block = t.stride(block_before_head ? 1 : 2);
  d.stride_row = t.stride(block_before_head ? 2 : 3);
  d.n_blocks = n;
  d.ring_start = ring_start;
  d.block = block;
  d.top_k = top_k;
  return d;
}

// MemLMCacheStorage.retrieve_for_query with blocks in the cache (mem_cache.py:51-109): (att_prefix [B,H,T,P], values
// [B,H,T,P,D]); undefined where the kernels do not take the problem or a gradient is asked for (of the queries, or of the unfinished
// block, whose rows belong to the graph of the chunk that stored them).  kc, vc: the block buffers in either layout; lm: dense
// landmark keys [B,H,capacity,D]; tail_k, tail_v [B,H,>=inc,D].  mode: 0 per token and head, 1 maximum over the
// tokens, 2 over the heads.
std::tuple<Tensor, Tensor> cache_retrieve(const Tensor& q_, const Tensor& kc, const Tensor& vc, const Tensor& lm, bool block_first,
                                          int64_t n, int64_t ring_start, int64_t block, int64_t top_k, const Tensor& cos,
                                          const Tensor& sin, int64_t mode, const Tensor& tail_k, const Tensor& tail_v, int64_t inc,
                                          int64_t tail_pos) {
  const auto st = q_.scalar_type();
  const auto B = q_.size(0), H = q_.size(1), T = q_.size(2), D = q_.size(3);
  if (!q_.is_cuda() || (st != at::kHalf && st != at::kBFloat16) || B * H > 65535) return {};
  if (needs_grad({q_}) || (inc && needs_grad({tail_k, tail_v}))) return {};
  for (const Tensor* t : {&kc, &vc, &lm, &cos, &sin, &tail_k, &tail_v})
    if (!t->is_cuda() || t->scalar_type() != st || t->stride(-1) != 1 || (reinterpret_cast<uintptr_t>(t->data_ptr()) & 15)) return {};
  const int code = dtype_code(q_);
  if (tail_k.strides() != tail_v.strides() || !lib.lmk_prefix_gather_supported(D, block, top_k, T, inc, code)) return {};
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = q_.contiguous();
  void* stream = stream_of(q);
  const float scale = 1.0 / std::sqrt((double)D);
  const lmk_cache_desc kd = block_desc(kc, block_first, n, ring_start, block, top_k), vd = block_desc(vc, block_first, n, ring_start, block, top_k);
  lmk_cache_desc ld{};
  ld.stride_b = lm.stride(0);
  ld.stride_h = lm.stride(1);
  ld.stride_block = lm.stride(2);
  ld.n_blocks = n;
  ld.ring_start = ring_start;
  ld.block = block;
  ld.top_k = top_k;
  const auto i32 = q.options().requires_grad(false).dtype(at::kInt);
  const bool small = lib.lmk_block_select_supported(D, n, top_k, code);
  Tensor idx, probs;
  if (mode == 0 && small) idx = at::empty({B, H, T, top_k}, i32);
  else probs = empty_f32({B, H, T, n}, q);
  if (small) {
    check(lib.lmk_block_select(q.data_ptr(), lm.data_ptr(), &ld, cos.data_ptr(), sin.data_ptr(), cos.size(0), LMK_ROTARY_INTERLEAVED,
                               probs.defined() ? probs.data_ptr<float>() : nullptr, idx.defined() ? idx.data_ptr<int>() : nullptr,
                               B, H, T, D, scale, code, stream),
          "lmk_block_select");
  } else {
    const size_t need = lib.lmk_landmark_scores_workspace(B, H, T, D, n, code);
    Tensor ws = need ? at::empty({(int64_t)need}, i32.dtype(at::kByte)) : Tensor();
    check(lib.lmk_landmark_scores(q.data_ptr(), lm.data_ptr(), &ld, cos.data_ptr(), sin.data_ptr(), cos.size(0), LMK_ROTARY_INTERLEAVED,
                                  probs.data_ptr<float>(), B, H, T, D, scale, 1, code, need ? ws.data_ptr() : nullptr, need, stream),
          "lmk_landmark_scores");
  }
  int64_t is[3] = {H * T * top_k, T * top_k, top_k};
  if (!idx.defined()) {
    const float* s = probs.data_ptr<float>();
    if (mode == 0) {
      idx = at::empty({B, H, T, top_k}, i32);
      check(lib.lmk_topk_sorted(s, idx.data_ptr<int>(), B * H * T, 1, n, 0, 1, 0, n, top_k, ring_start, stream), "lmk_topk_sorted");
    } else if (mode == 1) {
      idx = at::empty({B, H, 1, top_k}, i32);
      check(lib.lmk_topk_sorted(s, idx.data_ptr<int>(), B * H, 1, T * n, 0, T, n, n, top_k, ring_start, stream), "lmk_topk_sorted");
      is[0] = H * top_k, is[1] = top_k, is[2] = 0;
    } else {
      idx = at::empty({B, 1, T, top_k}, i32);
      check(lib.lmk_topk_sorted(s, idx.data_ptr<int>(), B, T, H * T * n, n, H, T * n, n, top_k, ring_start, stream), "lmk_topk_sorted");
      is[0] = T * top_k, is[1] = 0, is[2] = top_k;
    }
  }
  const int64_t P = top_k * block + inc;
  Tensor att = empty_like_dtype({B, H, T, P}, q), v = empty_like_dtype({B, H, T, P, D}, q);
  check(lib.lmk_prefix_gather(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), &kd, &vd, idx.data_ptr<int>(), is, cos.data_ptr(), sin.data_ptr(),
                              cos.size(0), LMK_ROTARY_INTERLEAVED, tail_k.data_ptr(), tail_v.data_ptr(), S3(tail_k).v, inc, tail_pos,
                              att.data_ptr(), v.data_ptr(), B, H, T, D, scale, code, stream),
        "lmk_prefix_gather");
  return {att, v};
}

// y += probs[..., :P] @ v per token (lmk_prefix_pv); false where the kernel does not take the tensors or a gradient of them is asked for
bool prefix_pv(const Tensor& probs, const Tensor& v, const Tensor& y) {
  const auto st = v.scalar_type();
  const auto B = y.size(0), H = y.size(1), T = y.size(2), D = y.size(3), P = v.size(3);
  if (needs_grad({probs, v}) || !v.is_cuda() || (st != at::kHalf && st != at::kBFloat16) || y.scalar_type() != st || D != 128 ||
      P > 8192 || B * H > 65535 ||
      P == 0 || !probs.is_contiguous() || !y.is_contiguous() || v.stride(4) != 1 || v.stride(3) != D || v.stride(0) % 8 ||
      v.stride(1) % 8 || v.stride(2) % 8 || (reinterpret_cast<uintptr_t>(v.data_ptr()) & 15))
    return false;
  c10::cuda::OptionalCUDAGuard guard(v.device());
  check(lib.lmk_prefix_pv(probs.data_ptr<float>(), probs.size(3), v.data_ptr(), S3(v).v, y.data_ptr(), B, H, T, P, D, dtype_code(v),
                          stream_of(v)),
        "lmk_prefix_pv");
  return true;
}

// ---- a chunk of a prompt behind a block cache (llama/llama_mem.py:318-430, 447-474), 16-bit types, head dim 128
struct Chunk {
  Tensor q, k, v;                 // rows of 16-byte vectors
  int64_t B = 0, H = 0, T = 0, D = 0;
  int code = 0;
  float scale = 0.f;
  void* stream = nullptr;
};
bool table_ok(const Tensor& t, const Tensor& q) {
  return t.is_cuda() && t.scalar_type() == q.scalar_type() && t.is_contiguous() && t.dim() == 2 && t.size(1) == q.size(3) &&
         (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}
bool rows_ok(const Tensor& t) {      // a cache [B, H, rows, D]
  return t.dim() == 4 && t.stride(3) == 1 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0 &&
         (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}
bool chunk_of(Chunk* c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& kc, const Tensor& vc, const Tensor& cos,
              const Tensor& sin) {
  const auto st = q.scalar_type();
  if (!q.is_cuda() || (st != at::kHalf && st != at::kBFloat16) || q.dim() != 4 || q.size(3) != 128 || k.sizes() != q.sizes() ||
      v.sizes() != q.sizes() || k.scalar_type() != st || v.scalar_type() != st || !k.is_cuda() || !v.is_cuda() ||
      kc.scalar_type() != st || vc.scalar_type() != st || !rows_ok(kc) || !rows_ok(vc) || kc.strides() != vc.strides() ||
      kc.size(0) != q.size(0) || kc.size(1) != q.size(1) || kc.size(3) != q.size(3) || !table_ok(cos, q) || !table_ok(sin, q) ||
      q.size(0) * q.size(1) > 65535)
    return false;
  c->B = q.size(0), c->H = q.size(1), c->T = q.size(2), c->D = q.size(3);
  c->q = vector_rows(q), c->k = vector_rows(k), c->v = vector_rows(v);
  c->code = dtype_code(q);
  c->scale = 1.0 / std::sqrt((double)c->D);
  c->stream = stream_of(q);
  return true;
}
lmk_cache_desc rows_desc(const Tensor& cache, int64_t n, int64_t block, int64_t top_k) {
  lmk_cache_desc d{};
  d.stride_b = cache.stride(0);
  d.stride_h = cache.stride(1);
  d.stride_block = cache.stride(2) * block;
  d.stride_row = cache.stride(2);
  d.n_blocks = n;
  d.block = block;
  d.top_k = top_k;
  d.pos_base = (n - top_k - 1) * block;
  return d;
}
Tensor landmark_scores(const Chunk& c, const Tensor& q_rot, const Tensor& keys, const lmk_cache_desc& d, const Tensor& cos,
                       const Tensor& sin, bool softmax) {
  Tensor s = empty_f32({c.B, c.H, c.T, d.n_blocks}, q_rot);
  if (softmax && lib.lmk_block_select_supported(c.D, d.n_blocks, d.top_k, c.code)) {
    check(lib.lmk_block_select(q_rot.data_ptr(), keys.data_ptr(), &d, cos.data_ptr(), sin.data_ptr(), cos.size(0), LMK_ROTARY_HALF,
                               s.data_ptr<float>(), nullptr, c.B, c.H, c.T, c.D, c.scale, c.code, c.stream), "lmk_block_select");
    return s;
  }
  const size_t need = lib.lmk_landmark_scores_workspace(c.B, c.H, c.T, c.D, d.n_blocks, c.code);
  Tensor ws = need ? at::empty({(int64_t)need}, q_rot.options().dtype(at::kByte)) : Tensor();
  check(lib.lmk_landmark_scores(q_rot.data_ptr(), keys.data_ptr(), &d, cos.data_ptr(), sin.data_ptr(), cos.size(0), LMK_ROTARY_HALF,
                                s.data_ptr<float>(), c.B, c.H, c.T, c.D, c.scale, softmax, c.code, need ? ws.data_ptr() : nullptr, need,
                                c.stream), "lmk_landmark_scores");
  return s;
}

// A chunk behind a retrieved prefix (lmk_cached_rows, lmk_prefix_pv); undefined where the kernels do not take it or a gradient is asked for.
Tensor cached_attend(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& prefix, const Tensor& values, const Tensor& flags,
                     int64_t max_groups, double scale) {
  const auto st = q_.scalar_type();
  if (!q_.is_cuda() || q_.dim() != 4 || k_.sizes() != q_.sizes() || v_.sizes() != q_.sizes() || prefix.dim() != 4 || values.dim() != 5 ||
      needs_grad({q_, k_, v_, prefix, values}))
    return Tensor();
  const auto B = q_.size(0), H = q_.size(1), T = q_.size(2), D = q_.size(3), P = prefix.size(3);
  for (const Tensor* t : {&k_, &v_, &prefix, &values})
    if (!t->is_cuda() || t->scalar_type() != st) return Tensor();
  if ((st != at::kHalf && st != at::kBFloat16) || D != 128 || B * H > 65535 || values.size(3) != P || !prefix.is_contiguous() ||
      prefix.size(0) != B || prefix.size(1) != H || prefix.size(2) != T || !flags.is_cuda() || flags.scalar_type() != at::kBool ||
      flags.dim() != 2 || flags.size(0) != B || flags.size(1) != P + T || flags.stride(1) != 1 || max_groups < 1 || max_groups > 2048 ||
      !lib.lmk_cached_rows_supported(D, T, P, dtype_code(q_)))
    return Tensor();
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const Tensor q = vector_rows(q_), k = vector_rows(k_), v = vector_rows(v_);
  Tensor probs = empty_f32({B, H, T, P}, q), y = empty_like_dtype({B, H, T, D}, q);
  check(lib.lmk_cached_rows(q.data_ptr(), k.data_ptr(), v.data_ptr(), S3(q).v, S3(k).v, S3(v).v, prefix.data_ptr(),
                            (const uint8_t*)flags.data_ptr(), flags.stride(0), probs.data_ptr<float>(), y.data_ptr(), B, H, T, P, D,
                            max_groups, scale, dtype_code(q), stream_of(q)), "lmk_cached_rows");
  return prefix_pv(probs, values, y) ? y : Tensor();
}

// A second stream for the part of a call that nothing else in it waits for, with the events of the fork and the join (one set per
// thread and device, reused: a wait refers to the event's state when it is enqueued).
struct Fork {
  c10::cuda::CUDAStream side;
  cudaEvent_t begin, end;
};
Fork fork_of(int dev) {
  constexpr int kMax = 64;
  static thread_local cudaEvent_t events[kMax][2] = {};
  TORCH_CHECK(dev >= 0 && dev < kMax, "device index out of range");
  for (auto& e : events[dev])
    if (e == nullptr) C10_CUDA_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  return {c10::cuda::getStreamFromPool(false, dev), events[dev][0], events[dev][1]};
}

// Makes `main` wait for what a call put on its side stream, also where the call ends in an exception: its tensors are given back to
// main's allocator, and its destination may be written again by what main does next.
class Join {
 public:
  Join(const Fork& fork, cudaStream_t main) : fork_(fork), main_(main) {}
  ~Join() {
    if (done_) return;
    (void)cudaEventRecord(fork_.end, fork_.side.stream());
    (void)cudaStreamWaitEvent(main_, fork_.end, 0);
  }
  Join(const Join&) = delete;
  Join& operator=(const Join&) = delete;
  void now() {                        // with `end` recorded behind the last thing that matters
    C10_CUDA_CHECK(cudaStreamWaitEvent(main_, fork_.end, 0));
    done_ = true;
  }

 private:
  const Fork fork_;
  const cudaStream_t main_;
  bool done_ = false;
};

// One selection per (head, token); `len` whole-block tokens in the caches; append: k, v stored behind them.
Tensor chunk_attend(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& kc, const Tensor& vc, int64_t len, bool append,
                    int64_t block, int64_t top_k, const Tensor& cos, const Tensor& sin, int64_t rotary) {
  if (block < 2 || block > 64 || len % block != 0 || len < block || (q_.size(2) - 1) / block > 64 || top_k < 1 || top_k > 32) return Tensor();
  const int64_t n = len / block;
  Chunk c;
  if (n > 49152 || kc.size(2) < len + (append ? q_.size(2) : 0) || !kc.is_cuda() || !vc.is_cuda() || !chunk_of(&c, q_, k_, v_, kc, vc, cos, sin))
    return Tensor();
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  // the values go to the attention as they are, and TMA addresses neither broadcast heads nor overlapping rows
  if (!tma_rows(c.v)) c.v = c.v.clone(at::MemoryFormat::Contiguous);
  const lmk_cache_desc d = rows_desc(kc, n, block, top_k);
  Tensor qr = empty_like_dtype({c.B, c.H, c.T, c.D}, c.q), kr = empty_like_dtype({c.B, c.H, c.T, c.D}, c.q);
  check(lib.lmk_chunk_rotate(c.q.data_ptr(), c.k.data_ptr(), c.v.data_ptr(), S3(c.q).v, S3(c.k).v, S3(c.v).v, cos.data_ptr(),
                             sin.data_ptr(), cos.size(0), len, qr.data_ptr(), kr.data_ptr(), nullptr, c.T * c.D,
                             append ? kc.data_ptr() : nullptr, append ? vc.data_ptr() : nullptr, append ? S3(kc).v : nullptr, len, c.B,
                             c.H, c.T, c.D, c.code, c.stream), "lmk_chunk_rotate");
  // The chunk's local attention runs beside the scores and the selection: it has 96 CTAs at 32 heads of 258
  // tokens (the whole call 158 -> 147 us), and neither needs the other's results.
  Tensor o = empty_like_dtype({c.B, c.H, c.T, c.D}, c.q), R = empty_f32({c.B * c.H, c.T}, c.q);
  const Fork fork = fork_of(q_.get_device());
  C10_CUDA_CHECK(cudaEventRecord(fork.begin, (cudaStream_t)c.stream));
  const Tensor s = landmark_scores(c, qr, kc, d, cos, sin, false);
  Tensor idx = at::empty({c.B, c.H, c.T, top_k}, c.q.options().requires_grad(false).dtype(at::kInt));
  check(lib.lmk_topk_sorted(s.data_ptr<float>(), idx.data_ptr<int>(), c.B * c.H * c.T, 1, n, 0, 1, 0, n, top_k, 0, c.stream), "lmk_topk_sorted");
  C10_CUDA_CHECK(cudaStreamWaitEvent(fork.side.stream(), fork.begin, 0));
  const int local = lib.lmk_attn_fwd_lse(qr.data_ptr(), kr.data_ptr(), c.v.data_ptr(), o.data_ptr(), R.data_ptr<float>(), c.B, c.H, c.T,
                                         c.T, c.D, S3(qr).v, S3(kr).v, S3(c.v).v, block, c.scale, c.code, fork.side.stream());
  C10_CUDA_CHECK(cudaEventRecord(fork.end, fork.side.stream()));
  C10_CUDA_CHECK(cudaStreamWaitEvent((cudaStream_t)c.stream, fork.end, 0));
  check(local, "lmk_attn_fwd_lse");
  Tensor out = empty_like_dtype({c.B, c.H, c.T, c.D}, c.q);
  check(lib.lmk_selected_attend(qr.data_ptr(), kc.data_ptr(), &d, vc.data_ptr(), &d, idx.data_ptr<int>(), cos.data_ptr(), sin.data_ptr(),
                                cos.size(0), rotary, o.data_ptr(), R.data_ptr<float>(), c.T, out.data_ptr(), c.B, c.H, c.T, c.D, c.scale,
                                c.code, c.stream), "lmk_selected_attend");
  return out;
}

// One selection per head, the maximum over the chunk's tokens; the chunk then attends to [selected blocks | chunk].  The caches hold
// n blocks, on the device (lm undefined: landmarks are read from kc; append: k, v stored behind the n blocks) or in pinned host memory
// (lm: their landmark keys; append: the chunk's whole blocks stored, on a second stream, because the writes over the host link
// do not depend on the attention and run against the direction of its reads).  Undefined where the kernels do not take the call or a
// gradient is asked for: the tensor formulation of the same call is differentiable.  It also takes blocks above 64: their attention runs
// on the two-pass tensor-core kernels there (H8, 100 tokens, blocks of 128, top 4: 355 us; 550 on the general kernels, which
// attn_fwd takes and which end at blocks of 128).
Tensor per_head_attend(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& kc, const Tensor& vc, const Tensor& lm, int64_t n,
                       bool append, int64_t block, int64_t top_k, const Tensor& cos, const Tensor& sin) {
  if (block > 64 || needs_grad({q_, k_, v_, cos, sin})) return Tensor();
  const bool host = lm.defined();
  Chunk c;
  if (block < 1 || n < 1 || n > 49152 || top_k < 1 || top_k > 32 || kc.is_cuda() == host || vc.is_cuda() == host ||
      kc.size(2) < n * block + (append ? q_.size(2) : 0) || !chunk_of(&c, q_, k_, v_, kc, vc, cos, sin))
    return Tensor();
  if (host && (!kc.is_pinned() || !vc.is_pinned() || kc.stride(2) != c.D || lm.scalar_type() != q_.scalar_type() || !rows_ok(lm) ||
               lm.size(2) < n || (append && c.T % block != 0)))
    return Tensor();
  c10::cuda::OptionalCUDAGuard guard(q_.device());
  const lmk_cache_desc d = rows_desc(kc, n, block, top_k);
  lmk_cache_desc ld = d;
  if (host) {
    ld.stride_b = lm.stride(0);
    ld.stride_h = lm.stride(1);
    ld.stride_block = lm.stride(2);
    ld.stride_row = 0;
  }
  std::optional<Fork> fork;
  std::optional<Join> join;
  if (host && append) {
    // by the copy engine: the same stores from a kernel fill the memory system's queues towards the host link and slow down
    // everything that runs beside them (the rotary kernel 4 -> 35 us)
    c.k = c.k.contiguous(), c.v = c.v.contiguous();
    fork = fork_of(q_.get_device());
    join.emplace(*fork, (cudaStream_t)c.stream);
    C10_CUDA_CHECK(cudaEventRecord(fork->begin, (cudaStream_t)c.stream));
    C10_CUDA_CHECK(cudaStreamWaitEvent(fork->side.stream(), fork->begin, 0));
    const size_t width = (size_t)c.T * c.D * 2, pitch = (size_t)kc.stride(1) * 2, at = (size_t)n * block * c.D * 2;
    const bool one = kc.stride(0) == c.H * kc.stride(1);      // one copy for all (batch, head) pairs
    for (int64_t b = 0; b < (one ? 1 : c.B); ++b)
      for (const auto& [dst, src] : {std::pair(&kc, &c.k), std::pair(&vc, &c.v)})
        C10_CUDA_CHECK(cudaMemcpy2DAsync(static_cast<char*>(dst->data_ptr()) + b * dst->stride(0) * 2 + at, pitch,
                                         static_cast<const char*>(src->data_ptr()) + b * src->stride(0) * 2, width, width,
                                         one ? c.B * c.H : c.H, cudaMemcpyDeviceToHost, fork->side.stream()));
    C10_CUDA_CHECK(cudaEventRecord(fork->end, fork->side.stream()));
    lm.narrow(2, n, c.T / block).copy_(c.k.slice(2, block - 1, c.T, block));
  }
  const bool device_append = append && !host;
  const int64_t P = top_k * block, W = P + c.T;
  Tensor qr = empty_like_dtype({c.B, c.H, c.T, c.D}, c.q);
  Tensor keys = empty_like_dtype({c.B, c.H, W, c.D}, c.q), vals = empty_like_dtype({c.B, c.H, W, c.D}, c.q);
  auto behind = [&](const Tensor& t) { return static_cast<uint16_t*>(t.data_ptr()) + P * c.D; };
  check(lib.lmk_chunk_rotate(c.q.data_ptr(), c.k.data_ptr(), c.v.data_ptr(), S3(c.q).v, S3(c.k).v, S3(c.v).v, cos.data_ptr(),
                             sin.data_ptr(), cos.size(0), n * block, qr.data_ptr(), behind(keys), behind(vals), W * c.D,
                             device_append ? kc.data_ptr() : nullptr, device_append ? vc.data_ptr() : nullptr,
                             device_append ? S3(kc).v : nullptr, n * block, c.B, c.H, c.T, c.D, c.code, c.stream), "lmk_chunk_rotate");
  const Tensor probs = landmark_scores(c, qr, host ? lm : kc, ld, cos, sin, true);
  Tensor idx = at::empty({c.B, c.H, 1, top_k}, c.q.options().requires_grad(false).dtype(at::kInt));
  check(lib.lmk_topk_sorted(probs.data_ptr<float>(), idx.data_ptr<int>(), c.B * c.H, 1, c.T * n, 0, c.T, n, n, top_k, 0, c.stream),
        "lmk_topk_sorted");
  check(lib.lmk_gather_kv_to(kc.data_ptr(), vc.data_ptr(), &d, &d, idx.data_ptr<int>(), cos.data_ptr(), sin.data_ptr(), cos.size(0), LMK_ROTARY_HALF,
                             keys.data_ptr(), vals.data_ptr(), W * c.D, c.B, c.H, 1, c.D, c.code, c.stream), "lmk_gather_kv");
  Tensor stats;
  Tensor out = attn_fwd(qr, keys, vals, c.scale, block, LMK_PATH_AUTO, &stats);
  if (join) join->now();
  return out;
}

// ------------------------------------------------------------------------------------------------ Python entry points
const Tensor& tensor_arg(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a tensor", name);
    throw python_error();
  }
  return THPVariable_Unpack(o);
}
Tensor opt_tensor_arg(PyObject* o, const char* name) { return o == Py_None ? Tensor() : tensor_arg(o, name); }
int64_t int_arg(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
double float_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
void need_args(Py_ssize_t n, Py_ssize_t want) {
  if (n != want) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
    throw python_error();
  }
}
PyObject* wrap_opt(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
template <typename... Ts> PyObject* wrap_tuple(const Ts&... ts) {
  PyObject* out = PyTuple_New(sizeof...(ts));
  if (!out) throw python_error();
  Py_ssize_t i = 0;
  (PyTuple_SET_ITEM(out, i++, wrap_opt(ts)), ...);
  return out;
}

PyObject* py_init(PyObject*, PyObject* arg) {
  HANDLE_TH_ERRORS
  const char* path = PyUnicode_AsUTF8(arg);
  if (!path) throw python_error();
  void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(h != nullptr, "cannot load ", path, ": ", dlerror());
#define X(name)                                                             \
  lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(h, #name));         \
  TORCH_CHECK(lib.name != nullptr, path, " does not export " #name);
  LMK_FUNCS(X)
#undef X
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// fused_attention(q, k, v, is_mem | None, scale | None, block, path)
PyObject* py_fused_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 7);
  const Tensor &q = tensor_arg(a[0], "q"), &k = tensor_arg(a[1], "k"), &v = tensor_arg(a[2], "v");
  const double scale = a[4] == Py_None ? 1.0 / std::sqrt((double)q.size(-1)) : float_arg(a[4]);
  const int64_t block = int_arg(a[5]), path = int_arg(a[6]);
  std::optional<RegularCheck> mask;
  if (a[3] != Py_None) mask.emplace(tensor_arg(a[3], "is_mem"), block);
  const int64_t history = k.size(-2) - q.size(-2);
  LMK_ASSERT(history % block == 0, "key history must be whole blocks");
  Tensor o = fused_attention(q, k, v, history / block, scale, block, path);
  if (mask) LMK_ASSERT(!mask->failed(), "is_mem must mark the last token of every block");
  return THPVariable_Wrap(std::move(o));
  END_HANDLE_TH_ERRORS
}

// check_regular(is_mem, block): the reference's assertion on the landmark mask (flash_landmark_attention.py:393-394)
PyObject* py_check_regular(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 2);
  const Tensor& m = tensor_arg(a[0], "is_mem");
  c10::cuda::OptionalCUDAGuard guard;
  if (m.is_cuda()) guard.set_device(m.device());
  LMK_ASSERT(!RegularCheck(m, int_arg(a[1])).failed(), "is_mem must mark the last token of every block");
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// masked_attention(q, k, v, is_mem, scale, max_groups) -> (o, R, A)
PyObject* py_masked_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 6);
  auto [o, R, A] = masked_fwd_autograd(tensor_arg(a[0], "q"), tensor_arg(a[1], "k"), tensor_arg(a[2], "v"),
                                       tensor_arg(a[3], "is_mem"), float_arg(a[4]), int_arg(a[5]));
  return wrap_tuple(o, R, A);
  END_HANDLE_TH_ERRORS
}

// rotary_apply(q, k, cos, sin, pos0, mode)
PyObject* py_rotary_apply(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 6);
  auto [q, k] = rotary_apply(tensor_arg(a[0], "q"), tensor_arg(a[1], "k"), tensor_arg(a[2], "cos"), tensor_arg(a[3], "sin"),
                             int_arg(a[4]), int_arg(a[5]));
  return wrap_tuple(q, k);
  END_HANDLE_TH_ERRORS
}

// grouped_softmax(x, is_mem, last, hidden | None, guards, max_groups, max_mem_cnt) -> (probs, group_prob | None)
PyObject* py_grouped_softmax(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 7);
  auto [p, gp] = grouped_softmax(tensor_arg(a[0], "x"), tensor_arg(a[1], "is_mem"), tensor_arg(a[2], "last"),
                                 opt_tensor_arg(a[3], "hidden"), int_arg(a[4]) != 0, int_arg(a[5]), int_arg(a[6]));
  return wrap_tuple(p, gp);
  END_HANDLE_TH_ERRORS
}

// grouped_softmax_causal(x, is_mem_row, max_groups)
PyObject* py_grouped_softmax_causal(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 3);
  return THPVariable_Wrap(grouped_softmax_causal(tensor_arg(a[0], "x"), tensor_arg(a[1], "is_mem_row"), int_arg(a[2])));
  END_HANDLE_TH_ERRORS
}

// (out, (keys, values)) with the cache's tokens up to `len` where the call appended to it, else out; None if out is undefined
PyObject* wrap_appended(const Tensor& out, bool append, const Tensor& kc, const Tensor& vc, int64_t len) {
  if (!out.defined() || !append) return wrap_opt(out);
  PyObject *o = THPVariable_Wrap(out), *k = THPVariable_Wrap(kc.narrow(2, 0, len)), *v = THPVariable_Wrap(vc.narrow(2, 0, len));
  PyObject* kv = PyTuple_Pack(2, k, v);
  PyObject* r = PyTuple_Pack(2, o, kv);
  for (PyObject* x : {o, k, v, kv}) Py_DECREF(x);
  return r;
}

// decode_attend(q, k_new, v_new, k_cache, v_cache, len, append, block, top_k, cos, sin) -> see wrap_appended
PyObject* py_decode_attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 11);
  const Tensor &q = tensor_arg(a[0], "q"), &kc = tensor_arg(a[3], "k_cache"), &vc = tensor_arg(a[4], "v_cache");
  const int64_t len = int_arg(a[5]);
  const bool append = int_arg(a[6]) != 0;
  return wrap_appended(decode_attend(q, tensor_arg(a[1], "k_new"), tensor_arg(a[2], "v_new"), kc, vc, len, append, int_arg(a[7]),
                                     int_arg(a[8]), tensor_arg(a[9], "cos"), tensor_arg(a[10], "sin")),
                       append, kc, vc, len + q.size(2));
  END_HANDLE_TH_ERRORS
}

// cache_retrieve(q, k, v, landmark keys, block_first, n, ring_start, block, top_k, cos, sin, mode, tail_k, tail_v, inc, tail_pos)
// -> (att_prefix, values) | (None, None)
PyObject* py_cache_retrieve(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 16);
  auto [att, v] = cache_retrieve(tensor_arg(a[0], "q"), tensor_arg(a[1], "k_cache"), tensor_arg(a[2], "v_cache"),
                                 tensor_arg(a[3], "landmark_keys"), int_arg(a[4]) != 0, int_arg(a[5]), int_arg(a[6]), int_arg(a[7]),
                                 int_arg(a[8]), tensor_arg(a[9], "cos"), tensor_arg(a[10], "sin"), int_arg(a[11]),
                                 tensor_arg(a[12], "tail_k"), tensor_arg(a[13], "tail_v"), int_arg(a[14]), int_arg(a[15]));
  return wrap_tuple(att, v);
  END_HANDLE_TH_ERRORS
}

// prefix_pv(probs, v, y) -> bool
PyObject* py_prefix_pv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 3);
  return PyBool_FromLong(prefix_pv(tensor_arg(a[0], "probs"), tensor_arg(a[1], "v"), tensor_arg(a[2], "y")));
  END_HANDLE_TH_ERRORS
}

// cached_attend(q, k, v, att_prefix, values, is_mem_row, max_groups, scale) -> out | None
PyObject* py_cached_attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 8);
  return wrap_opt(cached_attend(tensor_arg(a[0], "q"), tensor_arg(a[1], "k"), tensor_arg(a[2], "v"), tensor_arg(a[3], "att_prefix"),
                                tensor_arg(a[4], "values"), tensor_arg(a[5], "is_mem"), int_arg(a[6]), float_arg(a[7])));
  END_HANDLE_TH_ERRORS
}

// chunk_attend(q, k_new, v_new, k_cache, v_cache, len, append, block, top_k, cos, sin, rotary) -> see wrap_appended
PyObject* py_chunk_attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 12);
  const Tensor &q = tensor_arg(a[0], "q"), &kc = tensor_arg(a[3], "k_cache"), &vc = tensor_arg(a[4], "v_cache");
  const int64_t len = int_arg(a[5]);
  const bool append = int_arg(a[6]) != 0;
  return wrap_appended(chunk_attend(q, tensor_arg(a[1], "k_new"), tensor_arg(a[2], "v_new"), kc, vc, len, append, int_arg(a[7]),
                                    int_arg(a[8]), tensor_arg(a[9], "cos"), tensor_arg(a[10], "sin"), int_arg(a[11])),
                       append, kc, vc, len + q.size(2));
  END_HANDLE_TH_ERRORS
}

// per_head_attend(q, k_new, v_new, k_cache, v_cache, landmark keys | None, n_blocks, append, block, top_k, cos, sin) -> out | None
PyObject* py_per_head_attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  need_args(n, 12);
  return wrap_opt(per_head_attend(tensor_arg(a[0], "q"), tensor_arg(a[1], "k_new"), tensor_arg(a[2], "v_new"), tensor_arg(a[3], "k_cache"),
                                  tensor_arg(a[4], "v_cache"), opt_tensor_arg(a[5], "landmark keys"), int_arg(a[6]), int_arg(a[7]) != 0,
                                  int_arg(a[8]), int_arg(a[9]), tensor_arg(a[10], "cos"), tensor_arg(a[11], "sin")));
  END_HANDLE_TH_ERRORS
}

#define FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"init", py_init, METH_O, nullptr},
                         FAST("fused_attention", py_fused_attention),
                         FAST("check_regular", py_check_regular),
                         FAST("masked_attention", py_masked_attention),
                         FAST("rotary_apply", py_rotary_apply),
                         FAST("grouped_softmax", py_grouped_softmax),
                         FAST("grouped_softmax_causal", py_grouped_softmax_causal),
                         FAST("decode_attend", py_decode_attend),
                         FAST("cached_attend", py_cached_attend),
                         FAST("chunk_attend", py_chunk_attend),
                         FAST("per_head_attend", py_per_head_attend),
                         FAST("cache_retrieve", py_cache_retrieve),
                         FAST("prefix_pv", py_prefix_pv),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_lmk_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

TORCH_LIBRARY(lmk, m) {
  m.def("masked_attention_fwd(Tensor q, Tensor k, Tensor v, Tensor is_mem, float sm_scale, int max_groups) -> (Tensor, Tensor, Tensor)");
  m.def("masked_attention_bwd(Tensor q, Tensor k, Tensor v, Tensor is_mem, Tensor o, Tensor do, Tensor R, Tensor A, "
        "float sm_scale, int max_groups) -> (Tensor, Tensor, Tensor)");
}
TORCH_LIBRARY_IMPL(lmk, CUDA, m) {
  m.impl("masked_attention_fwd", masked_fwd_cuda);
  m.impl("masked_attention_bwd", masked_bwd_cuda);
}
TORCH_LIBRARY_IMPL(lmk, Autograd, m) { m.impl("masked_attention_fwd", masked_fwd_autograd); }

PyMODINIT_FUNC PyInit__lmk_host(void) { return PyModule_Create(&module); }
