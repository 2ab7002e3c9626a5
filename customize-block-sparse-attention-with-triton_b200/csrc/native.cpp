// Native host path of the public op: checks, workspaces, launches and the autograd node in C++, so that
// a call costs a few microseconds of host time instead of forty (the kernels of a short sequence take
// less than ten).  Everything on the device is done by the C-ABI library (include/bsattn.h); this file
// only knows torch tensors.
//
// A call that is out of the ordinary in any way (wrong types or shapes, no mask, a library call that
// refuses) is answered with None, and the Python layer takes it, which also raises the errors.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <mutex>
#include <unordered_map>

#include "../../include/bsattn.h"

namespace {

using at::Tensor;
constexpr int64_t kBlock = 64;

// ---------------------------------------------------------------------------------------------
// Per (device, stream): the zeroed work counter of the persistent kernels (they leave it at zero, also
// after a bounded wait gave up), and a status word in pinned host memory, which the device can write
// and the host can read without a synchronisation.
// ---------------------------------------------------------------------------------------------
struct StreamState {
  Tensor counter, dq_counter, status;
  int32_t *counter_ptr, *dq_counter_ptr;  // (the dQ kernel runs beside the dK/dV kernel, and has its own)
  volatile int32_t* word;
};

struct StreamKey {
  int device;
  cudaStream_t stream;
  bool operator==(const StreamKey& o) const { return device == o.device && stream == o.stream; }
};
struct StreamHash {
  size_t operator()(const StreamKey& k) const {
    return std::hash<void*>()(k.stream) * 31u + static_cast<size_t>(k.device);
  }
};

// nullptr: the stream is being captured and has no state yet (nothing that outlives the graph is allocated
// inside a capture: no report).  `device` is the current device.
StreamState* stream_state(int device, cudaStream_t stream) {
  thread_local StreamKey last_key{-1, nullptr};
  thread_local StreamState* last = nullptr;
  const StreamKey key{device, stream};
  if (last != nullptr && last_key == key) return last;
  static std::mutex mutex;
  static auto* states = new std::unordered_map<StreamKey, StreamState*, StreamHash>();  // never torn down
  std::lock_guard<std::mutex> lock(mutex);
  auto it = states->find(key);
  if (it == states->end()) {
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return nullptr;
    auto* st = new StreamState;
    // ordinary tensors whatever the mode of the call that comes first: both layers write to them later
    const c10::InferenceMode no_inference(false);
    // zeroed on the stream that will use it, so no cross-stream ordering is needed
    st->counter = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
    st->dq_counter = at::zeros_like(st->counter);
    st->status = at::zeros({1}, at::TensorOptions().dtype(at::kInt)).pin_memory();
    st->counter_ptr = st->counter.data_ptr<int32_t>();
    st->dq_counter_ptr = st->dq_counter.data_ptr<int32_t>();
    st->word = st->status.data_ptr<int32_t>();
    it = states->emplace(key, st).first;
  }
  last_key = key;
  return last = it->second;
}

// The work counters of a call's n kernels (two: dK/dV's and dQ's) for `blocks` blocks; none when a CTA has one of
// them at most.  A captured call may be replayed on any stream, beside calls on this one, and two kernels must
// not draw from one counter: it gets words of its own (*own, out of the graph's memory, zeroed by one node of
// the graph).  B200, replayed calls with this stream's counter / zeroed words / none: forward of one head,
// N = 17536, a tenth of the blocks 20.5 / 22.0 / 22.5 us; forward and backward of 4 heads, N = 6400, causal, a
// quarter 65.5 / 67.6 / 67.6 us (67.8 with a node for each word).
void work_counters(StreamState* state, int64_t blocks, const at::TensorOptions& options, int n, Tensor* own,
                   int32_t** counters) {
  for (int i = 0; i < n; ++i) counters[i] = nullptr;
  if (blocks <= at::cuda::getDeviceProperties(options.device().index())->multiProcessorCount) return;
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None) {
    if (state == nullptr) return;
    counters[0] = state->counter_ptr;
    if (n > 1) counters[1] = state->dq_counter_ptr;
    return;
  }
  *own = at::zeros({n}, options.dtype(at::kInt));
  for (int i = 0; i < n; ++i) counters[i] = own->mutable_data_ptr<int32_t>() + i;
}

// ---------------------------------------------------------------------------------------------
// Arguments
// ---------------------------------------------------------------------------------------------
// TMA needs a unit inner stride, 16-byte aligned base and outer strides.
Tensor tma_ready(const Tensor& t) {
  bool ok = t.stride(3) == 1 && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
  for (int i = 0; ok && i < 3; ++i) ok = t.stride(i) > 0 && t.stride(i) % 8 == 0;
  return ok ? t : t.contiguous();
}

// (Plain pointers and strides: each view of a tensor costs the host as much as a tenth of a small call.)
struct Mask {
  Tensor owner;                // what the block mask was reduced into, if it was
  const uint8_t* block;        // bytes [Bm,Hm,nb,nb]
  int64_t Bm, Hm, block_strides[4];
  Tensor dense;                // the mask of [Bm,Hm,N,N] elements (or an aligned copy of it), or undefined
  const uint8_t* dense_ptr = nullptr;
  int64_t dense_strides[4];    // (0 for a broadcast axis)
};

// The op's mask argument; false when it is nothing that this path takes.
bool read_mask(const Tensor& mask, int64_t B, int64_t H, int64_t N, const Tensor& q, void* stream, Mask* out) {
  const int64_t dims = mask.dim(), nb = N / kBlock;
  if (dims < 2 || dims > 4 || mask.device() != q.device()) return false;
  if (mask.scalar_type() != at::kBool && mask.scalar_type() != at::kByte) return false;
  // axes that are missing in front have size 1
  int64_t sizes[4], strides[4];
  const auto look_at = [&](const Tensor& m) {
    for (int64_t i = 0; i < 4; ++i) {
      const int64_t d = i - (4 - dims);
      sizes[i] = d < 0 ? 1 : m.size(d);
      strides[i] = d < 0 ? m.size(0) * m.stride(0) : m.stride(d);
    }
  };
  look_at(mask);
  if ((sizes[0] != 1 && sizes[0] != B) || (sizes[1] != 1 && sizes[1] != H)) return false;
  out->Bm = sizes[0];
  out->Hm = sizes[1];
  if (sizes[2] == nb && sizes[3] == nb) {
    out->block = static_cast<const uint8_t*>(mask.const_data_ptr());
    for (int i = 0; i < 4; ++i) out->block_strides[i] = strides[i];
    return true;
  }
  if (sizes[2] != N || sizes[3] != N) return false;
  // a dense mask: reduced to blocks, the partly kept ones marked 2, and applied inside those
  bool ok = strides[3] == 1 && reinterpret_cast<uintptr_t>(mask.const_data_ptr()) % 16 == 0;
  for (int i = 0; ok && i < 3; ++i) ok = strides[i] % 16 == 0;
  out->dense = ok ? mask : mask.contiguous();
  if (!ok) look_at(out->dense);
  out->owner = at::empty({sizes[0], sizes[1], nb, nb}, mask.options().dtype(at::kByte));
  uint8_t* block = out->owner.mutable_data_ptr<uint8_t>();
  out->block = block;
  out->dense_ptr = static_cast<const uint8_t*>(out->dense.const_data_ptr());
  for (int i = 0; i < 4; ++i) {
    out->dense_strides[i] = strides[i];
    out->block_strides[i] = out->owner.stride(i);
  }
  if (bsa_mask_reduce(out->dense_ptr, out->dense_strides, sizes[0], sizes[1], N, block, nullptr, 1, stream) != 0)
    return false;
  for (int i = 0; i < 2; ++i)
    if (sizes[i] == 1) out->dense_strides[i] = 0;  // broadcast
  return true;
}

int dtype_code(const Tensor& t) { return t.scalar_type() == at::kHalf ? BSA_F16 : BSA_BF16; }

// The tile lists of one call in one buffer of words: counts of the row and column lists, then their
// entries, every list in a place of nb words.
struct Lists {
  int64_t col_cnt, col_idx, row_idx, words;
  Lists(int64_t Bm, int64_t Hm, int64_t nb) {
    const int64_t rows = Bm * Hm * nb;
    col_cnt = rows;
    col_idx = (2 * rows + 3) & ~int64_t{3};
    row_idx = col_idx + rows * nb;
    words = row_idx + rows * nb;
  }
};

// Runs the forward; with lse2 and lists also what a backward needs.  False when the library refused.  (The
// forward lists each mask row inside the kernel.  The lists are written while it is still running, so their
// memory has to be allocated before the copies that q, k, v may be are given back.)
bool run_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Mask& m, double scale,
                 StreamState* state, void* stream, Tensor* o, Tensor* lse2, Tensor* lists) {
  const int64_t B = q.size(0), H = q.size(1), N = q.size(2), D = q.size(3);
  *o = at::empty({B, H, N, D}, q.options());
  Tensor own;
  int32_t* counter;
  work_counters(state, B * H * (N / kBlock), q.options(), 1, &own, &counter);
  int32_t* status = state ? const_cast<int32_t*>(state->word) : nullptr;
  const int64_t* dense_strides = m.dense_ptr ? m.dense_strides : nullptr;
  if (lists == nullptr)
    return bsa_attn_fwd_block_mask_output(
               q.const_data_ptr(), q.strides().data(), k.const_data_ptr(), k.strides().data(),
               v.const_data_ptr(), v.strides().data(), o->mutable_data_ptr(), o->strides().data(), m.block,
               m.block_strides, m.Bm, m.Hm, static_cast<float>(scale), dtype_code(q), B, H, N, D, m.dense_ptr,
               dense_strides, counter, status, stream) == 0;
  *lse2 = at::empty({B, H, N}, q.options().dtype(at::kFloat));
  const Lists at(m.Bm, m.Hm, N / kBlock);
  *lists = at::empty({at.words}, q.options().dtype(at::kInt));
  int32_t* p = lists->mutable_data_ptr<int32_t>();
  return bsa_attn_fwd_block_mask_lists(
             q.const_data_ptr(), q.strides().data(), k.const_data_ptr(), k.strides().data(),
             v.const_data_ptr(), v.strides().data(), o->mutable_data_ptr(), o->strides().data(),
             lse2->mutable_data_ptr<float>(), m.block, m.block_strides, m.Bm, m.Hm, static_cast<float>(scale),
             dtype_code(q), B, H, N, D, m.dense_ptr, dense_strides, p, p + at.col_idx, p + at.col_cnt,
             p + at.row_idx, counter, status, stream) == 0;
}

// ---------------------------------------------------------------------------------------------
// Errors of the backward: raised by the Python layer's function (fn, status, what a kernel reported), on
// whatever thread
// ---------------------------------------------------------------------------------------------
PyObject* raise_error = nullptr;

[[noreturn]] void raise_in_python(const char* fn, int status, int code = 0) {
  pybind11::gil_scoped_acquire gil;
  PyObject* r = PyObject_CallFunction(raise_error, "sii", fn, status, code);
  Py_XDECREF(r);  // (it always raises)
  python_error err;
  err.persist();
  throw err;
}
void check(const char* fn, int rc) {
  if (rc != 0) raise_in_python(fn, rc);
}

// Raises what an earlier kernel reported on this stream, if anything.  The report is taken: the word is
// zero again, and of several threads that look at the same time one raises.
void raise_if_reported(StreamState* state) {
  if (state == nullptr || *state->word == 0) return;
  const int code = __atomic_exchange_n(state->word, 0, __ATOMIC_RELAXED);
  if (code != 0) raise_in_python("flash_attention_custom_mask", BSA_ERR_DEVICE_TIMEOUT, code);
}

// ---------------------------------------------------------------------------------------------
// Autograd
// ---------------------------------------------------------------------------------------------
// (A node of its own and not torch::autograd::Function: that keeps what is saved in a map of boxed values,
// which costs a small call another 10 us.)
struct AttentionBackward : torch::autograd::Node {
  torch::autograd::SavedVariable q_, k_, v_, o_, lse2_, lists_;
  Tensor dense;  // the caller's mask (or an aligned copy of it): not to be changed before backward
  int64_t Bm, Hm, nb, dense_strides[4];
  float scale;

  std::string name() const override { return "AttentionBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto* s : {&q_, &k_, &v_, &o_, &lse2_, &lists_}) s->reset_data();
    dense.reset();
  }

  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    // (unpacking raises when the buffers have been released or an input was modified in place)
    const Tensor q = tma_ready(q_.unpack()), k = tma_ready(k_.unpack()), v = tma_ready(v_.unpack());
    const Tensor o = o_.unpack(shared_from_this()), lse2 = lse2_.unpack(), lists = lists_.unpack();
    at::AutoDispatchBelowADInplaceOrView no_autograd;
    const int64_t B = q.size(0), H = q.size(1), N = q.size(2), D = q.size(3);
    if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor()};
    const Tensor dout = tma_ready(grads[0].to(q.scalar_type()));
    const Lists at(Bm, Hm, nb);
    const uint8_t* dense_ptr = dense.defined() ? static_cast<const uint8_t*>(dense.const_data_ptr()) : nullptr;
    const c10::cuda::CUDAGuard guard(q.device());
    const cudaStream_t stream = at::cuda::getCurrentCUDAStream(q.device().index());
    StreamState* state = stream_state(q.device().index(), stream);
    raise_if_reported(state);
    Tensor own;
    int32_t* counters[2];
    work_counters(state, B * H * nb, q.options(), 2, &own, counters);
    int32_t* status = state ? const_cast<int32_t*>(state->word) : nullptr;
    // the gradients are laid out like the tensors they belong to, gaps included
    const auto like = [](const Tensor& t) { return at::empty_strided(t.sizes(), t.strides(), t.options()); };
    Tensor dq = like(q), dk = like(k), dv = like(v);
    const Tensor delta = at::empty({B, H, N}, lse2.options());
    const float* lse_p = lse2.const_data_ptr<float>();
    float* delta_p = delta.mutable_data_ptr<float>();
    const int32_t* p = lists.const_data_ptr<int32_t>();
    const int code = dtype_code(q), sb = Bm > 1 ? Hm : 0, sh = Hm > 1 ? 1 : 0;
    check("bsa_attn_bwd_delta_strided",
          bsa_attn_bwd_delta_strided(o.const_data_ptr(), o.strides().data(), dout.const_data_ptr(),
                                     dout.strides().data(), delta_p, code, B, H, N, D, stream));
    check("bsa_attn_bwd_strided",
          bsa_attn_bwd_strided(
              q.const_data_ptr(), q.strides().data(), k.const_data_ptr(), k.strides().data(),
              v.const_data_ptr(), v.strides().data(), dout.const_data_ptr(), dout.strides().data(), lse_p,
              delta_p, dq.mutable_data_ptr(), dq.strides().data(), dk.mutable_data_ptr(), dk.strides().data(),
              dv.mutable_data_ptr(), dv.strides().data(), p, p + at.col_idx, p + at.col_cnt, p + at.row_idx, nb, sb,
              sh, scale, code, B, H, N, D, dense_ptr, dense_ptr ? dense_strides : nullptr, counters[0], counters[1],
              status, stream));
    return {dq, dk, dv};
  }
};

// The forward with its node; undefined when the library refused.
Tensor forward_with_grad(const Tensor& q0, const Tensor& k0, const Tensor& v0, const Mask& m, double scale,
                         StreamState* state, void* stream) {
  std::shared_ptr<AttentionBackward> node(new AttentionBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(q0, k0, v0));
  Tensor o, lse2, lists;
  {
    at::AutoDispatchBelowADInplaceOrView no_autograd;
    if (!run_forward(tma_ready(q0), tma_ready(k0), tma_ready(v0), m, scale, state, stream, &o, &lse2, &lists))
      return Tensor();
  }
  node->Bm = m.Bm;
  node->Hm = m.Hm;
  node->nb = q0.size(2) / kBlock;
  node->dense = m.dense;
  for (int i = 0; i < 4; ++i) node->dense_strides[i] = m.dense_strides[i];
  node->scale = static_cast<float>(scale);
  node->q_ = torch::autograd::SavedVariable(q0, false);
  node->k_ = torch::autograd::SavedVariable(k0, false);
  node->v_ = torch::autograd::SavedVariable(v0, false);
  // (saved like the rest, so that offloading and checkpointing hooks get hold of all the memory)
  node->lse2_ = torch::autograd::SavedVariable(lse2, false);
  node->lists_ = torch::autograd::SavedVariable(lists, false);
  torch::autograd::set_history(o, node);
  node->o_ = torch::autograd::SavedVariable(o, true);
  return o;
}

std::optional<Tensor> attention(const Tensor& q, const Tensor& k, const Tensor& v,
                                const std::optional<Tensor>& mask, double scale) {
  if (!mask.has_value() || !q.is_cuda() || q.dim() != 4 || k.sizes() != q.sizes() || v.sizes() != q.sizes())
    return std::nullopt;
  const auto type = q.scalar_type();
  if ((type != at::kHalf && type != at::kBFloat16) || k.scalar_type() != type || v.scalar_type() != type ||
      k.device() != q.device() || v.device() != q.device())
    return std::nullopt;
  // the tracer would see the outputs being allocated and no kernel; the Python layer refuses to be traced
  if (torch::jit::tracer::isTracing()) return std::nullopt;
  // there is no forward derivative: the Python layer's Function says so, where this path would lose the tangent
  if (q._fw_grad(0).defined() || k._fw_grad(0).defined() || v._fw_grad(0).defined()) return std::nullopt;
  const int64_t B = q.size(0), H = q.size(1), N = q.size(2), D = q.size(3);
  if ((D != 16 && D != 32 && D != 64) || B == 0 || H == 0 || N == 0 || N % kBlock != 0) return std::nullopt;
  const c10::cuda::CUDAGuard guard(q.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream(q.device().index());
  StreamState* state = stream_state(q.device().index(), stream);
  if (state != nullptr && *state->word != 0) return std::nullopt;  // a report of an earlier kernel
  Mask m;
  if (!read_mask(*mask, B, H, N, q, stream, &m)) return std::nullopt;
  if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad())) {
    Tensor o = forward_with_grad(q, k, v, m, scale, state, stream);
    return o.defined() ? std::optional<Tensor>(o) : std::nullopt;
  }
  Tensor o;
  if (!run_forward(tma_ready(q), tma_ready(k), tma_ready(v), m, scale, state, stream, &o, nullptr, nullptr))
    return std::nullopt;
  return o;
}

// The image tokens (those behind the first n_text) of one to three tensors [B,heads,tokens,D] reordered in
// place; false when the tensors, the plan or the grid are nothing that one launch takes, or an earlier
// kernel has left a report.
bool permute_tokens(const std::vector<Tensor>& tensors, const Tensor& plan, int64_t F, int64_t Hh, int64_t W,
                    int64_t n_text, bool inverse) {
  const Tensor& t0 = tensors[0];
  if (tensors.size() > 3 || !t0.is_cuda() || t0.dim() != 4 || plan.device() != t0.device() || plan.dim() != 1 ||
      (plan.scalar_type() != at::kLong && plan.scalar_type() != at::kInt) || plan.size(0) != t0.size(1) ||
      n_text < 0 || t0.size(2) - n_text != F * Hh * W)
    return false;
  void* ptrs[3];
  int64_t strides[12];
  for (size_t i = 0; i < tensors.size(); ++i) {
    const Tensor& t = tensors[i];
    if (t.sizes() != t0.sizes() || t.scalar_type() != t0.scalar_type() || t.device() != t0.device() ||
        (t.requires_grad() && at::GradMode::is_enabled()))
      return false;
    for (size_t j = 0; j < i; ++j)
      if (t.is_alias_of(tensors[j])) return false;  // they may overlap, or be one tensor given twice
    ptrs[i] = static_cast<char*>(t.mutable_data_ptr()) + n_text * t.stride(2) * t.element_size();
    for (int d = 0; d < 4; ++d) strides[4 * i + d] = t.stride(d);
    // rows that overlap (expanded tensors) cannot be reordered in place
    for (int d = 0; d < 3; ++d)
      if (t.size(d) > 1 && t.stride(d) < t.size(3)) return false;
  }
  const c10::cuda::CUDAGuard guard(t0.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream(t0.device().index());
  StreamState* state = stream_state(t0.device().index(), stream);
  if (state != nullptr && *state->word != 0) return false;
  if (bsa_permute_in_place_status(ptrs, strides, tensors.size(), plan.const_data_ptr(), plan.element_size(),
                                  plan.stride(0), inverse ? 1 : 0, t0.size(0), t0.size(1), F * Hh * W, t0.size(3),
                                  F, Hh, W, t0.element_size(),
                                  state ? const_cast<int32_t*>(state->word) : nullptr, stream) != 0)
    return false;
  for (const Tensor& t : tensors)
    if (!t.is_inference()) t.unsafeGetTensorImpl()->bump_version();  // (inference tensors have no version)
  return true;
}

std::optional<std::pair<Tensor, Tensor>> state_tensors(int64_t device, int64_t stream) {
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
  StreamState* st = stream_state(static_cast<int>(device), reinterpret_cast<cudaStream_t>(stream));
  if (st == nullptr) return std::nullopt;
  return std::make_pair(st->counter, st->status);
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  m.def("attention", &attention);
  m.def("permute_tokens", &permute_tokens);
  m.def("state_tensors", &state_tensors);
  m.def("set_raise", [](pybind11::object f) { raise_error = f.release().ptr(); });
}
