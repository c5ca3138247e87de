// Torch side of the streaming runtime: the state on the GPU (StreamCore), the custom class
// torch.classes.rosa_soft.RosaRuntime with the reference's constructor and methods
// (rosa_soft/csrc/rosa_runtime.cpp:300-331, 333-482, 484-582) and the Python class behind
// rosa_soft_b200.RosaRuntime.  Every update is one rosa_b200_stream_update_chained call on the
// current stream.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime_api.h>
#include <torch/custom_class.h>
#include <torch/extension.h>

#include <algorithm>
#include <limits>
#include <mutex>
#include <optional>
#include <tuple>
#include <vector>

#include "autograd_binding.h"
#include "rosa_soft_b200.h"

namespace {

using torch::Tensor;
using Pair = std::tuple<Tensor, Tensor>;

constexpr int64_t kInt32Max = std::numeric_limits<int32_t>::max();
constexpr int64_t kMinCapacity = 256;
constexpr int kPacked = -1;

int element_type(torch::ScalarType t) {   // -2: not taken by the kernels
  switch (t) {
    case torch::kUInt8: return kPacked;
    case torch::kFloat32: return ROSA_B200_F32;
    case torch::kFloat16: return ROSA_B200_F16;
    case torch::kBFloat16: return ROSA_B200_BF16;
    default: return -2;
  }
}

// The state of a runtime and its update.  Callers have validated what they pass.
class StreamCore {
 public:
  StreamCore(int64_t heads, int64_t payload_heads, int64_t qk_bits, int64_t payload_bits, int64_t horizon)
      : heads_(heads), payload_heads_(payload_heads), qk_bits_(qk_bits), payload_bits_(payload_bits),
        horizon_(horizon) {}

  int64_t slots() const { return slots_; }
  int64_t capacity() const { return capacity_; }
  const std::vector<int64_t>& lengths() const { return lengths_; }
  bool on(const c10::Device& device) const { return device == device_; }

  void clear() {
    query_ = key_ = payload_ = links_ = tables_ = lens_ = scratch_ = Tensor();
    lengths_.clear();
    slots_ = -1;
    capacity_ = 0;
    phase_ = 0;
    longest_ = 0;
    ordered_ = false;
    last_ = at::cuda::CUDAEvent();   // an event stays with the device of its first record
    home_.reset();
    last_stream_.reset();
  }

  // The first update fixes the slots of a fresh runtime, unless it fails.
  struct Opening {
    Opening(StreamCore* core, int64_t slots, const c10::Device& device)
        : core_(core->slots_ == -1 ? core : nullptr) {
      if (core_ != nullptr) core_->open(slots, device);
    }
    ~Opening() {
      if (core_ != nullptr) core_->clear();
    }
    void keep() const { core_ = nullptr; }
    Pair done(Pair result) const {
      keep();
      return result;
    }
    mutable StreamCore* core_;
  };

  // Fixes the slots of a fresh runtime.
  void open(int64_t slots, const c10::Device& device) {
    slots_ = slots;
    device_ = device;
    lengths_.assign(static_cast<size_t>(slots), 0);
  }

  // Appends one chunk.  `offsets` undefined: `max_chunk` tokens for every slot; otherwise device
  // int32 offsets, and `chunk[s]` the host's view of the same chunk lengths.  The state is shared by
  // all updates: whatever stream the previous one ran on, this one starts after it.
  Pair append(const Tensor& query, const Tensor& key, const Tensor& payload, const Tensor& offsets,
              const std::vector<int64_t>* chunk, int64_t tokens, int64_t max_chunk,
              torch::ScalarType out_type, torch::IntArrayRef shape) {
    const auto stream = at::cuda::getCurrentCUDAStream(device_.index());
    if (ordered_ && stream != *last_stream_) last_.block(stream);
    int64_t after = longest_ + max_chunk;
    if (chunk != nullptr) {
      after = 0;
      for (size_t s = 0; s < lengths_.size(); ++s) after = std::max(after, lengths_[s] + (*chunk)[s]);
    }
    TORCH_CHECK(after <= kInt32Max - 31, "ROSA sequence length exceeded int32 range");
    grow(after, stream);
    const Tensor q = query.contiguous(), k = key.contiguous(), p = payload.contiguous();
    const bool packed = out_type == torch::kUInt8;
    std::vector<int64_t> out_shape = shape.vec();
    Tensor end = torch::empty(out_shape, lens_.options().dtype(torch::kInt64));
    if (!packed) out_shape.push_back(payload_bits_);
    Tensor out = torch::empty(out_shape, lens_.options().dtype(out_type));
    const size_t bytes = rosa_b200_stream_chained_workspace_bytes(tokens, (int)heads_);
    const bool step = bytes <= (size_t)scratch_.numel();
    Tensor ws = step ? scratch_
                     : torch::empty({static_cast<int64_t>(bytes)}, lens_.options().dtype(torch::kUInt8));
    rosa_b200_stream_call u = state_of_call();
    u.query = q.data_ptr(); u.key = k.data_ptr(); u.payload = p.data_ptr();
    u.input_type = element_type(q.scalar_type());
    u.output_type = element_type(out_type);
    u.chunk_offsets = offsets.defined() ? offsets.data_ptr<int32_t>() : nullptr;
    u.chunk_tokens = tokens; u.max_chunk = max_chunk; u.max_length_after = after;
    u.output = out.data_ptr(); u.matched_key_end = end.data_ptr<int64_t>();
    const int rc = rosa_b200_stream_update_chained(&u, ws.data_ptr(), (size_t)ws.numel(), stream.stream());
    TORCH_CHECK(rc == 0, "RosaRuntime update: ", rosa_b200_last_error());
    touched_on(stream);
    // committed only once the update has been enqueued
    if (chunk == nullptr) {
      for (auto& n : lengths_) n += max_chunk;
    } else {
      for (size_t s = 0; s < lengths_.size(); ++s) lengths_[s] += (*chunk)[s];
    }
    longest_ = after;
    phase_ ^= 1;
    return {out, end};
  }

  // The update of [slots, tokens, heads(, bits)] tensors if it is plainly valid, else nothing: the
  // caller then finds out what is wrong (or takes the general way).
  std::optional<Pair> dense(const Tensor& query, const Tensor& key, const Tensor& payload,
                            bool return_packed, std::optional<torch::ScalarType> out_type) {
    const auto type = query.scalar_type();
    const bool logits = type != torch::kUInt8;
    const int64_t rank = logits ? 4 : 3;
    if (element_type(type) == -2 || key.scalar_type() != type || payload.scalar_type() != type ||
        query.dim() != rank || payload.dim() != rank || query.sizes() != key.sizes())
      return std::nullopt;
    const auto out = return_packed ? torch::kUInt8 : out_type.value_or(type);
    if (element_type(out) == -2 || (!return_packed && out == torch::kUInt8)) return std::nullopt;
    const int64_t B = query.size(0), T = query.size(1);
    if (B < 1 || payload.size(0) != B || payload.size(1) != T || query.size(2) != heads_ ||
        payload.size(2) != payload_heads_ ||
        (logits && (query.size(3) != qk_bits_ || payload.size(3) != payload_bits_)))
      return std::nullopt;
    const auto device = query.device();
    if (!device.is_cuda() || key.device() != device || payload.device() != device ||
        B * T * heads_ > kInt32Max || (slots_ != -1 && (slots_ != B || device != device_)))
      return std::nullopt;
    const c10::cuda::OptionalCUDAGuard guard(device);
    const Opening opening(this, B, device);
    return opening.done(append(query, key, payload, Tensor(), nullptr, B * T, T, out,
                               query.sizes().slice(0, 3)));
  }

  // Chunks of host-known lengths: offsets[s] .. offsets[s + 1] of the token axis; `device_offsets`
  // (int32, optional) holds the same numbers on the GPU already.
  Pair packed(const Tensor& query, const Tensor& key, const Tensor& payload,
              const std::vector<int64_t>& offsets, const std::optional<Tensor>& device_offsets,
              torch::ScalarType out_type, torch::IntArrayRef shape) {
    const c10::Device device = query.device();
    const c10::cuda::OptionalCUDAGuard guard(device);
    const int64_t slots = (int64_t)offsets.size() - 1;
    const Opening opening(this, slots, device);
    std::vector<int64_t> chunk(static_cast<size_t>(slots));
    int64_t longest = 0, shortest = kInt32Max;
    for (int64_t s = 0; s < slots; ++s) {
      chunk[s] = offsets[s + 1] - offsets[s];
      longest = std::max(longest, chunk[s]);
      shortest = std::min(shortest, chunk[s]);
    }
    Tensor dev;
    if (longest != shortest) {
      if (device_offsets.has_value()) {
        dev = device_offsets->contiguous();
      } else {
        Tensor host = torch::empty({slots + 1}, torch::kInt32);
        std::copy(offsets.begin(), offsets.end(), host.data_ptr<int32_t>());
        dev = host.to(device, /*non_blocking=*/true);
      }
    }
    return opening.done(append(query, key, payload, dev, &chunk, offsets.back(), longest, out_type, shape));
  }

  // Copies on the current stream, after the last update and before the next.
  std::tuple<Tensor, Tensor, Tensor> export_histories() {
    const c10::cuda::OptionalCUDAGuard guard(device_);
    const auto stream = at::cuda::getCurrentCUDAStream(device_.index());
    if (ordered_ && stream != *last_stream_) last_.block(stream);
    const int64_t used = longest_;
    auto cut = [&](const Tensor& t) { return t.narrow(2, 0, used).clone(); };
    std::tuple<Tensor, Tensor, Tensor> copies{cut(query_), cut(key_), cut(payload_)};
    touched_on(stream);
    return copies;
  }

  void import_histories(const std::vector<int64_t>& lengths, const Tensor& query, const Tensor& key,
                        const Tensor& payload) {
    clear();
    const c10::Device device = query.device();
    const c10::cuda::OptionalCUDAGuard guard(device);
    const Opening opening(this, (int64_t)lengths.size(), device);   // a load that fails leaves nothing
    const int64_t used = query.size(2);
    const auto stream = at::cuda::getCurrentCUDAStream(device_.index());
    grow(std::max(used, *std::max_element(lengths.begin(), lengths.end())), stream);
    query_.narrow(2, 0, used).copy_(query);
    key_.narrow(2, 0, used).copy_(key);
    payload_.narrow(2, 0, used).copy_(payload);
    Tensor host = torch::empty({(int64_t)lengths.size()}, torch::kInt32);
    std::copy(lengths.begin(), lengths.end(), host.data_ptr<int32_t>());
    lens_.select(0, phase_).copy_(host);
    lengths_ = lengths;
    longest_ = *std::max_element(lengths.begin(), lengths.end());
    reindex(stream);
    touched_on(stream);
    opening.keep();
  }

 private:
  rosa_b200_stream_call state_of_call() const {
    rosa_b200_stream_call u{};
    u.slots = (int)slots_; u.num_heads = (int)heads_; u.num_payload_heads = (int)payload_heads_;
    u.qk_bits = (int)qk_bits_; u.payload_bits = (int)payload_bits_;
    u.max_suffix_length = horizon_; u.capacity = capacity_;
    u.query_history = query_.data_ptr<uint8_t>();
    u.key_history = key_.data_ptr<uint8_t>();
    u.payload_history = payload_.data_ptr<uint8_t>();
    u.chain_links = reinterpret_cast<uint32_t*>(links_.data_ptr<int32_t>());
    u.tables = tables_.data_ptr();
    u.lengths = lens_.data_ptr<int32_t>() + phase_ * slots_;
    u.lengths_after = lens_.data_ptr<int32_t>() + (phase_ ^ 1) * slots_;
    return u;
  }

  // Work on `stream` touches the state: its memory, allocated on another stream perhaps, may not be
  // handed out again before that work is done.
  void used_on(const c10::cuda::CUDAStream& stream) const {
    if (stream == *home_) return;
    for (const Tensor& t : {query_, key_, payload_, links_, tables_, lens_, scratch_})
      c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), stream);
  }

  // ... and whatever touches the state next starts after it.
  void touched_on(const c10::cuda::CUDAStream& stream) {
    used_on(stream);
    last_.record(stream);
    last_stream_ = stream;
    ordered_ = true;
  }

  void reindex(const c10::cuda::CUDAStream& stream) {
    rosa_b200_stream_call u = state_of_call();
    u.chunk_tokens = -1;
    const int rc = rosa_b200_stream_update_chained(&u, scratch_.data_ptr(), (size_t)scratch_.numel(),
                                                   stream.stream());
    TORCH_CHECK(rc == 0, "RosaRuntime index: ", rosa_b200_last_error());
  }

  // Room for `needed` tokens per slot: the capacity doubles, old contents are kept.  All copies are
  // enqueued on the update's stream.
  void grow(int64_t needed, const c10::cuda::CUDAStream& stream) {
    if (needed <= capacity_ && capacity_ > 0) return;
    int64_t capacity = std::max<int64_t>(kMinCapacity, capacity_);
    while (capacity < needed) capacity *= 2;
    const auto u8 = torch::TensorOptions().device(device_).dtype(torch::kUInt8);
    const auto i32 = u8.dtype(torch::kInt32);
    auto moved = [&](const Tensor& old, int64_t heads, const torch::TensorOptions& options) {
      Tensor t = torch::empty({slots_, heads, capacity}, options);
      if (capacity_ > 0) {
        const size_t item = t.element_size();
        C10_CUDA_CHECK(cudaMemcpy2DAsync(t.data_ptr(), capacity * item, old.data_ptr(), capacity_ * item,
                                         capacity_ * item, slots_ * heads, cudaMemcpyDeviceToDevice,
                                         stream.stream()));
      }
      return t;
    };
    Tensor query = moved(query_, heads_, u8), key = moved(key_, heads_, u8);
    Tensor payload = moved(payload_, payload_heads_, u8), links = moved(links_, heads_, i32);
    const int64_t table = (int64_t)rosa_b200_stream_table_bytes((int)qk_bits_, horizon_, capacity);
    const bool rebuilt = capacity_ > 0 && table != table_bytes_;
    Tensor tables = tables_, lens = lens_, scratch = scratch_;
    if (capacity_ == 0) {
      lens = torch::zeros({2, slots_}, i32);
      scratch = torch::empty({kScratchBytes}, u8);
    } else if (stream != *home_) {
      lens = lens_.clone();
      scratch = torch::empty({kScratchBytes}, u8);
      if (!rebuilt) tables = tables_.clone();
    }
    if (capacity_ == 0 || rebuilt) tables = torch::zeros({slots_, heads_, table}, u8);
    // everything is allocated: an update that runs out of memory leaves the state as it was.  The old
    // tensors are read by copies on this stream, whatever stream they go back to.
    if (capacity_ > 0) used_on(stream);
    query_ = query; key_ = key; payload_ = payload; links_ = links;
    tables_ = tables; lens_ = lens; scratch_ = scratch;
    table_bytes_ = table;
    capacity_ = capacity;
    home_ = stream;
    // recorded here, not only by the update that grows: if that one fails after this, the next may come
    // on the stream of the one before
    touched_on(stream);
    if (rebuilt) {
      reindex(stream);
      touched_on(stream);
    }
  }

  // workspace of an update that is one kernel, and of any update of up to 8000 token-heads
  static constexpr int64_t kScratchBytes = 64 * 1024;

  const int64_t heads_, payload_heads_, qk_bits_, payload_bits_, horizon_;
  int64_t slots_ = -1, capacity_ = 0, longest_ = 0, table_bytes_ = 0;
  int phase_ = 0;                  // which half of lens_ is current
  c10::Device device_{c10::kCPU};
  std::vector<int64_t> lengths_;
  Tensor query_, key_, payload_, links_, tables_, lens_, scratch_;
  std::optional<c10::cuda::CUDAStream> home_, last_stream_;   // of the allocation, of the last update
  at::cuda::CUDAEvent last_;
  bool ordered_ = false;
};

// torch.classes.rosa_soft.RosaRuntime: update_packed(cu_seqlens, query, key, payload) -> (output
// uint8 [total, H], matched_key_end int64 [total, H]), reset, close, stats.  cu_seqlens is read on
// the host (int32 or int64, CPU or CUDA) like the reference reads it, because the chunk lengths size
// the state.
class RosaRuntimeClass : public torch::CustomClassHolder {
 public:
  RosaRuntimeClass(int64_t num_heads, int64_t num_payload_heads, int64_t qk_bits,
                   int64_t payload_bits, int64_t max_suffix_length)
      : heads_(num_heads), payload_heads_(num_payload_heads), qk_bits_(qk_bits),
        core_(num_heads, num_payload_heads, qk_bits, payload_bits, max_suffix_length) {
    enforce({{heads_ > 0, "num_heads must be positive"},
             {payload_heads_ > 0, "num_payload_heads must be positive"},
             {payload_heads_ > 0 && heads_ % payload_heads_ == 0,
              "num_heads must be divisible by num_payload_heads"},
             {qk_bits > 0 && qk_bits <= 8, "qk_bits must be in [1, 8]"},
             {payload_bits > 0 && payload_bits <= 8, "payload_bits must be in [1, 8]"},
             {max_suffix_length > 0 && max_suffix_length <= kInt32Max,
              "max_suffix_length must be in [1, int32_max]"}});
  }

  std::tuple<Tensor, Tensor> update_packed(const Tensor& cu_seqlens, const Tensor& query,
                                           const Tensor& key, const Tensor& payload) {
    std::lock_guard<std::mutex> lock(mutex_);
    TORCH_CHECK(!closed_, "RosaRuntime is closed");
    enforce({{query.is_cuda() && key.is_cuda() && payload.is_cuda(),
              "RosaRuntime keeps its state on the GPU: query, key and payload must be CUDA tensors"},
             {query.scalar_type() == torch::kUInt8 && key.scalar_type() == torch::kUInt8 &&
                  payload.scalar_type() == torch::kUInt8,
              "query, key and payload must have dtype uint8"},
             {query.dim() == 2 && key.dim() == 2 && payload.dim() == 2,
              "query, key and payload must be two-dimensional (total_tokens, heads)"},
             {cu_seqlens.dim() == 1 && cu_seqlens.numel() >= 2,
              "cu_seqlens must be one-dimensional with at least two entries"},
             {cu_seqlens.scalar_type() == torch::kInt32 || cu_seqlens.scalar_type() == torch::kInt64,
              "cu_seqlens must be int32 or int64"}});
    enforce({{query.sizes() == key.sizes(), "query/key shape mismatch"},
             {query.size(1) == heads_, "query head count must equal num_heads"},
             {payload.size(1) == payload_heads_, "payload head count must equal num_payload_heads"},
             {payload.size(0) == query.size(0), "query/payload token mismatch"},
             {query.device() == key.device() && query.device() == payload.device(),
              "query, key and payload must be on the same CUDA device"}});
    const Tensor host_cu = cu_seqlens.to(torch::kCPU, torch::kInt64).contiguous();
    const int64_t* cu = host_cu.data_ptr<int64_t>();
    const int64_t slots = host_cu.numel() - 1;
    const int64_t total = query.size(0);
    TORCH_CHECK(cu[0] == 0, "cu_seqlens must start at 0");
    for (int64_t s = 0; s < slots; ++s)
      TORCH_CHECK(cu[s + 1] >= cu[s], "cu_seqlens must be non-decreasing");
    TORCH_CHECK(cu[slots] == total, "cu_seqlens[-1] must equal the total token count");
    if (core_.slots() >= 0) {
      TORCH_CHECK(slots == core_.slots(), "RosaRuntime slot count is fixed after the first update");
      TORCH_CHECK(core_.on(query.device()), "RosaRuntime state lives on another device");
    }
    return core_.packed(query, key, payload, std::vector<int64_t>(cu, cu + slots + 1), std::nullopt,
                        torch::kUInt8, query.sizes());
  }

  void reset() {
    std::lock_guard<std::mutex> lock(mutex_);
    TORCH_CHECK(!closed_, "RosaRuntime is closed");
    core_.clear();
  }

  void close() {
    std::lock_guard<std::mutex> lock(mutex_);
    core_.clear();
    closed_ = true;
  }

  // (states, edges, payload_symbols, automata, sequences, logical_bytes): there is no
  // automaton, so the first two are zero; the bytes are those of the histories and chain links.
  std::tuple<int64_t, int64_t, int64_t, int64_t, int64_t, int64_t> stats() const {
    std::lock_guard<std::mutex> lock(mutex_);
    int64_t tokens = 0;
    for (int64_t n : core_.lengths()) tokens += n;
    const int64_t slots = std::max<int64_t>(0, core_.slots());
    return {0, 0, tokens * payload_heads_, slots * heads_, slots,
            tokens * (heads_ * kTokenHeadBytes + payload_heads_)};
  }

 private:
  static void enforce(std::initializer_list<std::pair<bool, const char*>> rules) {
    for (const auto& rule : rules) TORCH_CHECK(rule.first, rule.second);
  }
  static constexpr int64_t kTokenHeadBytes = 6;   // query and key symbol, chain link

  const int64_t heads_, payload_heads_, qk_bits_;
  bool closed_ = false;
  StreamCore core_;
  mutable std::mutex mutex_;
};

torch::ScalarType scalar_type(const py::object& dtype) {
  return dtype.is_none() ? torch::kUInt8 : torch::python::detail::py_object_to_dtype(dtype);
}

}  // namespace

TORCH_LIBRARY_FRAGMENT(rosa_soft, m) {
  m.class_<RosaRuntimeClass>("RosaRuntime")
      .def(torch::init<int64_t, int64_t, int64_t, int64_t, int64_t>())
      .def("update_packed", &RosaRuntimeClass::update_packed)
      .def("reset", &RosaRuntimeClass::reset)
      .def("close", &RosaRuntimeClass::close)
      .def("stats", &RosaRuntimeClass::stats);
}

PYBIND11_MODULE(_C, m) {
  m.doc() = "rosa_soft_b200 operator registration, differentiable operator and streaming state";
  bind_autograd(m);
  py::class_<StreamCore>(m, "StreamCore")
      .def(py::init<int64_t, int64_t, int64_t, int64_t, int64_t>())
      .def_property_readonly("slots", &StreamCore::slots)
      .def_property_readonly("capacity", &StreamCore::capacity)
      .def_property_readonly("lengths", &StreamCore::lengths)
      .def("on", [](const StreamCore& c, const torch::Device& device) { return c.on(device); })
      .def("clear", &StreamCore::clear)
      // packed results: out_type None; values of the payload's type: dense(..., False, None)
      .def("dense",
           [](StreamCore& c, const Tensor& q, const Tensor& k, const Tensor& p, bool return_packed,
              const py::object& out_type) {
             return c.dense(q, k, p, return_packed,
                            out_type.is_none() ? std::nullopt
                                               : std::optional<torch::ScalarType>(scalar_type(out_type)));
           })
      .def("packed",
           [](StreamCore& c, const Tensor& q, const Tensor& k, const Tensor& p,
              const std::vector<int64_t>& offsets, const std::optional<Tensor>& device_offsets,
              const py::object& out_type, const std::vector<int64_t>& shape) {
             return c.packed(q, k, p, offsets, device_offsets, scalar_type(out_type), shape);
           })
      .def("export_histories", &StreamCore::export_histories)
      .def("import_histories", &StreamCore::import_histories);
}
