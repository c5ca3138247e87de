// Streaming hard inference over occurrence chains: the state of a (slot, head) is its query and key
// symbol histories, the chain links of its keys and the tables of chain_match.cuh, all of which only
// grow.  Indexing n tokens costs n steps whatever the length of the history; a row then walks the chain of
// its context, length / 2^13 members in a stream without structure, and looks at the whole history once
// where they lie closer (the bitmaps of rosa_b200_stream_update cost n * length / 32 word reads always).
// Semantics as there: reference rosa_soft/csrc/rosa_runtime.cpp:333-482 (chunked update_packed),
// :103-133, :455-467.
//
// Two schedules.  Up to kStepTokens tokens per slot (generation): ONE kernel, one warp per (slot,
// head), does everything from the logits to the unpacked result.  More (prompts): pack and append,
// index (one CTA per slot and head, tables staged in shared memory), match (one thread per row).
#include <algorithm>

#include "chain_kernels.cuh"

namespace rosa {

namespace {

constexpr int kStepTokens = 16;
constexpr int kPacked = -1;            // element type of packed uint8 symbols

struct StreamCall {
  const void *query, *key, *payload;   // token-major [tokens][heads](bits of logits)
  const int32_t* offsets;              // [slots + 1]; null: uniform_chunk tokens per slot
  int64_t tokens;
  int uniform_chunk, slots, H, Hp, group, qk_bits, payload_bits, W;
  uint8_t *query_history, *key_history, *payload_history;
  uint32_t* prev;                      // [slots][H][capacity]
  void* tables;                        // [slots][H][table entries]
  const int32_t* lengths;
  int32_t* lengths_after;
  int64_t capacity, longest;           // longest: of the histories after the update
  int context, hash_bits, entries;
  ChainPatience patience;
  int vec_qk, vec_payload;             // logit rows are whole aligned 16-byte words
  void* output;
  int64_t* matched_end;
};

__device__ __forceinline__ void chunk_of(const StreamCall& c, int s, int* off, int* n) {
  if (c.offsets == nullptr) {
    *off = s * c.uniform_chunk;
    *n = c.uniform_chunk;
  } else {
    *off = c.offsets[s];
    *n = c.offsets[s + 1] - *off;
  }
}

// Symbol of (token, head): packed, or bit d set iff logit d is positive.
template <typename In>
__device__ __forceinline__ uint32_t load_symbol(const void* base, int64_t index, int bits, int vec) {
  if constexpr (sizeof(In) == 1) {
    return (uint32_t)static_cast<const In*>(base)[index] & ((1u << bits) - 1u);
  } else {
    const In* row = static_cast<const In*>(base) + index * bits;
    uint32_t w = 0;
    if (vec) {
      constexpr int kPer = 16 / (int)sizeof(In);
#pragma unroll
      for (int c = 0; c < 8 / kPer; ++c) {
        if (c * kPer >= bits) break;
        const uint4 raw = __ldg(reinterpret_cast<const uint4*>(row) + c);
        const In* e = reinterpret_cast<const In*>(&raw);
#pragma unroll
        for (int x = 0; x < kPer; ++x) w |= (uint32_t)((float)e[x] > 0.0f) << (c * kPer + x);
      }
    } else {
      for (int d = 0; d < bits; ++d) w |= (uint32_t)((float)row[d] > 0.0f) << d;
    }
    return w;
  }
}

// Result of one (token, head): the packed successor symbol, or its bits as +-1 (zeros for no match).
template <typename Out>
__device__ __forceinline__ void store_symbol(void* base, int64_t index, int bits, int vec, bool hit,
                                             uint32_t symbol) {
  if constexpr (sizeof(Out) == 1) {
    static_cast<Out*>(base)[index] = (Out)(hit ? symbol : 0u);
  } else {
    Out* row = static_cast<Out*>(base) + index * bits;
    auto value = [&](int d) { return !hit ? (Out)0.0f : (symbol >> d & 1u) ? (Out)1.0f : (Out)-1.0f; };
    if (vec) {
      constexpr int kPer = 16 / (int)sizeof(Out);
#pragma unroll
      for (int c = 0; c < 8 / kPer; ++c) {
        if (c * kPer >= bits) break;
        alignas(16) Out v[kPer];
#pragma unroll
        for (int x = 0; x < kPer; ++x) v[x] = value(c * kPer + x);
        reinterpret_cast<uint4*>(row)[c] = *reinterpret_cast<const uint4*>(v);
      }
    } else {
      for (int d = 0; d < bits; ++d) row[d] = value(d);
    }
  }
}

// ------------------------------------------------------------------- generation
// One warp per (slot, head).  The tables stay in global memory: a few entries are touched.  What
// bounds it is the latency of about ten dependent reads.
template <typename Entry, typename In, typename Out>
__global__ void __launch_bounds__(128, 4) stream_step_kernel(StreamCall c, int vec_out) {
  __shared__ uint32_t links[4][2][2 * kStepTokens];      // per warp: chained, shorter lengths
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pair = blockIdx.x * 4 + warp;
  if (pair >= c.slots * c.H) return;
  const int s = pair / c.H, h = pair - s * c.H;
  int off, n;
  chunk_of(c, s, &off, &n);
  const int len = c.lengths[s];
  if (h == 0 && lane == 0) c.lengths_after[s] = len + n;
  if (len < 0 || n <= 0 || n > kStepTokens || (int64_t)len + n > c.capacity) return;
  uint8_t* q = c.query_history + (int64_t)pair * c.capacity;
  uint8_t* k = c.key_history + (int64_t)pair * c.capacity;
  uint32_t* prev = c.prev + (int64_t)pair * c.capacity;
  const int hp = c.group == 1 ? h : h / c.group;
  uint8_t* pay = c.payload_history + ((int64_t)s * c.Hp + hp) * c.capacity;
  uint32_t payload = 0u;
  if (lane < n) {
    const int64_t t = (int64_t)off + lane;
    q[len + lane] = (uint8_t)load_symbol<In>(c.query, t * c.H + h, c.qk_bits, c.vec_qk);
    k[len + lane] = (uint8_t)load_symbol<In>(c.key, t * c.H + h, c.qk_bits, c.vec_qk);
    payload = load_symbol<In>(c.payload, t * c.Hp + hp, c.payload_bits, c.vec_payload);
    if (h == hp * c.group) pay[len + lane] = (uint8_t)payload;
  }
  uint32_t* chained = links[warp][0];
  uint32_t* shorter = links[warp][1];
  shorter[lane] = 0u;
  __syncwarp();
  Entry* tables = static_cast<Entry*>(c.tables) + (int64_t)pair * c.entries;
  chain_index_warp<Entry, false, true>(q, k, len, len + n, c.context, c.qk_bits, true, c.hash_bits,
                                       tables, prev, chained - len);
  for (int L = c.context - 1; L >= 1; --L)
    chain_index_warp<Entry, true, true>(
        q, k, len, len + n, L, c.qk_bits, false, c.hash_bits,
        tables + (1 << c.hash_bits) + chain_low_entries(c.qk_bits, L), prev, shorter - len);
  __syncwarp();
  const int i = len + lane;
  int best_len, best_route;
  const bool gave_up = chain_walk<uint8_t>(q, k, prev, lane < n ? chained[lane] : 0u, lane < n ? 0 : -1, i,
                                           c.W, c.patience, lane, best_len, best_route);
  if (!gave_up && best_len < c.context) {
    best_route = (int)(shorter[lane] & 0x0fffffffu);
  }
  for (unsigned rows = __ballot_sync(0xffffffffu, gave_up); rows != 0u; rows &= rows - 1u) {
    const int r = __ffs(rows) - 1;
    int length, route;
    scan_row<uint8_t>(q, k, len + r, c.W, lane, length, route);
    if (lane == r) best_route = route;
  }
  // successors inside the chunk come from the lane that holds them: their history bytes may be
  // on their way from another warp
  const int local = best_route - len;
  const uint32_t fresh = __shfl_sync(0xffffffffu, payload, local & 31);
  if (lane < n) {
    const bool hit = best_route > 0;
    const int64_t row = ((int64_t)off + lane) * c.H + h;
    const uint32_t symbol = !hit ? 0u : local >= 0 ? fresh : (uint32_t)pay[best_route];
    store_symbol<Out>(c.output, row, c.payload_bits, vec_out, hit, symbol);
    c.matched_end[row] = (int64_t)best_route - 1;
  }
}

// ---------------------------------------------------------------------- prompts
// Appends the chunk: one thread per (slot, 16 aligned positions, column), columns being the query,
// key and payload heads, so that a warp reads neighbouring heads of one token after another and
// stores 16 bytes of its own history row.
template <typename In>
__global__ void __launch_bounds__(256) stream_append_chunk_kernel(StreamCall c, int steps_upper) {
  const int columns = 2 * c.H + c.Hp;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t st = idx / columns;
  const int col = (int)(idx - st * columns);
  const int s = (int)(st / steps_upper);
  if (s >= c.slots) return;
  int off, n;
  chunk_of(c, s, &off, &n);
  const int len = c.lengths[s];
  const int step = len / kChainStep + (int)(st - (int64_t)s * steps_upper);
  if (col == 0 && st == (int64_t)s * steps_upper) c.lengths_after[s] = len + n;
  const int begin = max(len, step * kChainStep), end = min(len + n, (step + 1) * kChainStep);
  if (len < 0 || begin >= end || (int64_t)len + n > c.capacity) return;
  const void* src;
  uint8_t* dst;
  int heads, head, bits, vec;
  if (col < 2 * c.H) {
    heads = c.H;
    head = col < c.H ? col : col - c.H;
    src = col < c.H ? c.query : c.key;
    dst = (col < c.H ? c.query_history : c.key_history) + ((int64_t)s * c.H + head) * c.capacity;
    bits = c.qk_bits;
    vec = c.vec_qk;
  } else {
    heads = c.Hp;
    head = col - 2 * c.H;
    src = c.payload;
    dst = c.payload_history + ((int64_t)s * c.Hp + head) * c.capacity;
    bits = c.payload_bits;
    vec = c.vec_payload;
  }
  const int64_t first = (int64_t)(off + begin - len) * heads + head;
  if (end - begin == kChainStep) {
    uint32_t w[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      w[x] = 0u;
#pragma unroll
      for (int y = 0; y < 4; ++y)
        w[x] |= load_symbol<In>(src, first + (int64_t)(4 * x + y) * heads, bits, vec) << (8 * y);
    }
    *reinterpret_cast<uint4*>(dst + begin) = make_uint4(w[0], w[1], w[2], w[3]);
  } else {
    for (int p = begin; p < end; ++p)
      dst[p] = (uint8_t)load_symbol<In>(src, first + (int64_t)(p - begin) * heads, bits, vec);
  }
}

// One CTA per (slot, head), one warp per context length: the tables of the pair are staged in
// shared memory for the chunk.  tokens < 0: the whole histories (after they were loaded or moved).
template <typename Entry, bool kMerge>
__global__ void __maxnreg__(kChainIndexRegisters)
    stream_index_kernel(StreamCall c, int segments, uint32_t* __restrict__ start,
                        uint32_t* __restrict__ low, int32_t* flag) {
  extern __shared__ uint4 staged_words[];
  Entry* staged = reinterpret_cast<Entry*>(staged_words);
  const int pair = blockIdx.x;
  const int s = pair / c.H, h = pair - s * c.H;
  if (pair == 0 && threadIdx.x == 0 && flag != nullptr) *flag = 0;
  const bool whole = c.tokens < 0;
  int off = 0, n = 0;
  if (!whole) chunk_of(c, s, &off, &n);
  const int len = c.lengths[s];
  const int begin = whole ? 0 : len, end = whole ? len : len + n;
  if (len < 0 || begin >= end || (int64_t)end > c.capacity) return;
  Entry* tables = static_cast<Entry*>(c.tables) + (int64_t)pair * c.entries;
  constexpr int kPer = 16 / (int)sizeof(Entry);       // c.entries is a multiple of it
  uint4* outside = reinterpret_cast<uint4*>(tables);
  if (begin == 0) {                                   // a fresh stream: nothing to read
    for (int e = threadIdx.x; e < c.entries / kPer; e += blockDim.x)
      staged_words[e] = make_uint4(0u, 0u, 0u, 0u);
  } else {
    for (int e = threadIdx.x; e < c.entries / kPer; e += blockDim.x) staged_words[e] = outside[e];
  }
  __syncthreads();
  const int64_t at = (int64_t)pair * c.capacity;
  const int64_t row = (int64_t)h * c.tokens + off - len;
  if (!whole)
    chain_index_block<Entry, kMerge, true>(c.query_history + at, c.key_history + at, begin, end, c.context,
                                           c.qk_bits, c.hash_bits, c.entries, segments, staged, c.prev + at,
                                           start + row, low + row);
  else   // keys only: the query lanes index the keys a second time and leave nothing
    chain_index_block<Entry, false, true>(c.key_history + at, c.key_history + at, begin, end, c.context,
                                          c.qk_bits, c.hash_bits, c.entries, segments, staged, c.prev + at,
                                          (uint32_t*)nullptr, (uint32_t*)nullptr);
  __syncthreads();
  // the set of the last piece has seen everything (of the pieces that are not empty)
  const int steps = (end - 1) / kChainStep - begin / kChainStep + 1;
  const int per = (steps + segments - 1) / segments;
  const uint4* newest = staged_words + (int64_t)((steps - 1) / per) * (c.entries / kPer);
  for (int e = threadIdx.x; e < c.entries / kPer; e += blockDim.x) outside[e] = newest[e];
}

// Rows of a chunk over the histories of their slots.
struct StreamAxis {
  StreamCall c;

  __device__ __forceinline__ int locate(int64_t g, int* start, int* i) const {
    int s, off;
    if (c.offsets == nullptr) {
      s = (int)((uint32_t)g / (uint32_t)c.uniform_chunk);
      off = s * c.uniform_chunk;
    } else {
      int lo = 0, hi = c.slots;             // the last slot with offsets[s] <= g
      while (lo + 1 < hi) {
        const int mid = (lo + hi) >> 1;
        if ((int64_t)c.offsets[mid] <= g) lo = mid; else hi = mid;
      }
      s = lo;
      off = c.offsets[s];
    }
    *start = s;
    *i = c.lengths[s] + (int)(g - off);
    return *i >= 0 && (int64_t)*i < c.capacity ? s : -1;
  }
  __device__ __forceinline__ int64_t symbols(int s, int h, int) const {
    return ((int64_t)s * c.H + h) * c.capacity;
  }
  __device__ __forceinline__ int64_t links(int64_t, int64_t g, int h, int) const {
    return (int64_t)h * c.tokens + g;
  }
};

template <typename Out>
struct SymbolEmit {
  StreamCall c;
  int vec;

  __device__ __forceinline__ bool pending(int64_t th) const { return c.matched_end[th] == -2; }

  __device__ __forceinline__ void operator()(int64_t g, int h, int H, int s, int length, int route) const {
    const int64_t th = g * H + h;
    c.matched_end[th] = length < 0 ? -2 : (int64_t)route - 1;
    uint32_t symbol = 0u;
    if (route > 0)
      symbol = c.payload_history[((int64_t)s * c.Hp + (c.group == 1 ? h : h / c.group)) * c.capacity + route];
    store_symbol<Out>(c.output, th, c.payload_bits, vec, route > 0, symbol);
  }
};

template <typename Entry, typename In>
int run_chunk(const StreamCall& c, int out_type, int vec_out, int max_chunk, char* ws,
              cudaStream_t stream) {
  const int64_t rows = c.tokens * c.H;
  int32_t* flag = reinterpret_cast<int32_t*>(ws);
  uint32_t* start = reinterpret_cast<uint32_t*>(ws + 256);
  uint32_t* low = start + rows;
  {
    ProfileScope prof("stream_append", stream);
    const int steps = max_chunk / kChainStep + 2;
    const int64_t threads = (int64_t)c.slots * steps * (2 * c.H + c.Hp);
    stream_append_chunk_kernel<In><<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(c, steps);
    ROSA_CUDA_OK(cudaGetLastError());
  }
  {
    ProfileScope prof("stream_index", stream);
    if (c.context > 2) ROSA_CUDA_OK(cudaMemsetAsync(low, 0, (size_t)rows * sizeof(uint32_t), stream));
    const int set_bytes = c.entries * (int)sizeof(Entry);
    const int segments = chain_segments((int64_t)c.slots * c.H, max_chunk, set_bytes, c.context);
    const int bytes = set_bytes * segments;
    auto kernel = c.context > 2 ? stream_index_kernel<Entry, true> : stream_index_kernel<Entry, false>;
    if (bytes > 48 * 1024)
      ROSA_CUDA_OK(allow_shared(kernel));
    kernel<<<(unsigned)(c.slots * c.H), 32 * c.context * segments, bytes, stream>>>(c, segments, start, low,
                                                                                  flag);
    ROSA_CUDA_OK(cudaGetLastError());
  }
  auto match = [&](auto emit) -> int {
    {
      ProfileScope prof("stream_match", stream);
      if (int rc = launch_chain_match_t<uint8_t>(StreamAxis{c}, c.query_history, c.key_history, c.tokens,
                                                 c.H, c.W, c.context, start, c.prev, low, c.patience,
                                                 flag, emit, stream))
        return rc;
    }
    if (c.longest <= kChainShort) return 0;        // nobody gives up
    return launch_run_match_t<uint8_t>(StreamAxis{c}, c.query_history, c.key_history, c.tokens, c.H, c.W,
                                       flag, emit, stream);
  };
  if (out_type == kPacked) return match(SymbolEmit<uint8_t>{c, vec_out});
  if (out_type == ROSA_B200_F32) return match(SymbolEmit<float>{c, vec_out});
  if (out_type == ROSA_B200_F16) return match(SymbolEmit<__half>{c, vec_out});
  return match(SymbolEmit<__nv_bfloat16>{c, vec_out});
}

template <typename Entry, typename In>
int run_step(const StreamCall& c, int out_type, int vec_out, cudaStream_t stream) {
  ProfileScope prof("stream_step", stream);
  const unsigned grid = (unsigned)((c.slots * c.H + 3) / 4);
  if (out_type == kPacked)
    stream_step_kernel<Entry, In, uint8_t><<<grid, 128, 0, stream>>>(c, vec_out);
  else if (out_type == ROSA_B200_F32)
    stream_step_kernel<Entry, In, float><<<grid, 128, 0, stream>>>(c, vec_out);
  else if (out_type == ROSA_B200_F16)
    stream_step_kernel<Entry, In, __half><<<grid, 128, 0, stream>>>(c, vec_out);
  else
    stream_step_kernel<Entry, In, __nv_bfloat16><<<grid, 128, 0, stream>>>(c, vec_out);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

template <typename Entry>
int run_update(const StreamCall& c, int in_type, int out_type, int vec_out, int max_chunk, char* ws,
               cudaStream_t stream) {
#define ROSA_STREAM_IN(In)                                                    \
  (max_chunk <= kStepTokens ? run_step<Entry, In>(c, out_type, vec_out, stream) \
                            : run_chunk<Entry, In>(c, out_type, vec_out, max_chunk, ws, stream))
  if (in_type == kPacked) return ROSA_STREAM_IN(uint8_t);
  if (in_type == ROSA_B200_F32) return ROSA_STREAM_IN(float);
  if (in_type == ROSA_B200_F16) return ROSA_STREAM_IN(__half);
  return ROSA_STREAM_IN(__nv_bfloat16);
#undef ROSA_STREAM_IN
}

// The tables follow the horizon as it was asked for and the capacity: a state of up to 512 tokens per slot
// holds contexts of 9 bits in 512 buckets (8-bit symbols: 3 KB per slot and head), a larger one the full
// tables (34 KB), with wider entries where a position outgrows them.  The state's owner indexes the
// histories anew when the size of the tables changes.
constexpr int64_t kSmallState = 512;

int stream_context(int qk_bits, int64_t W, int64_t capacity) {
  if (capacity > kSmallState) return chain_context(qk_bits, W, capacity);
  const int c = (9 + qk_bits - 1) / qk_bits;
  return (int64_t)c < W ? c : (int)W;
}

int stream_hash_bits(int qk_bits, int context, int64_t capacity) {
  return chain_hash_bits(qk_bits, context, capacity <= kSmallState ? kSmallState : (int64_t)1 << 30);
}

int table_entries(int qk_bits, int64_t W, int64_t capacity) {
  const int context = stream_context(qk_bits, W, capacity);
  const int n = (1 << stream_hash_bits(qk_bits, context, capacity)) + chain_low_entries(qk_bits, context);
  return (n + 3) / 4 * 4;
}

}  // namespace

}  // namespace rosa

using namespace rosa;

extern "C" {

ROSA_B200_API size_t rosa_b200_stream_table_bytes(int qk_bits, int64_t max_suffix_length, int64_t capacity) {
  if (qk_bits < 1 || qk_bits > 8 || max_suffix_length < 1) return 0;
  return (size_t)table_entries(qk_bits, max_suffix_length, capacity) * (capacity <= kChainNarrow ? 4 : 8);
}

ROSA_B200_API size_t rosa_b200_stream_chained_workspace_bytes(int64_t chunk_tokens, int num_heads) {
  if (chunk_tokens < 0 || num_heads < 1) return 0;
  return 256 + 2 * (size_t)chunk_tokens * (size_t)num_heads * sizeof(uint32_t);
}

ROSA_B200_API int rosa_b200_stream_update_chained(const rosa_b200_stream_call* u, void* workspace,
                                                  size_t workspace_bytes, void* stream) {
  ROSA_REQUIRE(u != nullptr && workspace != nullptr, "null pointer argument");
  ROSA_REQUIRE(u->slots >= 1, "slot count must be >= 1");
  ROSA_REQUIRE(u->num_heads >= 1 && u->num_payload_heads >= 1, "head counts must be >= 1");
  ROSA_REQUIRE(u->num_heads % u->num_payload_heads == 0,
               "num_heads must be divisible by num_payload_heads");
  ROSA_REQUIRE(u->qk_bits >= 1 && u->qk_bits <= 8, "qk_bits must be in [1, 8]");
  ROSA_REQUIRE(u->payload_bits >= 1 && u->payload_bits <= 8, "payload_bits must be in [1, 8]");
  ROSA_REQUIRE(u->max_suffix_length >= 1, "max_suffix_length must be >= 1");
  ROSA_REQUIRE(u->capacity >= 32 && u->capacity % 32 == 0 && u->capacity <= 0x7fffffff - 31,
               "history capacity must be a multiple of 32 in [32, 2^31)");
  const bool reindex = u->chunk_tokens < 0;
  ROSA_REQUIRE(reindex || (u->max_length_after >= 0 && u->max_length_after <= u->capacity),
               "max_length_after exceeds the history capacity");
  ROSA_REQUIRE(u->query_history && u->key_history && u->payload_history && u->chain_links && u->tables &&
                   u->lengths && (reindex || u->lengths_after),
               "null pointer argument");
  ROSA_REQUIRE((reinterpret_cast<uintptr_t>(u->query_history) | reinterpret_cast<uintptr_t>(u->key_history) |
                reinterpret_cast<uintptr_t>(u->payload_history) | reinterpret_cast<uintptr_t>(u->tables)) % 16 == 0,
               "state pointers must be 16-byte aligned");
  ROSA_REQUIRE((int64_t)u->slots * u->num_heads <= 0x7fffffff, "slots * num_heads exceeds the int32 range");
  StreamCall c{};
  c.tokens = reindex ? -1 : u->chunk_tokens;
  c.slots = u->slots; c.H = u->num_heads; c.Hp = u->num_payload_heads;
  c.group = u->num_heads / u->num_payload_heads;
  c.qk_bits = u->qk_bits; c.payload_bits = u->payload_bits;
  c.W = (int)std::min<int64_t>(u->max_suffix_length, u->capacity);
  c.query_history = u->query_history; c.key_history = u->key_history;
  c.payload_history = u->payload_history;
  c.prev = u->chain_links; c.tables = u->tables;
  c.lengths = u->lengths; c.lengths_after = u->lengths_after;
  c.capacity = u->capacity;
  c.context = stream_context(u->qk_bits, u->max_suffix_length, u->capacity);
  c.hash_bits = stream_hash_bits(u->qk_bits, c.context, u->capacity);
  c.entries = table_entries(u->qk_bits, u->max_suffix_length, u->capacity);
  const bool wide = u->capacity > kChainNarrow;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (reindex) {
    const int bytes = c.entries * (wide ? 8 : 4);
    auto kernel = wide ? stream_index_kernel<unsigned long long, false> : stream_index_kernel<uint32_t, false>;
    if (bytes > 48 * 1024)
      ROSA_CUDA_OK(allow_shared(kernel));
    kernel<<<(unsigned)(c.slots * c.H), 32 * c.context, bytes, st>>>(c, 1, nullptr, nullptr, nullptr);
    ROSA_CUDA_OK(cudaGetLastError());
    return 0;
  }
  const size_t need = rosa_b200_stream_chained_workspace_bytes(u->chunk_tokens, u->num_heads);
  ROSA_REQUIRE(workspace_bytes >= need, "workspace too small: need %zu bytes, got %zu", need, workspace_bytes);
  ROSA_REQUIRE(u->chunk_tokens * (int64_t)u->num_heads <= 0x7fffffff,
               "chunk_tokens * num_heads exceeds the int32 range");
  ROSA_REQUIRE(u->input_type >= kPacked && u->input_type <= ROSA_B200_BF16 && u->output_type >= kPacked &&
                   u->output_type <= ROSA_B200_BF16,
               "element types must be packed (-1), float32, float16 or bfloat16");
  ROSA_REQUIRE(u->chunk_tokens == 0 || (u->query && u->key && u->payload && u->output && u->matched_key_end),
               "null pointer argument");
  ROSA_REQUIRE(u->max_chunk >= 0 && u->max_chunk <= u->max_length_after, "max_chunk exceeds max_length_after");
  ROSA_REQUIRE(u->chunk_offsets != nullptr || u->max_chunk * (int64_t)u->slots == u->chunk_tokens,
               "without chunk_offsets every slot gets max_chunk tokens");
  c.longest = u->max_length_after;
  c.patience = chain_patience(c.qk_bits, c.context, c.longest);
  // A step is one kernel with a warp per row: a member (two reads one after the other) takes as long as a
  // round of 128 positions of the scan.
  if (u->max_chunk <= kStepTokens)
    c.patience = {(int)std::max<int64_t>(32, 4 * (c.longest >> c.hash_bits)), 0};
  c.query = u->query; c.key = u->key; c.payload = u->payload;
  c.offsets = u->chunk_offsets;
  c.uniform_chunk = (int)std::max<int64_t>(1, u->max_chunk);
  c.output = u->output; c.matched_end = u->matched_key_end;
  const auto size_of = [](int type) { return type == kPacked ? 1 : type == ROSA_B200_F32 ? 4 : 2; };
  const auto whole = [](const void* p, int bytes) {
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && bytes % 16 == 0;
  };
  c.vec_qk = whole(u->query, c.qk_bits * size_of(u->input_type)) &&
             whole(u->key, c.qk_bits * size_of(u->input_type));
  c.vec_payload = whole(u->payload, c.payload_bits * size_of(u->input_type));
  const int vec_out = whole(u->output, c.payload_bits * size_of(u->output_type));
  if (u->chunk_tokens == 0) {     // nothing to append: the lengths still move to their next place
    ROSA_CUDA_OK(cudaMemcpyAsync(u->lengths_after, u->lengths, (size_t)u->slots * sizeof(int32_t),
                                 cudaMemcpyDeviceToDevice, st));
    return 0;
  }
  char* ws = static_cast<char*>(workspace);
  const int max_chunk = (int)u->max_chunk;
  return wide ? run_update<unsigned long long>(c, u->input_type, u->output_type, vec_out, max_chunk, ws, st)
              : run_update<uint32_t>(c, u->input_type, u->output_type, vec_out, max_chunk, ws, st);
}

}  // extern "C"
