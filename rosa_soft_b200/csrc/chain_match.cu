// Hard matching of whole sequences through occurrence chains (chain_match.cuh): an index kernel
// that links the positions, and a match kernel that resolves the rows and writes the result of
// the call (routed value signs, or payload rows and matched positions).
#include "common.cuh"
#include "chain_match.cuh"
#include "row_emit.cuh"

namespace rosa {

namespace {

// One CTA per (sequence, head), one warp per context length.  A warp takes 16 positions at a
// time: lanes 0..15 hold the key contexts that end there, lanes 16..31 the query contexts.  One
// match.any finds the lanes of equal bucket; a lane's predecessor is the nearest lower key lane
// of its bucket, or, without one, the table entry that earlier steps left.  Only the newest key
// lane of a bucket writes the table, after all lanes have read it, so the links are those of a
// strictly sequential pass.  What bounds it is the latency of a step (a table read, the vote and
// a table write, about 150 cycles) times len / 16; the context words of the next four steps are
// requested before the current ones are processed, which keeps global latency out of that chain.
__global__ void chain_index_kernel(Plan plan, const int32_t* __restrict__ qsym,
                                   const int32_t* __restrict__ ksym, int64_t sym_seq_stride,
                                   int64_t sym_head_stride, int H, int bits, int context,
                                   int hash_bits, uint32_t* __restrict__ start,
                                   uint32_t* __restrict__ prev, uint32_t* __restrict__ low) {
  extern __shared__ uint32_t tables[];
  if (plan.cu_seqlens == nullptr && blockIdx.x == 0 && threadIdx.x < 4) plan.status[threadIdx.x] = 0;
  const int seq = blockIdx.x / H, h = blockIdx.x - seq * H;
  int64_t base = (int64_t)seq * sym_seq_stride + (int64_t)h * sym_head_stride;
  int len = plan.uniform_len;
  if (plan.cu_seqlens != nullptr) {
    if (plan.status[0] != 0) return;
    base += plan.seg_start[seq];
    len = plan.seg_len[seq];
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int L = context - warp;                    // warp 0: the chained length
  const int entries = (1 << hash_bits) + chain_low_entries(bits, context);
  for (int e = threadIdx.x; e < entries; e += blockDim.x) tables[e] = 0u;
  __syncthreads();
  uint32_t* __restrict__ table = warp == 0 ? tables : tables + (1 << hash_bits) + chain_low_entries(bits, L);
  const bool is_query = lane >= kChainStep;
  const int l = lane & (kChainStep - 1);
  const int32_t* __restrict__ sym = (is_query ? qsym : ksym) + base;
  const int context_bits = bits * L;
  const uint32_t context_mask = context_bits >= 32 ? 0xffffffffu : (1u << context_bits) - 1u;
  const int first_valid = is_query ? L : L - 1;    // a query at i needs a key context at j < i
  // bucket of the context that ends at p from its newest two symbols; lanes without one get a
  // value of their own that matches nobody
  auto bucket_of = [&](int p, int newest, int second) -> uint32_t {
    if (p < first_valid || p >= len) return 0x80000000u | (unsigned)lane;
    uint32_t w = (uint32_t)newest;
    if (L > 1) w |= (uint32_t)second << bits;
    for (int u = 2; u < L; ++u) w |= (uint32_t)__ldg(sym + p - u) << (bits * u);
    w &= context_mask;
    return warp == 0 ? chain_bucket(w, context_bits, hash_bits) : w;
  };
  auto newest_at = [&](int p) { return p < len ? __ldg(sym + p) : 0; };
  auto second_at = [&](int p) { return L > 1 && p >= 1 && p < len ? __ldg(sym + p - 1) : 0; };
  constexpr int kAhead = 4;
  uint32_t bucket[kAhead];
#pragma unroll
  for (int s = 0; s < kAhead; ++s) {
    const int p = s * kChainStep + l;
    bucket[s] = bucket_of(p, newest_at(p), second_at(p));
  }
  for (int p0 = 0; p0 < len; p0 += kAhead * kChainStep) {
    int a[kAhead], b[kAhead];
#pragma unroll
    for (int s = 0; s < kAhead; ++s) {
      const int p = p0 + (kAhead + s) * kChainStep + l;
      a[s] = newest_at(p);
      b[s] = second_at(p);
    }
#pragma unroll
    for (int s = 0; s < kAhead; ++s) {
      const int p = p0 + s * kChainStep + l;
      const uint32_t own = bucket[s];
      const bool valid = (int)own >= 0;
      const unsigned keys = __match_any_sync(0xffffffffu, own) & 0xffffu;
      const unsigned below = keys & ((1u << l) - 1u);
      uint32_t link = 0u;                          // position + 1 of the predecessor
      if (below != 0u) link = (uint32_t)(p - l + 32 - __clz(below));
      else if (valid) link = table[own];
      __syncwarp();
      if (!is_query && valid && (keys >> l) == 1u) table[own] = (uint32_t)p + 1u;
      __syncwarp();
      if (p < len) {
        if (warp == 0) {
          (is_query ? start : prev)[base + p] = link;
        } else if (is_query) {
          // one shorter length: its warp owns the array; several: the longest that occurs wins
          const uint32_t key = link != 0u ? ((uint32_t)L << 28) | link : 0u;
          if (context == 2) low[base + p] = key;
          else if (key != 0u) atomicMax(low + base + p, key);
        }
      }
    }
#pragma unroll
    for (int s = 0; s < kAhead; ++s)
      bucket[s] = bucket_of(p0 + (kAhead + s) * kChainStep + l, a[s], b[s]);
  }
}

// One thread per row: a warp takes 32 consecutive tokens of one head (its symbol and link reads
// coalesce), a CTA eight heads of them; the winners change places in shared memory so that the
// results go out with the heads of a token side by side.  Bound by the latency and the sector
// rate of the dependent chain reads in L2; many rows in flight hide it.
constexpr int kChainRows = 32;
constexpr int kChainHeads = 8;

template <typename Emit>
__global__ void __launch_bounds__(kChainRows * kChainHeads)
    chain_match_kernel(Plan plan, const int32_t* __restrict__ qsym, const int32_t* __restrict__ ksym,
                       int64_t sym_seq_stride, int64_t sym_head_stride, int64_t N, int H, int W,
                       int context, const uint32_t* __restrict__ start_link,
                       const uint32_t* __restrict__ prev, const uint32_t* __restrict__ low,
                       int head_blocks, unsigned long long gave_up_key, int32_t* flag, Emit emit) {
  __shared__ uint2 s_win[kChainRows][kChainHeads + 1];   // (length, route)
  __shared__ int s_start[kChainRows];
  const int heads = blockDim.x / kChainRows;             // heads of this CTA
  const int tile = blockIdx.x / head_blocks;
  const int h0 = (blockIdx.x - tile * head_blocks) * heads;
  const int64_t g0 = (int64_t)tile * kChainRows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int h = h0 + warp;
  const int64_t g = g0 + lane;
  int start = 0, len = 0, best_len = 0, best_route = 0;
  int seq = -1;
  bool gave_up = false;
  if (g < N) seq = find_segment(plan, g, &start, &len);
  if (seq >= 0 && h < H) {
    const int i = (int)(g - start);
    const int64_t base = (int64_t)seq * sym_seq_stride + (int64_t)h * sym_head_stride +
                         (plan.cu_seqlens == nullptr ? 0 : start);
    const uint32_t first = start_link[base + i];
    const uint32_t shorter = context > 1 ? low[base + i] : 0u;
    chain_walk<int32_t>(qsym + base, ksym + base, prev + base, first, i, W, best_len, best_route,
                        gave_up);
    if (best_len < context && !gave_up) {
      best_len = (int)(shorter >> 28);
      best_route = (int)(shorter & 0x0fffffffu);
    }
  }
  if (gave_up) {
    best_len = (int)(gave_up_key >> 32);
    best_route = (int)(gave_up_key & 0xffffffffull);
    *flag = 1;
  }
  s_win[lane][warp] = make_uint2((unsigned)best_len, (unsigned)best_route);
  if (warp == 0) s_start[lane] = start;
  __syncthreads();
  const int r = threadIdx.x / heads, hh = threadIdx.x - r * heads;
  if (g0 + r < N && h0 + hh < H) {
    const uint2 win = s_win[r][hh];
    emit(g0 + r, h0 + hh, H, s_start[r], (int)win.x, (int)win.y);
  }
}

template <typename Emit>
int launch_chain_match_t(const FwdArgs& a, unsigned long long gave_up_key, Emit emit,
                         cudaStream_t stream) {
  const int heads = a.H < kChainHeads ? a.H : kChainHeads;
  const int head_blocks = (a.H + heads - 1) / heads;
  const int64_t tiles = (a.N + kChainRows - 1) / kChainRows;
  chain_match_kernel<Emit><<<(unsigned)(tiles * head_blocks), kChainRows * heads, 0, stream>>>(
      a.plan, a.packed_q, a.packed_k, a.sym_seq_stride, a.sym_head_stride, a.N, a.H, a.W,
      chain_context(a.D, a.W), a.chain_start, a.chain_prev, a.chain_low, head_blocks, gave_up_key,
      a.plan.status + 2, emit);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace

int launch_chain_index(const FwdArgs& a, int64_t max_len, cudaStream_t stream) {
  ProfileScope prof("chain_index", stream);
  const int context = chain_context(a.D, a.W);
  const int hash_bits = chain_hash_bits(a.D, context, max_len);
  if (context > 2)   // several shorter lengths merge their results into zeroed words
    ROSA_CUDA_OK(cudaMemsetAsync(a.chain_low, 0, (size_t)a.N * a.H * sizeof(uint32_t), stream));
  const size_t smem = ((size_t)(1 << hash_bits) + chain_low_entries(a.D, context)) * sizeof(uint32_t);
  chain_index_kernel<<<(unsigned)(a.plan.S * a.H), 32 * context, smem, stream>>>(
      a.plan, a.packed_q, a.packed_k, a.sym_seq_stride, a.sym_head_stride, a.H, a.D, context,
      hash_bits, a.chain_start, a.chain_prev, a.chain_low);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

int launch_chain_forward(const FwdArgs& a, unsigned long long gave_up_key, cudaStream_t stream) {
  ProfileScope prof("hard_match", stream);
  return with_sign_emit(a, [&](auto emit) {
    return launch_chain_match_t(a, gave_up_key, emit, stream);
  });
}

int launch_chain_inference(const FwdArgs& a, const float* payload, float* out, int64_t* matched_end,
                           cudaStream_t stream) {
  ProfileScope prof("hard_match", stream);
  const auto aligned = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
  PayloadEmit emit{payload, out, matched_end, a.best, a.Hv, a.Dv,
                   a.Dv % 4 == 0 && aligned(payload) && aligned(out)};
  return launch_chain_match_t(a, 0ull, emit, stream);
}

}  // namespace rosa
