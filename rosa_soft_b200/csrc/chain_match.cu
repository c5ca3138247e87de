// Hard matching of whole sequences through occurrence chains (chain_match.cuh): an index kernel
// that links the positions, and a match kernel that resolves the rows and writes the result of
// the call (routed value signs, or payload rows and matched positions).
#include "common.cuh"
#include "chain_match.cuh"
#include "row_emit.cuh"

namespace rosa {

namespace {

// One CTA per (sequence, head), one warp per context length.  A warp takes 16 positions at a
// time: lanes 0..15 hold the key contexts that end there, lanes 16..31 the query contexts.  A table
// entry is the last step in which a key context fell into the bucket and the mask of its lanes in
// that step, so one read gives both the latest earlier position and the equal lanes of the step
// itself.  A step reads the old entry, stores its own and reads back; key lanes whose bit was
// overwritten by another lane of the same bucket then add it.  The links are those of a strictly
// sequential pass.  What bounds it is the latency of that chain of three shared-memory accesses
// times len / 16 (finding the equal lanes with match.any instead took 330-380 ns a step); the
// symbols of the next eight steps are requested before the current ones are processed, which keeps
// global latency out of it.  The results of a step are selected, not branched on: 128 ns a step
// against 315 with branches (4096 tokens, 128 streams: 81 us before).
template <typename Entry, bool kMerge>
__global__ void chain_index_kernel(Plan plan, const int32_t* __restrict__ qsym,
                                   const int32_t* __restrict__ ksym, int64_t sym_seq_stride,
                                   int64_t sym_head_stride, int H, int bits, int context,
                                   int hash_bits, uint32_t* __restrict__ start,
                                   uint32_t* __restrict__ prev, uint32_t* __restrict__ low) {
  extern __shared__ unsigned long long table_words[];
  Entry* tables = reinterpret_cast<Entry*>(table_words);
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
  for (int e = threadIdx.x; e < entries; e += blockDim.x) tables[e] = 0;
  __syncthreads();
  Entry* table = warp == 0 ? tables : tables + (1 << hash_bits) + chain_low_entries(bits, L);
  const bool is_query = lane >= kChainStep;
  const int l = lane & (kChainStep - 1);
  const int32_t* __restrict__ sym = (is_query ? qsym : ksym) + base;
  const int context_bits = bits * L;
  const uint32_t context_mask = context_bits >= 32 ? 0xffffffffu : (1u << context_bits) - 1u;
  const int first_valid = is_query ? L : L - 1;    // a query at i needs a key context at j < i
  // bucket of the context that ends at p from its newest two symbols; ~0 where there is none
  auto bucket_of = [&](int p, int newest, int second) -> uint32_t {
    uint32_t w = (uint32_t)newest;
    if (L > 1) w |= (uint32_t)second << bits;
    if (kMerge)
      for (int u = 2; u < L; ++u)
        if (p >= first_valid && p < len) w |= (uint32_t)__ldg(sym + p - u) << (bits * u);
    w &= context_mask;
    if (warp == 0) w = chain_bucket(w, context_bits, hash_bits);
    return p >= first_valid && p < len ? w : 0xffffffffu;
  };
  auto newest_at = [&](int p) { return p < len ? __ldg(sym + p) : 0; };
  auto second_at = [&](int p) { return L > 1 && p >= 1 && p < len ? __ldg(sym + p - 1) : 0; };
  // where this lane's links go: the chained length writes both kinds, a shorter one the queries'
  uint32_t* dst = (warp > 0 ? low : is_query ? start : prev) + base;
  const bool writes = warp == 0 || is_query;
  const uint32_t tag = warp == 0 ? 0u : (uint32_t)L << 28;
  uint32_t bucket[kChainAhead];
#pragma unroll
  for (int s = 0; s < kChainAhead; ++s) {
    const int p = s * kChainStep + l;
    bucket[s] = bucket_of(p, newest_at(p), second_at(p));
  }
  const unsigned own_bit = 1u << l;
  for (int p0 = 0; p0 < len; p0 += kChainAhead * kChainStep) {
    int a[kChainAhead], b[kChainAhead];
#pragma unroll
    for (int s = 0; s < kChainAhead; ++s) {
      const int p = p0 + (kChainAhead + s) * kChainStep + l;
      a[s] = newest_at(p);
      b[s] = second_at(p);
    }
#pragma unroll
    for (int s = 0; s < kChainAhead; ++s) {
      const int p = p0 + s * kChainStep + l;
      const bool valid = bucket[s] != 0xffffffffu;
      const bool is_key = valid && !is_query;
      Entry* slot = table + (valid ? bucket[s] : 0u);
      const Entry step = (Entry)(p0 / kChainStep + s + 1) << 16;
      const Entry old = *slot;
      __syncwarp();
      if (is_key) *slot = step | own_bit;
      __syncwarp();
      Entry now = *slot;
      if (__any_sync(0xffffffffu, is_key && ((unsigned)now & own_bit) == 0u)) {
        if (is_key && ((unsigned)now & own_bit) == 0u) atomicOr(slot, (Entry)own_bit);
        __syncwarp();
        now = *slot;
      }
      // the newest key lane below this one, else the newest of the bucket's last step
      const unsigned below = (now >> 16) == (step >> 16) ? (unsigned)now & (own_bit - 1u) : 0u;
      const Entry from = below != 0u ? step | below : old;
      // position + 1 of the predecessor: bit b of step n (from 1) is position 16 (n - 1) + b
      uint32_t link = (uint32_t)(from >> 16) * kChainStep + 16u - (uint32_t)__clz((unsigned)from & 0xffffu);
      link = from != 0 && valid ? link | tag : 0u;
      if (writes && p < len) {
        // one shorter length: its warp owns the array; several: the longest that occurs wins
        if (kMerge && warp > 0) {
          if (link != 0u) atomicMax(dst + p, link);
        } else {
          dst[p] = link;
        }
      }
    }
#pragma unroll
    for (int s = 0; s < kChainAhead; ++s)
      bucket[s] = bucket_of(p0 + (kChainAhead + s) * kChainStep + l, a[s], b[s]);
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
                       int head_blocks, int limit, int32_t* flag, Emit emit) {
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
  if (g < N && h < H) seq = find_segment(plan, g, &start, &len);
  const int i = (int)(g - start);
  int64_t base = 0;
  uint32_t first = 0u, shorter = 0u;
  if (seq >= 0) {
    base = (int64_t)seq * sym_seq_stride + (int64_t)h * sym_head_stride +
           (plan.cu_seqlens == nullptr ? 0 : start);
    first = start_link[base + i];
    if (context > 1) shorter = low[base + i];
  }
  if (chain_walk<int32_t>(qsym + base, ksym + base, prev + base, first, seq, i, W, limit, lane,
                          best_len, best_route)) {
    best_len = (int)(kChainGaveUp >> 32);          // resolved by a matcher of whole warps
    best_route = 0;
    *flag = 1;
  } else if (best_len < context) {
    best_len = (int)(shorter >> 28);
    best_route = (int)(shorter & 0x0fffffffu);
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

// A warp resolves a row that gave up by a look at every earlier position, newest first, 32 at a
// time: lanes whose position agrees with the row here and at the distance of the best length so far
// extend it.  Cost per row: len / 32 coalesced reads, whatever the chains look like.
constexpr int kScanWarps = 8;

template <typename Emit>
__global__ void __launch_bounds__(kScanWarps * 32)
    scan_match_kernel(Plan plan, const int32_t* __restrict__ qsym, const int32_t* __restrict__ ksym,
                      int64_t sym_seq_stride, int64_t sym_head_stride, int64_t N, int H, int W,
                      const int32_t* __restrict__ run_flag, Emit emit) {
  if (*run_flag == 0) return;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * kScanWarps, count = N * H;
  for (int64_t th0 = ((int64_t)blockIdx.x * kScanWarps + (threadIdx.x >> 5)) * 32; th0 < count;
       th0 += warps * 32) {
    const bool mine = th0 + lane < count && emit.pending(th0 + lane);
    for (unsigned rows = __ballot_sync(0xffffffffu, mine); rows != 0u; rows &= rows - 1u) {
      const int64_t th = th0 + __ffs(rows) - 1;
      const int64_t g = th / H;
      const int h = (int)(th - g * H);
      int start = 0, len = 0;
      const int seq = find_segment(plan, g, &start, &len);
      const int i = (int)(g - start);
      const int64_t base = (int64_t)seq * sym_seq_stride + (int64_t)h * sym_head_stride +
                           (plan.cu_seqlens == nullptr ? 0 : start);
      const int32_t* __restrict__ q = qsym + base;
      const int32_t* __restrict__ k = ksym + base;
      const int q_i = q[i];
      int best_len = 0, best_route = 0;              // the same in every lane
      for (int top = i - 1; top >= 0 && best_len < min(W, top + 1); top -= 32) {
        const int j = top - lane;
        int length = 0;
        if (j >= best_len && k[j] == q_i && k[j - best_len] == q[i - best_len])
          length = chain_extend<int32_t>(q, k, i, j, 1, min(W, j + 1));
        const int longest = __reduce_max_sync(0xffffffffu, length);
        if (longest > best_len) {
          best_len = longest;
          best_route = __reduce_max_sync(0xffffffffu, length == longest ? j + 1 : 0);
        }
      }
      if (lane == 0) emit(g, h, H, start, best_len, best_route);
    }
  }
}

template <typename Emit>
int launch_scan_match_t(const FwdArgs& a, const int32_t* run_flag, Emit emit, cudaStream_t stream) {
  ProfileScope prof("hard_match_scan", stream);
  // a grid that fills the GPU: it is launched whether or not a row gave up
  scan_match_kernel<Emit><<<148 * 8, kScanWarps * 32, 0, stream>>>(
      a.plan, a.packed_q, a.packed_k, a.sym_seq_stride, a.sym_head_stride, a.N, a.H, a.W,
      run_flag, emit);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

template <typename Emit>
int launch_chain_match_t(const FwdArgs& a, int limit, Emit emit, cudaStream_t stream) {
  const int heads = a.H < kChainHeads ? a.H : kChainHeads;
  const int head_blocks = (a.H + heads - 1) / heads;
  const int64_t tiles = (a.N + kChainRows - 1) / kChainRows;
  chain_match_kernel<Emit><<<(unsigned)(tiles * head_blocks), kChainRows * heads, 0, stream>>>(
      a.plan, a.packed_q, a.packed_k, a.sym_seq_stride, a.sym_head_stride, a.N, a.H, a.W,
      a.context, a.chain_start, a.chain_prev, a.chain_low, head_blocks, limit,
      a.plan.status + 2, emit);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace

int launch_chain_index(const FwdArgs& a, int64_t max_len, cudaStream_t stream) {
  ProfileScope prof("chain_index", stream);
  const int hash_bits = chain_hash_bits(a.D, a.context, max_len);
  if (a.context > 2)   // several shorter lengths merge their results into zeroed words
    ROSA_CUDA_OK(cudaMemsetAsync(a.chain_low, 0, (size_t)a.N * a.H * sizeof(uint32_t), stream));
  const size_t entries = (size_t)(1 << hash_bits) + chain_low_entries(a.D, a.context);
  const unsigned grid = (unsigned)(a.plan.S * a.H);
  const bool merge = a.context > 2, wide = max_len > 65535 * kChainStep;   // step beyond 16 bits
  const size_t bytes = entries * (wide ? sizeof(unsigned long long) : sizeof(uint32_t));
  auto kernel = wide ? (merge ? chain_index_kernel<unsigned long long, true>
                              : chain_index_kernel<unsigned long long, false>)
                     : (merge ? chain_index_kernel<uint32_t, true> : chain_index_kernel<uint32_t, false>);
  if (bytes > 48 * 1024)
    ROSA_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  kernel<<<grid, 32 * a.context, bytes, stream>>>(
      a.plan, a.packed_q, a.packed_k, a.sym_seq_stride, a.sym_head_stride, a.H, a.D, a.context,
      hash_bits, a.chain_start, a.chain_prev, a.chain_low);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

int launch_chain_forward(const FwdArgs& a, int limit, cudaStream_t stream) {
  ProfileScope prof("hard_match", stream);
  return with_sign_emit(a, [&](auto emit) {
    return launch_chain_match_t(a, limit, emit, stream);
  });
}

int launch_chain_inference(const FwdArgs& a, const float* payload, float* out, int64_t* matched_end,
                           int limit, cudaStream_t stream) {
  ProfileScope prof("hard_match", stream);
  return launch_chain_match_t(a, limit, make_payload_emit(a, payload, out, matched_end), stream);
}

int launch_scan_forward(const FwdArgs& a, const int32_t* run_flag, cudaStream_t stream) {
  return with_sign_emit(a, [&](auto emit) { return launch_scan_match_t(a, run_flag, emit, stream); });
}

int launch_scan_inference(const FwdArgs& a, const float* payload, float* out, int64_t* matched_end,
                          const int32_t* run_flag, cudaStream_t stream) {
  return launch_scan_match_t(a, run_flag, make_payload_emit(a, payload, out, matched_end), stream);
}

}  // namespace rosa
