// Kernels of the chained matcher (chain_match.cuh), over whole sequences (chain_match.cu) or over
// the histories of the streaming runtime (stream_chain.cu).
//
// An Axis says where a row lives: locate(g) gives the sequence (or slot) of token g, its `start`
// (what the result functor wants to know of the sequence) and the position i inside it; symbols()
// the offset of position 0 of a head in the symbol and link arrays; links() the offset of the row in
// the arrays that the index pass wrote for the query positions.
#pragma once

#include "chain_match.cuh"
#include "common.cuh"

namespace rosa {
namespace {

// How many pieces per head: as many warps as the GPU holds of these CTAs, pieces of at least 256
// positions, at most 8 (a table set each in shared memory), at most kChainIndexWarps warps a CTA:
// the index kernels are compiled for the registers a thread that this leaves.  (As a bound on the threads
// the same limit made the pass 19 % slower: 0.70 -> 0.83 ms at 64 x 16384 x 64 wide symbols.)
constexpr int kChainSharedBytes = 200 * 1024;
constexpr int kChainIndexWarps = 24;
constexpr int kChainIndexRegisters = 80;
static_assert(32 * kChainIndexWarps * kChainIndexRegisters <= 65536, "more registers than an SM has");

inline int chain_segments(int64_t heads, int64_t positions, size_t set_bytes, int context) {
  int n = 1;
  while (n < 8 && heads * n * 2 <= kSMs * 8 && positions >= 256 * n * 2 &&
         (size_t)n * 2 * set_bytes <= kChainSharedBytes && context * n * 2 <= kChainIndexWarps)
    n *= 2;
  return n;
}

// Indexes positions [begin, end) of one head for context length L; all lanes of a warp call.
//
// A warp takes 16 positions at a time: lanes 0..15 hold the key contexts that end there, lanes
// 16..31 the query contexts.  A table entry is the last step in which a key context fell into the
// bucket and the mask of its lanes in that step, so one read gives both the latest earlier position
// and the equal lanes of the step itself.  A step reads the old entry, stores its own and reads back;
// key lanes whose bit was overwritten by another lane of the same bucket then add it.  The links are
// those of a strictly sequential pass.  What bounds it is the latency of that chain of three
// shared-memory accesses times the number of steps (finding the equal lanes with match.any instead
// took 330-380 ns a step); the symbols of the next eight steps are requested before the current ones
// are processed, which keeps global latency out of it.  The results of a step are selected, not
// branched on: 128 ns a step against 315 with branches (4096 tokens, 128 streams: 81 us before).
//
// kResume: the table holds the entries of the positions below `begin`, the first step may hold some.
// kMerge: a shorter length leaves the larger of its own result and the one that is there (the longest
// length that occurs wins).  q, k, key_links and query_links are addressed by position; query_links
// null: the keys alone are indexed.
template <typename Entry, bool kMerge, bool kResume, typename Sym>
__device__ __forceinline__ void chain_index_warp(const Sym* q, const Sym* k, int begin, int end, int L,
                                                 int bits, bool chained, int hash_bits, Entry* table,
                                                 uint32_t* key_links, uint32_t* query_links) {
  const int lane = threadIdx.x & 31;
  const bool is_query = lane >= kChainStep;
  const int l = lane & (kChainStep - 1);
  const Sym* sym = is_query ? q : k;
  const int context_bits = bits * L;
  const uint32_t context_mask = context_bits >= 32 ? 0xffffffffu : (1u << context_bits) - 1u;
  // a query at i needs a key context at j < i
  const int first_valid = max(begin, is_query ? L : L - 1);
  // buckets of the contexts of the next steps from their newest two symbols (requested earlier) and
  // the older ones, all steps of one distance at a time; ~0 where there is no context
  uint32_t bucket[kChainAhead];
  auto fill_buckets = [&](int p0, const int (&newest)[kChainAhead], const int (&second)[kChainAhead]) {
#pragma unroll
    for (int s = 0; s < kChainAhead; ++s)
      bucket[s] = (uint32_t)newest[s] | (L > 1 ? (uint32_t)second[s] << bits : 0u);
    for (int u = 2; u < L; ++u) {
#pragma unroll
      for (int s = 0; s < kChainAhead; ++s) {
        const int p = p0 + s * kChainStep + l;
        if (p >= first_valid && p < end) bucket[s] |= (uint32_t)sym[p - u] << (bits * u);
      }
    }
#pragma unroll
    for (int s = 0; s < kChainAhead; ++s) {
      const int p = p0 + s * kChainStep + l;
      const uint32_t w = bucket[s] & context_mask;
      bucket[s] = p < first_valid || p >= end ? 0xffffffffu
                  : chained ? chain_bucket(w, context_bits, hash_bits) : w;
    }
  };
  auto request = [&](int p0, int (&newest)[kChainAhead], int (&second)[kChainAhead]) {
#pragma unroll
    for (int s = 0; s < kChainAhead; ++s) {
      const int p = p0 + s * kChainStep + l;
      newest[s] = p < end ? (int)sym[p] : 0;
      second[s] = L > 1 && p >= 1 && p < end ? (int)sym[p - 1] : 0;
    }
  };
  uint32_t* dst = is_query ? query_links : key_links;
  const bool writes = (chained || is_query) && dst != nullptr;
  const uint32_t tag = chained ? 0u : (uint32_t)L << 28;
  const int base = begin / kChainStep * kChainStep;
  int newest[kChainAhead], second[kChainAhead];
  request(base, newest, second);
  fill_buckets(base, newest, second);
  const unsigned own_bit = 1u << l;
  for (int p0 = base; p0 < end; p0 += kChainAhead * kChainStep) {
    request(p0 + kChainAhead * kChainStep, newest, second);
#pragma unroll
    for (int s = 0; s < kChainAhead; ++s) {
      if (s > 0 && p0 + s * kChainStep >= end) break;
      const int p = p0 + s * kChainStep + l;
      const bool valid = bucket[s] != 0xffffffffu;
      const bool is_key = valid && !is_query;
      Entry* slot = table + (valid ? bucket[s] : 0u);
      const Entry step = (Entry)(p0 / kChainStep + s + 1) << 16;
      const Entry old = *slot;
      __syncwarp();
      if (is_key) *slot = (kResume && (old >> 16) == (step >> 16) ? old : step) | own_bit;
      __syncwarp();
      Entry now = *slot;
      if (__any_sync(0xffffffffu, is_key && ((unsigned)now & own_bit) == 0u)) {
        if (is_key && ((unsigned)now & own_bit) == 0u) atomicOr(slot, (Entry)own_bit);
        __syncwarp();
        now = *slot;
      }
      // the newest key lane below this one, else the newest of the bucket's last step
      const unsigned below = (now >> 16) == (step >> 16) ? (unsigned)now & (own_bit - 1u) : 0u;
      // (an old entry of this very step holds positions before `begin`: they are in `below`)
      const Entry from = below != 0u ? step | below : old;
      // position + 1 of the predecessor: bit b of step n (from 1) is position 16 (n - 1) + b
      uint32_t link = (uint32_t)(from >> 16) * kChainStep + 16u - (uint32_t)__clz((unsigned)from & 0xffffu);
      link = from != 0 && valid ? link | tag : 0u;
      if (writes && p >= begin && p < end) {
        if (kMerge && !chained) {
          if (link != 0u) atomicMax(dst + p, link);
        } else {
          dst[p] = link;
        }
      }
    }
    fill_buckets(p0 + kChainAhead * kChainStep, newest, second);
  }
}

// Indexes positions [begin, end) of one head by a whole CTA of context * segments warps.  `tables`
// are `segments` table sets of `entries` entries each; the first holds the positions below `begin`.
//
// One warp per context length is all the parallelism a sequential pass has, so a call with few heads
// leaves the GPU idle for len / 16 steps.  With more segments the positions are cut into as many
// pieces: all threads together leave the newest key position of every bucket and piece in the table
// set of the next piece (a maximum, in any order), the sets are made cumulative, and every piece
// then runs its own pass from the table of everything before it.
template <typename Entry, bool kMerge, bool kResume, typename Sym>
__device__ __forceinline__ void chain_index_block(const Sym* q, const Sym* k, int begin, int end,
                                                  int context, int bits, int hash_bits, int entries,
                                                  int segments, Entry* tables, uint32_t* key_links,
                                                  uint32_t* start, uint32_t* low) {
  const int first_step = begin / kChainStep, steps = (end - 1) / kChainStep - first_step + 1;
  const int per = (steps + segments - 1) / segments;
  const auto piece = [&](int g) { return max(begin, (first_step + g * per) * kChainStep); };
  const auto table_at = [&](int g, int L) {
    return tables + (int64_t)g * entries +
           (L == context ? 0 : (1 << hash_bits) + chain_low_entries(bits, L));
  };
  if (segments > 1) {
    for (int e = threadIdx.x; e < (segments - 1) * entries; e += blockDim.x) tables[entries + e] = 0;
    __syncthreads();
    const int last = min(end, piece(segments - 1));
    constexpr int kBatch = 4;                        // positions of a thread whose loads overlap
    for (int p0 = begin + threadIdx.x; p0 < last; p0 += kBatch * blockDim.x) {
      uint32_t w[kBatch] = {0u, 0u, 0u, 0u};
      for (int L = 1; L <= context; ++L) {
        const int context_bits = bits * L;
        int symbol[kBatch];
#pragma unroll
        for (int x = 0; x < kBatch; ++x) {
          const int p = p0 + x * blockDim.x;
          symbol[x] = p < last && p >= L - 1 ? (int)k[p - L + 1] : 0;
        }
#pragma unroll
        for (int x = 0; x < kBatch; ++x) {
          const int p = p0 + x * blockDim.x;
          w[x] |= (uint32_t)symbol[x] << (context_bits - bits);
          if (p >= last || p < L - 1) continue;
          const int g = (p / kChainStep - first_step) / per + 1;
          const Entry entry = (Entry)(p / kChainStep + 1) << 16 | 1u << (p & (kChainStep - 1));
          const uint32_t c = context_bits >= 32 ? w[x] : w[x] & ((1u << context_bits) - 1u);
          atomicMax(table_at(g, L) + (L == context ? chain_bucket(c, context_bits, hash_bits) : c), entry);
        }
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < entries; e += blockDim.x) {
      Entry newest = tables[e];
      for (int g = 1; g < segments; ++g) {
        Entry* t = tables + (int64_t)g * entries + e;
        newest = max(newest, *t);
        *t = newest;
      }
    }
    __syncthreads();
  }
  const int warp = threadIdx.x >> 5;
  const int level = warp / segments, g = warp - level * segments;
  if (level >= context) return;                      // a short sequence of a pack takes fewer pieces
  const int L = context - level;                     // level 0: the chained length
  const int from = piece(g), to = g + 1 < segments ? min(end, piece(g + 1)) : end;
  if (from < to)
    chain_index_warp<Entry, kMerge, kResume>(q, k, from, to, L, bits, level == 0, hash_bits, table_at(g, L),
                                             key_links, level == 0 ? start : low);
}

// Rows of whole sequences over packed symbols ([sequence][head][position] or [head][token]).
struct SequenceAxis {
  Plan plan;
  int64_t seq_stride, head_stride;

  __device__ __forceinline__ int locate(int64_t g, int* start, int* i) const {
    int len = 0;
    const int seq = find_segment(plan, g, start, &len);
    *i = (int)(g - *start);
    return seq;
  }
  __device__ __forceinline__ int64_t symbols(int seq, int h, int start) const {
    return (int64_t)seq * seq_stride + (int64_t)h * head_stride +
           (plan.cu_seqlens == nullptr ? 0 : start);
  }
  __device__ __forceinline__ int64_t links(int64_t base, int64_t, int, int i) const { return base + i; }
};

// One thread per row: a warp takes 32 consecutive tokens of one head (its symbol and link reads
// coalesce), a CTA eight heads of them; the winners change places in shared memory so that the
// results go out with the heads of a token side by side.  Bound by the latency and the sector
// rate of the dependent chain reads in L2; many rows in flight hide it.
constexpr int kChainRows = 32;
constexpr int kChainHeads = 8;

template <typename Sym, typename Axis, typename Emit>
__global__ void __launch_bounds__(kChainRows * kChainHeads)
    chain_match_kernel(Axis axis, const Sym* __restrict__ qsym, const Sym* __restrict__ ksym,
                       int64_t N, int H, int W, int context, const uint32_t* __restrict__ start_link,
                       const uint32_t* __restrict__ prev, const uint32_t* __restrict__ low,
                       int head_blocks, ChainPatience patience, int32_t* flag, Emit emit) {
  __shared__ uint2 s_win[kChainRows][kChainHeads + 1];   // (length, route)
  __shared__ int s_start[kChainRows];
  const int heads = blockDim.x / kChainRows;             // heads of this CTA
  const int tile = blockIdx.x / head_blocks;
  const int h0 = (blockIdx.x - tile * head_blocks) * heads;
  const int64_t g0 = (int64_t)tile * kChainRows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int h = h0 + warp;
  const int64_t g = g0 + lane;
  int start = 0, i = 0, best_len = 0, best_route = 0;
  int seq = -1;
  if (g < N && h < H) seq = axis.locate(g, &start, &i);
  int64_t base = 0;
  uint32_t first = 0u, shorter = 0u;
  if (seq >= 0) {
    base = axis.symbols(seq, h, start);
    const int64_t at = axis.links(base, g, h, i);
    first = start_link[at];
    if (context > 1) shorter = low[at];
  }
  if (chain_walk<Sym>(qsym + base, ksym + base, prev + base, first, seq, i, W, patience, lane, best_len,
                      best_route)) {
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

template <typename Sym, typename Axis, typename Emit>
int launch_chain_match_t(Axis axis, const Sym* q, const Sym* k, int64_t N, int H, int W, int context,
                         const uint32_t* start, const uint32_t* prev, const uint32_t* low,
                         ChainPatience patience, int32_t* flag, Emit emit, cudaStream_t stream) {
  const int heads = H < kChainHeads ? H : kChainHeads;
  const int head_blocks = (H + heads - 1) / heads;
  const int64_t tiles = (N + kChainRows - 1) / kChainRows;
  chain_match_kernel<Sym, Axis, Emit><<<(unsigned)(tiles * head_blocks), kChainRows * heads, 0, stream>>>(
      axis, q, k, N, H, W, context, start, prev, low, head_blocks, patience, flag, emit);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------------ rows that gave up
// The newest kSymbols symbols that end at a position, compared at once.
template <typename Sym>
struct Probe;

template <>
struct Probe<uint8_t> {
  static constexpr int kSymbols = 8;
  uint32_t older, newer;
  // the eight bytes that end at p[0], from the aligned words that hold one of them or the byte after it
  __device__ __forceinline__ static Probe of(const uint8_t* p) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(p - 7);
    const uint32_t* words = reinterpret_cast<const uint32_t*>(at & ~(uintptr_t)3);
    const unsigned shift = 8u * (unsigned)(at & 3);
    const uint32_t a = words[0], b = words[1], c = words[2];
    return {__funnelshift_r(a, b, shift), __funnelshift_r(b, c, shift)};
  }
  // whether the newest n symbols agree (n from 1 to 8)
  __device__ __forceinline__ bool agrees(const Probe& o, int n) const {
    const uint32_t lo = n <= 4 ? 0u : ~0u << (64 - 8 * n), hi = n >= 4 ? ~0u : ~0u << (32 - 8 * n);
    return (((older ^ o.older) & lo) | ((newer ^ o.newer) & hi)) == 0u;
  }
};

template <>
struct Probe<int32_t> {
  static constexpr int kSymbols = 4;
  int32_t w[4];
  __device__ __forceinline__ static Probe of(const int32_t* p) { return {{p[0], p[-1], p[-2], p[-3]}}; }
  __device__ __forceinline__ bool agrees(const Probe& o, int n) const {
    return w[0] == o.w[0] && (n < 2 || w[1] == o.w[1]) && (n < 3 || w[2] == o.w[2]) &&
           (n < 4 || w[3] == o.w[3]);
  }
};

// A warp resolves one row by a look at every earlier position, newest first, 128 at a time: a position
// is worth extending only if it agrees in one symbol more than the best match has so far, which a probe
// or the symbol at that distance decides.  Cost: i / 128 rounds of coalesced reads, whatever the chains
// look like.  (A byte history is a row of whole words.)  All lanes call and get the result.
template <typename Sym>
__device__ __forceinline__ void scan_row(const Sym* q, const Sym* k, int i, int W, int lane,
                                         int& best_len, int& best_route) {
  constexpr int kProbe = Probe<Sym>::kSymbols;
  const Sym q_i = q[i];
  Probe<Sym> newest{};
  if (i >= kProbe) newest = Probe<Sym>::of(q + i);
  best_len = best_route = 0;
  const auto take = [&](int j, int length) {
    const int longest = __reduce_max_sync(0xffffffffu, length);
    if (longest > best_len) {
      best_len = longest;
      best_route = __reduce_max_sync(0xffffffffu, length == longest ? j + 1 : 0);
    }
  };
  int top = i - 1;
  while (top >= 0 && best_len < min(W, top + 1)) {
    if (top - 127 >= max(best_len, kProbe)) {
      const int n = min(best_len + 1, kProbe);
      const Sym q_b = q[i - best_len];
      bool candidate[4], any = false;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = top - 32 * u - lane;
        candidate[u] = Probe<Sym>::of(k + j).agrees(newest, n) && k[j - best_len] == q_b;
        any = any || candidate[u];
      }
      if (__any_sync(0xffffffffu, any)) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = top - 32 * u - lane;
          take(j, candidate[u] ? chain_extend<Sym>(q, k, i, j, n, min(W, j + 1)) : 0);
        }
      }
      top -= 128;
    } else {
      const int j = top - lane;
      int length = 0;
      if (j >= best_len && k[j] == q_i && k[j - best_len] == q[i - best_len])
        length = chain_extend<Sym>(q, k, i, j, 1, min(W, j + 1));
      take(j, length);
      top -= 32;
    }
  }
}

// Tiles of up to 256 rows of one sequence in which many rows gave up: the run-length recurrence
//     len(i, j) = (q_i == k_j) ? min(len(i - 1, j - 1) + 1, W) : 0
// along the diagonals, newest first in bands of 2048.  A thread owns eight neighbouring diagonals, so
// that the key symbols of eight rows are fifteen consecutive ones in registers; a pair costs a compare, an
// add with the cap, a select and a maximum over (run << 11 | how late the diagonal is), whatever the data
// are.  The run that enters the tile is counted backwards once per diagonal.  A band is the last when no
// older match can be longer.  What bounds it is instruction issue.  Streams of two symbols, against the
// matchers that took these rows before (a scan per row; bitmaps of the symbols, of up to 8 bits):
//   8 x 8192 x 32 inference, wide symbols       43.9 -> 3.1 ms
//   4 x 4096 x 32 scoring, 8 bits               1.48 -> 0.52 ms, 4 x 4096 x 16, 24 bits 3.59 -> 0.30 ms
//   16 x 8192 x 32 stream in chunks of 1024     78.1 -> 6.5 ms
constexpr int kRunRows = 256;          // most rows of a tile, threads of the CTA
constexpr int kRunPer = 8;
constexpr int kRunBits = 11;
constexpr int kRunBand = kRunRows * kRunPer;
static_assert(kRunBand == 1 << kRunBits, "a key holds the diagonal of a band");
constexpr int kRunMaxHorizon = 1 << 19;      // runs of a 32-bit key
// With at most this many pending rows a warp scans for each instead (a row of a scan costs as much as
// 6 to 40 rows of the runs, as the symbols go).
constexpr int kRunFew = 12;

// run[e]: key of the thread's diagonal e, its run << 11 | how late it is in the band.
__device__ __forceinline__ void run_rows(const int* s_q, const int* s_k, unsigned* s_best, int nrows, int W,
                                         int tid, int (&run)[kRunPer]) {
  const int lane = tid & 31;
  const int base = kRunBand - kRunPer - kRunPer * tid;       // column of (row 0, the oldest diagonal)
  int none[kRunPer], most[kRunPer], kw[2 * kRunPer];
#pragma unroll
  for (int e = 0; e < kRunPer; ++e) {
    none[e] = base + kRunPer - 1 - e;
    most[e] = none[e] + (W << kRunBits);
  }
  const auto load = [&](int at, int column) {
#pragma unroll
    for (int x = 0; x < kRunPer; x += 4) {
      const int4 w = *reinterpret_cast<const int4*>(s_k + column + x);
      kw[at + x] = w.x; kw[at + x + 1] = w.y; kw[at + x + 2] = w.z; kw[at + x + 3] = w.w;
    }
  };
  load(0, base);
#pragma unroll 1
  for (int r0 = 0; r0 < nrows; r0 += kRunPer) {
    load(kRunPer, base + r0 + kRunPer);
    int q[kRunPer];
#pragma unroll
    for (int x = 0; x < kRunPer; ++x) q[x] = s_q[r0 + x];
    unsigned mine = 0u;
#pragma unroll
    for (int rr = 0; rr < kRunPer; ++rr) {
      int key = 0;
#pragma unroll
      for (int e = 0; e < kRunPer; ++e) {
        run[e] = kw[rr + kRunPer - 1 - e] == q[rr] ? min(run[e] + kRunBand, most[e]) : none[e];
        key = max(key, run[e]);
      }
      const unsigned longest = __reduce_max_sync(0xffffffffu, (unsigned)key);
      if (lane == rr) mine = longest;
    }
    if (lane < kRunPer && mine >= (unsigned)kRunBand) atomicMax(s_best + r0 + lane, mine);
#pragma unroll
    for (int x = 0; x < kRunPer; ++x) kw[x] = kw[x + kRunPer];
  }
}

// The rows that gave up, tile by tile: longest first, as many CTAs as fill the GPU.
template <typename Sym, typename Axis, typename Emit>
__global__ void __launch_bounds__(kRunRows, 2)
    run_match_kernel(Axis axis, const Sym* __restrict__ qsym, const Sym* __restrict__ ksym, int64_t N,
                     int H, int W, int tile_rows, const int32_t* __restrict__ run_flag, Emit emit) {
  __shared__ __align__(16) int s_k[kRunBand + kRunRows];
  __shared__ int s_q[kRunRows];
  __shared__ unsigned s_best[kRunRows];
  __shared__ bool s_mine[kRunRows];
  __shared__ unsigned s_used[kRunRows / 32];
  __shared__ int s_first, s_last, s_count, s_seq, s_start, s_i0;
  if (*run_flag == 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t tiles = (N + tile_rows - 1) / tile_rows;
  for (int64_t task = blockIdx.x; task < tiles * H; task += gridDim.x) {
    const int h = (int)(task % H);
    const int64_t g0 = (tiles - 1 - task / H) * tile_rows;
    int seq = -1, start = 0, row = 0;
    bool pending = false;
    if (tid < tile_rows && g0 + tid < N && emit.pending((g0 + tid) * H + h)) {
      seq = axis.locate(g0 + tid, &start, &row);
      pending = seq >= 0;
    }
    // one sequence (or slot) of the tile at a time
    while (__syncthreads_or(pending)) {
      if (tid == 0) {
        s_first = kRunRows;
        s_last = s_count = 0;
      }
      __syncthreads();
      if (pending) atomicMin(&s_first, tid);
      __syncthreads();
      const int first = s_first;
      if (tid == first) {
        s_seq = seq;
        s_start = start;
        s_i0 = row;
      }
      __syncthreads();
      const bool mine = pending && seq == s_seq;
      s_mine[tid] = mine;
      if (mine) {
        atomicMax(&s_last, tid);
        atomicAdd(&s_count, 1);
      }
      __syncthreads();
      const int n = s_last - first + 1, i0 = s_i0;
      const int64_t at = axis.symbols(s_seq, h, s_start);
      const Sym* q = qsym + at;
      const Sym* k = ksym + at;
      if (s_count <= kRunFew || W > kRunMaxHorizon) {
        for (int r = first + warp; r <= s_last; r += kRunRows / 32) {
          if (!s_mine[r]) continue;
          int length, route;
          scan_row<Sym>(q, k, i0 + r - first, W, lane, length, route);
          if (lane == 0) emit(g0 + r, h, H, s_start, length, route);
        }
      } else {
        // thread t owns row i0 + t of the sequence as well as diagonals db + 8 t .. db + 8 t + 7
        const bool own = tid < n && s_mine[min(first + tid, kRunRows - 1)];
        const int i = i0 + tid, newest_row = i0 + n - 1;
        int best_len = 0, best_route = 0;
        // positions before the sequence hold a symbol that no row of the tile has: one of 0 .. 256
        if (tid < kRunRows / 32) s_used[tid] = 0u;
        __syncthreads();
        const int symbol = tid < n ? (int)q[i] : 0;
        s_q[tid] = symbol;
        if (symbol >= 0 && symbol < kRunRows) atomicOr(s_used + (symbol >> 5), 1u << (symbol & 31));
        __syncthreads();
        int absent = kRunRows;
        for (int x = kRunRows / 32 - 1; x >= 0; --x)
          if (~s_used[x] != 0u) absent = 32 * x + __ffs(~s_used[x]) - 1;
        for (int db = 1; db <= newest_row; db += kRunBand) {
          const int j0 = i0 - db - (kRunBand - 1);        // key position of column 0
          s_best[tid] = 0u;
          for (int c = tid; c < kRunBand + n; c += kRunRows) {
            const int j = j0 + c;
            s_k[c] = j >= 0 && j < newest_row ? (int)k[j] : absent;
          }
          __syncthreads();
          if (db + kRunPer * 32 * warp <= newest_row) {    // a warp of diagonals that exist
            int run[kRunPer];
#pragma unroll
            for (int e = 0; e < kRunPer; ++e) {
              const int d = db + kRunPer * tid + e;
              run[e] = kRunBand - 1 - kRunPer * tid - e;
              if (d < i0)
                run[e] += chain_extend<Sym>(q, k, i0 - 1, i0 - 1 - d, 0, min(W, i0 - d)) << kRunBits;
            }
            run_rows(s_q, s_k, s_best, n, W, tid, run);
          }
          __syncthreads();
          const int key = (int)s_best[tid];
          if (own && key >> kRunBits > best_len) {         // older bands only with a longer match
            best_len = key >> kRunBits;
            best_route = i - (db + kRunBand - 1 - (key & (kRunBand - 1))) + 1;
          }
          // the matches of the next band start at position i - db - 2048 at best
          if (__syncthreads_and(!own || best_len >= W || best_len >= i - db - kRunBand + 1)) break;
        }
        if (own) emit(g0 + first + tid, h, H, s_start, best_len, best_route);
      }
      pending = pending && !mine;
    }
  }
}

template <typename Sym, typename Axis, typename Emit>
int launch_run_match_t(Axis axis, const Sym* q, const Sym* k, int64_t N, int H, int W,
                       const int32_t* run_flag, Emit emit, cudaStream_t stream) {
  ProfileScope prof("hard_match_runs", stream);
  // launched whether or not a row gave up; short tiles where the tall ones would not fill the GPU
  const int tile_rows = (N + kRunRows - 1) / kRunRows * H < kSMs * 2 ? 64 : kRunRows;
  run_match_kernel<Sym, Axis, Emit><<<kSMs * 2, kRunRows, 0, stream>>>(axis, q, k, N, H, W, tile_rows,
                                                                      run_flag, emit);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace
}  // namespace rosa
