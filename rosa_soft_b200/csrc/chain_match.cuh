// Latest-longest suffix matching through occurrence chains, shared by the training forward, the
// batched inference (chain_match.cu) and the streaming runtime (stream_chain.cu).
//
// The context of length c at position p is the c symbols that end there.  Every key position is
// linked to the previous key position whose context falls into the same bucket, every query
// position to the latest earlier key position of its bucket.  A match of at least c symbols ends
// at a member of that chain, so a row visits the few positions that share its context instead of
// all the positions before it.  Rows whose best match is shorter than c need only the latest
// earlier occurrence of their context of length L < c for the largest such L: one table of
// 2^(L * bits) entries per L, without chains, because among matches of exactly that length the
// latest wins.
//
// c is the smallest length whose contexts span 12 bits (one symbol when it has 12 or more): the
// chains of a stream without structure then hold a few positions per 10^4 tokens, and the tables of
// the shorter lengths stay below 4096 entries in total.
#pragma once

#include <cstdint>

namespace rosa {

constexpr int kChainHashBits = 13;    // buckets of the chained contexts: at most 2^13
constexpr int kChainStep = 16;        // positions a warp indexes at a time
constexpr int kChainAhead = 8;        // steps between the request of a symbol and its use
// Longest history whose step numbers fit a 32-bit table entry beside the mask of 16 lanes.
constexpr int64_t kChainNarrow = (int64_t)65535 * kChainStep;
// When a row leaves its chain to the matchers whose cost does not depend on the data (run_match_kernel,
// scan_row): after `steps` members, or when they lie close together (streams of few distinct symbols): at
// the 24th less than 6 positions apart, at the `trial`-th (24th or 64th) or a later one less than 20;
// `trial` 0: the first rule alone.  A member is two dependent reads, 4 to 9 ps with all rows of a launch in
// flight, a position of the run matcher 0.3 ps, on short sequences 0.8.  Alphabet of 16, 8 x 8192 x 32
// inference: 3.2 ms when the rows leave, 5.0 when they walk on; 16 x 1024 x 16 scoring: 160 us when they
// leave after 24 members, 105 after 64.
struct ChainPatience {
  int steps, trial;
};
constexpr int kChainTrial = 24;
// Sequences up to here walk their chains to the end: the launch that stands by for the rows that give up
// would cost more.
constexpr int64_t kChainShort = 512;
// Winner that such a row leaves behind (a match length no real row has).
constexpr unsigned long long kChainGaveUp = 0xffffffffull << 32;

// (The results of the shorter lengths carry a position in 28 bits.)
inline int chain_context(int bits, int64_t W, int64_t max_len) {
  const int c = bits >= 12 || max_len >= ((int64_t)1 << 28) ? 1 : (12 + bits - 1) / bits;
  return (int64_t)c < W ? c : (int)W;
}

// log2 of the bucket count for streams of at most `len` tokens: exact contexts where they fit,
// otherwise about one bucket per token up to 2^13.
__host__ __device__ inline int chain_hash_bits(int bits, int c, int64_t len) {
  int n = 8;
  while (n < kChainHashBits && ((int64_t)1 << n) < len) ++n;
  return bits * c < n ? bits * c : n;
}

inline ChainPatience chain_patience(int bits, int c, int64_t len) {
  if (len <= kChainShort) return {0x7fffffff, 0};
  const int64_t expected = len >> chain_hash_bits(bits, c, len);    // members without structure
  return {(int)(4 * expected > 1024 ? 4 * expected : 1024), len <= 2048 ? 64 : kChainTrial};
}

__host__ __device__ inline uint32_t chain_bucket(uint32_t context, int context_bits, int hash_bits) {
  return context_bits <= hash_bits ? context : (context * 0x9E3779B1u) >> (32 - hash_bits);
}

// Entries of the tables of the lengths below L (exact contexts of 1 .. L - 1 symbols).
__host__ __device__ inline int chain_low_entries(int bits, int L) {
  int n = 0;
  for (int l = 1; l < L; ++l) n += 1 << (bits * l);
  return n;
}

// Number of equal symbols ending at k[j] and q[i], at most `cap`, of which `length` are known.
// Four at a time: the loads of a group do not wait for one another.
template <typename Sym>
__device__ __forceinline__ int chain_extend(const Sym* q, const Sym* k, int i, int j, int length,
                                            int cap) {
  while (length + 4 <= cap) {
    const Sym* kp = k + (j - length);
    const Sym* qp = q + (i - length);
    const bool e0 = kp[0] == qp[0], e1 = kp[-1] == qp[-1], e2 = kp[-2] == qp[-2],
               e3 = kp[-3] == qp[-3];
    if (!(e0 && e1 && e2 && e3)) return length + (!e0 ? 0 : !e1 ? 1 : !e2 ? 2 : 3);
    length += 4;
  }
  while (length < cap && k[j - length] == q[i - length]) ++length;
  return length;
}

// Resolves the rows of a warp: 32 consecutive positions of one head, lane by lane (`row` is the
// sequence of the lane's position, negative for none; q, k and prev start at it).  `first` is the
// latest candidate + 1 (0: none), prev[j] the next older candidate + 1.
//
// Newest candidates first: neighbouring rows inside a repeated passage have neighbouring newest
// candidates, i.e. they lie on one diagonal, where the match grows by one symbol per row.  Only the
// first lane of such a run extends its candidate symbol by symbol, the others count from it.  Then
// every lane walks the rest of its chain: candidates come newest first, so only a strictly longer
// match replaces the best one, and a candidate is worth extending only if it also agrees at the
// distance of the best length so far.  Returns the length and the route (position + 1) of the latest
// among the longest; the result is true when the row ran out of patience.  All lanes call.
template <typename Sym>
__device__ __forceinline__ bool chain_walk(const Sym* q, const Sym* k, const uint32_t* prev,
                                           uint32_t first, int row, int i, int W, ChainPatience patience, int lane,
                                           int& best_len, int& best_route) {
  best_len = 0;
  best_route = 0;
  int j = (int)first - 1;
  bool equal = false;
  if (first != 0u) {
    first = prev[j];
    equal = k[j] == q[i];
  }
  const int diagonal = equal ? i - j : 0;          // positive for a match
  const int up_diagonal = __shfl_up_sync(0xffffffffu, diagonal, 1);
  const int up_row = __shfl_up_sync(0xffffffffu, row, 1);
  const bool leads = lane == 0 || up_diagonal != diagonal || up_row != row;
  if (equal && leads) best_len = chain_extend<Sym>(q, k, i, j, 1, min(W, j + 1));
  const unsigned leaders = __ballot_sync(0xffffffffu, leads) & (0xffffffffu >> (31 - lane));
  const int leader = 31 - __clz(leaders);          // lane 0 leads
  const int counted = __shfl_sync(0xffffffffu, best_len, leader) + lane - leader;
  if (equal) {
    best_len = min(W, counted);
    best_route = j + 1;
  }
  int steps = 0, check = patience.trial > 0 ? kChainTrial : patience.steps;
  while (first != 0u && best_len < W) {
    j = (int)first - 1;
    const int cap = min(W, j + 1);                 // a match cannot start before the sequence
    if (cap <= best_len) break;                    // nor can that of any older candidate
    first = prev[j];
    if (k[j - best_len] == q[i - best_len]) {      // best_len < cap <= j + 1 <= i
      const int length = chain_extend<Sym>(q, k, i, j, 0, cap);
      if (length > best_len) {
        best_len = length;
        best_route = j + 1;
      }
    }
    if (++steps == check) {                        // now and then: the loop is as long as its chain
      if (steps >= patience.steps || i - j < (steps < patience.trial ? 6 : 20) * steps) return first != 0u;
      check += 40;
    }
  }
  return false;
}

}  // namespace rosa
