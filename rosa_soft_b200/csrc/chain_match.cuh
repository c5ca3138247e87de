// Latest-longest suffix matching through occurrence chains, shared by the training forward, the
// batched inference (hard_forward.cu) and the streaming runtime (stream_runtime.cu).
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
// A row gives up after this many chain members (streams of very few distinct symbols) and is
// resolved by the matcher whose cost does not depend on the data.
constexpr int kChainLimit = 256;
// Winner that such a row leaves behind (a match length no real row has).
constexpr unsigned long long kChainGaveUp = 0xffffffffull << 32;

__host__ __device__ inline int chain_context(int bits, int64_t W) {
  const int c = bits >= 12 ? 1 : (12 + bits - 1) / bits;
  return (int64_t)c < W ? c : (int)W;
}

// log2 of the bucket count for streams of at most `len` tokens: exact contexts where they fit,
// otherwise about one bucket per token up to 2^13.
__host__ __device__ inline int chain_hash_bits(int bits, int c, int64_t len) {
  int n = 8;
  while (n < kChainHashBits && ((int64_t)1 << n) < len) ++n;
  return bits * c < n ? bits * c : n;
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

// Walks the chain of one row.  `first` is the latest candidate + 1 (0: none), prev[j] the next
// older candidate + 1.  Candidates come newest first, so only a strictly longer match replaces
// the best one, and a candidate is worth extending only if it also agrees at the distance of the
// best length so far.  Returns the length and the route (position + 1) of the latest among the
// longest; `gave_up` is set when the chain was longer than kChainLimit.
template <typename Sym>
__device__ __forceinline__ void chain_walk(const Sym* __restrict__ q, const Sym* __restrict__ k,
                                           const uint32_t* __restrict__ prev, uint32_t first, int i,
                                           int W, int& best_len, int& best_route, bool& gave_up) {
  best_len = 0;
  best_route = 0;
  gave_up = false;
  int steps = 0;
  Sym q_next = first != 0u ? q[i] : (Sym)0;        // the symbol at the distance of the best length
  while (first != 0u) {
    const int j = (int)first - 1;
    const int cap = min(W, j + 1);                 // a match cannot start before the sequence
    if (cap <= best_len) break;                    // nor can that of any older candidate
    first = prev[j];
    if (k[j - best_len] == q_next) {
      int length = 0;
      while (length < cap && k[j - length] == q[i - length]) ++length;
      if (length > best_len) {
        best_len = length;
        best_route = j + 1;
        if (length >= W) break;
        q_next = q[i - length];   // length < W, and length <= j < i: inside the sequence
      }
    }
    if (++steps == kChainLimit && first != 0u) {
      gave_up = true;
      break;
    }
  }
}

}  // namespace rosa
