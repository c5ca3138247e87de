// Pieces shared by the surrogate-VJP kernels: work-item geometry, the online-softmax merge,
// the transposing warp reduction and the flush-to-zero cutoff of the window product.
#pragma once

#include <math_constants.h>

#include "common.cuh"

namespace rosa {
namespace {

constexpr float kSqrtScale = 2.41421356237309504880f;  // sqrt(2) + 1

// ------------------------------------------------------------- item geometry
struct Item {
  int seq, it, h, start, len;
  int nitems;            // items of this sequence (per head)
  int w_begin, w_end;    // bands walked by this CTA
  int64_t rowslot;       // first partial-row slot of this (item, head)
  int64_t ck_base;       // first checkpoint block of this (sequence, head)
  int64_t item_linear;   // dense index over (sequence, head, item)
};

__device__ __forceinline__ void merge_stats(float& m, float& z, float& e, float m2, float z2,
                                            float e2) {
  if (m2 == -CUDART_INF_F) return;
  if (m == -CUDART_INF_F) {
    m = m2; z = z2; e = e2;
    return;
  }
  const float mm = fmaxf(m, m2);
  const float s1 = __expf(m - mm), s2 = __expf(m2 - mm);
  z = z * s1 + z2 * s2;
  e = e * s1 + e2 * s2;
  m = mm;
}

// Sum of eight per-lane values across a warp in 9 shuffles instead of 40: each step
// exchanges half of the remaining values with the partner lane.  On return every lane
// holds the warp total of value index ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 +
// ((lane >> 2) & 1).
__device__ __forceinline__ float warp_reduce8(const float (&v)[8], int lane) {
  const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
  float a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float send = h16 ? v[i] : v[i + 4];
    const float keep = h16 ? v[i + 4] : v[i];
    a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float send = h8 ? a[i] : a[i + 2];
    const float keep = h8 ? a[i + 2] : a[i];
    b[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  float c = (h4 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h4 ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;
}

// Work item of a 1-D grid.  Heads vary fastest; for a dense batch the sequences vary next and
// the item index slowest, so that the longest items (the bands next to the main diagonal) of ALL
// sequences and heads are scheduled first and the tail of the launch consists of the shortest
// ones (with the sequence slowest, the long items of the last sequences would start late and
// finish alone).  Packed batches keep sequence-major order.
__device__ __forceinline__ bool load_item_1d(const VjpArgs& a, Item* o) {
  const int slot = blockIdx.x / a.H;
  if (a.plan.cu_seqlens == nullptr) {
    const int per = dense_items(a.plan);            // items of every sequence
    if (per <= 0 || slot >= per * a.plan.S) return false;
    o->it = slot / a.plan.S;
    o->seq = slot - o->it * a.plan.S;
  } else if (!find_item(a.plan, slot, &o->seq, &o->it)) {
    return false;
  }
  o->h = blockIdx.x - slot * a.H;
  segment_bounds(a.plan, o->seq, &o->start, &o->len);
  int64_t items_before, rows_before, cks_before;
  sequence_offsets(a.plan, o->seq, o->len, &o->nitems, &items_before, &rows_before, &cks_before);
  const int nbands = (int)vjp_bands(o->len);
  o->w_begin = o->it * a.bands_per_item;
  o->w_end = min(nbands, o->w_begin + a.bands_per_item);
  o->rowslot = rows_before * a.H +
               ((int64_t)o->h * o->nitems + o->it) * (int64_t)o->len;
  o->ck_base = cks_before * a.H + (int64_t)o->h * vjp_ck_count(o->len);
  o->item_linear = items_before * a.H + (int64_t)o->h * o->nitems + o->it;
  return true;
}

// How much work a launch of one CTA per item holds: the row blocks of all items per SM over those of
// the longest item.  Items run next to each other but a block of an item follows the block before it,
// so a launch of little work is as long as the longest item takes by itself (few, short blocks are
// what counts), one of much work as long as the SMs are busy.  The lengths of a packed batch are on
// the GPU: its longest sequence is taken to be twice as long as the average.
inline float vjp_fill(const VjpArgs& a) {
  const int64_t N = a.plan.N > 0 ? a.plan.N : 1;
  const int64_t S = a.plan.S > 0 ? a.plan.S : 1;
  int64_t longest = a.plan.cu_seqlens == nullptr ? a.plan.uniform_len : 2 * N / S;
  longest = longest < 2 ? 2 : longest > N ? N : longest;
  const float items = (float)vjp_bands(longest) / (float)a.bands_per_item;
  return (float)a.H * (float)N / (float)longest * 0.5f * (items + 1.0f) / kSMs;
}

}  // namespace

// Adds four accumulator values to a partial gradient row that this CTA alone writes: the first
// touch stores, later ones go out as one vector reduction to L2 instead of a load, four adds and
// a store, so no thread waits for the old value.  The touches of one address come from different
// threads of the CTA in different row blocks, always with a CTA barrier in between, which orders
// them; the sum is therefore still formed in a fixed order.  (The reduction unit flushes
// subnormal float32 values to zero.)
__device__ __forceinline__ void accumulate_row4(float4* p, bool first, float a, float b, float c,
                                                float d) {
  if (first) {
    *p = make_float4(a, b, c, d);
  } else {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c),
                 "f"(d)
                 : "memory");
  }
}

// One component of such a row (rows whose width is not a multiple of four).
__device__ __forceinline__ void accumulate_row1(float* p, bool first, float a) {
  if (first) {
    *p = a;
  } else {
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(a) : "memory");
  }
}

}  // namespace rosa
