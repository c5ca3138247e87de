// Register-tiled sweeps of the dense surrogate VJP (same math and schedule as
// surrogate_vjp.cu: evidence recurrence along diagonals, online softmax with the analytic
// reference, dropout counter, checkpoints every 16 rows).
//
// One thread owns R = FOUR (or two, or one: see launch_s1_tiled) consecutive diagonals and walks
// them down the rows together.  On block row r the R cells of a thread sit on R consecutive key
// columns, and one row further down the same diagonals sit one column to the right, so the
// key-side tables (key symbol, the symbol leaving the horizon window, value sign bits, first
// dropout hash round) of a group of four rows are R + 3 consecutive columns: for R = 4 two aligned
// 128-bit shared-memory loads per table and sixteen cells, kept in registers and indexed at
// compile time.  Everything that depends on the row only (query symbols, hash word of the query
// position, utility table base) is loaded once per row and thread and shared by R cells; the row
// sums of four cells are added in registers before the warp reduction.  Rows of a block always start
// at a multiple of 16 (rows that do not exist are masked), interior blocks -- every cell active and past the
// horizon -- run without any per-cell predicate.
#include "common.cuh"
#include "vjp_shared.cuh"
#include "vjp_tiled.cuh"

namespace rosa {

namespace {

constexpr int kTBand = kVjpBand;                // diagonals per band
constexpr int s1_threads(int R) { return kTBand / R; }         // threads per CTA, R diagonals each
constexpr int kTRows = kVjpRows;                // rows per checkpointed block
constexpr int kTWin = kTBand + kTRows;          // window columns of a block
// The column tables of a block (key symbols, symbols leaving the horizon, first hash round of the
// route, value sign nibbles) cover 272 key positions; the next block of the band needs the same
// positions moved by 16.  The tables therefore SLIDE inside a longer buffer: a block computes
// only its 16 entering columns and moves the base up; every 17th block the surviving 256 columns
// go back to the start (source [272, 528), destination [0, 256) and the entering columns
// [256, 272) are pairwise disjoint, so the step needs no barrier of its own).
constexpr int kTSlide = kTBand;
constexpr int kTTab = kTWin + kTSlide;          // entries per table
static_assert(kTRows == 16 && kTBand % 128 == 0, "geometry assumed by the register windows");

struct S1Smem {
  int* s_k;          // [kTWin] key symbols of the column window
  int* s_kold;       // [kTWin] key symbols W + 1 columns earlier
  uint32_t* s_h1;    // [kTWin] first dropout hash round of route j + 1
  uint32_t* s_vb0;   // [kTWin] spread value sign nibbles, groups 0..3
  uint32_t* s_vb1;   // [kTWin] groups 4..7
  int* s_q;          // [kTRows]
  int* s_qold;       // [kTRows]
  float* glut;       // [64] gate per mismatch count
  float2* wstat;     // four diagonals a thread: [kTRows][warps] sums of (e, e d u); else the cells'
                     // (e, d u), [kTRows][kTBand] in the order of s1_cell
  float* ulut;       // [kTRows][NG][16]
};

__host__ __device__ constexpr int s1_stat_words(int R) {
  return 2 * kTRows * (R == 4 ? s1_threads(R) / 32 : kTBand);
}
__host__ __device__ constexpr int s1_smem_words(int ng, int R) {
  return 5 * kTTab + 2 * kTRows + 64 + s1_stat_words(R) + kTRows * ng * 16;
}

__device__ __forceinline__ S1Smem s1_carve(float* base, int R) {
  S1Smem s;
  int* w = reinterpret_cast<int*>(base);
  s.s_k = w;                                        w += kTTab;
  s.s_kold = w;                                     w += kTTab;
  s.s_h1 = reinterpret_cast<uint32_t*>(w);          w += kTTab;
  s.s_vb0 = reinterpret_cast<uint32_t*>(w);         w += kTTab;
  s.s_vb1 = reinterpret_cast<uint32_t*>(w);         w += kTTab;
  s.s_q = w;                                        w += kTRows;
  s.s_qold = w;                                     w += kTRows;
  s.glut = reinterpret_cast<float*>(w);             w += 64;
  s.wstat = reinterpret_cast<float2*>(w);           w += s1_stat_words(R);
  s.ulut = reinterpret_cast<float*>(w);
  return s;
}

// bits 0 .. 15 of x on the even bits
__device__ __forceinline__ uint32_t spread_bits(uint32_t x) {
  x &= 0xffffu;
  x = (x | x << 8) & 0x00ff00ffu;
  x = (x | x << 4) & 0x0f0f0f0fu;
  x = (x | x << 2) & 0x33333333u;
  return (x | x << 1) & 0x55555555u;
}

// The column windows of one group of four rows: consecutive table entries, cell (row rr, diagonal e)
// reads entry rr + R - 1 - e.  The last kept(R) entries are the first ones of the next group.
__host__ __device__ constexpr int s1_kept(int R) { return R == 1 ? 0 : R; }

template <int NG, int R, bool kWindowed, bool kDropout>
struct ColWindow {
  static constexpr int E = 4 + s1_kept(R);
  int k[E];
  int kold[kWindowed ? E : 1];
  uint32_t h1[kDropout ? E : 1];
  uint32_t v0[E];
  uint32_t v1[NG > 4 ? E : 1];
};

// n entries from column `src` (a multiple of R) with loads of R entries
template <int R, typename T>
__device__ __forceinline__ void load_cols(T* dst, const T* src, int n) {
#pragma unroll
  for (int x = 0; x < n; x += R) {
    if constexpr (R == 4) {
      const int4 w = *reinterpret_cast<const int4*>(src + x);
      dst[x] = (T)w.x; dst[x + 1] = (T)w.y; dst[x + 2] = (T)w.z; dst[x + 3] = (T)w.w;
    } else if constexpr (R == 2) {
      const int2 w = *reinterpret_cast<const int2*>(src + x);
      dst[x] = (T)w.x; dst[x + 1] = (T)w.y;
    } else {
      dst[x] = src[x];
    }
  }
}

template <int NG, int R, bool kWindowed, bool kDropout>
__device__ __forceinline__ void load_window(ColWindow<NG, R, kWindowed, kDropout>& cw, const S1Smem& sm,
                                            int col, int at, int n) {
  load_cols<R>(cw.k + at, sm.s_k + col, n);
  if (kWindowed) load_cols<R>(cw.kold + at, sm.s_kold + col, n);
  if (kDropout) load_cols<R>(cw.h1 + at, sm.s_h1 + col, n);
  load_cols<R>(cw.v0 + at, sm.s_vb0 + col, n);
  if (NG > 4) load_cols<R>(cw.v1 + at, sm.s_vb1 + col, n);
}

struct S1Params {
  int W, hs_cut, len;
  float neg_md, mul2, bias2;
};

// The sums of a row are formed in one order whatever R is: four neighbouring diagonals one after the
// other, then 32 such groups as warp_reduce8 pairs its lanes, then the two halves of the band.  A
// sequence then gives the same bits in a launch of any size, alone, in a batch or in a slice.  With
// four diagonals a thread holds a group and a warp half a band; with fewer the cells go to shared
// memory and the sums are formed behind the barrier that closes the block (s1_row_sums).
//
// Where the cells of a row lie: neighbouring pairs change places in half of the groups, those that
// the lanes of a quarter warp would otherwise read from the same banks in s1_row_sums.
template <int R>
__device__ __forceinline__ int s1_swap(int group) {
  return (R == 1 ? group >> 2 : group >> 5) & 1;
}
template <int R>
__device__ __forceinline__ int s1_cell(int diagonal) {
  return diagonal ^ 2 * s1_swap<R>(diagonal >> 2);
}

// Sum of e and of e d u over 4 neighbouring diagonals from their (e, d u); a dropped cell's d u is 0
// and leaves the second sum as it is.
template <int R>
__device__ __forceinline__ float2 s1_group_sums(const float4* row, int group) {
  const int swap = s1_swap<R>(group);
  const float4 a = row[2 * group + swap], b = row[2 * group + 1 - swap];
  return make_float2(a.x + a.z + b.x + b.z,
                     fmaf(b.z, b.w, fmaf(b.x, b.y, fmaf(a.z, a.w, a.x * a.y))));
}

// Totals of row `row` of the block by 16 / R neighbouring lanes, half of them for each half of the
// band; every lane gets them.  The pairing is that of warp_reduce8: 16, 8, 4, 2, 1 groups apart.
template <int R>
__device__ __forceinline__ float2 s1_row_sums(const float2* wstat, int row, int lane) {
  constexpr int kHalf = 8 / R, kGroups = 32 / kHalf;
  const int u = lane & (kHalf - 1), half = (lane / kHalf) & 1;
  const float4* cells = reinterpret_cast<const float4*>(wstat + row * kTBand);
  float2 v[kGroups];                       // groups u, u + kHalf, ...
#pragma unroll
  for (int g = 0; g < kGroups; ++g) v[g] = s1_group_sums<R>(cells, 32 * half + u + kHalf * g);
#pragma unroll
  for (int n = kGroups / 2; n >= 1; n /= 2)
#pragma unroll
    for (int g = 0; g < n; ++g) v[g] = make_float2(v[g].x + v[g + n].x, v[g].y + v[g + n].y);
  float2 t = v[0];
#pragma unroll
  for (int x = kHalf / 2; x >= 1; x /= 2) {
    t.x += __shfl_xor_sync(0xffffffffu, t.x, x);
    t.y += __shfl_xor_sync(0xffffffffu, t.y, x);
  }
  return make_float2(t.x + __shfl_xor_sync(0xffffffffu, t.x, kHalf),
                     t.y + __shfl_xor_sync(0xffffffffu, t.y, kHalf));
}

// 4 R cells: rows r0 .. r0 + 3 of the block, the thread's R diagonals.  kEdge adds the
// predicates of blocks that touch the start of a diagonal, the first W + 1 key columns or the
// end of the sequence.  Returns the keep flags as bits (row rr, diagonal e at bit 4 rr + e); R = 4
// adds the row sums to es / eds, fewer diagonals store the thread's cells at `cells`.
template <int NG, int R, bool kWindowed, bool kDropout, bool kEdge>
__device__ __forceinline__ uint32_t s1_group(const ColWindow<NG, R, kWindowed, kDropout>& cw,
                                             const S1Smem& sm, const S1Params& p,
                                             const DropoutKey& dkey, int r0, int i0, int j_first,
                                             uint32_t qword0, float (&S)[R], int (&hs)[R],
                                             float (&es)[4], float (&eds)[4], float2* cells) {
  int q[4], qo[4];
  {
    const int4 q4 = *reinterpret_cast<const int4*>(sm.s_q + r0);
    q[0] = q4.x; q[1] = q4.y; q[2] = q4.z; q[3] = q4.w;
    if (kWindowed) {
      const int4 o4 = *reinterpret_cast<const int4*>(sm.s_qold + r0);
      qo[0] = o4.x; qo[1] = o4.y; qo[2] = o4.z; qo[3] = o4.w;
    }
  }
  // mismatch counts and the sliding window sums of all cells first: whether any window
  // product of the warp survives flush-to-zero is decided once per group
  int ham[4][R];
  int hsv[4][R];
  bool alive = false;
#pragma unroll
  for (int rr = 0; rr < 4; ++rr) {
#pragma unroll
    for (int e = 0; e < R; ++e) {
      const int idx = rr + R - 1 - e;
      ham[rr][e] = __popc(q[rr] ^ cw.k[idx]);
      if (kWindowed) {
        const int old = __popc(qo[rr] ^ cw.kold[idx]);
        if (kEdge) {
          const int j = j_first + rr - e;        // key column of the cell
          const bool act = j >= 0 && i0 + r0 + rr <= p.len - 1;
          hs[e] += act ? ham[rr][e] - (j > p.W ? old : 0) : 0;
          alive |= j >= p.W && hs[e] <= p.hs_cut;
        } else {
          hs[e] += ham[rr][e] - old;
          alive |= hs[e] <= p.hs_cut;
        }
        hsv[rr][e] = hs[e];
      }
    }
  }
  float P[4][R];
#pragma unroll
  for (int rr = 0; rr < 4; ++rr)
#pragma unroll
    for (int e = 0; e < R; ++e) P[rr][e] = 0.0f;
  if (kWindowed && __any_sync(0xffffffffu, alive)) {
#pragma unroll
    for (int rr = 0; rr < 4; ++rr)
#pragma unroll
      for (int e = 0; e < R; ++e) {
        bool on = hsv[rr][e] <= p.hs_cut;
        if (kEdge) on = on && (j_first + rr - e) >= p.W;
        P[rr][e] = on ? __expf(p.neg_md * (float)hsv[rr][e]) : 0.0f;
      }
  }
  uint32_t keepbits = 0;
#pragma unroll
  for (int rr = 0; rr < 4; ++rr) {
    const float* lut = sm.ulut + (r0 + rr) * NG * 16;
    const uint32_t qword = qword0 ^ (uint32_t)(r0 + rr);   // block rows start at a multiple of 16
    float ev[R], dv[R];
#pragma unroll
    for (int e = 0; e < R; ++e) {
      const int idx = rr + R - 1 - e;
      const float x = sm.glut[ham[rr][e]];
      const float Sn = x * (1.0f + S[e]) - P[rr][e];
      bool act = true;
      if (kEdge) act = (j_first + rr - e) >= 0 && i0 + r0 + rr <= p.len - 1;
      S[e] = act ? Sn : 0.0f;
      // the log i term cancels in the softmax, so the fixed reference drops it too
      float ex = exp2f(fmaf(sqrtf(1.0f + S[e]), p.mul2, p.bias2));
      if (kEdge) ex = act ? ex : 0.0f;
      const float du = tiled_utility<NG>(lut, cw.v0[idx], NG > 4 ? cw.v1[idx] : 0u);
      const bool keep = !kDropout || (act && dropout_keep_open(dkey, cw.h1[idx], qword));
      if constexpr (R == 4) {
        es[rr] += ex;
        if (keep) {       // predicated: one logic operation and one fused multiply-add
          if (kDropout) keepbits |= 1u << (4 * rr + e);
          eds[rr] = fmaf(ex, du, eds[rr]);
        }
      } else {
        if (kDropout) keepbits |= keep ? 1u << (4 * rr + e) : 0u;
        ev[e] = ex;
        dv[e] = keep ? du : 0.0f;
      }
    }
    if constexpr (R == 2)
      *reinterpret_cast<float4*>(cells + rr * kTBand) = make_float4(ev[0], dv[0], ev[1], dv[1]);
    if constexpr (R == 1) cells[rr * kTBand] = make_float2(ev[0], dv[0]);
  }
  return keepbits;
}

// Sweep 1, R diagonals per thread.  Writes the same checkpoints and per-item row partials as
// vjp_sweep1_kernel<NG, true, ...> (analytic softmax reference only); the dropout keep flags go
// out as one 64-bit word per four diagonals and block, the layout vjp_sweep2_tiled_kernel reads, or
// (kBallot) as the row ballots that the one-diagonal-per-thread second sweep reads.
template <int NG, int R, bool kWindowed, bool kDropout, bool kBallot>
__global__ void __launch_bounds__(s1_threads(R), 2 * R) vjp_sweep1_tiled_kernel(VjpArgs a) {
  constexpr int kTThreads = s1_threads(R), kTWarps = kTThreads / 32;
  extern __shared__ float4 smem_raw[];
  const S1Smem sm = s1_carve(reinterpret_cast<float*>(smem_raw), R);
  Item it;
  if (!load_item_1d(a, &it)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool dense = a.plan.cu_seqlens == nullptr;
  const int64_t sym_base = (int64_t)it.seq * a.sym_seq_stride + (int64_t)it.h * a.sym_head_stride +
                           (dense ? 0 : it.start);
  const int32_t* __restrict__ q = a.qsym + sym_base;
  const int32_t* __restrict__ k = a.ksym + sym_base;
  const int vh = it.h / a.group;
  const uint32_t* __restrict__ vb = a.vbits + ((int64_t)vh * a.N + it.start) * a.vwords;
  const int W = a.W;
  S1Params p;
  p.W = W;
  p.len = it.len;
  p.neg_md = -a.mismatch_scale / (float)a.D;
  p.hs_cut = a.window_cut;
  const float logit_mul = kSqrtScale * a.scale;
  const float top_root = sqrtf(1.0f + (float)W) - 1.0f;
  const float ref_top = a.scale * kSqrtScale * top_root;
  p.mul2 = logit_mul * 1.4426950408889634f;
  p.bias2 = -(logit_mul + ref_top) * 1.4426950408889634f;
  const DropoutKey dkey = make_dropout_key((uint32_t)it.h + a.head_offset,
                                           (uint32_t)it.seq + a.batch_offset, a.seed, a.dropout_p);
  if (tid <= a.D) sm.glut[tid] = expf(p.neg_md * (float)tid);
  const int vslot = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);

  for (int w = it.w_begin; w < it.w_end; ++w) {
    const int dmin = 1 + w * kTBand;
    const int dmax = dmin + kTBand - 1;
    float S[R];
    int hs[R];
#pragma unroll
    for (int e = 0; e < R; ++e) {
      S[e] = 0.0f;
      hs[e] = 0;
    }
    const int rb_lo = dmin / kTRows, rb_hi = (it.len - 1) / kTRows;
    int tab_base = 0;                           // window column 0 inside the table buffers
    const int64_t ck_band = it.ck_base + vjp_ck_before(it.len, w);
    for (int rb = rb_lo; rb <= rb_hi; ++rb) {
      const int i0 = rb * kTRows;                 // rows i0 .. i0 + 15, masked where absent
      const int jwin0 = i0 - dmax;                // key column of window index 0
      const int first_row = max(i0, dmin);        // rows below it belong to no cell of the band
      const int skew = first_row - i0;
      const int64_t ck_idx = ck_band + (rb - rb_lo);
      // No barrier here: every warp has passed the barrier that closes the previous block (all
      // table reads done), and the threads that still read the sums or cells of its rows after it
      // are through before they reach the barrier below, ahead of which nobody writes new ones.
      // ---- block tables: entry `at` of the buffers describes window column c.  Every global
      // load of the block (entering columns, row symbols, grad_output of the utility tables) is
      // issued before the first result is used, so the section costs one round trip to L2, not
      // three in a row.
      struct ColRaw { int k, kold; uint32_t bits; };
      auto load_col = [&](int c) {
        const int j = jwin0 + c;
        const bool in = j >= 0 && j < it.len - 1;
        const int jo = j - W - 1;
        ColRaw r;
        r.k = in ? __ldg(k + j) : 0;
        r.kold = (kWindowed && jo >= 0 && jo < it.len) ? __ldg(k + jo) : 0;
        r.bits = in ? __ldg(vb + j + 1) : 0u;
        return r;
      };
      auto store_col = [&](int at, int c, const ColRaw& r) {
        sm.s_k[at] = r.k;
        sm.s_kold[at] = r.kold;
        if (kDropout) sm.s_h1[at] = dropout_route_open((uint32_t)(jwin0 + c + 1));
        sm.s_vb0[at] = spread_nibbles(r.bits & 0xffffu);
        if (NG > 4) sm.s_vb1[at] = spread_nibbles(r.bits >> 16);
      };
      // raw grad_output element (converted after all loads are under way)
      auto go_raw = [&](int64_t idx) -> uint32_t {
        return a.dtype == ROSA_B200_F32 ? __ldg(static_cast<const uint32_t*>(a.go) + idx)
                                        : (uint32_t)__ldg(static_cast<const uint16_t*>(a.go) + idx);
      };
      auto go_value = [&](uint32_t bits) {
        if (a.dtype == ROSA_B200_F32) return __uint_as_float(bits);
        if (a.dtype == ROSA_B200_F16) return __half2float(__ushort_as_half((unsigned short)bits));
        return __uint_as_float(bits << 16);
      };
      // utility table of (row, value group) e from its four raw elements
      auto store_ulut = [&](int e, const uint32_t (&raw)[4]) {
        float gv[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) gv[b] = go_value(raw[b]);
        float4* dst = reinterpret_cast<float4*>(sm.ulut + e * 16);
#pragma unroll
        for (int n4 = 0; n4 < 4; ++n4) {
          // nibbles 4 n4 .. 4 n4 + 3: bits 2 and 3 fixed by n4, bits 0 and 1 vary
          const float hi = ((n4 & 1) ? gv[2] : -gv[2]) + ((n4 & 2) ? gv[3] : -gv[3]);
          dst[n4] = make_float4(hi - gv[0] - gv[1], hi + gv[0] - gv[1], hi - gv[0] + gv[1],
                                hi + gv[0] + gv[1]);
        }
      };
      auto load_go4 = [&](int e, uint32_t (&raw)[4]) {
        const int r = e / NG, g = e - r * NG;
        const int i = i0 + r;
#pragma unroll
        for (int b = 0; b < 4; ++b) raw[b] = 0u;     // +0.0 in every dtype
        if (e < kTRows * NG && i >= first_row && i <= it.len - 1) {
          const int64_t base = (((int64_t)it.start + i) * a.H + it.h) * a.Dv + 4 * g;
#pragma unroll
          for (int b = 0; b < 4; ++b)
            if (4 * g + b < a.Dv) raw[b] = go_raw(base + b);
        }
      };
      // -- loads
      ColRaw entering{0, 0, 0u};
      int q_new = 0, qold_new = 0;
      if (tid < kTRows) {
        if (rb != rb_lo) entering = load_col(kTBand + tid);
        const int i = i0 + tid;
        const bool in = i >= first_row && i <= it.len - 1;
        q_new = in ? __ldg(q + i) : 0;
        qold_new = (kWindowed && in && i - W - 1 >= 0) ? __ldg(q + i - W - 1) : 0;
      }
      uint32_t go_first[4];
      // the per-block chores are spread over the warps: the first fetches the entering columns and
      // the row symbols, the upper half builds the utility tables and closes the block's row sums
      const int ue = (tid + kTThreads / 2) & (kTThreads - 1);
      load_go4(ue, go_first);
      // -- shared-memory side
      if (rb == rb_lo) {                          // a band starts: the whole window
        tab_base = 0;
        for (int c = tid; c < kTWin; c += kTThreads) store_col(c, c, load_col(c));
      } else {                                    // the window moved up by 16 columns
        if (tab_base < kTSlide) {
          tab_base += kTRows;
        } else {
          for (int e = tid; e < kTWin - kTRows; e += kTThreads) {
            const int from = kTSlide + kTRows + e;
            sm.s_k[e] = sm.s_k[from];
            if (kWindowed) sm.s_kold[e] = sm.s_kold[from];
            if (kDropout) sm.s_h1[e] = sm.s_h1[from];
            sm.s_vb0[e] = sm.s_vb0[from];
            if (NG > 4) sm.s_vb1[e] = sm.s_vb1[from];
          }
          tab_base = 0;
        }
        if (tid < kTRows) store_col(tab_base + kTBand + tid, kTBand + tid, entering);
      }
      S1Smem win = sm;                            // the tables as the block's window sees them
      win.s_k += tab_base;
      win.s_kold += tab_base;
      win.s_h1 += tab_base;
      win.s_vb0 += tab_base;
      win.s_vb1 += tab_base;
      if (tid < kTRows) {
        sm.s_q[tid] = q_new;
        sm.s_qold[tid] = qold_new;
      }
      // nibble tables: one thread per (row, value group) builds its sixteen signed sums
      if (ue < kTRows * NG) store_ulut(ue, go_first);
      for (int e = ue + kTThreads; e < kTRows * NG; e += kTThreads) {
        uint32_t raw[4];
        load_go4(e, raw);
        store_ulut(e, raw);
      }
      __syncthreads();
      // ---- checkpoint of the thread's diagonals
      {
        auto* ck = a.ckpt + ck_idx * kTBand + R * tid;
        if constexpr (R == 1) {
          *reinterpret_cast<int2*>(ck) = make_int2(__float_as_int(S[0]), hs[0]);
        } else {
#pragma unroll
          for (int e = 0; e < R; e += 2)
            reinterpret_cast<int4*>(ck)[e / 2] =
                make_int4(__float_as_int(S[e]), hs[e], __float_as_int(S[e + 1]), hs[e + 1]);
        }
      }
      const bool interior = jwin0 >= (kWindowed ? W + 1 : 0) && i0 + kTRows - 1 <= it.len - 1;
      const uint32_t qword0 = dropout_query_word((uint32_t)i0);
      // window column of (row 0, last diagonal of this thread); a multiple of R
      const int col0 = kTBand - R - R * tid;
      constexpr int kKept = s1_kept(R);
      ColWindow<NG, R, kWindowed, kDropout> cw;
      load_window<NG, R, kWindowed, kDropout>(cw, win, col0, 0, kKept);
      uint32_t keep_lo = 0u, keep_hi = 0u;
#pragma unroll 1
      for (int r0 = 0; r0 < kTRows; r0 += 4) {
        load_window<NG, R, kWindowed, kDropout>(cw, win, col0 + r0 + kKept, kKept, 4);
        float es[4] = {0.0f, 0.0f, 0.0f, 0.0f}, eds[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        // key column of (row r0, diagonal 0 of this thread)
        const int j_first = jwin0 + col0 + r0 + R - 1;
        float2* cells = R == 4 ? nullptr : sm.wstat + r0 * kTBand + s1_cell<R>(R * tid);
        uint32_t keep;
        if (interior)
          keep = s1_group<NG, R, kWindowed, kDropout, false>(cw, sm, p, dkey, r0, i0, j_first, qword0, S,
                                                          hs, es, eds, cells);
        else
          keep = s1_group<NG, R, kWindowed, kDropout, true>(cw, sm, p, dkey, r0, i0, j_first, qword0, S,
                                                         hs, es, eds, cells);
        if constexpr (kDropout && kBallot) {
          // a word per row and 32 diagonals: [row][diagonal / 32], lane L writes row L / R (R = 2: the
          // even diagonals' flags and the odd ones' are interleaved)
          static_assert(R <= 2, "a word holds the flags of whole lanes of one or two diagonals");
          const int mine = (lane / R) & 3;
          uint32_t word[R];
#pragma unroll
          for (int rr = 0; rr < 4; ++rr)
#pragma unroll
            for (int e = 0; e < R; ++e) {
              const uint32_t ballot = __ballot_sync(0xffffffffu, keep >> (4 * rr + e) & 1u);
              if (rr == 0 || mine == rr) word[e] = ballot;
            }
          if constexpr (R == 2) {
            const int half = 16 * (lane & 1);
            word[0] = spread_bits(word[0] >> half) | spread_bits(word[1] >> half) << 1;
          }
          const int row = r0 + mine - skew;     // there the rows of a block count from its first one
          if (lane < 4 * R && row >= 0)
            a.keepbits[(ck_idx * kTRows + row) * (kTBand / 32) + R * warp + lane % R] = word[0];
        } else if (kDropout) {
          // the keep flags of this group: bit 4 r + e of the 64-bit word of the block
          if (r0 < 8) keep_lo |= keep << (4 * r0);
          else keep_hi |= keep << (4 * (r0 - 8));
        }
        if constexpr (R == 4) {
          float v[8];
#pragma unroll
          for (int rr = 0; rr < 4; ++rr) {
            v[2 * rr] = es[rr];
            v[2 * rr + 1] = eds[rr];
          }
          const float total = warp_reduce8(v, lane);
          if ((lane & 3) == 0)
            reinterpret_cast<float*>(sm.wstat + (r0 + (vslot >> 1)) * kTWarps + warp)[vslot & 1] = total;
        }
        // the upper entries become the lower ones of the next group
#pragma unroll
        for (int x = 0; x < kKept; ++x) {
          cw.k[x] = cw.k[x + 4];
          if (kWindowed) cw.kold[x] = cw.kold[x + 4];
          if (kDropout) cw.h1[x] = cw.h1[x + 4];
          cw.v0[x] = cw.v0[x + 4];
          if (NG > 4) cw.v1[x] = cw.v1[x + 4];
        }
      }
      // keep flags of the block: one 64-bit word per four diagonals (row r, diagonal e at bit
      // 4 r + e), put together by the 4 / R threads that own them
      if (kDropout && !kBallot) {
        if constexpr (R < 4) {
          const int part = tid & (4 / R - 1);
          keep_lo <<= R * part;
          keep_hi <<= R * part;
#pragma unroll
          for (int x = 1; x < 4 / R; x *= 2) {
            keep_lo |= __shfl_xor_sync(0xffffffffu, keep_lo, x);
            keep_hi |= __shfl_xor_sync(0xffffffffu, keep_hi, x);
          }
        }
        if ((tid & (4 / R - 1)) == 0)
          reinterpret_cast<uint2*>(a.keepbits)[ck_idx * (kTBand / 4) + tid / (4 / R)] =
              make_uint2(keep_lo, keep_hi);
      }
      __syncthreads();
      // row of the tail: R = 4 one thread of the second warp each, else 16 or 8 lanes each
      constexpr int kLanes = R == 4 ? 2 : kTThreads / kTRows;
      const int tr = R == 4 ? tid - kTThreads / 2 : tid / kLanes;
      float2 sum = make_float2(0.0f, 0.0f);
      if constexpr (R < 4) sum = s1_row_sums<R>(sm.wstat, tr, lane);
      if (tr >= 0 && tr < kTRows && (R == 4 || tid % kLanes == 0)) {
        const int i = i0 + tr;
        if (i >= first_row && i <= it.len - 1) {
          if constexpr (R == 4) {
            const float2 upper = sm.wstat[tr * kTWarps], lower = sm.wstat[tr * kTWarps + 1];
            sum = make_float2(upper.x + lower.x, upper.y + lower.y);
          }
          // ref_top - log i, rounded once; where both factors of ref_top are at hand the product
          // is fused and log i rounded, elsewhere log i is.  (One last bit of m is 2e-6 of a row's
          // sums: each variant keeps its rounding, so that gradients keep their bits.)
          constexpr bool kFusedTop = kWindowed && (kDropout || NG > 4);
          float m = kFusedTop ? fmaf(a.scale * kSqrtScale, top_root, -logf((float)i))
                              : fmaf(-__log2f((float)i), 0.69314718f, ref_top);
          float z = sum.x, e = sum.y * a.inv_keep;
          const int64_t slot = it.rowslot + i;
          if (w > it.w_begin) {
            const float4 prev = a.stat_part[slot];
            merge_stats(m, z, e, prev.x, prev.y, prev.z);
          }
          a.stat_part[slot] = make_float4(m, z, e, 0.0f);
        }
      }
    }
  }
}

template <int NG, int R, bool kBallot>
int launch_s1_tiled_r(const VjpArgs& a, unsigned grid, cudaStream_t stream) {
  constexpr int threads = s1_threads(R);
  constexpr int smem = s1_smem_words(NG, R) * (int)sizeof(float);
  const bool windowed = a.ring_slots > 0;
  const bool dropout = a.dropout_p > 0.0f;
  auto kernel = windowed ? (dropout ? vjp_sweep1_tiled_kernel<NG, R, true, true, kBallot>
                                    : vjp_sweep1_tiled_kernel<NG, R, true, false, false>)
                         : (dropout ? vjp_sweep1_tiled_kernel<NG, R, false, true, kBallot>
                                    : vjp_sweep1_tiled_kernel<NG, R, false, false, false>);
  if (smem > 48 * 1024)
    ROSA_CUDA_OK(allow_shared(kernel));
  kernel<<<grid, threads, smem, stream>>>(a);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

// Diagonals per thread.  Four share the most work (row values, column loads, row reductions), but a
// CTA is then two warps that need 7 us for a block of 16 rows; two or one have more warps work on a
// block.  Where the longest item decides that is the faster way (time with four / two / one):
//   1 x 256 x 4 float32 (fill 0.03)                    56 / 53 / 44 us
//   1 x 4096 x 16 (fill 0.9)                          1192 / 856 / 793 us
//   packed 3001 x 16, sequences up to 257             153 / 107 / 84 us
//   2 x 1024 x 64 (fill 2.2)                          451 / 347 / 358 us
//   4 x 1024 x 64 (fill 4.3)                          592 / 584 / 647 us
//   32 x 256 x 32 (fill 6.9)                          250 / 255 / 312 us
//   2 x 4096 x 64 (fill 7.4)                          2.76 / 2.86 / 3.66 ms
//   2 x 8192 x 64 (fill 14)                           9.48 / 10.4 / 13.7 ms
// Value rows of more than 16 components (two sign tables) never take four: their column windows and
// four sets of diagonals leave no registers to overlap anything (packed 32768 x 16, 32 components:
// 14.0 / 8.2 / 10.2 ms).
template <int NG>
int launch_s1_tiled(const VjpArgs& a, unsigned grid, cudaStream_t stream) {
  const float fill = vjp_fill(a);
  if (!vjp_tiled_applies(a)) {      // the second sweep is the one that reads ballots
    if (fill < 1.8f) return launch_s1_tiled_r<NG, 1, true>(a, grid, stream);
    return launch_s1_tiled_r<NG, 2, true>(a, grid, stream);
  }
  if (fill < 1.8f) return launch_s1_tiled_r<NG, 1, false>(a, grid, stream);
  if constexpr (NG > 4) {
    return launch_s1_tiled_r<NG, 2, false>(a, grid, stream);
  } else {
    if (fill < 7.0f) return launch_s1_tiled_r<NG, 2, false>(a, grid, stream);
    return launch_s1_tiled_r<NG, 4, false>(a, grid, stream);
  }
}

}  // namespace

// Value rows of up to 32 components (nibble tables), the analytic softmax reference, and not the
// testing flag that selects the one-diagonal-per-thread kernels.
bool vjp_sweep1_tiled_applies(const VjpArgs& a) {
  const float top = a.scale * kSqrtScale * (sqrtf(1.0f + (float)a.W) - 1.0f);
  return a.Dv <= 32 && top <= 80.0f && !a.force_cuda_core_contraction;
}

// The second sweep takes symbols of up to 16 bits (one MMA N).
bool vjp_tiled_applies(const VjpArgs& a) { return vjp_sweep1_tiled_applies(a) && a.D <= 16; }

int launch_vjp_sweep1_tiled(const VjpArgs& a, int items_upper, cudaStream_t stream) {
  const unsigned grid = (unsigned)((int64_t)items_upper * a.H);
  if (a.Dv <= 8) return launch_s1_tiled<2>(a, grid, stream);
  if (a.Dv <= 16) return launch_s1_tiled<4>(a, grid, stream);
  return launch_s1_tiled<8>(a, grid, stream);
}

}  // namespace rosa
