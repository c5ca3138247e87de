// Hard forward of the rosa_soft operator: sign-binarise Q/K into packed symbols, find the
// latest among the longest causal suffix matches within the horizon, gather the sign of
// the routed value row.  Replaces pack_sign_bits_pair_kernel, exact_suffix_length,
// merge_hard_route and hard_forward_kernel of the reference
// (rosa_soft/csrc/cuda/rosa_soft_kernels.cu:202-241, 311-531).
//
// Rows are resolved by the chained matcher (chain_match.cu).  Here: packing, and the matcher of the
// entry point without a workspace, the exact diagonal run-length recurrence
//     len(i, a) = (q_i == k_{a-1}) ? min(len(i-1, a-1) + 1, W) : 0
// where one thread owns several diagonals, a warp sits on one query row at a time, the per-row
// winner is reduced with redux.sync and merged across bands with one 64-bit integer atomicMax
// (order independent, hence exact and deterministic).
#include "common.cuh"
#include "chain_match.cuh"
#include "row_emit.cuh"

namespace rosa {

namespace {

// ------------------------------------------------------------------ packing
template <typename T>
__device__ __forceinline__ bool positive(T x);
template <>
__device__ __forceinline__ bool positive<float>(float x) { return x > 0.0f; }
template <>
__device__ __forceinline__ bool positive<__half>(__half x) { return __half2float(x) > 0.0f; }
template <>
__device__ __forceinline__ bool positive<__nv_bfloat16>(__nv_bfloat16 x) {
  return __bfloat162float(x) > 0.0f;
}

// Sign bits of one D-vector.  When the vector is a whole number of 16-byte words (and the tensor
// base is 16-byte aligned) it is read with 128-bit loads; bit d of the word is set iff
// component d is strictly positive (zero, -0 and NaN give 0).
template <typename T>
__device__ __forceinline__ uint32_t sign_word(const T* __restrict__ row, int D, bool vec) {
  uint32_t w = 0;
  if (vec) {
    constexpr int kPer = 16 / (int)sizeof(T);
    const uint4* p = reinterpret_cast<const uint4*>(row);
    for (int c = 0; c < D / kPer; ++c) {
      const uint4 raw = __ldg(p + c);
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int x = 0; x < kPer; ++x) w |= (uint32_t)positive<T>(e[x]) << (c * kPer + x);
    }
  } else {
    for (int d = 0; d < D; ++d) w |= (uint32_t)positive<T>(row[d]) << d;
  }
  return w;
}

// One thread per (token, head); threads of a warp read consecutive D-vectors.
template <typename T>
__global__ void pack_symbols_kernel(const T* __restrict__ q, const T* __restrict__ k, int64_t N,
                                    int H, int D, int dense, int64_t uniform_len, int vec,
                                    int32_t* __restrict__ pq, int32_t* __restrict__ pk,
                                    uint32_t* __restrict__ zeroed) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= N * H) return;
  if (zeroed != nullptr) zeroed[idx] = 0u;         // scratch of the matcher, one word per token-head
  const int64_t token = idx / H;
  const int h = (int)(idx - token * H);
  const uint32_t wq = sign_word<T>(q + idx * D, D, vec != 0);
  const uint32_t wk = k != nullptr ? sign_word<T>(k + idx * D, D, vec != 0) : 0u;
  int64_t dst;
  if (dense) {
    const int64_t b = token / uniform_len, t = token - b * uniform_len;
    dst = (b * H + h) * uniform_len + t;
  } else {
    dst = (int64_t)h * N + token;
  }
  pq[dst] = (int32_t)wq;
  if (k != nullptr) pk[dst] = (int32_t)wk;
}

// token-major [N, H] symbols -> head-major [H, N]
__global__ void transpose_symbols_kernel(const uint32_t* __restrict__ q,
                                         const uint32_t* __restrict__ k, int64_t N, int H,
                                         int32_t* __restrict__ qt, int32_t* __restrict__ kt) {
  __shared__ uint32_t tq[32][33], tk[32][33];
  const int64_t t0 = (int64_t)blockIdx.x * 32;
  const int h0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int64_t t = t0 + r;
    const int h = h0 + threadIdx.x;
    if (t < N && h < H) {
      tq[r][threadIdx.x] = q[t * H + h];
      tk[r][threadIdx.x] = k[t * H + h];
    }
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int h = h0 + r;
    const int64_t t = t0 + threadIdx.x;
    if (t < N && h < H) {
      qt[(int64_t)h * N + t] = (int32_t)tq[threadIdx.x][r];
      kt[(int64_t)h * N + t] = (int32_t)tk[threadIdx.x][r];
    }
  }
}

// ------------------------------------------------------------------ matching
// grid = (work items, heads); a work item is kFwdBand consecutive diagonals of one
// sequence; every warp of the CTA walks its own 256 diagonals independently.
__global__ void __launch_bounds__(kFwdWarps * 32)
    hard_match_kernel(Plan plan, const int32_t* __restrict__ qsym,
                      const int32_t* __restrict__ ksym, int64_t sym_seq_stride,
                      int64_t sym_head_stride, int H, int W,
                      unsigned long long* __restrict__ best) {
  int seq, local;
  if (!find_item(plan, blockIdx.x, &seq, &local)) return;
  const int h = blockIdx.y;
  int start, len;
  segment_bounds(plan, seq, &start, &len);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int delta0 = 1 + local * kFwdBand + warp * (32 * kFwdPerLane);
  if (delta0 > len - 1) return;
  const bool dense = plan.cu_seqlens == nullptr;
  const int64_t sym_base =
      (int64_t)seq * sym_seq_stride + (int64_t)h * sym_head_stride + (dense ? 0 : start);
  const int32_t* __restrict__ q = qsym + sym_base;
  const int32_t* __restrict__ k = ksym + sym_base;

  int run[kFwdPerLane];
#pragma unroll
  for (int r = 0; r < kFwdPerLane; ++r) run[r] = 0;

  for (int i = delta0; i < len; ++i) {
    const int qi = __ldg(q + i);
    int best_len = 0, best_route = 0;
    const int jbase = i - delta0 - lane;
#pragma unroll
    for (int r = 0; r < kFwdPerLane; ++r) {
      const int j = jbase - r * 32;
      int l = 0;
      if (j >= 0) {
        const int kj = __ldg(k + j);
        l = (kj == qi) ? min(run[r] + 1, W) : 0;
      }
      run[r] = l;
      if (l > best_len) {  // r ascending = route descending: strict > keeps the latest
        best_len = l;
        best_route = j + 1;
      }
    }
    const int row_len = __reduce_max_sync(0xffffffffu, best_len);
    if (row_len > 0) {
      const int row_route =
          __reduce_max_sync(0xffffffffu, best_len == row_len ? best_route : 0);
      if (lane == 0) {
        const unsigned long long key =
            ((unsigned long long)(unsigned)row_len << 32) | (unsigned)row_route;
        unsigned long long* slot = best + ((int64_t)(start + i) * H + h);
        if (*reinterpret_cast<volatile unsigned long long*>(slot) < key) atomicMax(slot, key);
      }
    }
  }
}

// Fast matcher for horizons below 2048 and sequences below 2^21 tokens: the candidate of a
// cell is one 32-bit key (run length << 21 | route), so the row winner is a plain integer
// max.  A CTA of 256 threads owns kFwdBand diagonals (four per thread), stages the key
// symbols of a 32-row block in shared memory, reduces the winner of a row with one
// redux.sync per warp, merges the warps through a shared-memory atomicMax and issues at most
// one global 64-bit atomicMax per row and block.
constexpr int kMatchRows = 32;
constexpr int kMatchThreads = 256;
constexpr int kMatchPerThread = kFwdBand / kMatchThreads;   // 4
constexpr int kMatchWin = kFwdBand + kMatchRows;

template <bool kRamp>
__device__ __forceinline__ void match_rows(int nrows, int tid, int lane, int W, int cmin,
                                           const int* s_q, const int* s_k, unsigned* s_best,
                                           int (&run)[kMatchPerThread], int abase) {
  for (int r = 0; r < nrows; ++r) {
    const int qi = s_q[r];
    unsigned best = 0;
#pragma unroll
    for (int u = 0; u < kMatchPerThread; ++u) {
      const int c = kFwdBand - 1 - tid - u * kMatchThreads + r;   // window column of this cell
      bool eq = s_k[c] == qi;
      if (kRamp) eq = eq && c >= cmin;                            // columns before the sequence
      const int l = eq ? min(run[u] + 1, W) : 0;
      run[u] = l;
      const unsigned key = ((unsigned)l << 21) + (unsigned)(abase + c);   // route = jwin0 + c + 1
      if (eq) best = max(best, key);
    }
    const unsigned wbest = __reduce_max_sync(0xffffffffu, best);
    if (lane == 0 && wbest > 0) atomicMax(s_best + r, wbest);
  }
}

__global__ void __launch_bounds__(kMatchThreads)
    hard_match_fast_kernel(Plan plan, const int32_t* __restrict__ qsym,
                           const int32_t* __restrict__ ksym, int64_t sym_seq_stride,
                           int64_t sym_head_stride, int H, int W,
                           unsigned long long* __restrict__ best) {
  __shared__ int s_k[kMatchWin];
  __shared__ int s_q[kMatchRows];
  __shared__ unsigned s_best[kMatchRows];
  const int slot = blockIdx.x / H;
  int seq, local;
  if (!find_item(plan, slot, &seq, &local)) return;
  const int h = blockIdx.x - slot * H;
  int start, len;
  segment_bounds(plan, seq, &start, &len);
  const int tid = threadIdx.x, lane = tid & 31;
  const int dmin = 1 + local * kFwdBand, dmax = dmin + kFwdBand - 1;
  const bool dense = plan.cu_seqlens == nullptr;
  const int64_t sym_base =
      (int64_t)seq * sym_seq_stride + (int64_t)h * sym_head_stride + (dense ? 0 : start);
  const int32_t* __restrict__ q = qsym + sym_base;
  const int32_t* __restrict__ k = ksym + sym_base;
  int run[kMatchPerThread];
#pragma unroll
  for (int u = 0; u < kMatchPerThread; ++u) run[u] = 0;

  for (int i0 = dmin; i0 < len; i0 = (i0 / kMatchRows + 1) * kMatchRows) {
    const int i1 = min((i0 / kMatchRows + 1) * kMatchRows - 1, len - 1);
    const int nrows = i1 - i0 + 1;
    const int jwin0 = i0 - dmax;   // key column of window index 0
    __syncthreads();
    for (int c = tid; c < nrows + kFwdBand - 1; c += kMatchThreads) {
      const int j = jwin0 + c;
      s_k[c] = (j >= 0 && j < len - 1) ? __ldg(k + j) : 0;
    }
    if (tid < nrows) {
      s_q[tid] = __ldg(q + i0 + tid);
      s_best[tid] = 0;
    }
    __syncthreads();
    if (jwin0 < 0)
      match_rows<true>(nrows, tid, lane, W, -jwin0, s_q, s_k, s_best, run, jwin0 + 1);
    else
      match_rows<false>(nrows, tid, lane, W, 0, s_q, s_k, s_best, run, jwin0 + 1);
    __syncthreads();
    if (tid < nrows && s_best[tid] > 0) {
      const unsigned key = s_best[tid];
      const unsigned long long wide =
          ((unsigned long long)(key >> 21) << 32) | (unsigned long long)(key & 0x1FFFFFu);
      atomicMax(best + ((int64_t)(start + i0 + tid) * H + h), wide);
    }
  }
}

// ------------------------------------------------------------------- gather
// One thread per (token, head, chunk of value components): 16 bytes of output per thread when
// the rows allow it (128-bit loads of the value row, one 128-bit store), else element by element.
// OutT = T writes the operator's output in the input dtype; OutT = int8_t writes -1 / 0 / +1
// bytes for a consumer that takes the routed signs as integers.
template <typename T, typename OutT>
__global__ void gather_output_kernel(Plan plan, const unsigned long long* __restrict__ best,
                                     const T* __restrict__ v, int64_t N, int H, int Hv, int Dv,
                                     int chunk, int vec, OutT* __restrict__ out,
                                     int32_t* __restrict__ route_token) {
  const int chunks = (Dv + chunk - 1) / chunk;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= N * H * chunks) return;
  const int c = (int)(idx % chunks);
  const int64_t th = idx / chunks;
  const int64_t token = th / H;
  const int h = (int)(th - token * H);
  const int route = (int)(best[th] & 0xffffffffull);
  int start = 0, len = 0;
  int64_t src_token = -1;
  if (route > 0 && find_segment(plan, token, &start, &len) >= 0) src_token = (int64_t)start + route;
  if (c == 0 && route_token) route_token[th] = (int32_t)src_token;
  OutT* o = out + th * Dv;
  const int d0 = c * chunk, d1 = min(Dv, d0 + chunk);
  const T* src = src_token < 0 ? nullptr : v + (src_token * Hv + h / (H / Hv)) * Dv;
  if (vec) {
    // `chunk` components: 16 bytes of OutT; the value row is read in 16-byte words
    constexpr int kOutPer = 16 / (int)sizeof(OutT);
    constexpr int kInPer = 16 / (int)sizeof(T);
    alignas(16) OutT vals[kOutPer];
#pragma unroll
    for (int x = 0; x < kOutPer; ++x) vals[x] = (OutT)0;
    if (src != nullptr) {
#pragma unroll
      for (int wd = 0; wd < kOutPer / kInPer; ++wd) {
        const uint4 raw = __ldg(reinterpret_cast<const uint4*>(src + d0) + wd);
        const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int x = 0; x < kInPer; ++x)
          vals[wd * kInPer + x] = positive<T>(e[x]) ? (OutT)1.0f : (OutT)-1.0f;
      }
    }
    *reinterpret_cast<uint4*>(o + d0) = *reinterpret_cast<const uint4*>(vals);
    return;
  }
  for (int d = d0; d < d1; ++d)
    o[d] = src == nullptr ? (OutT)0 : positive<T>(src[d]) ? (OutT)1.0f : (OutT)-1.0f;
}

// Splits the winners into the selected route (local index a, 0 = null) and its match length.
__global__ void route_inspect_kernel(const unsigned long long* __restrict__ best, int64_t count,
                                     int32_t* __restrict__ route, int32_t* __restrict__ length) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= count) return;
  const unsigned long long key = best[idx];
  if (route) route[idx] = (int32_t)(key & 0xffffffffull);
  if (length) length[idx] = (int32_t)(key >> 32);
}

}  // namespace

int launch_route_inspect(const unsigned long long* best, int64_t count, int32_t* route,
                         int32_t* length, cudaStream_t stream) {
  ProfileScope prof("route_inspect", stream);
  const int threads = 256;
  route_inspect_kernel<<<(unsigned)((count + threads - 1) / threads), threads, 0, stream>>>(
      best, count, route, length);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

int launch_pack_symbols(const void* q, const void* k, int dtype, int64_t N, int H, int D,
                        int dense, int64_t uniform_len, int32_t* pq, int32_t* pk, uint32_t* zeroed,
                        cudaStream_t stream) {
  ProfileScope prof("pack_symbols", stream);
  const int threads = 256;
  const int64_t blocks = (N * H + threads - 1) / threads;
  const int esize = dtype == ROSA_B200_F32 ? 4 : 2;
  const auto aligned = [](const void* p) { return p == nullptr || ((uintptr_t)p & 15u) == 0; };
  const int vec = (D * esize) % 16 == 0 && aligned(q) && aligned(k);
  if (dtype == ROSA_B200_F32)
    pack_symbols_kernel<float><<<(unsigned)blocks, threads, 0, stream>>>(
        (const float*)q, (const float*)k, N, H, D, dense, uniform_len, vec, pq, pk, zeroed);
  else if (dtype == ROSA_B200_F16)
    pack_symbols_kernel<__half><<<(unsigned)blocks, threads, 0, stream>>>(
        (const __half*)q, (const __half*)k, N, H, D, dense, uniform_len, vec, pq, pk, zeroed);
  else
    pack_symbols_kernel<__nv_bfloat16><<<(unsigned)blocks, threads, 0, stream>>>(
        (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, N, H, D, dense, uniform_len, vec, pq, pk, zeroed);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

int launch_transpose_symbols(const uint32_t* q, const uint32_t* k, int64_t N, int H, int32_t* qt,
                             int32_t* kt, cudaStream_t stream) {
  ProfileScope prof("transpose_symbols", stream);
  dim3 grid((unsigned)((N + 31) / 32), (unsigned)((H + 31) / 32)), block(32, 8);
  transpose_symbols_kernel<<<grid, block, 0, stream>>>(q, k, N, H, qt, kt);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

int launch_run_length_match(const FwdArgs& a, int items_upper, cudaStream_t stream) {
  if (items_upper <= 0) return 0;
  ProfileScope prof("hard_match_runs", stream);
  const int64_t max_len = a.plan.cu_seqlens == nullptr ? a.plan.uniform_len : a.N;
  if (a.W < 2048 && max_len < (1 << 21)) {
    // 32-bit candidate keys: run length in the top 11 bits, route in the low 21
    hard_match_fast_kernel<<<(unsigned)((int64_t)items_upper * a.H), kMatchThreads, 0, stream>>>(
        a.plan, a.packed_q, a.packed_k, a.sym_seq_stride, a.sym_head_stride, a.H, a.W, a.best);
    ROSA_CUDA_OK(cudaGetLastError());
    return 0;
  }
  dim3 grid((unsigned)items_upper, (unsigned)a.H);
  hard_match_kernel<<<grid, kFwdWarps * 32, 0, stream>>>(a.plan, a.packed_q, a.packed_k,
                                                        a.sym_seq_stride, a.sym_head_stride, a.H,
                                                        a.W, a.best);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

namespace {
template <typename T, typename OutT>
int launch_gather_t(const FwdArgs& a, OutT* out, cudaStream_t stream) {
  // vector path: a thread writes 16 bytes of output, i.e. 16 / sizeof(OutT) components, and
  // reads as many value components in 16-byte words
  constexpr int kOutPer = 16 / (int)sizeof(OutT);
  const auto aligned = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
  const bool vec = a.Dv % kOutPer == 0 && aligned(a.v) && aligned(out) &&
                   (a.Dv * (int)sizeof(T)) % 16 == 0 && kOutPer >= 16 / (int)sizeof(T);
  const int chunk = vec ? kOutPer : 8;
  const int chunks = (a.Dv + chunk - 1) / chunk;
  const int threads = 256;
  const int64_t blocks = (a.N * a.H * chunks + threads - 1) / threads;
  gather_output_kernel<T, OutT><<<(unsigned)blocks, threads, 0, stream>>>(
      a.plan, a.best, (const T*)a.v, a.N, a.H, a.Hv, a.Dv, chunk, vec ? 1 : 0, out, a.route_token);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}
}  // namespace

int launch_gather_output(const FwdArgs& a, cudaStream_t stream) {
  ProfileScope prof("gather_output", stream);
  if (a.out_i8 != nullptr) {
    if (a.dtype == ROSA_B200_F32) return launch_gather_t<float, int8_t>(a, a.out_i8, stream);
    if (a.dtype == ROSA_B200_F16) return launch_gather_t<__half, int8_t>(a, a.out_i8, stream);
    return launch_gather_t<__nv_bfloat16, int8_t>(a, a.out_i8, stream);
  }
  if (a.dtype == ROSA_B200_F32) return launch_gather_t<float, float>(a, (float*)a.out, stream);
  if (a.dtype == ROSA_B200_F16) return launch_gather_t<__half, __half>(a, (__half*)a.out, stream);
  return launch_gather_t<__nv_bfloat16, __nv_bfloat16>(a, (__nv_bfloat16*)a.out, stream);
}

}  // namespace rosa
