// Hard matching of whole sequences through occurrence chains (chain_match.cuh): an index kernel
// that links the positions, and a match kernel that resolves the rows and writes the result of
// the call (routed value signs, or payload rows and matched positions).
#include "chain_kernels.cuh"
#include "row_emit.cuh"

namespace rosa {

namespace {

// One CTA per (sequence, head), one warp per context length; the tables of a CTA in shared memory.
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
  const int entries = (1 << hash_bits) + chain_low_entries(bits, context);
  for (int e = threadIdx.x; e < entries; e += blockDim.x) tables[e] = 0;
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  const int L = context - warp;                    // warp 0: the chained length
  Entry* table = warp == 0 ? tables : tables + (1 << hash_bits) + chain_low_entries(bits, L);
  chain_index_warp<Entry, kMerge, false>(qsym + base, ksym + base, 0, len, L, bits, warp == 0, hash_bits,
                                         table, prev + base, (warp == 0 ? start : low) + base);
}

SequenceAxis sequence_axis(const FwdArgs& a) {
  return {a.plan, a.sym_seq_stride, a.sym_head_stride};
}

template <typename Emit>
int match_rows(const FwdArgs& a, int limit, Emit emit, cudaStream_t stream) {
  ProfileScope prof("hard_match", stream);
  return launch_chain_match_t(sequence_axis(a), a.packed_q, a.packed_k, a.N, a.H, a.W, a.context,
                              a.chain_start, a.chain_prev, a.chain_low, limit, a.plan.status + 2, emit,
                              stream);
}

template <typename Emit>
int scan_rows(const FwdArgs& a, const int32_t* run_flag, Emit emit, cudaStream_t stream) {
  return launch_scan_match_t(sequence_axis(a), a.packed_q, a.packed_k, a.N, a.H, a.W, run_flag, emit,
                             stream);
}

}  // namespace

int launch_chain_index(const FwdArgs& a, int64_t max_len, cudaStream_t stream) {
  ProfileScope prof("chain_index", stream);
  const int hash_bits = chain_hash_bits(a.D, a.context, max_len);
  if (a.context > 2)   // several shorter lengths merge their results into zeroed words
    ROSA_CUDA_OK(cudaMemsetAsync(a.chain_low, 0, (size_t)a.N * a.H * sizeof(uint32_t), stream));
  const size_t entries = (size_t)(1 << hash_bits) + chain_low_entries(a.D, a.context);
  const bool merge = a.context > 2, wide = max_len > kChainNarrow;
  const size_t bytes = entries * (wide ? sizeof(unsigned long long) : sizeof(uint32_t));
  auto kernel = wide ? (merge ? chain_index_kernel<unsigned long long, true>
                              : chain_index_kernel<unsigned long long, false>)
                     : (merge ? chain_index_kernel<uint32_t, true> : chain_index_kernel<uint32_t, false>);
  if (bytes > 48 * 1024)
    ROSA_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  kernel<<<(unsigned)(a.plan.S * a.H), 32 * a.context, bytes, stream>>>(
      a.plan, a.packed_q, a.packed_k, a.sym_seq_stride, a.sym_head_stride, a.H, a.D, a.context,
      hash_bits, a.chain_start, a.chain_prev, a.chain_low);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

int launch_chain_forward(const FwdArgs& a, int limit, cudaStream_t stream) {
  return with_sign_emit(a, [&](auto emit) { return match_rows(a, limit, emit, stream); });
}

int launch_chain_inference(const FwdArgs& a, const float* payload, float* out, int64_t* matched_end,
                           int limit, cudaStream_t stream) {
  return match_rows(a, limit, make_payload_emit(a, payload, out, matched_end), stream);
}

int launch_scan_forward(const FwdArgs& a, const int32_t* run_flag, cudaStream_t stream) {
  return with_sign_emit(a, [&](auto emit) { return scan_rows(a, run_flag, emit, stream); });
}

int launch_scan_inference(const FwdArgs& a, const float* payload, float* out, int64_t* matched_end,
                          const int32_t* run_flag, cudaStream_t stream) {
  return scan_rows(a, run_flag, make_payload_emit(a, payload, out, matched_end), stream);
}

}  // namespace rosa
