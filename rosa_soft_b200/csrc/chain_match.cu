// Hard matching of whole sequences through occurrence chains (chain_match.cuh): an index kernel
// that links the positions, and a match kernel that resolves the rows and writes the result of
// the call (routed value signs, or payload rows and matched positions).
#include "chain_kernels.cuh"
#include "row_emit.cuh"

namespace rosa {

namespace {

// One CTA per (sequence, head), one warp per context length and piece; the tables in shared memory.
template <typename Entry, bool kMerge>
__global__ void __maxnreg__(kChainIndexRegisters)
    chain_index_kernel(Plan plan, const int32_t* __restrict__ qsym, const int32_t* __restrict__ ksym,
                       int64_t sym_seq_stride, int64_t sym_head_stride, int H, int bits, int context,
                       int hash_bits, int segments, uint32_t* __restrict__ start,
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
    // the launch is sized for the longest sequence that the pack could hold: buckets (which the CTA has
    // to clear) and pieces by its own length
    hash_bits = min(hash_bits, chain_hash_bits(bits, context, len));
    if (len < 512) segments = 1;
  }
  const int entries = (1 << hash_bits) + chain_low_entries(bits, context);
  for (int e = threadIdx.x; e < entries; e += blockDim.x) tables[e] = 0;
  __syncthreads();
  chain_index_block<Entry, kMerge, false>(qsym + base, ksym + base, 0, len, context, bits, hash_bits,
                                          entries, segments, tables, prev + base, start + base,
                                          low + base);
}

SequenceAxis sequence_axis(const FwdArgs& a) {
  return {a.plan, a.sym_seq_stride, a.sym_head_stride};
}

template <typename Emit>
int match_rows(const FwdArgs& a, ChainPatience patience, Emit emit, cudaStream_t stream) {
  ProfileScope prof("hard_match", stream);
  return launch_chain_match_t(sequence_axis(a), a.packed_q, a.packed_k, a.N, a.H, a.W, a.context,
                              a.chain_start, a.chain_prev, a.chain_low, patience, a.plan.status + 2, emit,
                              stream);
}

template <typename Emit>
int run_rows_of(const FwdArgs& a, const int32_t* run_flag, Emit emit, cudaStream_t stream) {
  return launch_run_match_t(sequence_axis(a), a.packed_q, a.packed_k, a.N, a.H, a.W, run_flag, emit,
                            stream);
}

}  // namespace

int launch_chain_index(const FwdArgs& a, int64_t max_len, cudaStream_t stream) {
  ProfileScope prof("chain_index", stream);
  const bool merge = a.context > 2, wide = max_len > kChainNarrow;
  int hash_bits = chain_hash_bits(a.D, a.context, max_len);
  const auto set_bytes = [&] {
    return ((size_t)(1 << hash_bits) + chain_low_entries(a.D, a.context)) *
           (wide ? sizeof(unsigned long long) : sizeof(uint32_t));
  };
  const int64_t heads = (int64_t)a.plan.S * a.H;
  int segments = chain_segments(heads, max_len, set_bytes(), a.context);
  if (hash_bits == kChainHashBits && segments > 1 && segments < 8) {
    // half the buckets, if that doubles the pieces
    hash_bits = kChainHashBits - 1;
    const int more = chain_segments(heads, max_len, set_bytes(), a.context);
    if (more > segments) segments = more; else hash_bits = kChainHashBits;
  }
  if (merge && !a.low_is_zero)   // several shorter lengths merge their results into zeroed words
    ROSA_CUDA_OK(cudaMemsetAsync(a.chain_low, 0, (size_t)a.N * a.H * sizeof(uint32_t), stream));
  const size_t bytes = set_bytes() * segments;
  auto kernel = wide ? (merge ? chain_index_kernel<unsigned long long, true>
                              : chain_index_kernel<unsigned long long, false>)
                     : (merge ? chain_index_kernel<uint32_t, true> : chain_index_kernel<uint32_t, false>);
  if (bytes > 48 * 1024)
    ROSA_CUDA_OK(allow_shared(kernel));
  kernel<<<(unsigned)heads, 32 * a.context * segments, bytes, stream>>>(
      a.plan, a.packed_q, a.packed_k, a.sym_seq_stride, a.sym_head_stride, a.H, a.D, a.context,
      hash_bits, segments, a.chain_start, a.chain_prev, a.chain_low);
  ROSA_CUDA_OK(cudaGetLastError());
  return 0;
}

int launch_chain_forward(const FwdArgs& a, int64_t max_len, cudaStream_t stream) {
  const ChainPatience patience = chain_patience(a.D, a.context, max_len);
  return with_sign_emit(a, [&](auto emit) { return match_rows(a, patience, emit, stream); });
}

int launch_chain_inference(const FwdArgs& a, const float* payload, float* out, int64_t* matched_end,
                           int64_t max_len, cudaStream_t stream) {
  return match_rows(a, chain_patience(a.D, a.context, max_len),
                    make_payload_emit(a, payload, out, matched_end), stream);
}

int launch_pending_forward(const FwdArgs& a, const int32_t* run_flag, cudaStream_t stream) {
  return with_sign_emit(a, [&](auto emit) { return run_rows_of(a, run_flag, emit, stream); });
}

int launch_pending_inference(const FwdArgs& a, const float* payload, float* out, int64_t* matched_end,
                             const int32_t* run_flag, cudaStream_t stream) {
  return run_rows_of(a, run_flag, make_payload_emit(a, payload, out, matched_end), stream);
}

}  // namespace rosa
