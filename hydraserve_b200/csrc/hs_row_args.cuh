// What the row kernels are launched with, and how a row's result leaves them.
#pragma once

#include <cstddef>

#include "hs_common.cuh"
#include "hs_state.cuh"
#include "../../include/hs_sampler.h"

namespace hs {

enum SmallK {
  kSmallKList = 0,   // lists their candidates
  kSmallKOrder = 1,  // finishes them in token order like any other (samplers made for that alone)
  kSmallKLeave = 2,  // leaves them to the streaming kernel
};

struct RowKernelArgs {
  const void* logits;
  int dtype;
  long long row_stride;
  int vocab;
  int slice;            // elements per CTA slice (multiple of 8)
  const hs_row_params* params;
  hs_row_out* out;
  const float* noise;   // [batch, vocab] or null
  float* scores_out;    // [batch, vocab] or null
  float* gstage;        // [batch, slice * cluster] global stage, or null = shared memory
  Pool pool;            // token-count histograms
  uint32_t flags;
  int32_t* tokens_out;  // [batch] or null: the sampled ids once more, as the next step's input ids
  int small_k;          // what the resident kernel does with rows of a small top_k: SmallK
  int token_draw;       // bf16 counting rows draw near-flat rows by rejection on tokens (tuning / test switch)
};

// Parameters of a small batch travel in the launch itself (args.params is null then): no copy to
// wait for ahead of the kernel.  The block is part of every launch, used or not, so it ends at 64 rows:
// calls of 64 rows of 16,384 take 34.8 us with it and 36.0 with a copy, but with a block for 256 rows
// 36.9, those of 128 rows 40.9 (copied 40.2), and only 256 rows gain (49.7 against 50.3).
constexpr int kInlineRows = 64;
struct InlineRows {
  hs_row_params p[kInlineRows];
};
__device__ __forceinline__ hs_row_params row_params(const RowKernelArgs& a, const InlineRows& inl, int row) {
  return a.params ? a.params[row] : inl.p[row];
}

// A row's record is put together in shared memory (zero where nothing is to be said) and leaves in one
// piece (one warp): `out` may be pinned host memory, where every store is a transfer of its own.  When
// the host waits for the record itself (hs_step), its status goes last, behind everything else, and a
// row without log-probabilities leaves their place as it was.
constexpr uint32_t kHostWaits = 1u << 31;  // in RowKernelArgs.flags
constexpr int32_t kNoStatus = 0x7fffffff;  // what stands in the status until then
__device__ __forceinline__ void write_record(hs_row_out* out, const hs_row_out& rec, bool with_top, uint32_t flags) {
  static_assert(sizeof(hs_row_out) == 52 * 4 && offsetof(hs_row_out, top_ids) == 12 * 4, "words of a record");
  constexpr int kStatus = offsetof(hs_row_out, status) / 4;
  const bool last = flags & kHostWaits;
  const int n = with_top || !last ? 52 : 12;
  for (int i = threadIdx.x; i < n; i += 32)
    if (!last || i != kStatus) reinterpret_cast<uint32_t*>(out)[i] = reinterpret_cast<const uint32_t*>(&rec)[i];
  if (!last) return;
  __threadfence_system();
  __syncwarp();
  if (threadIdx.x == 0) *reinterpret_cast<volatile int32_t*>(&out->status) = rec.status;
}

constexpr int kTopKMax = 256;  // largest top_k served by the candidate paths

// Rows whose candidates (the top_k highest scores and the ties of the last) make a short list.
__host__ __device__ __forceinline__ bool is_candidate_row(const hs_row_params& P, int vocab) {
  return P.temperature != 0.0f && P.top_k > 0 && P.top_k <= kTopKMax && P.top_k < vocab;
}

struct KeptSet {
  uint32_t cut_key;  // kept: key > cut_key, or key == cut_key and global id <= tie_limit
  int tie_limit;
  __device__ __forceinline__ bool has(uint32_t k, int gid) const {
    return k > cut_key || (k == cut_key && gid <= tie_limit);
  }
};

}  // namespace hs
