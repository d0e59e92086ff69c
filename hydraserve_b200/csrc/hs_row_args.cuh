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
  hs_row_out* out;      // or null: the records go by mail alone
  const float* noise;   // [batch, vocab] or null
  float* scores_out;    // [batch, vocab] or null
  float* gstage;        // [batch, slice * cluster] global stage, or null = shared memory
  Pool pool;            // token-count histograms
  uint32_t flags;
  int32_t* tokens_out;  // [batch] or null: the sampled ids once more, as the next step's input ids
  int small_k;          // what the resident kernel does with rows of a small top_k: SmallK
  ulonglong2* mail;     // [batch, kMailPairs] in pinned host memory, where a host that waits looks for records, or null
  uint32_t mail_tag;    // this launch's
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
// piece (one warp): `out` may be pinned host memory, where every store is a transfer of its own.  A host
// that waits for the record itself (hs_step) finds it in the row's mail as well, sooner: there every word
// travels with the launch's tag in one 64-bit store, so the host sees for each word whether it has
// arrived, in whatever order they come, and no fence has to keep a last word behind the others.  Such a
// fence waits until the other stores have crossed the bus: it held a row's slot for 9.0 thousand cycles in
// a batch of 1,024 (1.2 thousand now), and calls of four fp32 rows took 49.7 us (46.6), of 32 81.5 (76.1), of one
// bf16 row 47.9 (46.9).  A row without log-probabilities leaves their place as it was then.
constexpr int kRecordWords = 52, kBareWords = 12;  // of a record; of one without log-probabilities
constexpr int kMailPairs = kRecordWords / 2;
__device__ __forceinline__ void write_record(hs_row_out* out, const hs_row_out& rec, bool with_top, ulonglong2* mail = nullptr,
                                             uint32_t tag = 0u) {
  static_assert(sizeof(hs_row_out) == kRecordWords * 4 && offsetof(hs_row_out, top_ids) == kBareWords * 4, "words of a record");
  const uint32_t* words = reinterpret_cast<const uint32_t*>(&rec);
  const int n = with_top || !mail ? kRecordWords : kBareWords, lane = threadIdx.x & 31;
  if (mail && lane < n / 2) {
    const u64 t = (u64)tag << 32;
    const u64 first = t | words[2 * lane], second = t | words[2 * lane + 1];
    asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(mail + lane), "l"(first), "l"(second) : "memory");
  }
  if (!out) return;
  for (int i = lane; i < n; i += 32) reinterpret_cast<uint32_t*>(out)[i] = words[i];
}
__device__ __forceinline__ hs_row_out* record_of(const RowKernelArgs& a, int row) { return a.out ? a.out + row : nullptr; }
__device__ __forceinline__ ulonglong2* mail_of(const RowKernelArgs& a, int row) {
  return a.mail ? a.mail + (size_t)row * kMailPairs : nullptr;
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
