// C ABI of the sampler (include/hs_sampler.h): handle management, launch planning and
// the host-buffer convenience call.  No torch types, no exceptions across the boundary.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <atomic>
#include <mutex>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "../../include/hs_sampler.h"
#include "hs_common.cuh"
#include "hs_pause.h"
#include "hs_state.cuh"
#include "hs_row_args.cuh"
#include "hs_row_v3.cuh"
#include "hs_row_topk.cuh"
#include "hs_sharded.cuh"
#include "hs_row_finish.cuh"
#include "hs_row_bf16_kernel.cuh"
#include "hs_row_f32_stream.cuh"
#include "hs_row_resident.cuh"

namespace {

using hs::u64;

constexpr int kMaxParts = 16;  // CTAs per counting row the hand-over can deal with
constexpr int kMaxSplit = 8;   // CTAs per candidate row: the parts' lists, top_k entries and ties each, meet in one list
constexpr int32_t kNoToken = -1;  // where a greedy step's id will stand
constexpr int kSideCapMax = 16384;  // side-list entries a CTA can keep in global scratch

struct DeviceGuard {
  int prev = -1;
  bool ok = true;
  explicit DeviceGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) { ok = false; return; }
    if (prev != dev && cudaSetDevice(dev) != cudaSuccess) ok = false;
  }
  ~DeviceGuard() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};

struct Plan {
  int cluster;
  int slice;
  size_t smem;
  bool global_stage;
};

inline size_t align16(size_t v) { return (v + 15) & ~size_t(15); }

// Shared memory of the resident kernel next to the slice: a candidate row's finisher takes the
// slice's place, so that never gets less than kResMerge bytes.
size_t fixed_smem(int cluster) {
  size_t off = align16(sizeof(hs::Exchange));
  off += sizeof(hs::Hist);
  off += (sizeof(u64) + sizeof(uint32_t)) * (hs::kBins / cluster);
  return align16(off);
}
size_t resident_smem(int cluster, int slice, bool global_stage) {
  const size_t stage = global_stage ? 0 : (size_t)slice * sizeof(float);
  return fixed_smem(cluster) + std::max(stage, (size_t)hs::kResMerge);
}

}  // namespace

struct hs_sampler {
  int device = 0;
  int vocab_max = 0, slots_user = 0, slots_total = 0, unique_cap = 0, batch_max = 0;
  int sm_count = 0;
  int smem_optin = 0;
  int force_cluster = 0;
  int force_general = 0;  // route bf16 rows through the general (fp32-stage) kernel too
  int force_split = 0;    // CTAs per candidate row (0 = chosen per call)
  int force_csplit = 0;   // CTAs per counting row (0 = chosen per call)
  int token_draw = 1;     // near-flat counting rows draw by rejection on tokens
  int ctab_tables = 0;    // parts of counting rows the hand-over scratch holds
  uint32_t* ctab = nullptr;   // [ctab_tables, kHandedCap]
  int2* crare = nullptr;      // [ctab_tables, kV3RareCap]
  int2* crare_n = nullptr;    // [ctab_tables]
  int split_tables = 0;   // parts of candidate rows
  int* count_ticket = nullptr;  // [batch_max]
  int resident_bf16 = 0;  // CTAs of the bf16 kernel that can be resident at once: CTAs per SM x SMs
  int2* side_pair = nullptr;  // [resident_bf16, side_cap] side lists too long for shared memory
  int* scratch_busy = nullptr;  // [resident_bf16] which of those scratch sets are in use
  unsigned long long* split_lists = nullptr;  // [split_tables, kSplitCap], a list per part
  int* split_n = nullptr;
  int* split_ticket = nullptr;
  int side_cap = 0;
  unsigned long long* phase_clocks = nullptr;  // HS_CREATE_PHASE_CLOCKS: per-row phase timestamps
  hs::Pool pool{};
  u64* greedy_best = nullptr;   // [batch_max] best element of a row so far (0 between calls)
  int* greedy_ticket = nullptr;  // [batch_max] its chunks that have arrived (0 between calls)
  float* gstage = nullptr;  // global stand-in for the on-chip row copy (very wide rows only)
  size_t gstage_elems = 0;
  // device + pinned staging for the host-buffer call
  void* d_logits = nullptr;
  size_t d_logits_bytes = 0;
  hs_row_params* d_params = nullptr;
  hs_row_out* d_out = nullptr;
  int32_t* d_hist = nullptr;
  size_t d_hist_elems = 0;
  int32_t* d_offsets = nullptr;
  int32_t* d_slots = nullptr;
  hs_row_params* h_params = nullptr;  // pinned
  int32_t* h_small = nullptr;         // pinned: offsets[batch_max+1] then slots[batch_max]
  // hs_step: the pinned block its caller fills, its copy on the device, and pinned results.  The first
  // blocks are part of h_held and d_held; larger ones, when a step needs them, are own allocations.
  unsigned char* h_block = nullptr;
  size_t h_block_bytes = 0;
  unsigned char* d_block = nullptr;
  size_t d_block_bytes = 0;
  void *h_block_own = nullptr, *d_block_own = nullptr;
  hs_row_out* h_out = nullptr;    // [batch_max]
  int32_t* h_tokens = nullptr;    // [batch_max]
  volatile u64* h_mail = nullptr;  // [batch_max, kRecordWords] a record's words as they arrive, each under its step's tag
  uint32_t mail_tag = 0;           // of the last hs_step
  std::vector<uint8_t> mail_words; // [batch_max] words of each row's record of that step
  std::vector<int> pending;        // [batch_max] rows hs_step_wait still looks for
  std::atomic<int> awaited_ids{0}, awaited_records{0};  // on their way into h_tokens and h_mail
  std::mutex mu;         // the staging buffers of hs_sample_host
  // Every launching call takes launch_mu, and work of one call is ordered after the previous
  // call's on the GPU (an event when the stream changed), because all calls share the
  // sampler's scratch memory and its histograms.
  std::mutex launch_mu;
  cudaEvent_t ev_done = nullptr;
  cudaStream_t last_stream = nullptr;
  bool have_last = false;
  void* h_held = nullptr;  // the one pinned allocation, likewise
  void* d_held = nullptr;  // the one allocation the arrays above live in (DeviceBlock)
  size_t device_bytes = 0;
  unsigned long long launches = 0;
};

namespace {

// The text of the calling thread's last failure (calls may come from several threads).
thread_local char g_last_error[512] = "";

int fail(hs_sampler*, int code, const char* what, cudaError_t e = cudaSuccess) {
  if (e != cudaSuccess)
    std::snprintf(g_last_error, sizeof g_last_error, "%s: %s", what, cudaGetErrorString(e));
  else
    std::snprintf(g_last_error, sizeof g_last_error, "%s", what);
  return code;
}

#define HS_CUDA(h, call)                                              \
  do {                                                                \
    cudaError_t e_ = (call);                                          \
    if (e_ != cudaSuccess) return fail((h), HS_ERR_CUDA, #call, e_);  \
  } while (0)

// Holds the sampler for one call's launches: calls on one sampler are serialised on the host
// (the mutex) and on the GPU (a call on another stream than the previous one first waits for
// that one's work), so they may come from any thread on any stream.
struct Serial {
  hs_sampler* h;
  cudaStream_t stream;
  std::unique_lock<std::mutex> lock;
  cudaError_t status = cudaSuccess;
  Serial(hs_sampler* h_, cudaStream_t s) : h(h_), stream(s), lock(h_->launch_mu) {
    if (h->have_last && h->last_stream != stream) status = cudaStreamWaitEvent(stream, h->ev_done, 0);
  }
  // records the end of this call's work; call once, after the last launch
  cudaError_t done() {
    const cudaError_t e = cudaEventRecord(h->ev_done, stream);
    if (e == cudaSuccess) { h->last_stream = stream; h->have_last = true; }
    return e;
  }
};

// What a sampler holds on the device from the start: ONE allocation (each takes the driver a
// round of mapping and a lock), what starts at zero in front, so that one memset clears it.
struct DeviceBlock {
  std::vector<std::pair<void**, size_t>> zeroed, others;
  template <class T>
  void add(T** p, size_t bytes, bool zero) {
    (zero ? zeroed : others).emplace_back(reinterpret_cast<void**>(p), (bytes + 255) & ~size_t(255));
  }
  bool allocate(hs_sampler* h) {
    size_t clear = 0, total = 0;
    for (auto& e : zeroed) clear += e.second;
    total = clear;
    for (auto& e : others) total += e.second;
    if (cudaMalloc(&h->d_held, total) != cudaSuccess) return false;
    h->device_bytes += total;
    unsigned char* at = static_cast<unsigned char*>(h->d_held);
    for (auto* list : {&zeroed, &others})
      for (auto& e : *list) { *e.first = at; at += e.second; }
    return cudaMemset(h->d_held, 0, clear) == cudaSuccess;
  }
};

// The resident kernel's geometry.  As many CTAs per row as leave each at least 4,096 tokens (below
// that a row's time is its barriers), eight at most (the portable cluster size): the row's passes
// over its slices are what takes time, and eight slices of up to about 19,000 tokens still sit two
// to an SM.  A batch that would run to more than four waves of two CTAs per SM gets fewer, larger
// slices (fewer merges per row), down to the smallest cluster whose shared memory holds the row.
bool make_plan(const hs_sampler* h, int vocab, int batch, Plan& p) {
  auto plan_of = [&](int c, bool global_stage) {
    const int slice = ((vocab + c - 1) / c + 7) & ~7;
    return Plan{c, slice, resident_smem(c, slice, global_stage), global_stage};
  };
  auto fits = [&](int c) {
    const Plan q = plan_of(c, false);
    return q.smem <= (size_t)h->smem_optin && q.slice <= hs::kMaxSliceElems;
  };
  if (h->force_cluster) {
    if (fits(h->force_cluster)) { p = plan_of(h->force_cluster, false); return true; }
  } else {
    int c = hs::kMaxCluster;
    while (c > 1 && vocab / c < 4096 && fits(c / 2)) c /= 2;
    while (c > 1 && (long long)batch * c > 8ll * h->sm_count && fits(c / 2)) c /= 2;
    if (fits(c)) { p = plan_of(c, false); return true; }
  }
  p = plan_of(hs::kMaxCluster, true);
  return p.slice <= hs::kMaxSliceElems;
}

int check_common(hs_sampler* h, const void* logits, int dtype, int batch, int vocab) {
  if (!h) return HS_ERR_INVALID;
  if (!logits && batch > 0) return fail(h, HS_ERR_INVALID, "logits is null");
  if (dtype != HS_DTYPE_F32 && dtype != HS_DTYPE_BF16) return fail(h, HS_ERR_INVALID, "unknown dtype");
  if (batch < 0 || vocab < 1) return fail(h, HS_ERR_INVALID, "batch must be >= 0 and vocab >= 1");
  if (vocab > h->vocab_max) return fail(h, HS_ERR_CAPACITY, "vocab exceeds vocab_max given to hs_create");
  if (batch > h->batch_max) return fail(h, HS_ERR_CAPACITY, "batch exceeds batch_max given to hs_create");
  return HS_OK;
}

// Launch attributes: `cluster` CTAs per cluster; `behind` = the kernel may get ready while the one
// launched before it on the stream is still running (it waits for that one's end by itself).
struct LaunchAttrs {
  cudaLaunchAttribute a[2];
  unsigned n = 0;
  LaunchAttrs(int cluster, bool behind) {
    if (cluster > 0) {
      a[n].id = cudaLaunchAttributeClusterDimension;
      a[n].val.clusterDim.x = (unsigned)cluster; a[n].val.clusterDim.y = 1; a[n].val.clusterDim.z = 1;
      ++n;
    }
    if (behind) {
      a[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      a[n].val.programmaticStreamSerializationAllowed = 1;
      ++n;
    }
  }
};
template <class... Params, class... Args>
cudaError_t launch(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, LaunchAttrs attrs,
                   Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attrs.a;
  cfg.numAttrs = attrs.n;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

int n_count_of(const hs_row_params* params, int batch, int vocab) {
  int n = 0;
  for (int r = 0; r < batch; ++r) n += hs::is_candidate_row(params[r], vocab) ? 0 : 1;
  return n;
}

const hs::InlineRows kNoInlineRows{};  // (stands in when the parameters are in device memory)

// `params` in device memory, or null with the rows' parameters in `inl`; n_count: how many rows are
// not candidate rows, or -1 when the host does not know; `behind`: the launch before
// this one on the stream is one of this sampler's histogram kernels.
int launch_rows(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
                const hs_row_params* params, const hs::InlineRows& inl, int n_count, hs_row_out* out, const float* noise,
                float* scores_out, int32_t* tokens_out, uint32_t flags, bool behind, cudaStream_t stream, bool mailed = false) {
  Plan plan;
  hs::RowKernelArgs a{};
  a.logits = logits; a.dtype = dtype; a.row_stride = row_stride; a.vocab = vocab; a.slice = 0;
  a.params = params; a.out = out; a.noise = noise; a.scores_out = scores_out; a.gstage = nullptr;
  a.pool = h->pool; a.flags = flags & HS_SAMPLE_APPEND_TOKEN; a.tokens_out = tokens_out;
  a.mail = mailed ? reinterpret_cast<ulonglong2*>(const_cast<u64*>(h->h_mail)) : nullptr;
  a.mail_tag = h->mail_tag;
  a.token_draw = h->token_draw;
  if (dtype == HS_DTYPE_BF16 && !h->force_general && !(flags & HS_SAMPLE_GENERAL_KERNEL)) {
    // One launch: the parts of the counting rows, then the parts of the candidate rows, two CTAs
    // resident per SM.  How many rows take which path is known when the parameters come from the
    // host (n_count >= 0).  Counting goes at the rate of an SM's shared atomics, so the rows are cut into as
    // many parts as give every SM one, eight at most and none below 32,768 tokens (one row of 248,320 in 1 / 2 /
    // 4 / 8 parts 58.2 / 54.5 / 51.1 / 50.5 us a call; whole or in four parts, one row and sixteen: of 98,304
    // 47.3 / 47.3 and 47.4 / 48.1, of 128,256 48.5 / 47.8 and 50.9 / 48.9, of 151,936 51.5 / 49.4 and 53.7 / 50.3).
    // Where that, or the hand-over scratch, makes less than four of them, the hand-over costs what the
    // shorter count saves (64 rows of 151,936 whole or in two: 58.3 / 61.8), unless so many candidate rows
    // share the SMs that whole counting rows wait for them and for each other: as many candidate rows as counting
    // ones and more CTAs than SMs, or a quarter as many and a third more CTAs than SMs (whole or in two, 64 among 96
    // rows 63.8 / 66.8, 80 among 100 63.6 / 67.9, but 64 among 128 70.8 / 69.4, 100 among 128 74.4 / 70.2), and rows of
    // 131,072 on (64 among 256, of 65,536 64.9 / 66.8, of 131,072 77.8 / 73.5, of 248,320 100.8 / 87.4).
    // Candidate rows get what the wave has left, up to eight CTAs each (a second, partial wave costs more
    // than idle SMs in the first), none below 16,384 tokens, its bound's sample.
    // When the host does not know, every row may be either: four parts as far as the hand-over
    // scratch goes, else whole rows (256 rows of 248,320, half of them counting: 61.9 us a step, 66.0 in two
    // parts), and a wave of candidate parts.
    const int resident = h->resident_bf16;
    const bool known = n_count >= 0;
    int csplit, split;
    if (known) {
      const int n_cand = batch - n_count;
      const int most = h->ctab_tables / batch;
      csplit = std::min({h->sm_count / std::max(1, n_count), 8, vocab / 32768, most});
      if (csplit < 4) {
        const int halves = 2 * n_count + n_cand;  // CTAs, the counting rows in two
        const bool mixed = 2 * n_count <= resident && ((n_cand >= n_count && halves > h->sm_count) ||
                                                       (4 * n_cand >= n_count && 3 * halves >= 4 * h->sm_count));
        csplit = mixed && vocab >= 131072 ? std::max(1, std::min(std::max(csplit, 2), most)) : 1;
      }
      split = (resident - std::min(resident, n_count * csplit)) / std::max(1, n_cand);
      split = std::max(1, std::min({split, kMaxSplit, vocab / hs::kSample}));
    } else {
      csplit = vocab < 65536 || (long long)batch * 4 > h->ctab_tables ? 1 : 4;
      split = std::max(1, std::min({resident / batch, 4, vocab / (2 * hs::kSample)}));
    }
    if (h->force_csplit) csplit = h->force_csplit;
    if (h->force_split) split = vocab < h->force_split * 2 * hs::kSample ? 1 : h->force_split;
    csplit = std::max(1, std::min(csplit, h->ctab_tables / batch));
    split = std::max(1, std::min(split, h->split_tables / batch));
    hs::RowV3Args a3{a, h->side_pair, h->side_cap, h->resident_bf16, h->scratch_busy, h->phase_clocks,
                     csplit, h->ctab, h->crare, h->crare_n, h->count_ticket,
                     split, h->split_lists, h->split_n, h->split_ticket, batch};
    const unsigned grid = (unsigned)batch * (unsigned)(csplit + split);
    HS_CUDA(h, launch(hs::row_kernel_bf16, dim3(grid), hs::kThreads, hs::bf16_kernel_smem(), stream, LaunchAttrs(0, behind), a3, inl));
    h->launches += 1;
    return HS_OK;
  }
  if (!make_plan(h, vocab, batch, plan)) return fail(h, HS_ERR_CAPACITY, "vocabulary too wide for the row kernel");
  // A row with a small top_k is drawn from its sorted list wherever it is sampled, so a row that another
  // kernel gave up (HS_SAMPLE_GENERAL_KERNEL) is listed here too: which token a seed names must not
  // depend on the kernel, which depends on the batch around the row.
  a.small_k = h->force_general ? hs::kSmallKOrder : hs::kSmallKList;
  // fp32 rows with a small top_k: as clusters while these are at most two waves of two CTAs per SM, one
  // CTA each in the streaming kernel beyond that (a row takes longer there, but 296 of them run side by
  // side: 64 rows are two waves less a little and 55 us here, 61 there; 75 would be a third, 70 against
  // 62).  Such a batch is too large for inline parameters.
  const bool may_stream = dtype == HS_DTYPE_F32 && !h->force_general && !(flags & HS_SAMPLE_GENERAL_KERNEL);
  if (may_stream && params && n_count != batch && (long long)batch * plan.cluster > 4ll * h->sm_count) {
    a.small_k = hs::kSmallKLeave;
    HS_CUDA(h, launch(hs::row_kernel_f32_stream, dim3((unsigned)batch), hs::kThreads, hs::layout_cand().total, stream,
                      LaunchAttrs(0, false), a));
    h->launches += 1;
    if (n_count == 0) return HS_OK;
    behind = false;  // (the launch before the resident kernel is not a histogram kernel any more)
  }
  if (plan.global_stage) {
    const size_t need = (size_t)batch * plan.slice * plan.cluster;
    if (need > h->gstage_elems) return fail(h, HS_ERR_CAPACITY, "global stage too small for this batch x vocab");
  }
  a.slice = plan.slice;
  a.gstage = plan.global_stage ? h->gstage : nullptr;

  HS_CUDA(h, launch(plan.global_stage ? hs::row_kernel<false> : hs::row_kernel<true>, dim3((unsigned)plan.cluster, (unsigned)batch), hs::kThreads, plan.smem, stream,
                    LaunchAttrs(plan.cluster, behind), a, inl));
  h->launches += 1;
  return HS_OK;
}

int launch_greedy(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
                  int32_t* tokens_out, cudaStream_t stream) {
  // enough CTAs to fill the SMs four times over (eight fit, but a shorter chunk than one load per
  // thread gains nothing)
  int chunks = (4 * h->sm_count + batch - 1) / batch;
  const int per = hs::kGreedyThreads * (dtype == HS_DTYPE_BF16 ? 8 : 4);
  chunks = std::max(1, std::min(chunks, (vocab + per - 1) / per));
  int chunk = ((vocab + chunks - 1) / chunks + 7) & ~7;
  chunks = (vocab + chunk - 1) / chunk;
  hs::greedy_kernel<<<dim3((unsigned)chunks, (unsigned)batch), hs::kGreedyThreads, 0, stream>>>(
      logits, dtype, row_stride, vocab, chunk, h->greedy_best, h->greedy_ticket, tokens_out);
  HS_CUDA(h, cudaGetLastError());
  h->launches += 1;
  return HS_OK;
}

int launch_append(hs_sampler* h, const int32_t* tokens, const int32_t* offsets, const int32_t* slots,
                  int n_slots, int vocab, int max_tokens, cudaStream_t stream) {
  if (n_slots == 0 || max_tokens <= 0) return HS_OK;
  const int threads = 256;
  int bx = std::max(1, std::min((max_tokens + threads - 1) / threads, 64));
  dim3 grid((unsigned)bx, (unsigned)n_slots);
  hs::slots_register_kernel<<<grid, threads, 0, stream>>>(h->pool, tokens, offsets, slots, n_slots, vocab);
  HS_CUDA(h, cudaGetLastError());
  hs::slots_count_kernel<<<grid, threads, 0, stream>>>(h->pool, tokens, offsets, slots, n_slots, vocab);
  HS_CUDA(h, cudaGetLastError());
  hs::slots_classify_kernel<<<grid, threads, 0, stream>>>(h->pool, tokens, offsets, slots, n_slots, vocab);
  HS_CUDA(h, cudaGetLastError());
  h->launches += 3;
  return HS_OK;
}

// hs_step_wait is for the step before it: what an earlier step left, whose caller waited for the stream
// instead, counts no more.
void nothing_awaited(hs_sampler* h) { h->awaited_ids = h->awaited_records = 0; }

void release(hs_sampler* h) {
  cudaFree(h->d_held); cudaFree(h->d_block_own); cudaFree(h->d_logits); cudaFree(h->d_hist);
  if (h->ev_done) cudaEventDestroy(h->ev_done);
  if (h->h_held) cudaFreeHost(h->h_held);
  if (h->h_block_own) cudaFreeHost(h->h_block_own);
}

}  // namespace

// ---- hs_greedy_noalloc: arg max per row with its scratch in a fixed device array --------
namespace {

constexpr int kNoAllocMaxBatch = HS_NOALLOC_MAX_BATCH;
constexpr int kNoAllocChunks = 16;
constexpr int kNoAllocMaxDevices = 64;

// One partial result per (row, chunk).  Every GPU that loads this library holds these
// 128 KB until the process exits.  In host code this name is only a handle for
// cudaGetSymbolAddress; kernels get the device address obtained from it.
static __device__ __align__(256) unsigned long long g_noalloc_partials[kNoAllocMaxBatch * kNoAllocChunks];

struct NoAllocDevice {
  u64* partials = nullptr;  // device address of g_noalloc_partials on that GPU
  bool ready = false;
};
NoAllocDevice g_noalloc_devices[kNoAllocMaxDevices];
std::mutex g_noalloc_mu;
thread_local char g_noalloc_error[256] = "";

int noalloc_fail(int code, const char* what, cudaError_t e = cudaSuccess) {
  if (e != cudaSuccess)
    std::snprintf(g_noalloc_error, sizeof g_noalloc_error, "%s: %s", what, cudaGetErrorString(e));
  else
    std::snprintf(g_noalloc_error, sizeof g_noalloc_error, "%s", what);
  return code;
}

}  // namespace

extern "C" {

const char* hs_greedy_noalloc_error(void) { return g_noalloc_error; }

int hs_greedy_noalloc(const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
                      int32_t* tokens_out, void* stream_) {
  g_noalloc_error[0] = 0;
  if (dtype != HS_DTYPE_F32 && dtype != HS_DTYPE_BF16) return noalloc_fail(HS_ERR_INVALID, "unknown dtype");
  if (batch < 0 || vocab < 1) return noalloc_fail(HS_ERR_INVALID, "batch must be >= 0 and vocab >= 1");
  if (batch > kNoAllocMaxBatch) {
    std::snprintf(g_noalloc_error, sizeof g_noalloc_error,
                  "batch %d exceeds HS_NOALLOC_MAX_BATCH (%d): split the call", batch, kNoAllocMaxBatch);
    return HS_ERR_CAPACITY;
  }
  if (batch == 0) return HS_OK;
  if (!logits || !tokens_out) return noalloc_fail(HS_ERR_INVALID, "logits / tokens_out is null");
  if (row_stride < vocab) return noalloc_fail(HS_ERR_INVALID, "row_stride smaller than vocab");
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return noalloc_fail(HS_ERR_CUDA, "cudaGetDevice", e);
  if (dev < 0 || dev >= kNoAllocMaxDevices) return noalloc_fail(HS_ERR_CAPACITY, "device index beyond 63");
  u64* partials = nullptr;
  {
    // Set-up, once per device, with that device current: resolve the array's device address.
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    NoAllocDevice& d = g_noalloc_devices[dev];
    if (!d.ready) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_noalloc_partials);
      if (e != cudaSuccess) return noalloc_fail(HS_ERR_CUDA, "cudaGetSymbolAddress(g_noalloc_partials)", e);
      d.partials = static_cast<u64*>(p);
      d.ready = true;
    }
    partials = d.partials;
  }
  cudaStream_t stream = (cudaStream_t)stream_;
  int chunks = kNoAllocChunks;
  int chunk = ((vocab + chunks - 1) / chunks + 7) & ~7;
  chunks = (vocab + chunk - 1) / chunk;
  // Every (row, chunk) slot that the final kernel reads is written by the partial kernel of
  // the same call, so nothing left over from an earlier call needs clearing.
  hs::greedy_partial_kernel<<<dim3((unsigned)chunks, (unsigned)batch), hs::kGreedyThreads, 0, stream>>>(
      logits, dtype, row_stride, vocab, chunk, partials);
  e = cudaGetLastError();
  if (e != cudaSuccess) return noalloc_fail(HS_ERR_CUDA, "greedy_partial_kernel launch", e);
  hs::greedy_final_kernel<<<(batch + 127) / 128, 128, 0, stream>>>(partials, chunks, batch, tokens_out);
  e = cudaGetLastError();
  if (e != cudaSuccess) return noalloc_fail(HS_ERR_CUDA, "greedy_final_kernel launch", e);
  return HS_OK;
}

int hs_abi_version(void) { return 1; }

const char* hs_status_string(int status) {
  switch (status) {
    case HS_OK: return "ok";
    case HS_ERR_INVALID: return "invalid argument";
    case HS_ERR_CAPACITY: return "capacity exceeded";
    case HS_ERR_CUDA: return "CUDA error";
    case HS_ERR_UNSUPPORTED: return "unsupported";
    default: return "unknown status";
  }
}

const char* hs_last_error(hs_sampler* h) { return h ? g_last_error : "null sampler"; }

int hs_create(int device, int vocab_max, int slots_max, int unique_cap, int batch_max, hs_sampler** out) {
  return hs_create_ex(device, vocab_max, slots_max, unique_cap, batch_max, 0u, out);
}

int hs_create_ex(int device, int vocab_max, int slots_max, int hist_cap, int batch_max, uint32_t flags,
                 hs_sampler** out) {
  if (!out) return HS_ERR_INVALID;
  *out = nullptr;
  if (vocab_max < 1 || slots_max < 0 || batch_max < 1 || hist_cap < 0) return HS_ERR_INVALID;
  if (batch_max > 65535) return HS_ERR_CAPACITY;
  hs_sampler* h = new (std::nothrow) hs_sampler();
  if (!h) return HS_ERR_INVALID;
  DeviceGuard guard(device);
  if (!guard.ok) { delete h; return HS_ERR_CUDA; }
  h->device = device;
  h->vocab_max = vocab_max;
  h->slots_user = slots_max;
  h->slots_total = slots_max + batch_max;  // the tail serves per-call (stateless) histories
  h->unique_cap = hist_cap == 0 ? vocab_max : std::min(hist_cap, vocab_max);
  h->batch_max = batch_max;
  h->force_general = (flags & HS_CREATE_FORCE_GENERAL) ? 1 : 0;
  {
    const int v = (int)((flags >> 8) & 0xfu);
    if (v == 1 || v == 2 || v == 4 || v == 8) h->force_cluster = v;
  }
  auto bail = [&](int code) { release(h); delete h; return code; };
  if (cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return bail(HS_ERR_CUDA);
  if (cudaDeviceGetAttribute(&h->smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) return bail(HS_ERR_CUDA);
  h->smem_optin -= 1024;  // (the kernels' static shared memory)
  if (cudaFuncSetAttribute(hs::row_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, h->smem_optin) != cudaSuccess) return bail(HS_ERR_CUDA);
  if (cudaFuncSetAttribute(hs::row_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, h->smem_optin) != cudaSuccess) return bail(HS_ERR_CUDA);
  if (cudaFuncSetAttribute(hs::row_kernel_bf16, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hs::bf16_kernel_smem()) != cudaSuccess) return bail(HS_ERR_CUDA);
  if (cudaFuncSetAttribute(hs::row_kernel_f32_stream, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hs::layout_cand().total) != cudaSuccess) return bail(HS_ERR_CUDA);
  if (cudaFuncSetAttribute(hs::shard_partial_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hs::layout_cand().total) != cudaSuccess) return bail(HS_ERR_CUDA);
  if (cudaFuncSetAttribute(hs::shard_merge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hs::layout_cand().total) != cudaSuccess) return bail(HS_ERR_CUDA);
  {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, hs::row_kernel_bf16, hs::kThreads,
                                                      hs::bf16_kernel_smem()) != cudaSuccess || per_sm < 1)
      return bail(HS_ERR_CUDA);
    h->resident_bf16 = per_sm * h->sm_count;
  }

  const size_t st = (size_t)h->slots_total;
  h->pool.slots_total = h->slots_total;
  h->pool.unique_cap = h->unique_cap;
  h->pool.pos_stride = vocab_max;
  h->pool.cls_stride = (vocab_max + 15) / 16 + 4;  // words; padded so 128-bit reads of the tail stay inside
  DeviceBlock held;
  held.add(&h->pool.pairs, st * h->unique_cap * sizeof(int2), false);
  held.add(&h->pool.n, st * sizeof(int32_t), true);
  held.add(&h->pool.n_heavy, st * sizeof(int32_t), true);
  held.add(&h->pool.heavy, st * h->unique_cap * sizeof(int32_t), false);
  held.add(&h->pool.cls, st * (size_t)h->pool.cls_stride * sizeof(uint32_t), true);
  held.add(&h->pool.pos, st * (size_t)vocab_max * sizeof(int32_t), true);
  held.add(&h->pool.error, sizeof(int32_t), true);
  held.add(&h->greedy_best, (size_t)batch_max * sizeof(u64), true);
  held.add(&h->greedy_ticket, (size_t)batch_max * sizeof(int), true);
  held.add(&h->d_params, (size_t)batch_max * sizeof(hs_row_params), false);
  held.add(&h->d_out, (size_t)batch_max * sizeof(hs_row_out), false);
  held.add(&h->d_offsets, ((size_t)batch_max + 1) * sizeof(int32_t), false);
  held.add(&h->d_slots, (size_t)batch_max * sizeof(int32_t), false);
  // scratch of the bf16 kernel, per resident CTA (not per row of the batch)
  h->side_cap = std::min((vocab_max + 7) & ~7, kSideCapMax);
  held.add(&h->side_pair, (size_t)h->resident_bf16 * h->side_cap * sizeof(int2), false);
  held.add(&h->scratch_busy, (size_t)h->resident_bf16 * sizeof(int), true);
  // hand-over scratch of rows split over several CTAs: two parts per resident CTA
  h->ctab_tables = 2 * h->resident_bf16;
  h->split_tables = std::max(2 * h->resident_bf16, 2 * batch_max);
  held.add(&h->ctab, (size_t)h->ctab_tables * hs::kHandedCap * sizeof(uint32_t), false);
  held.add(&h->crare, (size_t)h->ctab_tables * hs::kV3RareCap * sizeof(int2), false);
  held.add(&h->crare_n, (size_t)h->ctab_tables * sizeof(int2), false);
  held.add(&h->count_ticket, (size_t)batch_max * sizeof(int), true);
  held.add(&h->split_lists, (size_t)h->split_tables * hs::kSplitCap * sizeof(unsigned long long), false);
  held.add(&h->split_n, (size_t)h->split_tables * sizeof(int), false);
  held.add(&h->split_ticket, (size_t)batch_max * sizeof(int), true);
  if (flags & HS_CREATE_PHASE_CLOCKS)
    held.add(&h->phase_clocks, (size_t)batch_max * hs::kV3PhaseSlots * sizeof(unsigned long long), true);
  Plan plan;
  if (!make_plan(h, vocab_max, batch_max, plan)) return bail(HS_ERR_CAPACITY);
  if (plan.global_stage) {
    h->gstage_elems = (size_t)batch_max * plan.slice * plan.cluster;
    held.add(&h->gstage, h->gstage_elems * sizeof(float), false);
  }
  // a step of every row with a new token or two, or a quarter of a million history tokens: growing a
  // block costs a step 0.2 ms and more
  const size_t first_block = (size_t)batch_max * (sizeof(hs_row_params) + 32) + (1 << 20);
  held.add(&h->d_block, first_block, false);
  bool ok = held.allocate(h);
  ok = ok && cudaEventCreateWithFlags(&h->ev_done, cudaEventDisableTiming) == cudaSuccess;
  if (ok) {
    const size_t mail_bytes = (size_t)batch_max * hs::kRecordWords * sizeof(u64);
    const size_t sizes[6] = {(size_t)batch_max * sizeof(hs_row_params), (2 * (size_t)batch_max + 1) * sizeof(int32_t),
                             (size_t)batch_max * sizeof(hs_row_out), (size_t)batch_max * sizeof(int32_t), mail_bytes, first_block};
    size_t at[7] = {0};
    for (int i = 0; i < 6; ++i) at[i + 1] = (at[i] + sizes[i] + 255) & ~size_t(255);
    ok = cudaMallocHost(&h->h_held, at[6]) == cudaSuccess;
    if (ok) {
      unsigned char* base = static_cast<unsigned char*>(h->h_held);
      h->h_params = reinterpret_cast<hs_row_params*>(base);
      h->h_small = reinterpret_cast<int32_t*>(base + at[1]);
      h->h_out = reinterpret_cast<hs_row_out*>(base + at[2]);
      h->h_tokens = reinterpret_cast<int32_t*>(base + at[3]);
      h->h_mail = reinterpret_cast<u64*>(base + at[4]);
      std::memset(base + at[4], 0, mail_bytes);
      h->mail_words.assign((size_t)batch_max, 0);
      h->pending.assign((size_t)batch_max, 0);
      h->h_block = base + at[5];
      h->h_block_bytes = h->d_block_bytes = first_block;
    }
  }
  if (!ok) return bail(HS_ERR_CUDA);
  if (cudaDeviceSynchronize() != cudaSuccess) return bail(HS_ERR_CUDA);
  *out = h;
  return HS_OK;
}

int hs_destroy(hs_sampler* h) {
  if (!h) return HS_ERR_INVALID;
  {
    DeviceGuard guard(h->device);
    cudaDeviceSynchronize();
    release(h);
  }
  delete h;
  return HS_OK;
}

int hs_slots_reset(hs_sampler* h, const int32_t* slots, int n_slots, void* stream) {
  if (!h || n_slots < 0 || (!slots && n_slots)) return HS_ERR_INVALID;
  if (n_slots == 0) return HS_OK;
  DeviceGuard guard(h->device);
  Serial serial(h, (cudaStream_t)stream);
  HS_CUDA(h, serial.status);
  hs::slots_reset_kernel<<<n_slots, 256, 0, (cudaStream_t)stream>>>(h->pool, slots, n_slots);
  HS_CUDA(h, cudaGetLastError());
  h->launches += 1;
  HS_CUDA(h, serial.done());
  return HS_OK;
}

int hs_slots_append(hs_sampler* h, const int32_t* tokens, const int32_t* offsets, const int32_t* slots,
                    int n_slots, int vocab, int max_tokens_per_slot, void* stream) {
  if (!h || n_slots < 0 || (n_slots && (!offsets || !slots))) return HS_ERR_INVALID;
  if (vocab < 1 || vocab > h->vocab_max) return fail(h, HS_ERR_CAPACITY, "vocab exceeds vocab_max");
  if (n_slots > 65535) return fail(h, HS_ERR_CAPACITY, "too many slots in one call");
  DeviceGuard guard(h->device);
  Serial serial(h, (cudaStream_t)stream);
  HS_CUDA(h, serial.status);
  const int rc = launch_append(h, tokens, offsets, slots, n_slots, vocab, max_tokens_per_slot, (cudaStream_t)stream);
  if (rc != HS_OK) return rc;
  HS_CUDA(h, serial.done());
  return HS_OK;
}

int hs_slot_unique_count(hs_sampler* h, int slot, void* stream, int* out) {
  if (!h || !out || slot < 0 || slot >= h->slots_total) return HS_ERR_INVALID;
  DeviceGuard guard(h->device);
  Serial serial(h, (cudaStream_t)stream);
  HS_CUDA(h, serial.status);
  int32_t v = 0;
  HS_CUDA(h, cudaMemcpyAsync(&v, h->pool.n + slot, sizeof v, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  HS_CUDA(h, cudaStreamSynchronize((cudaStream_t)stream));
  *out = v;
  return HS_OK;
}

int hs_sample(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
              const hs_row_params* params, hs_row_out* out, const float* noise, float* scores_out,
              uint32_t flags, void* stream) {
  return hs_sample_ex(h, logits, dtype, row_stride, batch, vocab, params, out, noise, scores_out, nullptr,
                      flags, stream);
}

int hs_sample_ex(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
                 const hs_row_params* params, hs_row_out* out, const float* noise, float* scores_out,
                 int32_t* tokens_out, uint32_t flags, void* stream) {
  int rc = check_common(h, logits, dtype, batch, vocab);
  if (rc != HS_OK) return rc;
  if (batch == 0) return HS_OK;
  if (!params || !out) return fail(h, HS_ERR_INVALID, "params / out is null");
  if (row_stride < vocab) return fail(h, HS_ERR_INVALID, "row_stride smaller than vocab");
  DeviceGuard guard(h->device);
  Serial serial(h, (cudaStream_t)stream);
  HS_CUDA(h, serial.status);
  rc = launch_rows(h, logits, dtype, row_stride, batch, vocab, params, kNoInlineRows, -1, out, noise, scores_out,
                   tokens_out, flags, false, (cudaStream_t)stream);
  if (rc != HS_OK) return rc;
  HS_CUDA(h, serial.done());
  return HS_OK;
}

int hs_greedy(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
              int32_t* tokens_out, void* stream) {
  int rc = check_common(h, logits, dtype, batch, vocab);
  if (rc != HS_OK) return rc;
  if (batch == 0) return HS_OK;
  if (!tokens_out) return fail(h, HS_ERR_INVALID, "tokens_out is null");
  if (row_stride < vocab) return fail(h, HS_ERR_INVALID, "row_stride smaller than vocab");
  DeviceGuard guard(h->device);
  Serial serial(h, (cudaStream_t)stream);
  HS_CUDA(h, serial.status);
  rc = launch_greedy(h, logits, dtype, row_stride, batch, vocab, tokens_out, (cudaStream_t)stream);
  if (rc != HS_OK) return rc;
  HS_CUDA(h, serial.done());
  return HS_OK;
}

int hs_sample_host(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
                   hs_row_params* params, hs_row_out* out, const int32_t* hist_tokens,
                   const int32_t* hist_offsets, uint32_t flags, void* stream_) {
  int rc = check_common(h, logits, dtype, batch, vocab);
  if (rc != HS_OK) return rc;
  if (batch == 0) return HS_OK;
  if (!params || !out) return fail(h, HS_ERR_INVALID, "params / out is null");
  if (row_stride < vocab) return fail(h, HS_ERR_INVALID, "row_stride smaller than vocab");
  cudaStream_t stream = (cudaStream_t)stream_;
  std::lock_guard<std::mutex> lock(h->mu);  // one user of the staging buffers at a time
  DeviceGuard guard(h->device);
  Serial serial(h, stream);
  HS_CUDA(h, serial.status);

  const size_t esz = dtype == HS_DTYPE_BF16 ? 2 : 4;
  const size_t need = (size_t)batch * vocab * esz;
  if (need > h->d_logits_bytes) {
    HS_CUDA(h, cudaStreamSynchronize(stream));
    cudaFree(h->d_logits);
    h->d_logits = nullptr;
    h->d_logits_bytes = 0;
    HS_CUDA(h, cudaMalloc(&h->d_logits, need));
    h->d_logits_bytes = need;
  }
  HS_CUDA(h, cudaMemcpy2DAsync(h->d_logits, (size_t)vocab * esz, logits, (size_t)row_stride * esz,
                               (size_t)vocab * esz, (size_t)batch, cudaMemcpyHostToDevice, stream));

  // Rows marked slot == -2 are penalised with the history passed in this call: it is
  // counted into a per-row scratch slot on the device (the reference's stateless form).
  int32_t* h_offsets = h->h_small;
  int32_t* h_slots = h->h_small + (h->batch_max + 1);
  int n_temp = 0;
  int max_len = 0;
  long long total = 0;
  for (int r = 0; r < batch; ++r) {
    h->h_params[r] = params[r];
    if (params[r].slot == -2) {
      if (!hist_tokens || !hist_offsets) return fail(h, HS_ERR_INVALID, "slot -2 needs hist_tokens / hist_offsets");
      const int len = hist_offsets[r + 1] - hist_offsets[r];
      if (len < 0) return fail(h, HS_ERR_INVALID, "hist_offsets must not decrease");
      h_slots[n_temp] = h->slots_user + r;
      h->h_params[r].slot = h->slots_user + r;
      ++n_temp;
      max_len = std::max(max_len, len);
      total += len;
    } else if (params[r].slot >= h->slots_user || params[r].slot < -2) {
      return fail(h, HS_ERR_INVALID, "params.slot out of range");
    }
  }
  if (n_temp) {
    if ((size_t)total > h->d_hist_elems) {
      HS_CUDA(h, cudaStreamSynchronize(stream));
      cudaFree(h->d_hist);
      h->d_hist = nullptr;
      h->d_hist_elems = 0;
      HS_CUDA(h, cudaMalloc(&h->d_hist, (size_t)total * sizeof(int32_t)));
      h->d_hist_elems = (size_t)total;
    }
    // The append kernels index offsets by position in `slots`, so the participants'
    // tokens are packed back to back.
    long long cursor = 0;
    std::vector<int32_t> packed;
    packed.reserve((size_t)total);
    int idx = 0;
    for (int r = 0; r < batch; ++r) {
      if (params[r].slot != -2) continue;
      h_offsets[idx++] = (int32_t)cursor;
      const int b = hist_offsets[r], e = hist_offsets[r + 1];
      packed.insert(packed.end(), hist_tokens + b, hist_tokens + e);
      cursor += e - b;
    }
    h_offsets[idx] = (int32_t)cursor;
    if (cursor) HS_CUDA(h, cudaMemcpyAsync(h->d_hist, packed.data(), (size_t)cursor * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
    HS_CUDA(h, cudaMemcpyAsync(h->d_offsets, h_offsets, ((size_t)n_temp + 1) * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
    HS_CUDA(h, cudaMemcpyAsync(h->d_slots, h_slots, (size_t)n_temp * sizeof(int32_t), cudaMemcpyHostToDevice, stream));
    if (cursor) HS_CUDA(h, cudaStreamSynchronize(stream));  // `packed` is pageable and about to go away
    hs::slots_reset_kernel<<<n_temp, 256, 0, stream>>>(h->pool, h->d_slots, n_temp);
    HS_CUDA(h, cudaGetLastError());
    h->launches += 1;
    rc = launch_append(h, h->d_hist, h->d_offsets, h->d_slots, n_temp, vocab, max_len, stream);
    if (rc != HS_OK) return rc;
  }
  HS_CUDA(h, cudaMemcpyAsync(h->d_params, h->h_params, (size_t)batch * sizeof(hs_row_params), cudaMemcpyHostToDevice, stream));
  rc = launch_rows(h, h->d_logits, dtype, vocab, batch, vocab, h->d_params, kNoInlineRows, n_count_of(h->h_params, batch, vocab), h->d_out, nullptr, nullptr,
                   nullptr, flags, false, stream);
  if (rc != HS_OK) return rc;
  HS_CUDA(h, cudaMemcpyAsync(out, h->d_out, (size_t)batch * sizeof(hs_row_out), cudaMemcpyDeviceToHost, stream));
  HS_CUDA(h, serial.done());
  HS_CUDA(h, cudaStreamSynchronize(stream));
  return HS_OK;
}

int hs_step_block(hs_sampler* h, size_t bytes, void** block) {
  if (!h || !block) return HS_ERR_INVALID;
  *block = nullptr;
  if (bytes > h->h_block_bytes) {
    DeviceGuard guard(h->device);
    const size_t want = std::max<size_t>(2 * bytes, 64 << 10);
    if (h->h_block_own) cudaFreeHost(h->h_block_own);
    h->h_block_own = nullptr;
    h->h_block = nullptr;
    h->h_block_bytes = 0;
    HS_CUDA(h, cudaMallocHost(&h->h_block_own, want));
    h->h_block = static_cast<unsigned char*>(h->h_block_own);
    h->h_block_bytes = want;
  }
  *block = h->h_block;
  return HS_OK;
}

namespace {

// (awaited: the caller is going to call hs_step_wait, so the records go by mail alone)
int step(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
         const hs_step_desc* d, const hs_row_out** out, bool awaited, void* stream_) {
  int rc = check_common(h, logits, dtype, batch, vocab);
  if (rc != HS_OK) return rc;
  if (!d || !out) return fail(h, HS_ERR_INVALID, "desc / out is null");
  *out = nullptr;
  nothing_awaited(h);
  const bool repeats = d->repeats != 0;
  if (batch == 0) return HS_OK;
  if (row_stride < vocab) return fail(h, HS_ERR_INVALID, "row_stride smaller than vocab");
  if (d->n_resets < 0 || d->n_appends < 0 || d->n_appends > 65535 || d->n_resets > 65535)
    return fail(h, HS_ERR_CAPACITY, "too many slots in one call");
  if (d->bytes > h->h_block_bytes || d->bytes < (size_t)batch * sizeof(hs_row_params) ||
      d->resets_at + (size_t)d->n_resets * 4 > d->bytes || d->slots_at + (size_t)d->n_appends * 4 > d->bytes ||
      (d->n_appends && d->offsets_at + ((size_t)d->n_appends + 1) * 4 > d->bytes) || d->tokens_at > d->bytes)
    return fail(h, HS_ERR_INVALID, "the step's description does not fit its block");
  cudaStream_t stream = (cudaStream_t)stream_;
  DeviceGuard guard(h->device);
  Serial serial(h, stream);
  HS_CUDA(h, serial.status);

  *out = h->h_out;
  if (++h->mail_tag == 0) {
    // (around once: no word may still stand under a tag that comes again)
    HS_CUDA(h, cudaStreamSynchronize(stream));
    std::memset(const_cast<u64*>(h->h_mail), 0, (size_t)h->batch_max * hs::kRecordWords * sizeof(u64));
    h->mail_tag = 1;
  }

  // What a small step brings along goes into the launches themselves: 64 rows' parameters (3 KB)
  // and 256 (slot, token) pairs (2 KB) are cheaper there than one copy ahead of the kernel
  // (about 3 us of host and GPU time); anything larger is copied in one piece.
  const auto* params = reinterpret_cast<const hs_row_params*>(h->h_block);
  for (int r = 0; r < batch; ++r) h->mail_words[(size_t)r] = (uint8_t)(params[r].n_logprobs >= 0 ? hs::kRecordWords : hs::kBareWords);
  const bool counting = d->n_resets > 0 || d->n_appends > 0;
  const bool singles = d->n_resets == 0 && d->n_appends > 0 && d->max_tokens == 1 && !repeats;
  // a slot that is emptied and then filled again is one entry of the build (the two lists are in
  // the same order); what is only emptied stays in the list of resets
  int n_alone = 0;
  if (d->n_resets) {
    auto* resets = reinterpret_cast<int32_t*>(h->h_block + d->resets_at);
    auto* slots = reinterpret_cast<int32_t*>(h->h_block + d->slots_at);
    int j = 0;
    for (int i = 0; i < d->n_resets; ++i) {
      int k = j;
      while (!repeats && k < d->n_appends && slots[k] != resets[i]) ++k;
      if (!repeats && k < d->n_appends) { slots[k] |= hs::kResetFirst; j = k + 1; }
      else resets[n_alone++] = resets[i];
    }
  }
  const bool rows_inline = batch <= hs::kInlineRows;
  const bool appends_inline = singles && d->n_appends <= hs::kInlineAppends;
  if (!rows_inline || (counting && !appends_inline)) {
    const size_t bytes = counting && !appends_inline ? d->bytes : (size_t)batch * sizeof(hs_row_params);
    if (bytes > h->d_block_bytes) {
      HS_CUDA(h, cudaStreamSynchronize(stream));
      cudaFree(h->d_block_own);
      h->d_block_own = nullptr;
      h->d_block = nullptr;
      h->d_block_bytes = 0;
      const size_t want = std::max<size_t>(2 * bytes, 64 << 10);
      HS_CUDA(h, cudaMalloc(&h->d_block_own, want));
      h->d_block = static_cast<unsigned char*>(h->d_block_own);
      h->d_block_bytes = want;
    }
    HS_CUDA(h, cudaMemcpyAsync(h->d_block, h->h_block, bytes, cudaMemcpyHostToDevice, stream));
  }
  bool behind = false;
  const auto* h_slots = reinterpret_cast<const int32_t*>(h->h_block + d->slots_at);
  const auto* h_offsets = reinterpret_cast<const int32_t*>(h->h_block + d->offsets_at);
  const auto* h_tokens = reinterpret_cast<const int32_t*>(h->h_block + d->tokens_at);
  const auto* d_slots = reinterpret_cast<const int32_t*>(h->d_block + d->slots_at);
  const auto* d_offsets = reinterpret_cast<const int32_t*>(h->d_block + d->offsets_at);
  const auto* d_tokens = reinterpret_cast<const int32_t*>(h->d_block + d->tokens_at);
  if (appends_inline) {
    hs::InlineAppends in;
    in.n = d->n_appends;
    for (int i = 0; i < d->n_appends; ++i) { in.slot[i] = h_slots[i]; in.token[i] = h_tokens[h_offsets[i]]; }
    hs::slots_append_inline_kernel<<<(d->n_appends + 31) / 32, 32, 0, stream>>>(h->pool, in, vocab);
    HS_CUDA(h, cudaGetLastError());
    h->launches += 1;
    behind = true;
  } else if (singles) {
    hs::slots_append_single_kernel<<<(d->n_appends + 31) / 32, 32, 0, stream>>>(h->pool, d_tokens, d_offsets, d_slots,
                                                                               d->n_appends, vocab);
    HS_CUDA(h, cudaGetLastError());
    h->launches += 1;
    behind = true;
  } else {
    if (n_alone) {
      hs::slots_reset_kernel<<<n_alone, 256, 0, stream>>>(
          h->pool, reinterpret_cast<const int32_t*>(h->d_block + d->resets_at), n_alone);
      HS_CUDA(h, cudaGetLastError());
      h->launches += 1;
    }
    if (d->n_appends && repeats) {
      rc = launch_append(h, d_tokens, d_offsets, d_slots, d->n_appends, vocab, d->max_tokens, stream);
      if (rc != HS_OK) return rc;
    } else if (d->n_appends) {
      // one token per thread, as long as the CTAs are few enough to run side by side
      int c = 1;
      while (c < hs::kMaxCluster && c * hs::kBuildThreads < d->max_tokens && d->n_appends * c < 2 * h->sm_count) c *= 2;
      HS_CUDA(h, launch(hs::slots_build_kernel, dim3((unsigned)c, (unsigned)d->n_appends), hs::kBuildThreads, 0, stream,
                        LaunchAttrs(c, false), h->pool,
                        reinterpret_cast<int32_t*>(h->d_block + d->tokens_at), d_offsets, d_slots, d->n_appends, vocab));
      h->launches += 1;
      behind = true;
    }
  }
  hs::InlineRows inl;
  if (rows_inline) std::memcpy(inl.p, params, (size_t)batch * sizeof(hs_row_params));
  // (the records go straight to pinned memory: see write_record)
  rc = launch_rows(h, logits, dtype, row_stride, batch, vocab,
                   rows_inline ? nullptr : reinterpret_cast<const hs_row_params*>(h->d_block), rows_inline ? inl : kNoInlineRows,
                   n_count_of(params, batch, vocab), awaited ? nullptr : h->h_out, nullptr, nullptr, nullptr, 0u, behind, stream, true);
  if (rc != HS_OK) return rc;
  HS_CUDA(h, serial.done());
  h->awaited_records = batch;
  return HS_OK;
}

}  // namespace

int hs_step(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
            const hs_step_desc* d, const hs_row_out** out, void* stream) {
  return step(h, logits, dtype, row_stride, batch, vocab, d, out, false, stream);
}

int hs_step_awaited(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
                    const hs_step_desc* d, const hs_row_out** out, void* stream) {
  return step(h, logits, dtype, row_stride, batch, vocab, d, out, true, stream);
}

int hs_step_wait(hs_sampler* h, void* stream) {
  if (!h) return HS_ERR_INVALID;
  // A greedy row's id is one word in pinned memory, any other row's record comes word by word (see
  // write_record) and is put together here: all are there some microseconds before the stream reports
  // its end.  Rows are taken as they come: bound by the reads of memory the GPU has just written, about 10 ns
  // a row, which in the order of the rows were left for the end whenever an early row was a late one (256 rows of
  // 151,936: 20 counting rows among them 75.2 us a call in order, 72.6 this way, all counting 94.5 and 90.2,
  // none 59.7 and 57.1).  (For as long as a large step takes; then, or if something went wrong, the stream
  // has the word, and all mail is there.)
  const int ids = h->awaited_ids.exchange(0), records = h->awaited_records.exchange(0);
  const uint32_t tag = h->mail_tag;
  auto there = [&](int row) {
    if (ids) return *reinterpret_cast<volatile int32_t*>(h->h_tokens + row) != kNoToken;
    const volatile u64* mail = h->h_mail + (size_t)row * hs::kRecordWords;
    if ((uint32_t)(mail[0] >> 32) != tag) return false;
    const int n = h->mail_words[(size_t)row];
    uint32_t words[hs::kRecordWords], other = 0;
    for (int i = 0; i < n; ++i) {
      const u64 w = mail[i];
      other |= (uint32_t)(w >> 32) ^ tag;
      words[i] = (uint32_t)w;
    }
    if (other) return false;
    std::memcpy(h->h_out + row, words, (size_t)n * 4);
    return true;
  };
  int* const pending = h->pending.data();
  int left = ids + records;
  for (int row = 0; row < left; ++row) pending[row] = row;
  const bool awaited = left > 0;
  auto look = [&] {
    int kept = 0;
    for (int i = 0; i < left; ++i)
      if (!there(pending[i])) pending[kept++] = pending[i];
    left = kept;
  };
  for (int looks = 0; looks < 200000 && left > 0; looks += 1 + left / 64) {
    look();
    if (left > 0) hs_pause();
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  if (awaited && left == 0) return HS_OK;
  DeviceGuard guard(h->device);
  HS_CUDA(h, cudaStreamSynchronize((cudaStream_t)stream));
  look();
  if (records && left > 0) return fail(h, HS_ERR_CUDA, "a step's records did not come");
  return HS_OK;
}

int hs_step_greedy(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch, int vocab,
                   const int32_t** tokens, void* stream_) {
  int rc = check_common(h, logits, dtype, batch, vocab);
  if (rc != HS_OK) return rc;
  if (!tokens) return fail(h, HS_ERR_INVALID, "tokens is null");
  *tokens = nullptr;
  nothing_awaited(h);
  if (batch == 0) return HS_OK;
  if (row_stride < vocab) return fail(h, HS_ERR_INVALID, "row_stride smaller than vocab");
  cudaStream_t stream = (cudaStream_t)stream_;
  DeviceGuard guard(h->device);
  Serial serial(h, stream);
  HS_CUDA(h, serial.status);
  *tokens = h->h_tokens;
  std::fill_n(h->h_tokens, batch, kNoToken);
  rc = launch_greedy(h, logits, dtype, row_stride, batch, vocab, h->h_tokens, stream);
  if (rc != HS_OK) return rc;
  HS_CUDA(h, serial.done());
  h->awaited_ids = batch;
  return HS_OK;
}

int hs_sharded_partial(hs_sampler* h, const void* logits, int dtype, int64_t row_stride, int batch,
                       int vocab_local, int vocab_offset, const hs_row_params* params,
                       hs_shard_rec* recs_out, void* stream) {
  int rc = check_common(h, logits, dtype, batch, vocab_local);
  if (rc != HS_OK) return rc;
  if (dtype != HS_DTYPE_BF16) return fail(h, HS_ERR_UNSUPPORTED, "sharded sampling takes bf16 slices");
  if (batch == 0) return HS_OK;
  if (!params || !recs_out) return fail(h, HS_ERR_INVALID, "params / recs_out is null");
  if (row_stride < vocab_local || vocab_offset < 0) return fail(h, HS_ERR_INVALID, "bad row_stride / vocab_offset");
  DeviceGuard guard(h->device);
  hs::ShardArgs a{};
  a.base.logits = logits; a.base.dtype = dtype; a.base.row_stride = row_stride; a.base.vocab = vocab_local;
  a.base.params = params; a.base.pool = h->pool;
  a.vocab_offset = vocab_offset;
  a.recs = recs_out;
  Serial serial(h, (cudaStream_t)stream);
  HS_CUDA(h, serial.status);
  hs::shard_partial_kernel<<<(unsigned)batch, hs::kThreads, hs::layout_cand().total, (cudaStream_t)stream>>>(a);
  HS_CUDA(h, cudaGetLastError());
  h->launches += 1;
  HS_CUDA(h, serial.done());
  return HS_OK;
}

int hs_sharded_merge(hs_sampler* h, const hs_shard_rec* recs, int ranks, int batch, int vocab_total,
                     const hs_row_params* params, hs_row_out* out, const float* noise, float* full_lse,
                     void* stream) {
  if (!h) return HS_ERR_INVALID;
  if (batch < 0 || ranks < 1 || ranks > 64 || vocab_total < 1) return fail(h, HS_ERR_INVALID, "bad ranks / batch / vocab_total");
  if (ranks * HS_SHARD_CAND > hs::kCandCap) return fail(h, HS_ERR_CAPACITY, "too many ranks for one merge");
  if (batch == 0) return HS_OK;
  if (!recs || !params || !out) return fail(h, HS_ERR_INVALID, "recs / params / out is null");
  DeviceGuard guard(h->device);
  hs::MergeArgs a{recs, ranks, batch, vocab_total, params, out, noise, full_lse};
  Serial serial(h, (cudaStream_t)stream);
  HS_CUDA(h, serial.status);
  hs::shard_merge_kernel<<<(unsigned)batch, hs::kThreads, hs::layout_cand().total, (cudaStream_t)stream>>>(a);
  HS_CUDA(h, cudaGetLastError());
  h->launches += 1;
  HS_CUDA(h, serial.done());
  return HS_OK;
}

int hs_debug_phase_clocks(hs_sampler* h, int batch, unsigned long long* out_host) {
  if (!h || !out_host || batch < 0 || batch > h->batch_max) return HS_ERR_INVALID;
  if (!h->phase_clocks) return fail(h, HS_ERR_UNSUPPORTED, "create the sampler with HS_CREATE_PHASE_CLOCKS");
  DeviceGuard guard(h->device);
  HS_CUDA(h, cudaMemcpy(out_host, h->phase_clocks, (size_t)batch * hs::kV3PhaseSlots * sizeof(unsigned long long),
                        cudaMemcpyDeviceToHost));
  return HS_OK;
}

int hs_debug_set(hs_sampler* h, int what, int value) {
  if (!h) return HS_ERR_INVALID;
  std::lock_guard<std::mutex> lock(h->launch_mu);
  if (what == 0) {
    if (value != 0 && value != 1 && value != 2 && value != 4) return fail(h, HS_ERR_INVALID, "split must be 0, 1, 2 or 4");
    h->force_split = value;
    return HS_OK;
  }
  if (what == 1) {
    if (value < 0 || value > kMaxParts) return fail(h, HS_ERR_INVALID, "counting split must be 0 to 16");
    h->force_csplit = value;
    return HS_OK;
  }
  if (what == 4) {
    h->mail_tag = (uint32_t)value;
    return HS_OK;
  }
  if (what == 3) {
    h->token_draw = value ? 1 : 0;
    return HS_OK;
  }
  return fail(h, HS_ERR_INVALID, "unknown setting");
}

int hs_query(hs_sampler* h, int what, int vocab, int dtype) {
  if (!h) return HS_ERR_INVALID;
  Plan plan;
  const bool v3 = dtype == HS_DTYPE_BF16 && !h->force_general;
  switch (what) {
    case 0: return v3 ? 1 : (make_plan(h, vocab, 1, plan) ? plan.cluster : HS_ERR_CAPACITY);
    case 1: return v3 ? 0 : (make_plan(h, vocab, 1, plan) ? (plan.global_stage ? 0 : 1) : HS_ERR_CAPACITY);
    case 4: return v3 ? 1 : 0;
    case 2: return h->sm_count;
    case 3: return (int)(h->launches & 0x7fffffffull);
    case 5: return (int)std::min<size_t>(h->device_bytes >> 10, 0x7fffffffu);
    case 6: {
      const size_t per_slot = (size_t)h->unique_cap * (sizeof(int2) + sizeof(int32_t)) +
                              (size_t)h->pool.cls_stride * sizeof(uint32_t) + (size_t)h->vocab_max * sizeof(int32_t) +
                              2 * sizeof(int32_t);
      return (int)std::min<size_t>(per_slot, 0x7fffffffu);
    }
    case 7: return h->resident_bf16;
    case 8: {
      // the flag the append kernels raise when a histogram is asked to hold more distinct ids
      // than hist_cap (those ids were not counted); waits for the device
      DeviceGuard guard(h->device);
      int32_t raised = 0;
      HS_CUDA(h, cudaDeviceSynchronize());
      HS_CUDA(h, cudaMemcpy(&raised, h->pool.error, sizeof raised, cudaMemcpyDeviceToHost));
      return raised ? 1 : 0;
    }
    default: return HS_ERR_INVALID;
  }
}

}  // extern "C"
