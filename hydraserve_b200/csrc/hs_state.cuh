// Device-resident token-count histograms (one per request slot) and the plain-greedy
// arg-max kernels.
//
// A slot is the device form of the `counts` dict the reference rebuilds per row per step
// (sampling.py:106-110).  It holds
//   pairs[]   the distinct token ids seen so far with their counts, (id, count), 8 bytes each
//   pos[]     dense index: pos[token] = 1 + position in pairs (0 = unseen); touched only
//             when tokens are appended
//   cls[]     dense 2-bit class per token, min(count, 3), sixteen tokens per 32-bit word: what
//             the bf16 sampling kernel streams next to the logits (V/4 bytes per row)
//   heavy[]   positions in pairs of the ids whose count reached 3: the only tokens whose
//             exact count the bf16 kernels need (one look-up gives id and count)
#pragma once

#include "hs_common.cuh"
#include "../../include/hs_sampler.h"

namespace hs {

struct Pool {
  int2* pairs;     // [slots_total, unique_cap] (token id, count)
  int32_t* n;      // [slots_total]
  int32_t* pos;    // [slots_total, pos_stride]
  uint32_t* cls;   // [slots_total, cls_stride] 2-bit classes
  int32_t* heavy;  // [slots_total, unique_cap] positions in pairs
  int32_t* n_heavy;  // [slots_total]
  int32_t* error;  // [1] sticky: 1 = a slot overflowed unique_cap
  int slots_total;
  int unique_cap;
  long long pos_stride;
  long long cls_stride;  // words per slot
};

// Sets the 2-bit class of `token` to min(count, 3); returns the previous class.
__device__ __forceinline__ uint32_t set_class(uint32_t* cls, int token, int count) {
  const uint32_t want = (uint32_t)min(count, 3);
  uint32_t* word = cls + (token >> 4);
  const int shift = (token & 15) * 2;
  uint32_t old = __ldcg(word);
  while (true) {
    const uint32_t cur = (old >> shift) & 3u;
    if (cur >= want) return cur;  // classes only grow between resets
    const uint32_t next = (old & ~(3u << shift)) | (want << shift);
    const uint32_t seen = atomicCAS(word, old, next);
    if (seen == old) return cur;
    old = seen;
  }
}

// Empties each listed slot by walking its id list (no dense clear).
__global__ void slots_reset_kernel(Pool p, const int32_t* slots, int n_slots) {
  const int s = blockIdx.x < n_slots ? slots[blockIdx.x] : -1;
  if (s < 0 || s >= p.slots_total) return;
  const int n = min(p.n[s], p.unique_cap);
  const int2* pairs = p.pairs + (size_t)s * p.unique_cap;
  int32_t* pos = p.pos + (size_t)s * p.pos_stride;
  uint32_t* cls = p.cls + (size_t)s * p.cls_stride;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const int id = pairs[j].x;
    if (id >= 0 && id < p.pos_stride) {
      pos[id] = 0;
      cls[id >> 4] = 0;  // every non-zero field of the word belongs to a listed id
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) { p.n[s] = 0; p.n_heavy[s] = 0; }
}

// Pass 1 of an append: give every token id not yet in the slot a list position.
__global__ void slots_register_kernel(Pool p, const int32_t* tokens, const int32_t* offsets,
                                      const int32_t* slots, int n_slots, int vocab) {
  const int row = blockIdx.y;
  const int s = row < n_slots ? slots[row] : -1;
  if (s < 0 || s >= p.slots_total) return;
  const int t0 = offsets[row], t1 = offsets[row + 1];
  int2* pairs = p.pairs + (size_t)s * p.unique_cap;
  int32_t* pos = p.pos + (size_t)s * p.pos_stride;
  for (int j = t0 + blockIdx.x * blockDim.x + threadIdx.x; j < t1; j += gridDim.x * blockDim.x) {
    const int t = tokens[j];
    if (t < 0 || t >= vocab || t >= p.pos_stride) continue;  // ignored, as in the reference
    if (atomicCAS(&pos[t], 0, -1) == 0) {
      const int idx = atomicAdd(&p.n[s], 1);
      if (idx < p.unique_cap) {
        pairs[idx] = make_int2(t, 0);
        pos[t] = idx + 1;
      } else {
        atomicSub(&p.n[s], 1);
        pos[t] = 0;
        *p.error = 1;
      }
    }
  }
}

// Pass 2 of an append: count.
__global__ void slots_count_kernel(Pool p, const int32_t* tokens, const int32_t* offsets,
                                   const int32_t* slots, int n_slots, int vocab) {
  const int row = blockIdx.y;
  const int s = row < n_slots ? slots[row] : -1;
  if (s < 0 || s >= p.slots_total) return;
  const int t0 = offsets[row], t1 = offsets[row + 1];
  int2* pairs = p.pairs + (size_t)s * p.unique_cap;
  const int32_t* pos = p.pos + (size_t)s * p.pos_stride;
  for (int j = t0 + blockIdx.x * blockDim.x + threadIdx.x; j < t1; j += gridDim.x * blockDim.x) {
    const int t = tokens[j];
    if (t < 0 || t >= vocab || t >= p.pos_stride) continue;
    const int q = pos[t];
    if (q > 0) atomicAdd(&pairs[q - 1].y, 1);
  }
}

// Pass 3 of an append: with the counts final, refresh the 2-bit classes and list the ids
// whose count reached 3 (the thread that moves a class to 3 does the listing).
__global__ void slots_classify_kernel(Pool p, const int32_t* tokens, const int32_t* offsets,
                                      const int32_t* slots, int n_slots, int vocab) {
  const int row = blockIdx.y;
  const int s = row < n_slots ? slots[row] : -1;
  if (s < 0 || s >= p.slots_total) return;
  const int t0 = offsets[row], t1 = offsets[row + 1];
  const int2* pairs = p.pairs + (size_t)s * p.unique_cap;
  const int32_t* pos = p.pos + (size_t)s * p.pos_stride;
  uint32_t* cls = p.cls + (size_t)s * p.cls_stride;
  int32_t* heavy = p.heavy + (size_t)s * p.unique_cap;
  for (int j = t0 + blockIdx.x * blockDim.x + threadIdx.x; j < t1; j += gridDim.x * blockDim.x) {
    const int t = tokens[j];
    if (t < 0 || t >= vocab || t >= p.pos_stride) continue;
    const int q = pos[t];
    if (q <= 0) continue;
    const int count = pairs[q - 1].y;
    const uint32_t before = set_class(cls, t, count);
    if (count >= 3 && before < 3u) {
      const int idx = atomicAdd(&p.n_heavy[s], 1);
      if (idx < p.unique_cap) heavy[idx] = q - 1;
    }
  }
}

// One token appended by a single thread (the sampling kernel's epilogue).
__device__ __forceinline__ bool slot_append_one(const Pool& p, int s, int token) {
  int2* pairs = p.pairs + (size_t)s * p.unique_cap;
  int32_t* pos = p.pos + (size_t)s * p.pos_stride;
  uint32_t* cls = p.cls + (size_t)s * p.cls_stride;
  int count;
  const int q = pos[token];
  if (q > 0) {
    count = (pairs[q - 1].y += 1);
  } else {
    const int n = p.n[s];
    if (n >= p.unique_cap) return false;
    pairs[n] = make_int2(token, 1);
    pos[token] = n + 1;
    p.n[s] = n + 1;
    count = 1;
  }
  if (count <= 3) {
    uint32_t* word = cls + (token >> 4);
    const int shift = (token & 15) * 2;
    *word = (*word & ~(3u << shift)) | ((uint32_t)count << shift);
    if (count == 3) {
      const int h = p.n_heavy[s];
      if (h < p.unique_cap) { (p.heavy + (size_t)s * p.unique_cap)[h] = pos[token] - 1; p.n_heavy[s] = h + 1; }
    }
  }
  return true;
}

// A whole history into each listed slot in one launch, a cluster of CTAs per slot (gridDim.x).
// Bound by the latency of scattered reads and atomics, so what counts is how many of them follow
// one another.  A slot that is emptied first (kResetFirst, the usual case) takes two barriers: its
// old ids are cleared; every token is counted where its position will stand, and the token that
// found a zero there stands for its id from then on; those write id and count, position and class.
// Four tokens per thread are under way together.  One slot with an 8,192-token prompt, cold (ncu): 22 us
// to empty it (one CTA) and 16 us for the three passes above, 12.4 us here in all.
// A slot that keeps what it has goes through the three passes with barriers in between.
// Overwrites `tokens` (this sampler's own copy of them).
constexpr int kBuildThreads = 512;
constexpr int kBuildBatch = 4;
constexpr int kResetFirst = 1 << 30;  // in a slot number
__global__ void __launch_bounds__(kBuildThreads) slots_build_kernel(const Pool p, int32_t* tokens, const int32_t* offsets,
                                                                    const int32_t* slots, int n_slots, int vocab) {
  cudaTriggerProgrammaticLaunchCompletion();
  cg::cluster_group cluster = cg::this_cluster();
  const int row = blockIdx.y;
  const int entry = row < n_slots ? slots[row] : -1;
  const int s = entry < 0 ? -1 : entry & (kResetFirst - 1);
  if (s < 0 || s >= p.slots_total) return;  // (all CTAs of the cluster alike)
  const int at = (int)blockIdx.x * kBuildThreads + threadIdx.x, step = (int)gridDim.x * kBuildThreads;
  int2* pairs = p.pairs + (size_t)s * p.unique_cap;
  int32_t* pos = p.pos + (size_t)s * p.pos_stride;
  uint32_t* cls = p.cls + (size_t)s * p.cls_stride;
  int32_t* heavy = p.heavy + (size_t)s * p.unique_cap;
  auto sync = [&]() {
    __threadfence();
    if (gridDim.x > 1) cluster.sync(); else __syncthreads();
  };
  auto valid = [&](int t) { return t >= 0 && t < vocab && t < p.pos_stride; };  // (others are ignored, as in the reference)
  const int t0 = offsets[row], t1 = offsets[row + 1];
  // room for this warp's `mine` new ids in a counter of the slot: one atomic per warp
  auto room = [&](int32_t* counter, bool mine) {
    const uint32_t who = __ballot_sync(0xffffffffu, mine);
    int first = 0;
    if (who && (threadIdx.x & 31) == (unsigned)(__ffs(who) - 1)) first = atomicAdd(counter, __popc(who));
    first = __shfl_sync(0xffffffffu, first, who ? __ffs(who) - 1 : 0);
    return first + __popc(who & ((1u << (threadIdx.x & 31)) - 1u));
  };
  if (entry & kResetFirst) {
    const int n = min(__ldcg(p.n + s), p.unique_cap);
    int t[kBuildBatch];
    auto fetch = [&](int j) {
#pragma unroll
      for (int u = 0; u < kBuildBatch; ++u) t[u] = j + u * step < t1 ? __ldcg(tokens + j + u * step) : -1;
    };
    fetch(t0 + at);  // (on their way while the slot is emptied)
    for (int j = at; j < n; j += kBuildBatch * step) {
      int id[kBuildBatch];
#pragma unroll
      for (int u = 0; u < kBuildBatch; ++u) id[u] = j + u * step < n ? __ldcg(pairs + j + u * step).x : -1;
#pragma unroll
      for (int u = 0; u < kBuildBatch; ++u) {
        if (id[u] < 0 || id[u] >= p.pos_stride) continue;
        __stcg(pos + id[u], 0);
        __stcg(cls + (id[u] >> 4), 0u);  // every non-zero field of the word belongs to a listed id
      }
    }
    sync();
    if (at == 0) { __stcg(p.n + s, 0); __stcg(p.n_heavy + s, 0); }
    const bool one_batch = t1 - t0 <= kBuildBatch * step;
    for (int j = t0 + at;; ) {
      int old[kBuildBatch];
#pragma unroll
      for (int u = 0; u < kBuildBatch; ++u) old[u] = valid(t[u]) ? atomicAdd(pos + t[u], 1) : 1;
#pragma unroll
      for (int u = 0; u < kBuildBatch; ++u) {
        if (old[u] != 0) t[u] = -1;  // (another token stands for this id)
        if (!one_batch && j + u * step < t1) __stcg(tokens + j + u * step, t[u]);
      }
      j += kBuildBatch * step;
      if (j >= t1) break;
      fetch(j);
    }
    sync();
    if (!one_batch) fetch(t0 + at);
    for (int j0 = t0 + at - (int)(threadIdx.x & 31);; ) {  // (whole warps stay in the loop)
      int count[kBuildBatch];
#pragma unroll
      for (int u = 0; u < kBuildBatch; ++u) count[u] = t[u] >= 0 ? __ldcg(pos + t[u]) : 0;
#pragma unroll
      for (int u = 0; u < kBuildBatch; ++u) {
        const int idx = room(p.n + s, t[u] >= 0);
        const bool fits = t[u] >= 0 && idx < p.unique_cap;
        if (t[u] >= 0 && !fits) { __stcg(pos + t[u], 0); *p.error = 1; }
        if (fits) {
          __stcg(pairs + idx, make_int2(t[u], count[u]));
          __stcg(pos + t[u], idx + 1);
          atomicOr(cls + (t[u] >> 4), (uint32_t)min(count[u], 3) << ((t[u] & 15) * 2));
        }
        const bool often = fits && count[u] >= 3;
        if (__any_sync(0xffffffffu, often)) {
          const int h = room(p.n_heavy + s, often);
          if (often && h < p.unique_cap) heavy[h] = idx;
        }
      }
      j0 += kBuildBatch * step;
      if (j0 >= t1) break;
      fetch(j0 + (int)(threadIdx.x & 31));
    }
    // (ids beyond the capacity took numbers too: the count goes back to what is listed)
    sync();
    if (at == 0 && __ldcg(p.n + s) > p.unique_cap) __stcg(p.n + s, p.unique_cap);
    return;
  }
  for (int j = t0 + at; j < t1; j += step) {
    const int t = tokens[j];
    if (!valid(t) || atomicCAS(&pos[t], 0, -1) != 0) continue;
    const int idx = atomicAdd(&p.n[s], 1);
    if (idx < p.unique_cap) {
      __stcg(pairs + idx, make_int2(t, 0));
      __stcg(pos + t, idx + 1);
    } else {
      atomicSub(&p.n[s], 1);
      __stcg(pos + t, 0);
      *p.error = 1;
    }
  }
  sync();
  for (int j = t0 + at; j < t1; j += step) {
    const int t = tokens[j];
    if (!valid(t)) continue;
    const int q = __ldcg(pos + t);
    if (q > 0) atomicAdd(&pairs[q - 1].y, 1);
  }
  sync();
  for (int j = t0 + at; j < t1; j += step) {
    const int t = tokens[j];
    if (!valid(t)) continue;
    const int q = __ldcg(pos + t);
    if (q <= 0) continue;
    const int count = __ldcg(&pairs[q - 1].y);
    const uint32_t before = set_class(cls, t, count);
    if (count >= 3 && before < 3u) {
      const int idx = atomicAdd(&p.n_heavy[s], 1);
      if (idx < p.unique_cap) heavy[idx] = q - 1;
    }
  }
}

// One new token per listed slot (the common step of a decode loop: every request has gained the
// token sampled last), each by one thread: no slot is listed twice, so nothing is contended and
// the three passes above are one.  Up to kInlineAppends pairs travel in the launch's own
// parameters; without inline pairs they come from device memory as hs_slots_append takes them.
// Bound by three dependent scattered accesses: 2.4 us for one request, 3.9 us for 256 (three launches
// and a copy before).  Where the line lies, calls of 64 and 256 rows that gained a token each: 40.3 and
// 61.9 us with the pairs in the launch, 42.8 and 62.7 with a copy; room for 1,024 pairs costs every launch
// that has fewer (128 rows 49.6 us against 48.3).
constexpr int kInlineAppends = 256;
struct InlineAppends {
  int n;
  int slot[kInlineAppends];
  int token[kInlineAppends];
};
__device__ __forceinline__ void append_single(const Pool& p, int s, int t, int vocab) {
  if (s < 0 || s >= p.slots_total || t < 0 || t >= vocab || t >= p.pos_stride) return;
  if (!slot_append_one(p, s, t)) *p.error = 1;
}
__global__ void slots_append_inline_kernel(const Pool p, const __grid_constant__ InlineAppends in, int vocab) {
  // (the sampling kernel behind this one may get its CTAs ready meanwhile; it waits for this
  // grid's end before it looks at a histogram)
  cudaTriggerProgrammaticLaunchCompletion();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < in.n) append_single(p, in.slot[i], in.token[i], vocab);
}
__global__ void slots_append_single_kernel(const Pool p, const int32_t* tokens, const int32_t* offsets,
                                           const int32_t* slots, int n_slots, int vocab) {
  cudaTriggerProgrammaticLaunchCompletion();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_slots && offsets[i + 1] > offsets[i]) append_single(p, slots[i], tokens[offsets[i]], vocab);
}

// ---- plain greedy: arg max per row, lowest id on ties (reference sampling.py:69-73) ---
// Bound by HBM once the row chunks of a call fill the SMs, by latency below that.  A CTA takes
// one chunk of one row.  Values are compared as integers in their order (two bf16 values per
// 32-bit word: sign-magnitude to two's complement, which gives -0.0 and +0.0 one value; NaNs of
// positive sign come out on top, as the fp32 key order has them); a thread keeps its best value
// and the first 16 bytes it saw it in, and only the chunk's winner looks into those again.
constexpr int kGreedyThreads = 256;
constexpr int kGreedyUnroll = 8;  // 128-bit loads in flight per thread

__device__ __forceinline__ int greedy_image_f32(float f) {
  const uint32_t u = __float_as_uint(f);
  const int mag = (int)(u & 0x7fffffffu);
  return (int)u < 0 ? -mag : mag;
}
__device__ __forceinline__ int greedy_image_bf16(uint32_t raw) {
  const int mag = (int)(raw & 0x7fffu);
  return (raw & 0x8000u) ? -mag : mag;
}
// Highest of the eight values of a 16-byte chunk, as an integer image.
__device__ __forceinline__ int greedy_chunk_bf16(const uint4& w) {
  uint32_t best = 0x80018001u;  // below every image
  const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    uint32_t mask;
    asm("prmt.b32 %0, %1, 0, 0xBB99;" : "=r"(mask) : "r"(words[k]));  // 0xffff per negative half
    best = __viaddmax_s16x2((words[k] & 0x7fff7fffu) ^ mask, mask & 0x00010001u, best);
  }
  return max((int)(short)(best & 0xffffu), (int)best >> 16);
}
__device__ __forceinline__ int greedy_chunk_f32(const uint4& w) {
  return max(max(greedy_image_f32(__uint_as_float(w.x)), greedy_image_f32(__uint_as_float(w.y))),
             max(greedy_image_f32(__uint_as_float(w.z)), greedy_image_f32(__uint_as_float(w.w))));
}

// Best element of tokens [begin, begin + n) of a row, as (order-preserving value, ~id); valid in
// thread 0.
template <bool BF16>
__device__ u64 greedy_chunk_best(const void* logits, long long row_offset, int begin, int n) {
  __shared__ u64 warp_best[kGreedyThreads / 32];
  constexpr int kPer = BF16 ? 8 : 4;  // values per 16 bytes
  const int tid = threadIdx.x;
  const unsigned char* base = reinterpret_cast<const unsigned char*>(logits) + (row_offset + begin) * (BF16 ? 2 : 4);
  // (a row may start anywhere: whole chunks from the first boundary on, the elements around them one by one;
  // with every element read by itself 64 rows of 50,257 took 28.3 us a call and take 23.0, 16 fp32 rows of
  // 151,937 22.4 and 17.5)
  const int head = min((int)((0u - (uint32_t)reinterpret_cast<uintptr_t>(base)) & 15u) / (BF16 ? 2 : 4), n);
  const int n16 = (n - head) / kPer;
  const uint4* src = reinterpret_cast<const uint4*>(base + head * (BF16 ? 2 : 4));
  auto image = [&](int i) {
    return BF16 ? greedy_image_bf16(reinterpret_cast<const unsigned short*>(base)[i])
                : greedy_image_f32(reinterpret_cast<const float*>(base)[i]);
  };
  constexpr int kNone = (int)0x80000000;  // below every image (an fp32 image is at least -0x7fffffff)
  int best = kNone, at = 0;
  int i = tid;
  for (; i + (kGreedyUnroll - 1) * kGreedyThreads < n16; i += kGreedyUnroll * kGreedyThreads) {
    uint4 w[kGreedyUnroll];
#pragma unroll
    for (int u = 0; u < kGreedyUnroll; ++u) w[u] = __ldcs(src + i + u * kGreedyThreads);
#pragma unroll
    for (int u = 0; u < kGreedyUnroll; ++u) {
      const int v = BF16 ? greedy_chunk_bf16(w[u]) : greedy_chunk_f32(w[u]);
      if (v > best) { best = v; at = i + u * kGreedyThreads; }
    }
  }
  if (i < n16) {
    uint4 w[kGreedyUnroll];
#pragma unroll
    for (int u = 0; u < kGreedyUnroll - 1; ++u)
      if (i + u * kGreedyThreads < n16) w[u] = __ldcs(src + i + u * kGreedyThreads);
#pragma unroll
    for (int u = 0; u < kGreedyUnroll - 1; ++u) {
      if (i + u * kGreedyThreads >= n16) break;
      const int v = BF16 ? greedy_chunk_bf16(w[u]) : greedy_chunk_f32(w[u]);
      if (v > best) { best = v; at = i + u * kGreedyThreads; }
    }
  }
  // (value, ~first element of the chunk of 16 bytes it was seen in)
  u64 mine = best == kNone ? 0ull : ((u64)((uint32_t)best ^ 0x80000000u) << 32) | (uint32_t)(~(uint32_t)(head + at * kPer));
  const int loose = n - n16 * kPer;  // (at most seven ahead, seven behind)
  if (tid < loose) {
    const int k = tid < head ? tid : tid + n16 * kPer;
    const u64 e = ((u64)((uint32_t)image(k) ^ 0x80000000u) << 32) | (uint32_t)(~(uint32_t)k);
    mine = e > mine ? e : mine;
  }
  mine = warp_max_u64(mine);
  if ((tid & 31) == 0) warp_best[tid >> 5] = mine;
  __syncthreads();
  if (tid != 0) return 0;
#pragma unroll
  for (int k = 1; k < kGreedyThreads / 32; ++k) mine = warp_best[k] > mine ? warp_best[k] : mine;
  int id = (int)(~(uint32_t)mine);
  const int value = (int)((uint32_t)(mine >> 32) ^ 0x80000000u);
  if (id >= head && id < head + n16 * kPer)
    while (image(id) != value) ++id;  // (one of the chunk's eight or four)
  return (mine & 0xffffffff00000000ull) | (uint32_t)(~(uint32_t)(begin + id));
}

// The row's best over its chunks meets in best[row] (0 between calls); the CTA that draws the
// row's last ticket writes the id and puts both back to 0.  Bound by HBM on large batches and by one
// load's latency on small ones, so a row is cut into as many chunks as fill the SMs four times.
// One row of 151,936 bf16 tokens takes 4.6 us, 64 rows of 248,320 13.5 us (2.4 TB/s); with partial maxima and a
// second launch over them 7.9 and 21.2.
__global__ void __launch_bounds__(kGreedyThreads) greedy_kernel(
    const void* logits, int dtype, long long row_stride, int vocab, int chunk, u64* best, int* ticket, int32_t* tokens_out) {
  const int row = blockIdx.y, begin = blockIdx.x * chunk, n = max(0, min(chunk, vocab - begin));
  const u64 mine = dtype == HS_DTYPE_BF16 ? greedy_chunk_best<true>(logits, row * row_stride, begin, n)
                                          : greedy_chunk_best<false>(logits, row * row_stride, begin, n);
  if (threadIdx.x != 0) return;
  u64 top = mine;
  if (gridDim.x > 1) {
    atomicMax(&best[row], mine);
    __threadfence();
    if (atomicAdd(&ticket[row], 1) != (int)gridDim.x - 1) return;
    __threadfence();
    top = atomicExch(&best[row], 0ull);
    ticket[row] = 0;
  }
  // (one store, the CTA's last: a host that waits for it in pinned memory sees it when it has crossed the bus.  A
  // system-wide fence behind it made the kernel's end wait for that too, and with it the rows still to be
  // dispatched: 64 rows of 248,320 took 34.5 us a call and take 29.3.)
  *reinterpret_cast<volatile int32_t*>(tokens_out + row) = (int32_t)(~(uint32_t)(top & 0xffffffffu));
}

// The same in two launches, with nothing that has to hold a value between calls.
__global__ void __launch_bounds__(kGreedyThreads) greedy_partial_kernel(
    const void* logits, int dtype, long long row_stride, int vocab, int chunk, u64* partials) {
  const int row = blockIdx.y, begin = blockIdx.x * chunk, n = max(0, min(chunk, vocab - begin));
  const u64 mine = dtype == HS_DTYPE_BF16 ? greedy_chunk_best<true>(logits, row * row_stride, begin, n)
                                          : greedy_chunk_best<false>(logits, row * row_stride, begin, n);
  if (threadIdx.x == 0) partials[(size_t)row * gridDim.x + blockIdx.x] = mine;
}

__global__ void greedy_final_kernel(const u64* partials, int chunks, int batch, int32_t* tokens_out) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= batch) return;
  u64 best = 0;
  for (int g = 0; g < chunks; ++g) {
    const u64 t = partials[(size_t)row * chunks + g];
    best = t > best ? t : best;
  }
  tokens_out[row] = (int32_t)(~(uint32_t)(best & 0xffffffffu));
}

}  // namespace hs
