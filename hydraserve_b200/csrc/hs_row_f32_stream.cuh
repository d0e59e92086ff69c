// The streaming candidate kernel: fp32 rows with a small top_k in a batch of more rows than the
// resident kernel (hs_row_resident.cuh) holds side by side.
//
// One CTA per row, and no row kept on chip.  A lower bound of the row's k-th highest score comes from 512 groups
// of eight neighbouring tokens spread over the row (each thread scores one group and keeps the best: 512
// different tokens, so the k-th highest of them is a valid bound); the bound becomes, per count
// class, the lowest logit VALUE whose score reaches it (scores grow with the value inside a class: a
// search over the 2^32 ordered float patterns, 32 at a time with ballots); the row is streamed
// once, four values per 128-bit load, against the most permissive of those values.  A hit is
// listed as it is, and the listed hits are scored together whenever the list is looked at: looking a
// hit's count class up where it is found would stall the stream on a scattered load.  The list is
// cut back whenever it gets long, and finished exactly like a bf16 candidate row's.  A list
// that overflows (more ties than it holds) reports status 4, for the general kernel.
//
// What bounds it: the chain of bound, stream and finish of one row, the same 61 us for any batch that
// is one wave of two CTAs per SM, where the resident kernel's time grows with the waves of its
// clusters.  151,936 tokens, top_k 50, penalties, one plain greedy row for the resident kernel (us a
// step; streaming / resident): 32 rows 59 / 30, 64 rows 61 / 55, 74 rows 61 / 69, 128 rows 62 / 103, 256
// rows 76 / 246.
#pragma once

#include "hs_row_bf16_kernel.cuh"
#include "hs_sharded.cuh"

namespace hs {

// score of a token with logit x that the history holds `count` times
__device__ __forceinline__ float score_of_float(const Scorer& c, float x, int count) {
  float v = x;  // (a zero's sign goes at the end)
  if (count > 0) {
    v = v < 0.0f ? __fmul_rn(v, c.rp) : __fdiv_rn(v, c.rp);
    v = __fsub_rn(v, c.pp);
    v = __fsub_rn(v, __fmul_rn(c.fp, (float)count));
  }
  return c.score_of_value(v);
}

// Per count class (thr[0..2]), the lowest logit value whose score key reaches `bound`, NaN when
// none does.  Warp cc searches the ordered patterns from -inf to +inf.
__device__ __forceinline__ void f32_thresholds(const Scorer& c, uint32_t bound, float* thr) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < 3) {
    const u64 none = (u64)key_of(__int_as_float(0x7f800000)) + 1ull;  // one past +inf
    // every pattern below lo fails, every pattern from hi on passes (hi = none: nothing does)
    u64 lo = (u64)key_of(__int_as_float(0xff800000)), hi = none;
#pragma unroll 1
    while (lo < hi) {
      const u64 step = (hi - lo + 31ull) >> 5;
      const u64 t = lo + (u64)(lane + 1) * step - 1ull;  // last pattern of this lane's block
      const bool pass = t >= hi || key_of(score_of_float(c, score_of((uint32_t)t), warp)) >= bound;
      const uint32_t votes = __ballot_sync(0xffffffffu, pass);
      if (votes == 0) { lo = hi; break; }
      const int f = __ffs(votes) - 1;  // the answer lies in block f
      hi = min(lo + (u64)(f + 1) * step - 1ull, hi);
      lo = lo + (u64)f * step;
    }
    if (lane == 0) thr[warp] = lo >= none ? __int_as_float(0x7fc00000) : score_of((uint32_t)lo);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kThreads, 2) row_kernel_f32_stream(const __grid_constant__ RowKernelArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ hs_row_out rec;
  const int tid = threadIdx.x, row = blockIdx.x;
  const hs_row_params P = a.params[row];
  if (!is_candidate_row(P, a.vocab)) return;  // the resident kernel's row
  const LayoutCand lay = layout_cand();
  Ctx3 c;
  int* small = reinterpret_cast<int*>(smem_raw + lay.small);
  CandCtx L{reinterpret_cast<u64*>(smem_raw + lay.cand), small + 4, small + 5,
            reinterpret_cast<uint32_t*>(smem_raw + lay.count), small + 8, nullptr};
  float* thr = reinterpret_cast<float*>(small + 12);  // [3]
  c.row = row;
  c.vocab = a.vocab;
  c.greedy = false;
  const float* logits = reinterpret_cast<const float*>(a.logits) + (long long)row * a.row_stride;
  // the row in 16-byte chunks from its first boundary; up to six tokens lie before and behind them
  const int head = min((int)((0u - (uint32_t)reinterpret_cast<uintptr_t>(logits)) & 15u) >> 2, c.vocab);
  const int n4 = (c.vocab - head) >> 2;
  const float4* src4 = reinterpret_cast<const float4*>(logits + head);
  c.T = P.temperature; c.rp = P.repetition_penalty; c.pp = P.presence_penalty; c.fp = P.frequency_penalty;
  c.pool = a.pool;
  c.slot = P.slot;
  const bool slot_ok = P.slot >= 0 && P.slot < a.pool.slots_total;
  const bool penalised = slot_ok && (c.rp != 1.0f || c.pp != 0.0f || c.fp != 0.0f);
  c.cls = penalised ? a.pool.cls + (size_t)P.slot * a.pool.cls_stride : nullptr;
  if (tid < 16) small[tid] = 0;
  if (tid < (int)sizeof(hs_row_out) / 4) reinterpret_cast<uint32_t*>(&rec)[tid] = 0;
  __syncthreads();
  const int k = P.top_k;  // (0 < k <= kTopKMax and k < vocab)

  // 1. the first bound.  A group is eight neighbours (two 128-bit loads, one or two words of the class
  // map); the 512 groups do not overlap.  (A row of fewer than about 4,100 tokens goes without a
  // bound: everything is listed.)
  uint32_t bound = 0;
  {
    const bool sampled = n4 >= 2 * kThreads + 2;
    u64 best = 0;
    if (sampled) {
      const int i = (int)(((long long)tid * (n4 - 2)) / kThreads);  // groups at least two chunks apart
      const float4 a4 = src4[i], b4 = src4[i + 1];
      const float xs[8] = {a4.x, a4.y, a4.z, a4.w, b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int id = head + 4 * i + j;
        const int cc = c.class_of(id);
        if (cc == 3 || xs[j] != xs[j]) continue;  // (listed per request and taken below; NaN)
        const u64 e = cand_pack(key_of(score_of_float(c, xs[j], cc)), id);
        best = e > best ? e : best;
      }
    }
    L.cand[tid] = best;
    __syncthreads();
    if (sampled) bound = cand_kth_key(*c.x(), L, kThreads, k);
    __syncthreads();
  }
  // 2. tokens the history holds three times or more: from the request's list, with their count
  if (c.cls) {
    const int n_heavy = min(c.pool.n_heavy[c.slot], c.pool.unique_cap);
    const int32_t* heavy = c.pool.heavy + (size_t)c.slot * c.pool.unique_cap;
    const int2* pairs = c.pool.pairs + (size_t)c.slot * c.pool.unique_cap;
#pragma unroll 1
    for (int j = tid; j < n_heavy; j += kThreads) {
      const int q = heavy[j];
      if (q < 0 || q >= c.pool.unique_cap) continue;
      const int2 pr = pairs[q];  // (id, count)
      if (pr.x < 0 || pr.x >= c.vocab) continue;
      const float x = logits[pr.x];
      if (x != x) continue;
      const int slot = atomicAdd(L.n, 1);
      if (slot < kCandCap) L.cand[slot] = cand_pack(key_of(score_of_float(c, x, pr.y)), pr.x);
      else *L.lost = 1;
    }
  }
  __syncthreads();
  // (read by every thread before the barrier in f32_thresholds: after it the stream adds to the list)
  int n_scored = min(*L.n, kCandCap);  // the often-repeated tokens, scored when they were listed
  f32_thresholds(c, bound, thr);

  // 3. the row, once.  Listed hits are (value bits, id); a token of a penalised class that does not reach
  // its own threshold drops out when they are scored.
  auto look = [&](int id, float x) {
    const int slot = atomicAdd(L.n, 1);
    if (slot < kCandCap) L.cand[slot] = ((u64)__float_as_uint(x) << 32) | (uint32_t)id;
    else *L.lost = 1;
  };
  auto score_pending = [&](int from, int to) {
    // (left to the compiler to unroll: the hits' count classes are scattered reads, and one at a time
    // they make 128 rows take 82 us instead of 62)
    for (int i = from + tid; i < to; i += kThreads) {
      const u64 e = L.cand[i];
      const int id = (int)(uint32_t)e;
      const float x = __uint_as_float((uint32_t)(e >> 32));
      const int cc = c.class_of(id);
      const bool valid = cc != 3 && x >= thr[cc];  // (three times or more: listed above already)
      L.cand[i] = valid ? cand_pack(key_of(score_of_float(c, x, cc)), id) : 0ull;
    }
    __syncthreads();
  };
  auto lowest_threshold = [&] {
    return c.cls ? fminf(thr[0], fminf(thr[1], thr[2])) : thr[0];  // (a NaN threshold, "none", is ignored by fminf)
  };
  // One buffer: a chunk's successor is requested as soon as the chunk has been tested, so a
  // request has a whole pass of the loop to arrive, and the registers hold one batch only.
  constexpr int kBatch = 4;
  float4 w[kBatch];
#pragma unroll
  for (int u = 0; u < kBatch; ++u) {
    const int i = tid + u * kThreads;
    if (i < n4) w[u] = __ldcs(src4 + i);
  }
  int iteration = 0, next_look = 1, last_look = -1, last_seen = 0, turn = 0;
#pragma unroll 1
  for (int base = 0; base < n4; base += kBatch * kThreads, ++iteration) {
    const float t_min = lowest_threshold();
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int i = base + tid + u * kThreads;
      if (i < n4) {
        const float4 v = w[u];
        if (i + kBatch * kThreads < n4) w[u] = __ldcs(src4 + i + kBatch * kThreads);
        if (!(v.x >= t_min || v.y >= t_min || v.z >= t_min || v.w >= t_min)) continue;  // the common case
        const int id = head + 4 * i;
        if (v.x >= t_min) look(id, v.x);
        if (v.y >= t_min) look(id + 1, v.y);
        if (v.z >= t_min) look(id + 2, v.z);
        if (v.w >= t_min) look(id + 3, v.w);
      }
    }
    // a look at the list's length now and then, the sooner the faster it grows (each is a barrier,
    // which makes the batch wait for its slowest load)
    if (iteration != next_look) continue;
    // (two words in turn: one is written again only after the next look's barrier, when every thread has read it)
    turn ^= 1;
    if (tid == 0) L.lost[1 + turn] = *L.n;
    const bool refresh = __syncthreads_or(*L.n >= kCandSoft);
    {
      const int seen = L.lost[1 + turn];
      const int per_batch = max(0, seen - last_seen) / (iteration - last_look);
      last_seen = seen;
      last_look = iteration;
      constexpr int kRoom = (kCandCap - kCandSoft) / 2;
      next_look = iteration + (per_batch * 8 <= kRoom ? 8 : (per_batch * 4 <= kRoom ? 4 : (per_batch * 2 <= kRoom ? 2 : 1)));
    }
    // raise the bound when the list is getting long (block-uniform decision)
    if (refresh) {
      if (*L.lost) break;
      const int n_now = min(*L.n, kCandCap);
      score_pending(n_scored, n_now);
      bound = cand_kth_key(*c.x(), L, n_now, k);
      n_scored = last_seen = cand_compact(L, n_now, bound);
      f32_thresholds(c, bound, thr);
    }
  }
  __syncthreads();
  {
    const int n_loose = c.vocab - 4 * n4;
    if (tid < n_loose) {
      const int id = tid < head ? tid : tid + 4 * n4;
      const float x = logits[id];
      if (x >= lowest_threshold()) look(id, x);
    }
  }
  __syncthreads();
  if (*L.lost) {  // more ties than the list holds: the general kernel samples this row
    if (tid == 0) rec.status = 4;
    __syncthreads();
    if (tid < 32) write_record(record_of(a, row), rec, P.n_logprobs >= 0, mail_of(a, row), a.mail_tag);
    return;
  }
  int n = min(*L.n, kCandCap);
  score_pending(n_scored, n);
  // (without a cut the pass still drops the entries the scoring voided)
  n = cand_keep_sorted(L, reinterpret_cast<u64*>(smem_raw + lay.mass), n, n > k && n > kSortAll ? cand_kth_key(*c.x(), L, n, k) : 0u);
  if (n > k) {
    // a list that was sorted whole: top-k keeps the first k entries and the ties of the k-th
    const uint32_t cut = cand_key(L.cand[k - 1]);
    u64 keep = 0, unused = 0;
    for (int i = tid; i < n; i += kThreads) keep += cand_key(L.cand[i]) >= cut ? 1 : 0;
    block_sum2(*c.x(), keep, unused);
    n = (int)keep;
  }
  const float* noise_row = a.noise ? a.noise + (size_t)row * a.vocab : nullptr;
  FinishOut r = finish_sorted(*c.x(), L.cand, reinterpret_cast<u64*>(smem_raw + lay.mass), n, P, noise_row, &rec);
  if (P.slot >= a.pool.slots_total) r.status |= 64;  // a slot this sampler does not have: no penalties
  if (a.scores_out) {
    float* dst = a.scores_out + (size_t)row * a.vocab;
#pragma unroll 1
    for (int id = tid; id < c.vocab; id += kThreads) dst[id] = __int_as_float(0xff800000);
    __syncthreads();
#pragma unroll 1
    for (int i = tid; i < (int)r.n_kept; i += kThreads) dst[cand_id(L.cand[i])] = score_of(cand_key(L.cand[i]));
  }
  if (tid == 0) {
    if (a.tokens_out) a.tokens_out[row] = r.token;
    if ((a.flags & HS_SAMPLE_APPEND_TOKEN) && slot_ok && r.token >= 0 && r.token < a.vocab) {
      if (!slot_append_one(a.pool, P.slot, r.token)) r.status |= 2;
    }
    write_finish(r, &rec);
  }
  __syncthreads();
  if (tid < 32) write_record(record_of(a, row), rec, P.n_logprobs >= 0, mail_of(a, row), a.mail_tag);
}

}  // namespace hs
