// The resident row kernel: fp32 rows (but small top_k in large batches: hs_row_f32_stream.cuh), and
// bf16 rows another kernel gave up.
//
// One thread-block cluster owns a row.  The row is read from HBM once, scored on the way in (the
// 2-bit count classes travel along, so penalties need no second pass; tokens held three times or
// more follow from the request's list) and kept on chip as fp32 scores, a slice per CTA (global
// scratch stands in when the row is too wide for the cluster's shared memory).
//
// Rows with a small top_k: every CTA takes a lower bound of the row's k-th highest score from its
// threads' own maxima (see slice_bound), the few scores at or above the lowest of these bounds are
// listed, one CTA collects the lists and finishes the row as every candidate row is finished.
//
// The other rows: ONE histogram of count and exact mass over 1,024 buckets of equal width in
// score, between the row maximum and 30 below it (2^-40 units of mass end at 28.4) or the row
// minimum.  Every cut (top-k by count, top-p by mass, top-N) names a bucket; the bucket's members
// are gathered from all slices, sorted, and the cut is read off exactly.  The draw is an inverse
// CDF in token order: a thread adds up a contiguous run of the slice, and one warp looks into the
// run that holds the target.  What bounds it: shared-memory atomics and exponentials of the
// histogram (about two atomics and 40 instructions per token), then cluster barriers; with eight
// CTAs a row, two per SM, 32 rows of 151,936 are one wave.  With top_p over all tokens they take 56 us
// (113 us by radix descents, several passes a cut); four rows with top_k 50 24 us (72 us).
// A bucket with more members than a list holds (a row of few values) is resolved by radix
// descents over the keys instead, several passes each.
//
// Probability mass is an integer multiple of 2^-40 (hs::mass_of), so every sum is exact and
// independent of accumulation order: the same row always yields the same cut.
#pragma once

#include "hs_row_args.cuh"
#include "hs_row_topk.cuh"
#include "hs_select.cuh"
#include "hs_sharded.cuh"

#include <type_traits>

namespace hs {

constexpr int kResBuckets = 1024;
constexpr int kResList = 2048;      // members a gather can hold, over all slices
constexpr int kResMerge = 64 << 10; // bytes of the stage a candidate row's finisher needs: list and masses
static_assert(kResMerge >= 2 * kCandCap * (int)sizeof(u64), "the merged list and its masses fit the stage");
static_assert(sizeof(Hist) >= kCandCap * sizeof(u64) && sizeof(Hist) >= 16 * kResBuckets + 8 * kResList,
              "a slice's candidate list, or histogram and members, fit the radix histogram's place");

struct RowCtx : ClusterCtx {
  int row;
  int vocab;
  int slice;
  int base;      // global index of the first element of this CTA's slice
  int n_local;   // elements in this CTA's slice
  int seg;       // elements per warp in the id-ordered walks (multiple of 32)
  float* stage;  // this CTA's slice: final scores
  uint32_t turn = 0;  // exchanges so far (see cluster_exchange)
  template <int N>
  __device__ __forceinline__ void exchange(const u64 (&vals)[N], u64 (&got)[N]) {
    cluster_exchange<N>(cluster, *x, turn, vals, got);
  }
};

// Every element of the resident fp32 row, for descend_core.
template <bool WITH_MASS>
struct StageFill {
  const float* stage;
  int n_local;
  float m;
  template <class Add>
  __device__ __forceinline__ void operator()(int level, int shift, int bits, uint32_t prefix,
                                             uint32_t lo_key, const Add& add) const {
    const uint32_t mask = (1u << bits) - 1u;
    for (int i0 = threadIdx.x & ~31; i0 < n_local; i0 += kThreads) {
      const int i = i0 + (threadIdx.x & 31);
      bool valid = i < n_local;
      float s = 0.f;
      uint32_t k = 0;
      if (valid) {
        s = stage[i];
        k = key_of(s);
        valid = k >= lo_key && (level == 0 || (k >> (shift + bits)) == prefix);
      }
      add(valid, (k >> shift) & mask, 1u, (WITH_MASS && valid) ? mass_of(s, m) : 0ull);
    }
  }
};

template <bool BY_MASS, bool WITH_MASS>
__device__ Selection descend(RowCtx& c, uint32_t lo_key, u64 target_cnt, float top_p, float m) {
  StageFill<WITH_MASS> fill{c.stage, c.n_local, m};
  return descend_core<BY_MASS, WITH_MASS>(c, fill, lo_key, target_cnt, top_p);
}

// Count and mass of all elements with key >= lo_key, cluster wide.
__device__ void totals_above(RowCtx& c, uint32_t lo_key, float m, bool with_mass, u64& cnt, u64& mass) {
  u64 a = 0, b = 0;
  for (int i = threadIdx.x; i < c.n_local; i += kThreads) {
    const float s = c.stage[i];
    if (key_of(s) >= lo_key) {
      ++a;
      if (with_mass) b += mass_of(s, m);
    }
  }
  block_sum2(*c.x, a, b);
  u64 vals[2] = {a, b}, got[2];
  c.exchange<2>(vals, got);
  cnt = warp_sum_u64(got[0]);
  mass = warp_sum_u64(got[1]);
}

// Global id of the t-th (1-based) element, in ascending id order, whose key equals `key`.
__device__ int find_tth_equal(RowCtx& c, uint32_t key, u64 t) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int w0 = warp * c.seg;
  const int w1 = min(w0 + c.seg, c.n_local);
  u64 mine = 0;
  for (int i = w0 + lane; i < w1; i += 32) mine += key_of(c.stage[i]) == key;
  const u64 wtot = warp_sum_u64(mine);
  u64 pre, pre_unused, tot, tot_unused;
  block_warp_prefix2(*c.x, wtot, 0, pre, pre_unused, tot, tot_unused);
  u64 vals[1] = {tot}, got[1];
  c.exchange<1>(vals, got);
  if (threadIdx.x == 0) c.x->bcast[6] = 0;
  __syncthreads();
  const u64 before = ranks_below(got[0], c.rank) + pre;
  if (before < t && t <= before + wtot) {  // this warp holds the t-th
    u64 running = before;
    for (int i0 = w0; i0 < w1; i0 += 32) {
      const int i = i0 + lane;
      const bool hit = i < w1 && key_of(c.stage[i]) == key;
      const uint32_t ballot = __ballot_sync(0xffffffffu, hit);
      const u64 n = __popc(ballot);
      if (running + n >= t) {
        const int nth = (int)(t - running);  // 1-based among set bits
        const int pos = __fns(ballot, 0, nth);
        if (lane == 0) c.x->bcast[6] = (u64)(c.base + i0 + pos) + 1;
        break;
      }
      running += n;
    }
  }
  __syncthreads();
  u64 v2[1] = {c.x->bcast[6]};
  c.exchange<1>(v2, got);
  const u64 found = warp_max_u64(got[0]);  // (id + 1, on the one rank that has it)
  return found ? (int)(found - 1) : 0x7fffffff;
}

// arg max over the kept set of fl(fl(e / z) / noise), lowest id on ties: what
// torch.multinomial(p, 1) computes on CPU from its Exp(1) variates.
__device__ int draw_with_noise(RowCtx& c, const KeptSet& kept, float m, float zf,
                               const float* noise_row) {
  u64 best = 0;
  for (int i = threadIdx.x; i < c.n_local; i += kThreads) {
    const float s = c.stage[i];
    const int gid = c.base + i;
    if (!kept.has(key_of(s), gid)) continue;
    const float p = __fdiv_rn(expf(s - m), zf);
    const float ratio = __fdiv_rn(p, noise_row[gid]);
    const u64 packed = ((u64)__float_as_uint(ratio) << 32) | (uint32_t)(~(uint32_t)gid);
    best = packed > best ? packed : best;
  }
  best = block_max_u64(*c.x, best);
  u64 vals[1] = {best}, got[1];
  c.exchange<1>(vals, got);
  best = warp_max_u64(got[0]);
  return (int)(~(uint32_t)(best & 0xffffffffu));
}


// Inverse CDF over the kept set in ascending id order: the first kept element at which the
// running integer mass exceeds `target` (0 <= target < total kept mass), or -1.  Thread t adds up
// elements [t, t + 1) * run of the slice (run is odd: the threads' reads fall on different banks);
// it first marks the kept ones of 32 at a time, so that a warp spends an exponential per kept
// element and not per element.  The warp that owns the run with the target in it looks into it.
__device__ int draw_inverse_cdf(RowCtx& c, const KeptSet& kept, float m, u64 target) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int run = ((c.n_local + kThreads - 1) / kThreads) | 1;
  const int r0 = min(tid * run, c.n_local), r1 = min(r0 + run, c.n_local);
  auto mass_at = [&](int i) -> u64 {
    const float s = c.stage[i];
    return kept.has(key_of(s), c.base + i) ? mass_of(s, m) : 0ull;
  };
  u64 mine = 0;
  for (int b = r0; b < r1; b += 32) {
    uint32_t marks = 0;
    const int n = min(32, r1 - b);
#pragma unroll 8
    for (int j = 0; j < n; ++j) marks |= (kept.has(key_of(c.stage[b + j]), c.base + b + j) ? 1u : 0u) << j;
    while (marks) {
      const int j = __ffs(marks) - 1;
      marks &= marks - 1;
      mine += mass_of(c.stage[b + j], m);
    }
  }
  const u64 incl = warp_scan_u64(mine);
  u64 pre, pu, tot, tu;
  block_warp_prefix2(*c.x, shfl_u64(incl, 31), 0, pre, pu, tot, tu);
  u64 vals[1] = {tot}, got[1];
  c.exchange<1>(vals, got);
  const u64 before = ranks_below(got[0], c.rank) + pre + incl - mine;
  if (tid == 0) c.x->bcast[6] = 0;
  __syncthreads();
  const uint32_t votes = __ballot_sync(0xffffffffu, before <= target && target < before + mine);
  if (votes) {  // (this warp owns it)
    const int owner = __ffs(votes) - 1;
    const int b = __shfl_sync(0xffffffffu, r0, owner), e = __shfl_sync(0xffffffffu, r1, owner);
    u64 running = shfl_u64(before, owner);
    for (int i0 = b; i0 < e; i0 += 32) {
      const int i = i0 + lane;
      const u64 in = warp_scan_u64(i < e ? mass_at(i) : 0ull);
      const uint32_t past = __ballot_sync(0xffffffffu, running + in > target);
      if (past) {
        if (lane == 0) c.x->bcast[6] = (u64)(c.base + i0 + __ffs(past) - 1) + 1;
        break;
      }
      running += shfl_u64(in, 31);
    }
  }
  __syncthreads();
  u64 v2[1] = {c.x->bcast[6]};
  c.exchange<1>(v2, got);
  return (int)warp_max_u64(got[0]) - 1;
}

// ---- the one histogram ------------------------------------------------------------------
struct ResHist {
  float lo, scale;  // bucket = (score - lo) * scale, clamped: grows with the score
  __device__ __forceinline__ int bucket(float s) const {
    return min(max(__float2int_rz((s - lo) * scale), 0), kResBuckets - 1);
  }
};
// Scores that can be in buckets [first, last], with a bucket's width to spare on either side: two
// comparisons instead of a bucket number per element.
struct ResRange {
  float from, to;
  __device__ __forceinline__ ResRange(const ResHist& h, int first, int last) {
    const float width = __fdiv_rn(1.0f, h.scale);
    from = first <= 0 ? __int_as_float(0xff800000) : h.lo + ((float)first - 1.0f) * width;
    to = last >= kResBuckets - 1 ? __int_as_float(0x7f800000) : h.lo + ((float)last + 2.0f) * width;
  }
  __device__ __forceinline__ bool near(float s) const { return !(s < from || s > to); }  // (a NaN may be)
};
struct BucketHit {
  int bucket;
  u64 above_cnt, above_mass, bin_cnt, bin_mass;
};
// Fills the merged histogram: afterwards rank r holds buckets [r, r + 1) * kResBuckets / nranks
// in red_cnt / red_mass, and lane r of every warp holds rank r's totals in `seg`.
__device__ void res_histogram(RowCtx& c, const ResHist& rh, float m, u64 (&seg)[2]) {
  uint32_t* cnt = reinterpret_cast<uint32_t*>(c.hist);
  const int tid = threadIdx.x;
  for (int b = tid; b < 3 * kResBuckets; b += kThreads) cnt[b] = 0;
  __syncthreads();
  auto take = [&](float s) {
    const int b = rh.bucket(s);
    atomicAdd(&cnt[b], 1u);
    const u64 q = mass_of(s, m);  // (0 from 28.4 below the maximum on)
    shared_add_u64(&cnt[kResBuckets + b], &cnt[2 * kResBuckets + b], q);
  };
  int i = tid;
  for (; i + 3 * kThreads < c.n_local; i += 4 * kThreads) {
    float s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = c.stage[i + u * kThreads];
#pragma unroll
    for (int u = 0; u < 4; ++u) take(s[u]);
  }
  for (; i < c.n_local; i += kThreads) take(c.stage[i]);
  c.sync_all();
  const int per = kResBuckets / (int)c.nranks;
  u64 tc = 0, tm = 0;
  for (int b = tid; b < per; b += kThreads) {
    const int gb = (int)c.rank * per + b;
    uint32_t n = 0;
    u64 q = 0;
#pragma unroll
    for (unsigned r = 0; r < (unsigned)kMaxCluster; ++r) {
      if (r >= c.nranks) break;
      const uint32_t* h = c.nranks > 1 ? c.cluster.map_shared_rank(cnt, r) : cnt;
      n += h[gb];
      q += (u64)h[kResBuckets + gb] | ((u64)h[2 * kResBuckets + gb] << 32);
    }
    c.red_cnt[b] = n;
    c.red_mass[b] = q;
    tc += n;
    tm += q;
  }
  block_sum2(*c.x, tc, tm);
  u64 vals[2] = {tc, tm};
  c.exchange<2>(vals, seg);
}
// The bucket, from the top, at which the running count (or mass) reaches `want` (>= 1, at most the
// total).  Every CTA works it out for itself; no barrier between CTAs.
template <bool BY_MASS>
__device__ BucketHit res_find(RowCtx& c, const u64 (&seg)[2], u64 want) {
  const int per = kResBuckets / (int)c.nranks, lane = threadIdx.x & 31;
  __syncthreads();
  if (threadIdx.x < 32) {
    // the rank: what lies above rank r is the total less the ranks up to r
    const u64 ic = warp_scan_u64(seg[0]), im = warp_scan_u64(seg[1]);
    const u64 over_c = shfl_u64(ic, 31) - ic, over_m = shfl_u64(im, 31) - im;
    const u64 over = BY_MASS ? over_m : over_c;
    const uint32_t here = __ballot_sync(0xffffffffu, over < want && want <= over + seg[BY_MASS ? 1 : 0]);
    const unsigned r = here ? (unsigned)(__ffs(here) - 1) : 0u;
    u64 ac = shfl_u64(over_c, (int)r), am = shfl_u64(over_m, (int)r);
    const uint32_t* rc = c.nranks > 1 ? c.cluster.map_shared_rank(c.red_cnt, r) : c.red_cnt;
    const u64* rm = c.nranks > 1 ? c.cluster.map_shared_rank(c.red_mass, r) : c.red_mass;
    // its buckets: lane l owns per / 32 consecutive ones (a multiple of four), the highest lane 0
    const int mine = per >> 5, first = per - mine * (lane + 1);
    u64 sn = 0, sq = 0;
    uint4 n4 = make_uint4(0, 0, 0, 0);
    ulonglong2 qa = make_ulonglong2(0, 0), qb = qa;
    for (int u = 0; u < mine; u += 4) {
      n4 = *reinterpret_cast<const uint4*>(rc + first + u);
      qa = *reinterpret_cast<const ulonglong2*>(rm + first + u);
      qb = *reinterpret_cast<const ulonglong2*>(rm + first + u + 2);
      sn += (u64)n4.x + n4.y + n4.z + n4.w;
      sq += qa.x + qa.y + qb.x + qb.y;
    }
    const u64 in = warp_scan_u64(sn), iq = warp_scan_u64(sq);
    const uint32_t votes = __ballot_sync(0xffffffffu, want <= (BY_MASS ? am + iq : ac + in));
    if (lane == __ffs(votes) - 1) {
      ac += in - sn;
      am += iq - sq;
      for (int u = mine - 4; u >= 0; u -= 4) {
        if (mine > 4) {  // (else the four are at hand)
          n4 = *reinterpret_cast<const uint4*>(rc + first + u);
          qa = *reinterpret_cast<const ulonglong2*>(rm + first + u);
          qb = *reinterpret_cast<const ulonglong2*>(rm + first + u + 2);
        }
        const uint32_t n[4] = {n4.x, n4.y, n4.z, n4.w};
        const u64 q[4] = {qa.x, qa.y, qb.x, qb.y};
        bool done = false;
#pragma unroll
        for (int k = 3; k >= 0; --k) {
          if (done) continue;
          if (want <= (BY_MASS ? am + q[k] : ac + n[k])) {
            c.x->bcast[0] = (u64)((int)r * per + first + u + k);
            c.x->bcast[1] = ac;
            c.x->bcast[2] = am;
            c.x->bcast[3] = n[k];
            c.x->bcast[4] = q[k];
            done = true;
          } else {
            ac += n[k];
            am += q[k];
          }
        }
        if (done) break;
      }
    }
  }
  __syncthreads();
  BucketHit h{(int)c.x->bcast[0], c.x->bcast[1], c.x->bcast[2], c.x->bcast[3], c.x->bcast[4]};
  __syncthreads();
  return h;
}

// The CTAs' lists (lane r of every warp holds the length of rank r's) one behind the other into
// dst: one remote read per entry, all side by side.
__device__ __forceinline__ void res_collect(RowCtx& c, u64* list, u64 len, int total, u64* dst) {
  for (int i0 = threadIdx.x & ~31; i0 < total; i0 += kThreads) {
    const int i = i0 + (threadIdx.x & 31);
    int at = i;
    unsigned r = 0;
    for (unsigned k = 0; k + 1 < c.nranks; ++k) {
      const int n = (int)shfl_u64(len, (int)k);
      if (r == k && at >= n) { at -= n; r = k + 1; }
    }
    if (i < total) dst[i] = (c.nranks > 1 ? c.cluster.map_shared_rank(list, r) : list)[at];
  }
}
// Entries in all lists (a list that ran over counts as very long).
__device__ __forceinline__ int res_total(u64 len) { return (int)warp_sum_u64(min(len, (u64)1 << 20)); }

// All elements `take(score)` names, from all slices, sorted by (score descending, id ascending), in
// every CTA's own copy; returns how many, or -1 when they are more than a list holds.  `first` =
// no gather has run since the last barrier between the CTAs.
template <class Take>
__device__ int res_gather(RowCtx& c, bool& first, Take&& take) {
  u64* list = reinterpret_cast<u64*>(reinterpret_cast<unsigned char*>(c.hist) + 16 * kResBuckets);
  u64* members = reinterpret_cast<u64*>(c.hist);
  int* n_at = reinterpret_cast<int*>(&c.x->bcast[7]);
  if (!first) c.sync_all();  // (another CTA may still be reading this one's list)
  first = false;
  if (threadIdx.x == 0) *n_at = 0;
  __syncthreads();
  for (int i0 = threadIdx.x; i0 < c.n_local; i0 += 4 * kThreads) {
    float s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = i0 + u * kThreads < c.n_local ? c.stage[i0 + u * kThreads] : 0.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * kThreads;
      if (i >= c.n_local || !take(s[u], c.base + i)) continue;
      const int slot = atomicAdd(n_at, 1);
      if (slot < kResList) list[slot] = cand_pack(key_of(s[u]), c.base + i);
    }
  }
  __syncthreads();
  u64 vals[1] = {(u64)*n_at}, len[1];
  c.exchange<1>(vals, len);
  const int total = res_total(len[0]);
  if (total > kResList) return -1;
  res_collect(c, list, len[0], total, members);
  __syncthreads();
  CandCtx L{members, nullptr, nullptr, nullptr, nullptr, nullptr};
  cand_sort(L, total);
  return total;
}

// Reads a cut off a sorted member list: the key at which the running count (or mass) of the
// members in `in` reaches want (counted from the list's top), and what lies above and at it.
template <bool BY_MASS, class In>
__device__ Selection res_resolve(RowCtx& c, int n, float m, u64 want, In&& in) {
  const u64* members = reinterpret_cast<const u64*>(c.hist);
  const int per = (n + kThreads - 1) / kThreads, i0 = min((int)threadIdx.x * per, n), i1 = min(i0 + per, n);
  u64 sum = 0;
  auto weight = [&](u64 e) -> u64 {
    if (!in(score_of(cand_key(e)))) return 0ull;
    return BY_MASS ? mass_of(score_of(cand_key(e)), m) : 1ull;
  };
  for (int i = i0; i < i1; ++i) sum += weight(members[i]);
  const u64 incl = warp_scan_u64(sum);
  u64 pre, pu, tot, tu;
  block_warp_prefix2(*c.x, shfl_u64(incl, 31), 0, pre, pu, tot, tu);
  Selection sel{};
  sel.target = want;
  sel.ok = want >= 1 && want <= tot;
  if (!sel.ok) return sel;
  u64 run = pre + incl - sum;
  if (run < want && want <= run + sum) {
    for (int i = i0; i < i1; ++i) {
      run += weight(members[i]);
      if (want <= run) { c.x->bcast[0] = (u64)cand_key(members[i]); break; }
    }
  }
  __syncthreads();
  sel.key = (uint32_t)c.x->bcast[0];
  u64 ac = 0, am = 0, bc = 0, bm = 0;
  for (int i = i0; i < i1; ++i) {
    const uint32_t k = cand_key(members[i]);
    if (k < sel.key || !in(score_of(k))) continue;
    const u64 q = mass_of(score_of(k), m);
    if (k > sel.key) { ++ac; am += q; } else { ++bc; bm += q; }
  }
  block_sum2(*c.x, ac, am);
  block_sum2(*c.x, bc, bm);
  sel.above_cnt = ac;
  sel.above_mass = am;
  sel.bin_cnt = bc;
  sel.bin_mass = bm;
  return sel;
}

// A lower bound of the slice's j-th highest score key (0 when it has no j groups): the threads'
// maxima are maxima of disjoint groups of tokens, so the j-th highest of them (or of the maxima
// over eight threads, where 64 groups are enough) bounds the j-th highest token from below.
__device__ uint32_t slice_bound(RowCtx& c, uint32_t thread_max, int j) {
  uint32_t* keys = reinterpret_cast<uint32_t*>(c.hist);  // (not in use yet)
  const int tid = threadIdx.x, lane = tid & 31;
  const bool coarse = j <= 32;
  uint32_t v = thread_max;
  if (coarse) {
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, d));
    if ((lane & 7) == 0) keys[tid >> 3] = v;
  } else {
    keys[tid] = v;
  }
  if (tid == 0) c.x->bcast[6] = 0;
  __syncthreads();
  const int n = coarse ? kThreads / 8 : kThreads;
  if (tid < n) {
    const uint32_t mine = keys[tid];
    int greater = 0, at_least = 0;
    for (int k = 0; k < n; k += 4) {
      const uint4 o = *reinterpret_cast<const uint4*>(keys + k);
      greater += (o.x > mine) + (o.y > mine) + (o.z > mine) + (o.w > mine);
      at_least += (o.x >= mine) + (o.y >= mine) + (o.z >= mine) + (o.w >= mine);
    }
    if (greater < j && j <= at_least) c.x->bcast[6] = (u64)mine;  // (equal keys write the same value)
  }
  __syncthreads();
  return (uint32_t)c.x->bcast[6];
}

// ---- the kernel -----------------------------------------------------------------------
// ON_CHIP: the slices are in shared memory (else in global scratch).
template <bool ON_CHIP>
__global__ void __launch_bounds__(kThreads, 2) row_kernel(const __grid_constant__ RowKernelArgs a,
                                                          const __grid_constant__ InlineRows inl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ hs_row_params P;
  __shared__ hs_row_out record;
  if (threadIdx.x == 0) P = row_params(a, inl, blockIdx.y);
  if (threadIdx.x < sizeof(hs_row_out) / 4) reinterpret_cast<uint32_t*>(&record)[threadIdx.x] = 0u;
  RowCtx c{{cg::this_cluster()}};
  c.rank = c.cluster.block_rank();
  c.nranks = c.cluster.num_blocks();
  c.row = blockIdx.y;
  c.vocab = a.vocab;
  c.slice = a.slice;
  c.base = (int)c.rank * a.slice;
  c.n_local = max(0, min(a.slice, a.vocab - c.base));
  c.seg = ((c.n_local + kThreads - 1) / kThreads) * 32;

  size_t off = 0;
  c.x = reinterpret_cast<Exchange*>(smem_raw + off);
  off += (sizeof(Exchange) + 15) & ~size_t(15);
  c.hist = reinterpret_cast<Hist*>(smem_raw + off);
  off += sizeof(Hist);
  c.red_mass = reinterpret_cast<u64*>(smem_raw + off);
  off += sizeof(u64) * (kBins / c.nranks);
  c.red_cnt = reinterpret_cast<uint32_t*>(smem_raw + off);
  off += sizeof(uint32_t) * (kBins / c.nranks);
  off = (off + 15) & ~size_t(15);
  unsigned char* on_chip = smem_raw + off;
  if constexpr (ON_CHIP) c.stage = reinterpret_cast<float*>(on_chip);
  else c.stage = a.gstage + (size_t)c.row * ((size_t)a.slice * c.nranks) + c.base;
  cudaGridDependencySynchronize();  // (the histograms are up to date from here on)
  __syncthreads();

  const int tid = threadIdx.x;
  const bool greedy = P.temperature == 0.0f;
  const bool candidate = is_candidate_row(P, a.vocab) && a.small_k != kSmallKOrder;
  if (candidate && a.small_k == kSmallKLeave) return;  // (all CTAs of the cluster alike)
  const bool slot_ok = P.slot >= 0 && P.slot < a.pool.slots_total;
  const bool penalised = slot_ok && (P.repetition_penalty != 1.0f || P.presence_penalty != 0.0f ||
                                     P.frequency_penalty != 0.0f);
  // (in registers: the compiler cannot know that storing a score leaves P alone)
  const float rp = P.repetition_penalty, pp = P.presence_penalty, fp = P.frequency_penalty;
  const float T = P.temperature;
  const bool divide = !greedy && T != 1.0f;
  auto score = [&](float v, int count) {
    if (count > 0) {
      v = v < 0.0f ? __fmul_rn(v, rp) : __fdiv_rn(v, rp);
      v = __fsub_rn(v, pp);
      v = __fsub_rn(v, __fmul_rn(fp, (float)count));
    }
    if (divide) v = __fdiv_rn(v, T);
    return canonical(v);
  };
  auto score_new = [&](float v) { return canonical_number(divide ? __fdiv_rn(v, T) : v); };  // (held never, no NaN)

  // ---- A. the one read of the row from HBM, scored ------------------------------------
  uint32_t top_key = 0, low_key = 0xffffffffu;  // over this thread's elements
  int top_at = 0;                               // (the lowest with the highest key)
  auto note = [&](float s, int i) {
    const uint32_t k = key_of(s);
    if (k > top_key) { top_key = k; top_at = i; }  // (a thread's elements come in ascending order)
    low_key = min(low_key, k);
  };
  {
    const uint32_t* cls = penalised ? a.pool.cls + (size_t)P.slot * a.pool.cls_stride : nullptr;
    const long long gofs = (long long)c.row * a.row_stride + c.base;
    auto put = [&](float x, uint32_t cc, int i) {
      if (cc == 3u) { c.stage[i] = x; return; }  // (held three times or more: scored below, with its count)
      float v = score(x, (int)cc);
      if (candidate && v != v) v = __int_as_float(0xff800000);  // (a NaN is never a candidate)
      c.stage[i] = v;
      note(v, i);
    };
    // four neighbours at once: the common case (none of them in the history, no NaN) without a
    // branch per token, one 128-bit store
    auto put4 = [&](const float4& w, uint32_t cl, int i) {
      if ((cl & 0xffu) == 0u) {
        const float4 v = make_float4(score_new(w.x), score_new(w.y), score_new(w.z), score_new(w.w));
        const uint32_t k0 = key_of(v.x), k1 = key_of(v.y), k2 = key_of(v.z), k3 = key_of(v.w);
        const uint32_t hi = max(max(k0, k1), max(k2, k3)), lo = min(min(k0, k1), min(k2, k3));
        if (hi <= 0xff800000u && lo >= 0x007fffffu) {  // (keys of +inf and -inf)
          *reinterpret_cast<float4*>(c.stage + i) = v;
          low_key = min(low_key, lo);
          if (hi > top_key) {
            top_key = hi;
            top_at = i + (k0 == hi ? 0 : (k1 == hi ? 1 : (k2 == hi ? 2 : 3)));
          }
          return;
        }
      }
      put(w.x, cl & 3u, i); put(w.y, (cl >> 2) & 3u, i + 1); put(w.z, (cl >> 4) & 3u, i + 2); put(w.w, (cl >> 6) & 3u, i + 3);
    };
    if (a.dtype == HS_DTYPE_BF16) {
      const unsigned short* src = reinterpret_cast<const unsigned short*>(a.logits) + gofs;
#pragma unroll 4
      for (int i = tid; i < c.n_local; i += kThreads) {
        const int id = c.base + i;
        const uint32_t cc = cls ? (__ldcg(cls + (id >> 4)) >> ((id & 15) * 2)) & 3u : 0u;
        put(__uint_as_float((uint32_t)__ldcs(src + i) << 16), cc, i);
      }
    } else {
      const float* src = reinterpret_cast<const float*>(a.logits) + gofs;
      const bool vec = (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
      const int n4 = vec ? c.n_local / 4 : 0;
      const float4* src4 = reinterpret_cast<const float4*>(src);
      constexpr int kFlight = 6;  // 128-bit loads in flight per thread
      for (int i0 = tid; i0 < n4; i0 += kFlight * kThreads) {
        float4 w[kFlight];
        uint32_t cl[kFlight];
#pragma unroll
        for (int u = 0; u < kFlight; ++u) {
          const int i = i0 + u * kThreads;
          cl[u] = 0u;
          if (i < n4) {
            w[u] = __ldcs(src4 + i);
            const int id = c.base + 4 * i;  // (a multiple of four: the classes share a word)
            if (cls) cl[u] = __ldcg(cls + (id >> 4)) >> ((id & 15) * 2);
          }
        }
#pragma unroll
        for (int u = 0; u < kFlight; ++u) {
          const int i = i0 + u * kThreads;
          if (i >= n4) break;
          put4(w[u], cl[u], 4 * i);
        }
      }
#pragma unroll 8
      for (int i = n4 * 4 + tid; i < c.n_local; i += kThreads) {
        const int id = c.base + i;
        put(__ldcs(src + i), cls ? (__ldcg(cls + (id >> 4)) >> ((id & 15) * 2)) & 3u : 0u, i);
      }
    }
    if (penalised) {
      __syncthreads();
      const int n_heavy = min(a.pool.n_heavy[P.slot], a.pool.unique_cap);
      const int32_t* heavy = a.pool.heavy + (size_t)P.slot * a.pool.unique_cap;
      const int2* pairs = a.pool.pairs + (size_t)P.slot * a.pool.unique_cap;
      for (int j = tid; j < n_heavy; j += kThreads) {
        const int q = heavy[j];
        if (q < 0 || q >= a.pool.unique_cap) continue;
        const int2 e = pairs[q];  // (id, count)
        const int i = e.x - c.base;
        if (i < 0 || i >= c.n_local) continue;
        float v = score(c.stage[i], e.y);
        if (candidate && v != v) v = __int_as_float(0xff800000);
        c.stage[i] = v;
        // (these come in any order: an equal score at a lower id takes the place)
        if (key_of(v) == top_key) top_at = min(top_at, i);
        note(v, i);
      }
    }
  }

  // ---- B. row maximum, arg max, minimum -----------------------------------------------
  u64 best = c.n_local ? ((u64)top_key << 32) | (uint32_t)(~(uint32_t)(c.base + top_at)) : 0ull;
  if (top_key == 0) best = 0;
  best = block_max_u64(*c.x, best);
  low_key = ~block_max_u32(*c.x, ~low_key);
  uint32_t bound = 0;
  if (candidate) bound = slice_bound(c, top_key, (P.top_k + (int)c.nranks - 1) / (int)c.nranks);
  {
    u64 vals[3] = {best, (u64)low_key, (u64)bound}, got[3];
    c.exchange<3>(vals, got);
    best = warp_max_u64(got[0]);
    low_key = (uint32_t)ranks_min(got[1], c.nranks);
    bound = (uint32_t)ranks_min(got[2], c.nranks);
  }
  const uint32_t max_key = (uint32_t)(best >> 32);
  const int argmax_id = (int)(~(uint32_t)(best & 0xffffffffu));
  const float m = score_of(max_key);
  int status = P.slot >= a.pool.slots_total ? 64 : 0;  // a slot this sampler does not have: no penalties
  hs_row_out* out = record_of(a, c.row);

  // ---- C. rows with a small top_k -----------------------------------------------------
  if (candidate) {
    u64* list = reinterpret_cast<u64*>(c.hist);
    int* n_at = reinterpret_cast<int*>(&c.x->bcast[7]);
    u64 len[1];
    int total = 0;
    for (int attempt = 0; attempt < 2; ++attempt) {
      if (tid == 0) *n_at = 0;
      __syncthreads();
      for (int i0 = tid; i0 < c.n_local; i0 += 4 * kThreads) {
        uint32_t k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) k[u] = i0 + u * kThreads < c.n_local ? key_of(c.stage[i0 + u * kThreads]) : 0u;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = i0 + u * kThreads;
          if (i >= c.n_local || k[u] < bound) continue;
          const int slot = atomicAdd(n_at, 1);
          if (slot < kCandCap) list[slot] = cand_pack(k[u], c.base + i);
        }
      }
      __syncthreads();
      u64 vals[1] = {(u64)*n_at};
      c.exchange<1>(vals, len);
      total = res_total(len[0]);
      if (total <= kCandCap || attempt == 1) break;
      // (values that lie unevenly over the slices: once more from the exact k-th highest key)
      const Selection sk = descend<false, false>(c, 0u, (u64)P.top_k, 1.0f, m);
      bound = sk.ok ? sk.key : 0u;
      c.sync_all();
    }
    if (total <= kCandCap) {
      if (c.rank == 0) {
        u64* merged = reinterpret_cast<u64*>(on_chip);  // (the slice has served)
        __syncthreads();
        res_collect(c, list, len[0], total, merged);
      }
      c.sync_all();  // (the lists have been read: the other CTAs may leave)
      if (c.rank != 0) return;
      int* small = reinterpret_cast<int*>(c.red_mass);
      CandCtx L{reinterpret_cast<u64*>(on_chip), small, small + 1, reinterpret_cast<uint32_t*>(c.hist), small + 2, nullptr};
      int n = total;
      u64* mass = reinterpret_cast<u64*>(on_chip) + kCandCap;
      n = cand_keep_sorted(L, mass, n, n > P.top_k && n > kSortAll ? cand_kth_key(*c.x, L, n, P.top_k) : 0u);
      if (n > P.top_k) {
        // a list that was sorted whole: top-k keeps the first k entries and the ties of the k-th
        const uint32_t cut = cand_key(L.cand[P.top_k - 1]);
        u64 keep = 0, unused = 0;
        for (int i = tid; i < n; i += kThreads) keep += cand_key(L.cand[i]) >= cut ? 1 : 0;
        block_sum2(*c.x, keep, unused);
        n = (int)keep;
      }
      const float* noise_row = a.noise ? a.noise + (size_t)c.row * a.vocab : nullptr;
      FinishOut r = finish_sorted(*c.x, L.cand, mass, n, P, noise_row, &record);
      r.status |= status;
      if (a.scores_out) {
        float* dst = a.scores_out + (size_t)c.row * a.vocab;
        for (int id = tid; id < c.vocab; id += kThreads) dst[id] = __int_as_float(0xff800000);
        __syncthreads();
        for (int i = tid; i < (int)r.n_kept; i += kThreads) dst[cand_id(L.cand[i])] = score_of(cand_key(L.cand[i]));
      }
      if (tid == 0) {
        write_finish(r, &record);
        if (a.tokens_out) a.tokens_out[c.row] = r.token;
        if ((a.flags & HS_SAMPLE_APPEND_TOKEN) && slot_ok && r.token >= 0 && r.token < a.vocab) {
          if (!slot_append_one(a.pool, P.slot, r.token)) record.status = r.status | 2;
        }
      }
      __syncthreads();
      if (tid < 32) write_record(out, record, P.n_logprobs >= 0, mail_of(a, c.row), a.mail_tag);
      return;
    }
    // more ties at the k-th value than a list holds: in token order, like any other row
    c.sync_all();
  }

  // ---- D. the other rows --------------------------------------------------------------
  KeptSet kept{0u, 0x7fffffff};
  int token = argmax_id;
  u64 n_topk = (u64)a.vocab, n_minp = (u64)a.vocab, n_kept = (u64)a.vocab;
  u64 q_kept = 0;
  long long cut_ties = -1;
  const int n_want_all = P.n_logprobs >= 0 ? min(P.n_logprobs, a.vocab) : 0;
  int n_top_list = -1;  // members gathered for the log-probabilities, sorted; -1 = not yet

  if (!greedy || P.n_logprobs >= 0) {
    ResHist rh;
    rh.lo = fmaxf(score_of(low_key), m - 30.0f);
    const float range = m - rh.lo;
    bool hist_ok = range > 0.f && range < 3.0e38f;
    rh.scale = hist_ok ? __fdiv_rn((float)kResBuckets - 0.5f, range) : 0.f;
    u64 seg[2] = {0, 0};
    u64 cnt = 0, mass = 0;
    bool first = true;
    if (hist_ok) {
      res_histogram(c, rh, m, seg);
      cnt = warp_sum_u64(seg[0]);
      mass = warp_sum_u64(seg[1]);
    } else {
      totals_above(c, 0u, m, true, cnt, mass);
    }
    // the bucket that holds the last of the top-N
    int top_bucket = kResBuckets;
    if (hist_ok && n_want_all > 0) top_bucket = res_find<false>(c, seg, (u64)n_want_all).bucket;
    // A cut: by the histogram and the members of one bucket; by radix descents when that bucket
    // is too full (they take the histogram's place).  lo_key: only elements from there up count.
    auto select_cut = [&](auto by_mass, u64 want, float top_p, uint32_t lo_key) -> Selection {
      constexpr bool BY_MASS = decltype(by_mass)::value;
      if (hist_ok) {
        const BucketHit h = res_find<BY_MASS>(c, seg, want);
        const bool with_top = BY_MASS;  // (the last cut: the top-N come along in the same gather)
        const ResRange range_of(rh, h.bucket, with_top && top_bucket < kResBuckets ? kResBuckets - 1 : h.bucket);
        const int n = res_gather(c, first, [&](float s, int) {
          if (!range_of.near(s)) return false;
          const int b = rh.bucket(s);
          return (b == h.bucket && key_of(s) >= lo_key) || (with_top && b >= top_bucket);
        });
        if (n >= 0) {
          Selection sel = res_resolve<BY_MASS>(c, n, m, want - (BY_MASS ? h.above_mass : h.above_cnt), [&](float s) {
            return rh.bucket(s) == h.bucket && key_of(s) >= lo_key;
          });
          sel.above_cnt += h.above_cnt;
          sel.above_mass += h.above_mass;
          sel.target = want;
          if (with_top && n_want_all > 0) n_top_list = n;
          if (sel.ok) {
            // the t-th tie by ascending id, should top-p split the group: the list is sorted
            if (BY_MASS && sel.bin_cnt > 0) {
              const u64 qv = sel.bin_mass / sel.bin_cnt;
              u64 t = qv > 0 ? (want - sel.above_mass + qv - 1) / qv : sel.bin_cnt;
              t = min(max(t, (u64)1), sel.bin_cnt);
              if (t < sel.bin_cnt) {
                const u64* members = reinterpret_cast<const u64*>(c.hist);
                if (tid == 0) c.x->bcast[5] = 0x7fffffff;
                __syncthreads();
                for (int i = tid; i < n; i += kThreads)
                  if (cand_key(members[i]) == sel.key && (i == 0 || cand_key(members[i - 1]) != sel.key))
                    c.x->bcast[5] = (u64)cand_id(members[i + (int)t - 1]);
                __syncthreads();
                kept.tie_limit = (int)c.x->bcast[5];
                __syncthreads();
              }
            }
            return sel;
          }
        }
        hist_ok = false;
        n_top_list = -1;
        c.sync_all();
      }
      Selection sel = descend<BY_MASS, true>(c, lo_key, want, top_p, m);
      if (BY_MASS && sel.ok && sel.bin_cnt > 0) {
        const u64 qv = sel.bin_mass / sel.bin_cnt;
        u64 t = qv > 0 ? (sel.target - sel.above_mass + qv - 1) / qv : sel.bin_cnt;
        t = min(max(t, (u64)1), sel.bin_cnt);
        if (t < sel.bin_cnt) kept.tie_limit = find_tth_equal(c, sel.key, t);
      }
      return sel;
    };

    if (!greedy) {
      if (P.top_k > 0 && P.top_k < a.vocab) {
        const Selection sk = select_cut(std::integral_constant<bool, false>{}, (u64)P.top_k, 1.0f, 0u);
        if (!sk.ok) status |= 1;
        kept.cut_key = sk.key;
        if (sk.ok) { cnt = sk.above_cnt + sk.bin_cnt; mass = sk.above_mass + sk.bin_mass; }
        n_topk = sk.above_cnt + sk.bin_cnt;
      }
      if (P.min_p > 0.0f) {
        const float z1 = mass_to_float(mass);
        const float thr = __fmul_rn(__fdiv_rn(1.0f, z1), P.min_p);
        uint32_t lowest = 0xffffffffu;
        for (int i = tid; i < c.n_local; i += kThreads) {
          const float s = c.stage[i];
          const uint32_t k = key_of(s);
          if (k >= kept.cut_key && k < lowest && !(__fdiv_rn(expf(s - m), z1) < thr)) lowest = k;
        }
        lowest = ~block_max_u32(*c.x, ~lowest);
        u64 vals[1] = {(u64)lowest}, got[1];
        c.exchange<1>(vals, got);
        lowest = (uint32_t)ranks_min(got[0], c.nranks);
        first = true;
        if (lowest != 0xffffffffu && lowest > kept.cut_key) {
          kept.cut_key = lowest;
          totals_above(c, kept.cut_key, m, true, cnt, mass);
        }
      }
      n_minp = cnt;
      if (P.top_p < 1.0f) {
        const u64 target = top_p_target_warp(mass, P.top_p);
        Selection sp{};
        if (mass > 0) sp = select_cut(std::integral_constant<bool, true>{}, target, P.top_p, kept.cut_key);
        if (mass > 0 && sp.ok && sp.bin_cnt > 0) {
          const u64 qv = sp.bin_mass / sp.bin_cnt;  // all elements of the bin share one score
          u64 t = sp.bin_cnt;
          if (qv > 0) {
            const u64 need = sp.target - sp.above_mass;
            t = (need + qv - 1) / qv;
            if (t < 1) t = 1;
            if (t > sp.bin_cnt) t = sp.bin_cnt;
          }
          kept.cut_key = sp.key;
          cnt = sp.above_cnt + t;
          mass = sp.above_mass + t * qv;
          cut_ties = (long long)t;
        } else {
          status |= 1;
        }
      }
      n_kept = cnt;
    }
    q_kept = mass;

    // ---- log-probabilities: the first n_want members of the sorted list ---------------
    if (n_want_all > 0 && n_top_list < 0) {
      const int n_want = (int)min((u64)n_want_all, n_kept);
      if (hist_ok) {
        const ResRange range_of(rh, top_bucket, kResBuckets - 1);
        n_top_list = res_gather(c, first, [&](float s, int) { return range_of.near(s) && rh.bucket(s) >= top_bucket; });
      }
      if (n_top_list < 0) {
        hist_ok = false;
        c.sync_all();
        const Selection sn = descend<false, false>(c, kept.cut_key, (u64)n_want, 1.0f, m);
        if (sn.ok) {
          const int last = find_tth_equal(c, sn.key, (u64)n_want - sn.above_cnt);
          first = true;
          n_top_list = res_gather(c, first, [&](float s, int id) {
            const uint32_t k = key_of(s);
            return k > sn.key || (k == sn.key && id <= last);
          });
        }
        if (n_top_list < 0) status |= 1;
      }
    }
  }

  // ---- E. draw ------------------------------------------------------------------------
  if (!greedy) {
    if (q_kept == 0) {
      token = argmax_id;
      status |= 1;
    } else if (a.noise) {
      token = draw_with_noise(c, kept, m, mass_to_float(q_kept), a.noise + (size_t)c.row * a.vocab);
    } else {
      const Philox4 r = philox4x32_10(0u, 0u, 0u, 0u, (uint32_t)P.seed, (uint32_t)(P.seed >> 32));
      const u64 r64 = ((u64)r.v[0] << 32) | r.v[1];
      token = draw_inverse_cdf(c, kept, m, __umul64hi(r64, q_kept));
      if (token < 0) { token = argmax_id; status |= 1; }
    }
  }

  // ---- F. optional dump of the final scores (parity tests) ------------------------------
  if (a.scores_out) {
    float* dst = a.scores_out + (size_t)c.row * a.vocab + c.base;
    for (int i = tid; i < c.n_local; i += kThreads) {
      const float s = c.stage[i];
      dst[i] = (greedy || kept.has(key_of(s), c.base + i)) ? s : __int_as_float(0xff800000);
    }
  }

  // ---- G. the record, by the CTA that holds the token -----------------------------------
  if (c.rank == (unsigned)(token / a.slice)) {
    float log_z = 0.f;
    if (P.n_logprobs >= 0) {
      log_z = (float)(log((double)q_kept) - (double)kMassShift * 0.6931471805599453);
      const int n_want = n_top_list < 0 ? 0 : (int)min((u64)n_want_all, n_kept);
      const u64* members = reinterpret_cast<const u64*>(c.hist);
      if (tid < n_want) {
        record.top_ids[tid] = cand_id(members[tid]);
        record.top_logprobs[tid] = (score_of(cand_key(members[tid])) - m) - log_z;
      }
      if (tid == 0) {
        record.logprob = (c.stage[token - c.base] - m) - log_z;
        record.n_top = n_want;
      }
    }
    if (tid == 0) {
      record.token = token;
      record.status = status;
      record.n_kept = (int32_t)n_kept;
      record.n_after_topk = (int32_t)n_topk;
      record.n_after_minp = (int32_t)n_minp;
      record.n_after_topp = (int32_t)n_kept;
      record.cut_bits = __float_as_uint(score_of(kept.cut_key));
      record.n_cut_ties = (int32_t)cut_ties;
      record.row_max = m;
      record.log_z = log_z;
      if (a.tokens_out) a.tokens_out[c.row] = token;
      if ((a.flags & HS_SAMPLE_APPEND_TOKEN) && slot_ok && token >= 0 && token < a.vocab) {
        if (!slot_append_one(a.pool, P.slot, token)) record.status = status | 2;
      }
    }
    __syncthreads();
    if (tid < 32) write_record(out, record, P.n_logprobs >= 0, mail_of(a, c.row), a.mail_tag);
  }
  // No CTA may leave while a peer can still read its shared memory.
  c.sync_all();
}

}  // namespace hs
