// The fused per-row sampling kernel for bf16 logits (the serving default): one CTA per row.
//
// Everything the sampler needs to know about a bf16 row fits in COUNTS.  A token's final
// score is a function of its raw bf16 value and of how often the request's history holds
// it, so tokens fall into classes (count class c in {0, 1, 2}, value bin b), and all tokens
// of a class share one score and one probability mass.  The kernel streams the row from
// HBM once, 128 bits at a time, together with the request's dense 2-bit count classes
// (V/4 bytes), and counts tokens per class with shared-memory atomics: three tables of
// 6,144 one-value bins (2^-14 <= |x| < 2^10).  The few tokens that do not fit a class --
// history count >= 3 (listed per request), or a value outside the bin window -- become
// individual (id, score) entries of a small side list.
//
// Selection (top-k by count, min-p by threshold, top-p by probability mass, top-N for the
// log-probabilities) needs ONE pass over the count table: a histogram of count and mass over 1,024
// buckets of equal width in score.  Every cut names a bucket from the top, and the bucket's members
// are resolved exactly against one another; a bucket with too many members is spread over 1,024
// again.  Probability mass is an integer multiple of 2^-40, so all sums are exact and
// order-independent.
//
// Token ids are only needed at the very end ("a uniformly chosen member of this class",
// "the lowest ids of this tie group").  A class of more than kV3RejectMin tokens is sampled by
// rejection: Philox-drawn positions are probed until one belongs to the class (exactly
// uniform over its members); a lone CTA issues scattered reads slowly, so a smaller class,
// or one the probes keep missing, is found by scanning the row once more for its bit
// pattern.  Lowest-id tie-breaks walk the row hierarchically.
//
// A row's CTA keeps the count table, the histogram and a short side list in shared memory, 112.3 KB, so
// that two CTAs share an SM and one row's barrier-bound selection phases overlap another row's
// counting.  What is left of L1 is small, so the streaming loads go past it.
#pragma once

#include "hs_common.cuh"
#include "hs_select.cuh"
#include "hs_state.cuh"
#include "hs_row_args.cuh"
#include "../../include/hs_sampler.h"

namespace hs {

constexpr int kV3Half = 3072;                 // 24 binades x 128 mantissas
constexpr int kV3Bins = 2 * kV3Half;          // per count class
constexpr int kCells = 3 * kV3Bins;           // count classes 0, 1, 2
constexpr uint32_t kV3Base = 113u << 7;       // smallest binned magnitude: 2^-14
constexpr int kV3ListCap = 256;               // members of a bucket resolved against one another; top-N ids
constexpr int kV3RejectMin = 128;             // classes of up to this many tokens are found by scanning the row, larger ones by rejection
constexpr int kV3ScanCap = 1024;              // ids one class scan can hold
constexpr int kV3TieCap = 1536;               // token ids ranked in shared memory
constexpr int kV3Buckets = 1024;              // of a selection's histogram
constexpr int kV3Staged = 7168;               // (class, count) entries of a hand-over staged in shared memory
constexpr uint32_t kMostHanded = 0x1fffe;     // highest count of one such entry (17 bits beside a 15-bit class)
// Room for a part's list: an entry for every cell, and those a part of the widest row (eight slices) adds by
// counts above kMostHanded.
constexpr int kHandedCap = (kCells + kMaxCluster * kMaxSliceElems / (int)kMostHanded + 3) & ~3;
#ifndef HS_RARE_CAP
#define HS_RARE_CAP 512
#endif
#ifndef HS_SIDE_SHARED
#define HS_SIDE_SHARED 1024
#endif
constexpr int kV3RareCap = HS_RARE_CAP;               // out-of-window tokens remembered before a sweep
constexpr int kV3SideShared = HS_SIDE_SHARED;           // side-list entries kept in shared memory (else global scratch)
constexpr int kV3PhaseSlots = 64;
#ifndef HS_DEFER_CAP
#define HS_DEFER_CAP 2048
#endif
constexpr int kV3DeferCap = HS_DEFER_CAP;             // chunks the counting loop sets aside for the token-by-token pass
constexpr int kSplitCap = 4096;               // candidate entries one CTA of a split row can hand over

struct V3Entry {
  uint32_t key;  // 32-bit key of the score
  int32_t id;    // token id
};
// A member of a selection's deciding bucket: a class or a side element.
struct __align__(16) V3Member {
  uint32_t key, cnt;
  u64 w;  // mass of all its tokens
};

struct RowV3Args {
  RowKernelArgs base;
  int2* s_pair;   // [n_scratch, s_cap] side lists too long for shared memory: (token id or -1, fp32 bits of the score)
  int s_cap;
  int n_scratch;       // scratch sets: as many as CTAs of the kernel can be resident at once
  int* scratch_busy;   // [n_scratch] 1 while a CTA holds the set
  unsigned long long* phase_clocks;  // [batch, kV3PhaseSlots] or null
  int csplit;                        // CTAs per row on the counting path
  uint32_t* ctab;                    // [batch, csplit, kHandedCap] classes and counts handed over by the parts of a row
  int2* crare;                       // [batch, csplit, kV3RareCap] their rare lists
  int2* crare_n;                     // [batch, csplit] (classes, rare tokens)
  int* count_ticket;                 // [batch] arrival counter (returns to 0)
  int split;                         // CTAs per row on the candidate path
  unsigned long long* split_lists;   // [batch, split, kSplitCap] candidate lists of the row's CTAs
  int* split_n;                      // [batch, split] their lengths
  int* split_ticket;                 // [batch] arrival counter (returns to 0)
  int batch;                         // rows in the launch
};

// Shared memory of a counting row.  What only the counting needs (rare tokens, set-aside chunks, the
// staged hand-over) and what only the selections need (histogram, members, token ids) share a place.
constexpr size_t kStateBytes = 1024;  // CountState
struct LayoutV3 {
  size_t x, state, tab, side, hist, members, list, staged, rare, defer, small, total;
};
__host__ __device__ constexpr LayoutV3 layout_v3() {
  LayoutV3 l{};
  size_t off = 0;
  auto take = [&off](size_t bytes) {
    const size_t at = off;
    off = (off + bytes + 15) & ~size_t(15);
    return at;
  };
  l.x = take(sizeof(Exchange));
  l.state = take(kStateBytes);
  l.tab = take(sizeof(uint32_t) * kCells);
  l.side = take(sizeof(int2) * kV3SideShared);
  l.staged = take(sizeof(uint32_t) * kV3Staged);
  l.rare = l.staged;
  l.defer = l.rare + sizeof(int2) * kV3RareCap;
  l.hist = l.staged;
  l.members = l.hist + sizeof(uint32_t) * 3 * kV3Buckets;
  l.list = l.members + sizeof(V3Member) * kV3ListCap;
  l.small = take(sizeof(int) * 64);
  l.total = off;
  return l;
}
constexpr LayoutV3 kLayV3 = layout_v3();
constexpr int kPerClass = kV3Bins / kThreads;  // a thread's cells tid + u * kThreads: count class u / kPerClass
static_assert(kV3Bins % kThreads == 0, "a thread's u-th cell has the same count class for all threads");
static_assert(sizeof(uint32_t) * (3 * kV3Buckets + kV3TieCap) + sizeof(V3Member) * kV3ListCap <= sizeof(uint32_t) * kV3Staged &&
              sizeof(int2) * kV3RareCap + sizeof(int) * kV3DeferCap <= sizeof(uint32_t) * kV3Staged,
              "the two uses fit the shared place");

// Chunks of eight tokens a part of a counting row takes (the last one takes what is left): an even number, so
// that the count classes of every part start on a whole word.
__device__ __forceinline__ int chunks_per_part(int n8, int parts) { return ((n8 + parts - 1) / parts + 1) & ~1; }

__device__ __forceinline__ int v3_bin_of_raw(uint32_t raw) {
  const uint32_t idx = (raw & 0x7fffu) - kV3Base;
  if (idx >= (uint32_t)kV3Half) return -1;
  return (raw & 0x8000u) ? kV3Half - 1 - (int)idx : kV3Half + (int)idx;
}
__device__ __forceinline__ uint32_t v3_raw_of_bin(int b) {
  return b >= kV3Half ? (uint32_t)(b - kV3Half) + kV3Base
                      : 0x8000u | ((uint32_t)(kV3Half - 1 - b) + kV3Base);
}

// What turns a token's raw value and count into its score.
struct Scorer {
  float T, rp, pp, fp;
  bool greedy;
  template <bool NUMBER = false>
  __device__ __forceinline__ float score_of_value(float v) const {
    if (!greedy && T != 1.0f) v = __fdiv_rn(v, T);
    return NUMBER ? canonical_number(v) : canonical(v);
  }
  // score of a token with raw value bits `raw` (NUMBER: not a NaN's) that the history holds `count` times
  template <bool NUMBER = false>
  __device__ __forceinline__ float score_of(uint32_t raw, int count) const {
    float v = __uint_as_float(raw << 16);  // (a zero's sign goes at the end)
    if (count > 0) {
      if (rp != 1.0f) v = v < 0.0f ? __fmul_rn(v, rp) : __fdiv_rn(v, rp);
      v = __fsub_rn(v, pp);
      v = __fsub_rn(v, __fmul_rn(fp, (float)count));
    }
    return score_of_value<NUMBER>(v);
  }
  // score of a bin of count class k, and of a cell
  __device__ __forceinline__ float bin_score(int bin, int k) const { return score_of<true>(v3_raw_of_bin(bin), k); }
  __device__ __forceinline__ float cell_score(int cell) const {
    const int c = cell / kV3Bins;
    return bin_score(cell - c * kV3Bins, c);
  }
};
template <size_t AT, class T>
__device__ __forceinline__ T* at_smem() {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return reinterpret_cast<T*>(smem_raw + AT);
}
struct Ctx3 : Scorer {
  // (places in shared memory; the block primitives' scratch comes first in every kernel's layout)
  __device__ __forceinline__ Exchange* x() const { return at_smem<0, Exchange>(); }
  __device__ __forceinline__ uint32_t* tab() const { return at_smem<kLayV3.tab, uint32_t>(); }     // [kCells] tokens per class
  __device__ __forceinline__ uint32_t* hist() const { return at_smem<kLayV3.hist, uint32_t>(); }   // [3 * kV3Buckets] count, mass as low and high words
  __device__ __forceinline__ V3Member* members() const { return at_smem<kLayV3.members, V3Member>(); }  // [kV3ListCap] of a selection's deciding bucket
  __device__ __forceinline__ V3Entry* gbuf() const { return at_smem<kLayV3.members, V3Entry>(); }  // [kV3ListCap] top-N tokens (in the same place)
  __device__ __forceinline__ int* list() const { return at_smem<kLayV3.list, int>(); }             // [kV3TieCap] token ids
  __device__ __forceinline__ int2* rare() const { return at_smem<kLayV3.rare, int2>(); }           // [kV3RareCap] (id, raw bits | count class << 16)
  __device__ __forceinline__ int2* side() const { return at_smem<kLayV3.side, int2>(); }           // [kV3SideShared]
  // (of the small counters: 0 gbuf_n, 1 rare_n, 2 side_n, 3 low id / ties, 8..11 thresholds, 14 ticket,
  // 16..21 ends, 22 lowest side key, 24..25 step_n, 27 defer_n, 30..31 span, 40..45 range, 48..63 warps)
  __device__ __forceinline__ int* gbuf_n() const { return at_smem<kLayV3.small, int>(); }
  __device__ __forceinline__ int* step_n() const { return at_smem<kLayV3.small, int>() + 24; }     // [2] of a scan
  __device__ __forceinline__ uint32_t* span() const { return at_smem<kLayV3.small, uint32_t>() + 30; }  // lowest and highest key of a deciding bucket
  __device__ __forceinline__ int* range() const { return at_smem<kLayV3.small, int>() + 40; }      // [6] of for_classes_at
  __device__ __forceinline__ int* ends() const { return at_smem<kLayV3.small, int>() + 16; }       // [6] per count class: highest non-empty cell + 1 (0 = none), lowest
  int row, vocab;
  int lo, hi;                    // token range this CTA streams in the candidate path ...
  int chunk_lo, chunk_hi;        // ... and the whole chunks in it
  const unsigned short* logits;  // this row
  const uint32_t* cls;           // this row's 2-bit classes, or null (no penalties)
  // The row in 16-byte chunks of eight tokens: a row may start anywhere (an odd vocabulary shifts
  // every row by another two bytes), so the first `head` tokens (at most seven) lie before the
  // first 16-byte boundary, n8 whole chunks follow, and the rest lies behind them.  Chunk i holds
  // tokens head + 8 i to head + 8 i + 7; the up to fourteen others are "loose".
  // (Worked out from the pointer where it is needed.)
  __device__ __forceinline__ void set_row(const void* all_logits, long long row_stride) {
    logits = reinterpret_cast<const unsigned short*>(all_logits) + (long long)row * row_stride;
  }
  __device__ __forceinline__ int head() const {
    return min((int)((0u - (uint32_t)reinterpret_cast<uintptr_t>(logits)) & 15u) >> 1, vocab);
  }
  __device__ __forceinline__ int n8() const { return (vocab - head()) >> 3; }
  __device__ __forceinline__ const uint4* chunks() const { return reinterpret_cast<const uint4*>(logits + head()); }
  __device__ __forceinline__ int first_of(int chunk) const { return head() + 8 * chunk; }
  __device__ __forceinline__ int n_loose() const { return vocab - 8 * n8(); }
  __device__ __forceinline__ int loose(int j) const { return j < head() ? j : j + 8 * n8(); }
  // the eight 2-bit classes of a chunk (cls is not null); past L1
  __device__ __forceinline__ uint32_t chunk_classes(int chunk) const {
    if (head() == 0) return (uint32_t)__ldcg(reinterpret_cast<const unsigned short*>(cls) + chunk);
    const int id = first_of(chunk);
    return __funnelshift_r(__ldcg(cls + (id >> 4)), __ldcg(cls + (id >> 4) + 1), (uint32_t)(id & 15) * 2u) & 0xffffu;
  }
  Pool pool;
  int slot;
  int2* s_pair;
  int n_s, s_cap;
  float m;
  __device__ __forceinline__ int class_of(int id) const {
    return cls ? (int)((cls[id >> 4] >> ((id & 15) * 2)) & 3u) : 0;
  }
  // exact history count of a token of class 3
  __device__ __forceinline__ int heavy_count(int id) const {
    const int q = (pool.pos + (size_t)slot * pool.pos_stride)[id];
    return q > 0 ? (pool.pairs + (size_t)slot * pool.unique_cap)[q - 1].y : 0;
  }
  // score of the token at position id, whatever population it belongs to
  __device__ __forceinline__ float element_score(int id, uint32_t raw, int c) const {
    return score_of(raw, c == 3 ? heavy_count(id) : c);
  }
};

template <class F>
__device__ __forceinline__ void for_each_side3(const Ctx3& c, F&& f) {
  const int2* pairs = c.s_pair;
  const int n = c.n_s;
#pragma unroll 1
  for (int j = threadIdx.x; j < n; j += kThreads) {
    const int2 e = pairs[j];
    if (e.x >= 0) f(e.x, __int_as_float(e.y));
  }
}

// ---- the row's classes --------------------------------------------------------------------------
// Scores grow with the bin inside a count class, so a count class's cells, from its lowest to its
// highest non-empty one, are in the order of their scores.  Thread t owns cells t, t + kThreads, ... of
// each.  Calls f(valid, score, tokens, cell) for the non-empty ones, WHOLE WARPS together; empty cells
// cost a look, not a call (a pass is bound by the instructions it issues, and two cells in three
// may be empty), and neighbouring lanes have neighbouring cells, so they mostly go in step.
template <class F>
__device__ __forceinline__ void for_each_class(const Ctx3& c, F&& f) {
  const Scorer sc = c;
  const uint32_t* tab = c.tab() + threadIdx.x;
#pragma unroll 1
  for (int k = 0; k < 3; ++k) {
    if (c.ends()[k] == 0) continue;  // (nothing in this count class)
    uint32_t bits = 0;
#pragma unroll
    for (int u = 0; u < kPerClass; ++u) bits |= (tab[(k * kPerClass + u) * kThreads] ? 1u : 0u) << u;
#pragma unroll 1
    while (__any_sync(0xffffffffu, bits != 0u)) {
      const bool valid = bits != 0u;
      const int at = (k * kPerClass + (valid ? __ffs(bits) - 1 : 0)) * kThreads;
      bits &= bits - 1u;
      const int cell = at + (int)threadIdx.x;
      f(valid, sc.bin_score(cell - k * kV3Bins, k), tab[at], cell);
    }
  }
}

// Where a key falls among the buckets: by score, over equal widths from `lo` to the row maximum
// (lin), or by the key itself, over [klo, khi].  Both grow with the key.
struct V3Map {
  bool lin;
  float lo, scale;
  uint32_t klo, khi;
  int shift;
  __device__ __forceinline__ bool in(uint32_t key) const { return key >= klo && key <= khi; }
  __device__ __forceinline__ int bucket_of(float score) const {  // (lin)
    return min(max(__float2int_rz((score - lo) * scale), 0), kV3Buckets - 1);
  }
  __device__ __forceinline__ int bucket(uint32_t key) const {
    if (lin) return bucket_of(score_of(key));
    return key < klo ? -1 : (key > khi ? kV3Buckets : (int)((key - klo) >> shift));
  }
  // buckets over the keys of [from, to]
  __device__ __forceinline__ void by_key(uint32_t from, uint32_t to) {
    lin = false;
    klo = from;
    khi = to;
    shift = max(0, 32 - __clz(to - from) - 10);  // ((to - from) >> shift) < 1,024
  }
  // buckets over the scores from `lowest` (or 30 below the maximum m, where no mass is left) to m;
  // by key when the scores do not spread
  __device__ __forceinline__ void by_score(float lowest, float m) {
    by_key(0u, 0xffffffffu);
    lo = fmaxf(lowest, m - 30.0f);
    const float range = m - lo;
    lin = range > 0.f && range < 3.0e38f;
    scale = lin ? __fdiv_rn((float)kV3Buckets - 0.5f, range) : 0.f;
  }
};
// Where the cells of bucket b lie: c.range()[k] to c.range()[3 + k] of count class k (a bucket grows with
// the key, and keys grow with the cell).  Warp w looks for one end of class w % 3's range, 32 cells
// at a time.  Called by the whole CTA; barriers on both sides.
__device__ __noinline__ void locate_cells(const Ctx3& c, const V3Map map, int b) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (warp < 6) {
    const Scorer sc = c;
    const int k = warp % 3, top = c.ends()[k];
    const int want = warp < 3 ? b : b + 1;  // the first cell whose bucket is at least this
    int lo = top ? c.ends()[3 + k] : 0, hi = top;
#pragma unroll 1
    while (lo < hi) {
      const int step = (hi - lo + 31) >> 5;
      const int t = lo + (lane + 1) * step - 1;
      const bool pass = t >= hi || map.bucket(key_of(sc.bin_score(min(t, hi - 1) - k * kV3Bins, k))) >= want;
      const uint32_t votes = __ballot_sync(0xffffffffu, pass);
      if (votes == 0) { lo = hi; break; }
      const int first = __ffs(votes) - 1;
      hi = min(lo + (first + 1) * step - 1, hi);
      lo = lo + first * step;
    }
    if (lane == 0) c.range()[warp] = lo;
  }
  __syncthreads();
}
// Calls f(tokens, cell) for the non-empty cells that were located, one per thread and step.
template <class F>
__device__ __forceinline__ void for_located_cells(const Ctx3& c, F&& f) {
#pragma unroll 1
  for (int k = 0; k < 3; ++k) {
#pragma unroll 1
    for (int cell = c.range()[k] + (int)threadIdx.x; cell < c.range()[3 + k]; cell += kThreads) {
      const uint32_t n = c.tab()[cell];
      if (n) f(n, cell);
    }
  }
}

// ---- the tie group of a key: the classes (at most one per count class, scores grow with
// the bin) and the side elements whose score key equals it ---------------------------------
struct Group {
  uint32_t key;
  int cell0, cell1, cell2;  // class index per count class, or -1
  __device__ __forceinline__ int cell_of(int cc) const { return cc == 0 ? cell0 : (cc == 1 ? cell1 : cell2); }
};
__device__ __forceinline__ Group find_group(Ctx3& c, uint32_t key) {
  if (threadIdx.x < 3) c.x()->bcast[threadIdx.x] = 0;
  V3Map at_key;
  at_key.by_key(key, key);
  locate_cells(c, at_key, 0);
  for_located_cells(c, [&](uint32_t, int cell) { c.x()->bcast[cell / kV3Bins] = (u64)cell + 1; });
  __syncthreads();
  Group g;
  g.key = key;
  g.cell0 = (int)c.x()->bcast[0] - 1;
  g.cell1 = (int)c.x()->bcast[1] - 1;
  g.cell2 = (int)c.x()->bcast[2] - 1;
  __syncthreads();
  return g;
}
// Does the token at position id (raw bits, 2-bit class cc) belong to the group?
__device__ __forceinline__ bool in_group(const Ctx3& c, const Group& g, int id, uint32_t raw, int cc) {
  if (cc < 3) {
    const int b = v3_bin_of_raw(raw);
    if (b >= 0) return g.cell_of(cc) == cc * kV3Bins + b;
    return key_of(c.score_of(raw, cc)) == g.key;  // outside the bin window: a side element
  }
  return key_of(c.score_of(raw, c.heavy_count(id))) == g.key;
}

// Bit k set: token k of chunk i belongs to the group.
__device__ __forceinline__ uint32_t chunk_members(const Ctx3& c, const Group& g, int i, const uint4& w,
                                                  uint32_t cls16) {
  const uint32_t words[4] = {w.x, w.y, w.z, w.w};
  uint32_t memb = 0;
#pragma unroll 1
  for (int k = 0; k < 4; ++k) {
    memb |= (in_group(c, g, c.first_of(i) + 2 * k, words[k] & 0xffffu, (cls16 >> (4 * k)) & 3) ? 1u : 0u) << (2 * k);
    memb |= (in_group(c, g, c.first_of(i) + 2 * k + 1, words[k] >> 16, (cls16 >> (4 * k + 2)) & 3) ? 1u : 0u) << (2 * k + 1);
  }
  return memb;
}
// Members in chunks [b, e) seen by this lane (lanes of a warp interleave), four 128-bit
// loads in flight per lane.
__device__ __forceinline__ u64 count_members(const Ctx3& c, const Group& g, int b, int e) {
  const int lane = threadIdx.x & 31;
  const uint4* src4 = c.chunks();
  u64 mine = 0;
  for (int i0 = b + lane; i0 < e; i0 += 4 * 32) {
    uint4 w[4];
    uint32_t cl[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + 32 * u;
      if (i < e) { w[u] = __ldcg(src4 + i); cl[u] = c.cls ? c.chunk_classes(i) : 0u; }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + 32 * u;
      if (i < e) mine += __popc(chunk_members(c, g, i, w[u], cl[u]));
    }
  }
  return mine;
}

// Token id of the n-th (1-based, ascending id) member of the group (classes and side
// elements whose score key is g.key), or 0x7fffffff: for groups of any size.  The row is cut into one segment per
// warp, members are counted, and the segment that holds the n-th is cut again until one
// warp can rank its members with ballots.
__device__ __noinline__ int nth_in_large_group(Ctx3& c, const Group g, u64 n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
  int b = 0, e = c.n8();
  u64 before = 0;
  // the loose tokens ahead of the first chunk, by every warp alike
  {
    const bool mbr = lane < c.head() && in_group(c, g, lane, c.logits[lane], c.class_of(lane));
    const uint32_t ballot = __ballot_sync(0xffffffffu, mbr);
    if ((u64)__popc(ballot) >= n) return (int)__fns(ballot, 0, (int)n);
    before = (u64)__popc(ballot);
  }
  bool in_tail = false;
  int result = 0x7fffffff;
  while (true) {
    if (e - b <= 4 * 32) break;
    const int seg = (e - b + kWarps - 1) / kWarps;
    const int mb = min(b + warp * seg, e), me = min(mb + seg, e);
    const u64 wtot = warp_sum_u64(count_members(c, g, mb, me));
    u64 pre, pre_unused, tot, tot_unused;
    block_warp_prefix2(*c.x(), wtot, 0, pre, pre_unused, tot, tot_unused);
    if (before + tot < n) { before += tot; in_tail = true; break; }
    if (before + pre < n && n <= before + pre + wtot && lane == 0) {
      c.x()->bcast[4] = (u64)mb;
      c.x()->bcast[5] = (u64)me;
      c.x()->bcast[6] = before + pre;
    }
    __syncthreads();
    b = (int)c.x()->bcast[4];
    e = (int)c.x()->bcast[5];
    before = c.x()->bcast[6];
    __syncthreads();
  }
  if (tid == 0) c.x()->bcast[6] = 0;
  __syncthreads();
  if (warp == 0) {
    // at most 128 chunks, then the loose tokens behind the last one: rank members with warp scans
    const uint4* src4 = c.chunks();
    u64 running = before;
    for (int i0 = b; !in_tail && i0 < e && running < n; i0 += 32) {
      const int i = i0 + lane;
      uint32_t memb = 0;
      if (i < e) memb = chunk_members(c, g, i, __ldcg(src4 + i), c.cls ? c.chunk_classes(i) : 0u);
      const u64 incl = warp_scan_u64((u64)__popc(memb));
      u64 rank = running + incl - __popc(memb);
      for (int k = 0; k < 8; ++k) {
        if (!((memb >> k) & 1u)) continue;
        if (++rank == n) c.x()->bcast[6] = (u64)(c.first_of(i) + k) + 1;
      }
      running += shfl_u64(incl, 31);
    }
    if (running < n) {
      const int id = c.first_of(c.n8()) + lane;
      const bool mbr = id < c.vocab && in_group(c, g, id, c.logits[id], c.class_of(id));
      const uint32_t ballot = __ballot_sync(0xffffffffu, mbr);
      const u64 rank = running + __popc(ballot & ((1u << lane) - 1u)) + 1;
      if (mbr && rank == n) c.x()->bcast[6] = (u64)id + 1;
    }
  }
  __syncthreads();
  const u64 found = c.x()->bcast[6];
  __syncthreads();
  if (found) result = (int)(found - 1);
  return result;
}

// Token id of the n-th (1-based, ascending id) member of up to three classes, one per count class,
// of at most kV3ScanCap tokens together.  The row is walked from the end that is nearer to the n-th
// member, 16,384 tokens per step, and the walk stops soon after the step that reaches it (it looks
// every other step): members are spread evenly over the row, so on average a third of it is read.
// A class is one bf16 bit pattern and a normal number (the bin window holds neither zeros nor NaNs),
// so two tokens are compared with it by one native bf16x2 equality per 32-bit word; a hit looks its
// count class up in the 16 class bits that travel with its chunk.  The ids found are ranked among
// themselves.  Bound by the latency of the row's loads (out of L2, or HBM when the row has left it):
// a chunk's successor is requested as soon as the chunk has been compared, and one batch of four
// 128-bit registers is all that is held (two batches were spilled: 26 thousand cycles for a third of
// a 248,320-token row).
static_assert(kV3ScanCap <= kV3TieCap - 4, "scan ids fit the list of ids");
// (Not inlined, and handed plain values instead of the row's context: the registers of the kernel's
// main body are all taken.  And no more of them than a whole row needs: with a range's first chunk as a value of
// its own the walk of a row with penalties took 57.4 thousand cycles from the cuts to the token, 52.7 without; 200
// such rows of 248,320 among 256 137.2 us a call and 132.0.)
struct ScanArgs {
  const unsigned short* logits;
  const uint32_t* cls;
  int vocab, head, n8;
  int front;      // of the loose tokens ahead of the first chunk, how many are looked at: all (head) or none
  int* ids;       // [kV3TieCap]
  int* slot_n;    // ids in the list so far (the caller's own members first)
  int* step_n;    // [2]
  u64* result;    // id + 1 of the answer, or 0
};
constexpr uint32_t kNoRaw = 0x7fc0u;  // a NaN: equal to nothing
template <bool ONE>  // one class (cc0, raw0); else raw0 / raw1 / raw2 of the count classes 0 / 1 / 2
__device__ __noinline__ void scan_members(const ScanArgs c, uint32_t raw0, uint32_t raw1, uint32_t raw2, int cc0, int n, int members) {
  const int tid = threadIdx.x;
  auto pair_of = [](uint32_t raw) {
    const uint32_t v = raw | (raw << 16);
    return *reinterpret_cast<const __nv_bfloat162*>(&v);
  };
  const __nv_bfloat162 v0 = pair_of(raw0), v1 = pair_of(raw1), v2 = pair_of(raw2);
  auto member = [&](uint32_t raw, int cc) {
    if (ONE) return raw == raw0 && cc == cc0;
    return cc < 3 && raw == (cc == 0 ? raw0 : (cc == 1 ? raw1 : raw2));
  };
  int* ids = c.ids;
  const bool forward = 2 * n <= members + 1;
  const int need = forward ? n : members - n + 1;  // counted from the end the walk starts at
  if (tid == 0) { c.step_n[0] = 0; c.step_n[1] = 0; *c.result = 0; }
  __syncthreads();
  const int n8 = c.n8;
  const uint4* src4 = reinterpret_cast<const uint4*>(c.logits + c.head);
  // Members found are counted in two counters that take turns from one look to the next:
  // after a look's barrier every thread reads that turn's counter, which nobody adds to before
  // the barrier after next, so all threads see the same running total and leave together.
  auto note = [&](int id, int parity) {
    const int slot = atomicAdd(c.slot_n, 1);
    if (slot < kV3ScanCap) ids[slot] = id;
    atomicAdd(c.step_n + parity, 1);
  };
  // the loose tokens at the end the walk starts from, and later those at its other end
  auto loose = [&](int from, int to, int parity) {
    const int id = from + tid;
    if (id < to && member((uint32_t)c.logits[id], c.cls ? (int)((c.cls[id >> 4] >> ((id & 15) * 2)) & 3u) : 0)) note(id, parity);
  };
  const int tail_at = c.head + 8 * n8;
  if (forward) loose(0, c.front, 0); else loose(tail_at, c.vocab, 0);
  constexpr int kBatch = 4;
  constexpr int kStep = kBatch * kThreads;  // chunks per step
  constexpr int kCheckShift = 1;            // the walk looks whether it may stop every 2^kCheckShift steps
  const int n_steps = (n8 + kStep - 1) / kStep;
  uint4 w[kBatch];
  uint32_t cl[kBatch];
  // chunk u of step s for this thread (steps are numbered in walking order)
  auto chunk_of = [&](int s, int u) { return (forward ? s : n_steps - 1 - s) * kStep + u * kThreads + tid; };
  auto fetch = [&](int u, int s) {
    const int i = chunk_of(s, u);
    if (s >= n_steps || i >= n8) { w[u] = make_uint4(~0u, ~0u, ~0u, ~0u); return; }  // (NaNs: no hits)
    w[u] = __ldcg(src4 + i);
    if (!c.cls) return;
    if (c.head == 0) {
      cl[u] = (uint32_t)__ldcg(reinterpret_cast<const unsigned short*>(c.cls) + i);
    } else {
      const int id = c.head + 8 * i;
      cl[u] = __funnelshift_r(__ldcg(c.cls + (id >> 4)), __ldcg(c.cls + (id >> 4) + 1), (uint32_t)(id & 15) * 2u);
    }
  };
#pragma unroll
  for (int u = 0; u < kBatch; ++u) { cl[u] = 0u; fetch(u, 0); }
  bool reached = false;
  int total = 0, seen[2] = {0, 0};
  for (int s = 0; s < n_steps; ++s) {
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const uint4 cur = w[u];
      const uint32_t cur_cl = cl[u];
      fetch(u, s + 1);
      auto same = [&](uint32_t word) {
        const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(&word);
        uint32_t m = __heq2_mask(x, v0);
        if (!ONE) m |= __heq2_mask(x, v1) | __heq2_mask(x, v2);
        return m;
      };
      const uint32_t m0 = same(cur.x), m1 = same(cur.y), m2 = same(cur.z), m3 = same(cur.w);
      if (m0 | m1 | m2 | m3) {
        uint32_t hits = ((m0 & 1u) | ((m0 >> 15) & 2u)) | (((m1 & 1u) | ((m1 >> 15) & 2u)) << 2) |
                        (((m2 & 1u) | ((m2 >> 15) & 2u)) << 4) | (((m3 & 1u) | ((m3 >> 15) & 2u)) << 6);
        while (hits) {
          const int q = __ffs(hits) - 1;
          hits &= hits - 1;
          const uint32_t word = q < 2 ? cur.x : (q < 4 ? cur.y : (q < 6 ? cur.z : cur.w));
          if (member((word >> (16 * (q & 1))) & 0xffffu, (int)((cur_cl >> (2 * q)) & 3u)))
            note(c.head + 8 * chunk_of(s, u) + q, (s >> kCheckShift) & 1);
        }
      }
    }
    // (a look every few steps: a barrier after every step would make each one wait for its
    // slowest load)
    if ((s & ((1 << kCheckShift) - 1)) == (1 << kCheckShift) - 1) {
      const int turn = (s >> kCheckShift) & 1;
      __syncthreads();
      const int now = c.step_n[turn];
      total += now - seen[turn];
      seen[turn] = now;
      if (total >= need) { reached = true; break; }
    }
  }
  if (!reached) { if (forward) loose(tail_at, c.vocab, 0); else loose(0, c.front, 0); }
  __syncthreads();
  const int found = min(*c.slot_n, kV3ScanCap);
  if (tid < 4) ids[found + tid] = forward ? 0x7fffffff : -1;
  __syncthreads();
  // every member on the near side of the last step's far end was noted: the one that `need - 1`
  // others precede (follow, when walking backwards) is the answer
  for (int t = tid; t < found; t += kThreads) {
    const int mine = ids[t];
    int before = 0;
    for (int j = 0; j < found; j += 4) {
      const int4 o = *reinterpret_cast<const int4*>(ids + j);
      before += forward ? (o.x < mine) + (o.y < mine) + (o.z < mine) + (o.w < mine)
                        : (o.x > mine) + (o.y > mine) + (o.z > mine) + (o.w > mine);
    }
    if (before + 1 == need) *c.result = (u64)mine + 1;
  }
  __syncthreads();
}
__device__ __forceinline__ ScanArgs scan_args(const Ctx3& c) {
  return ScanArgs{c.logits, c.cls, c.vocab, c.head(), c.n8(), c.head(), c.list(), c.gbuf_n(), c.step_n(), &c.x()->bcast[6]};
}
// Token id of the n-th member of a group: by one scan when the group is small enough.
__device__ int nth_in_group(Ctx3& c, const Group& g, u64 n) {
  auto count = [&](int cell) { return cell >= 0 ? (u64)c.tab()[cell] : 0ull; };
  auto raw = [&](int cell, int cc) { return cell >= 0 ? v3_raw_of_bin(cell - cc * kV3Bins) : kNoRaw; };
  const u64 in_classes = count(g.cell0) + count(g.cell1) + count(g.cell2);
  if (in_classes <= (u64)kV3ScanCap) {
    // the group's side elements are noted first, whatever the walk will see
    __syncthreads();
    if (threadIdx.x == 0) *c.gbuf_n() = 0;
    __syncthreads();
    for_each_side3(c, [&](int id, float s) {
      if (key_of(s) != g.key) return;
      const int slot = atomicAdd(c.gbuf_n(), 1);
      if (slot < kV3ScanCap) c.list()[slot] = id;
    });
    __syncthreads();
    const u64 all = in_classes + (u64)*c.gbuf_n();
    if (all <= (u64)kV3ScanCap && n >= 1 && n <= all) {
      const int cc = g.cell0 >= 0 ? 0 : (g.cell1 >= 0 ? 1 : 2);
      if ((g.cell0 >= 0) + (g.cell1 >= 0) + (g.cell2 >= 0) == 1)
        scan_members<true>(scan_args(c), raw(g.cell_of(cc), cc), kNoRaw, kNoRaw, cc, (int)n, (int)all);
      else
        scan_members<false>(scan_args(c), raw(g.cell0, 0), raw(g.cell1, 1), raw(g.cell2, 2), 0, (int)n, (int)all);
      const u64 hit = c.x()->bcast[6];
      __syncthreads();
      if (hit) return (int)(hit - 1);
    }
  }
  return nth_in_large_group(c, g, n);
}

// Appends to the gather buffer the ids of all group members with id <= id_limit.
__device__ void emit_group_upto(Ctx3& c, const Group& g, int id_limit) {
  const int last = min(c.n8(), max(0, id_limit - c.head()) / 8 + 1);
  const uint4* src4 = c.chunks();
  auto emit = [&](int id) {
    const int slot = atomicAdd(c.gbuf_n(), 1);
    if (slot < kV3ListCap) c.gbuf()[slot] = V3Entry{g.key, id};
  };
  for (int i = threadIdx.x; i < last; i += kThreads) {
    uint32_t memb = chunk_members(c, g, i, __ldcg(src4 + i), c.cls ? c.chunk_classes(i) : 0u);
    while (memb) {
      const int k = __ffs(memb) - 1;
      memb &= memb - 1;
      if (c.first_of(i) + k <= id_limit) emit(c.first_of(i) + k);
    }
  }
  if ((int)threadIdx.x < c.n_loose()) {
    const int id = c.loose(threadIdx.x);
    if (id <= id_limit && in_group(c, g, id, c.logits[id], c.class_of(id))) emit(id);
  }
  __syncthreads();
}

// A uniformly chosen token of ONE class (count class and one-value bin `cell`) by rejection:
// Philox-drawn positions are probed, `trials` (<= kRandomTrials) per thread and round with
// their loads in flight together; trial t = (round * trials + j) * kThreads + thread, and
// the lowest hitting trial wins.  A lone CTA sustains well under one scattered load per
// clock, so a probe reads the value first and the class map only when the value matches.
// Returns -1 if max_rounds pass without a hit.
constexpr int kRandomTrials = 8;
__device__ int random_in_class(Ctx3& c, int cell, int trials, uint64_t seed, int max_rounds) {
  const int tid = threadIdx.x;
  const int cc = cell / kV3Bins;
  const uint32_t value = v3_raw_of_bin(cell - cc * kV3Bins);
  for (int round = 0; round < max_rounds; ++round) {
    int id[kRandomTrials];
    uint32_t raw[kRandomTrials];
#pragma unroll
    for (int j = 0; j < kRandomTrials / 2; ++j) {
      if (2 * j < trials) {
        const Philox4 r = philox4x32_10((uint32_t)round, (uint32_t)tid, 1u + (uint32_t)j, 0u, (uint32_t)seed,
                                        (uint32_t)(seed >> 32));
        id[2 * j] = (int)__umul64hi(((u64)r.v[0] << 32) | r.v[1], (u64)c.vocab);
        id[2 * j + 1] = (int)__umul64hi(((u64)r.v[2] << 32) | r.v[3], (u64)c.vocab);
      }
    }
#pragma unroll
    for (int j = 0; j < kRandomTrials; ++j) raw[j] = j < trials ? (uint32_t)c.logits[id[j]] : ~value;
    uint32_t key = 0;
    int mine = -1;
#pragma unroll
    for (int j = kRandomTrials - 1; j >= 0; --j) {
      if (j < trials && raw[j] == value && c.class_of(id[j]) == cc) {
        key = (uint32_t)((kRandomTrials - j) * kThreads - tid);
        mine = id[j];
      }
    }
    const uint32_t best = block_max_u32(*c.x(), key);
    if (best) {
      if (key == best) c.x()->bcast[6] = (u64)mine;
      __syncthreads();
      const int token = (int)c.x()->bcast[6];
      __syncthreads();
      return token;
    }
  }
  return -1;
}

// A token of the kept set drawn with probability proportional to its mass, by rejection on
// TOKENS: a Philox-drawn position is accepted when a second number, uniform on [0, 2^40), lies
// below the token's integer mass (2^40 stands for the row maximum) and the token is kept.  The
// first accepted trial wins (trial t = (round * kTokenTrials + j) * kThreads + thread), which
// makes the draw exact and reproducible.  The chance per trial is the kept mass over
// vocab * 2^40: high on near-flat rows -- exactly where the draw by classes is slow (many
// small classes, whose members must be looked for) -- and hopeless on peaked ones, so the
// caller asks for it only when a round is almost sure to succeed (with one trial per thread
// on the flattest rows, else two).  A top-p cut that splits a
// tie group keeps the group's `cut_ties` lowest ids: a member of the group that is hit stands
// for the group as a whole and is accepted with probability cut_ties / group_cnt; the caller
// then picks one of the kept members (group_hit).  Returns -1 if max_rounds pass without a hit.
constexpr int kTokenTrials = 2;
__device__ int draw_by_token_rejection(Ctx3& c, const KeptSet& kept, bool tie_split, u64 cut_ties, u64 group_cnt,
                                       uint64_t seed, int max_rounds, int trials, bool& group_hit) {
  const int tid = threadIdx.x;
  group_hit = false;
  for (int round = 0; round < max_rounds; ++round) {
    int id[kTokenTrials];
    u64 u[kTokenTrials];
    uint32_t raw[kTokenTrials];
    int cc[kTokenTrials];
#pragma unroll
    for (int j = 0; j < kTokenTrials; ++j) {
      if (j >= trials) break;
      const Philox4 r = philox4x32_10((uint32_t)round, (uint32_t)tid, (uint32_t)j, 2u, (uint32_t)seed, (uint32_t)(seed >> 32));
      id[j] = (int)__umul64hi(((u64)r.v[0] << 32) | r.v[1], (u64)c.vocab);
      u[j] = ((u64)r.v[2] << 8) | (r.v[3] >> 24);
    }
#pragma unroll
    for (int j = 0; j < kTokenTrials; ++j) {
      if (j >= trials) break;
      raw[j] = (uint32_t)c.logits[id[j]];
      cc[j] = c.class_of(id[j]);
    }
    u64 best = 0;
#pragma unroll
    for (int j = 0; j < kTokenTrials; ++j) {
      if (j >= trials) break;
      const float s = c.element_score(id[j], raw[j], cc[j]);
      const uint32_t k = key_of(s);
      if (k < kept.cut_key || !(u[j] < mass_of(s, c.m))) continue;
      bool group = false;
      if (k == kept.cut_key && tie_split) {
        const Philox4 r = philox4x32_10((uint32_t)round, (uint32_t)tid, (uint32_t)j, 3u, (uint32_t)seed, (uint32_t)(seed >> 32));
        if (!(__umul64hi(((u64)r.v[0] << 32) | r.v[1], group_cnt) < cut_ties)) continue;
        group = true;
      }
      const u64 packed = ((u64)((kTokenTrials - j) * kThreads - tid) << 33) | ((u64)(group ? 1u : 0u) << 32) | (uint32_t)id[j];
      best = packed > best ? packed : best;
    }
    best = block_max_u64(*c.x(), best);
    if (best) {
      group_hit = ((best >> 32) & 1ull) != 0;
      return (int)(uint32_t)best;
    }
  }
  return -1;
}

}  // namespace hs
